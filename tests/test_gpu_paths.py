"""Edges of the kernels' dispatch and of the host path around them, each against the CPU oracle
or a plain PyTorch reference of the same operation."""
import threading

import numpy as np
import pytest
import torch

from switchml_b200 import lib
from switchml_b200.ops.emulation import emulated_allreduce
from switchml_b200.ops.oracle import quant_allreduce_oracle

pytestmark = pytest.mark.gpu


def test_kept_staging_memory_serves_other_geometries_and_threads():
    """Staging memory of one emulated call is used again by the next, whatever its ranks, slots and
    algorithm, and by one call at a time."""
    rng = np.random.default_rng(5)
    cases = [(n, algo, block, slots, rng.standard_normal((n, 50_000 + 7 * n)).astype(np.float32))
             for n, algo, block, slots in [(2, "push", 64, 4), (4, "staged", 256, 2), (8, "oneshot", 64, 3),
                                           (2, "staged", 64, 4), (3, "push", 1024, 1)]]
    wanted = [quant_allreduce_oracle(list(c[4]), c[2]) for c in cases]
    errors = []

    def walk(start):
        try:
            for turn in range(2 * len(cases)):
                n, algo, block, slots, xs = cases[(start + turn) % len(cases)]
                outs = emulated_allreduce([torch.from_numpy(x).cuda() for x in xs], mode="quant", algo=algo,
                                          block_numel=block, slots_per_channel=slots, slot_bytes=65536)
                for o in outs:
                    assert np.array_equal(o.cpu().numpy(), wanted[(start + turn) % len(cases)]), (n, algo)
        except BaseException as e:  # noqa: B902 - handed to the main thread
            errors.append(e)

    walk(0)
    threads = [threading.Thread(target=walk, args=(s,)) for s in (1, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    lib().sml_emu_release()
    walk(2)
    assert not errors, errors[0]
