"""One worker, exact mode, tensors that begin anywhere between two 16-byte boundaries (csrc/kernels/local_pass.cuh): the
oracle's bits, and no other byte of the buffer they lie in is touched."""
import numpy as np
import pytest
import torch

import switchml_b200 as sml
from switchml_b200.ops.oracle import quant_allreduce_oracle

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 7, 9, 250, 1016, 1017, 1023, 1024, 1025, 1031, 2048, 8 * 1024 - 1, 8 * 1024 + 5, 20 * 1024 + 777]


@pytest.mark.parametrize("block", [32, 64, 128, 256, 512, 1024])
def test_slices_of_a_flat_buffer(block):
    ctx = sml.Context.get_instance()
    assert ctx.start(sml.make_config("cuda", packet_numel=block, mode="int32_quant", launch="inline"))
    try:
        for dtype, offsets in ((torch.float32, range(4)), (torch.bfloat16, range(8))):
            for off in offsets:
                for numel in SIZES:
                    g = torch.Generator().manual_seed(1000 * off + numel)
                    flat = (torch.randn(numel + off + 8, generator=g) * 10.0 ** torch.randint(-3, 4, (numel + off + 8,), generator=g)).to(dtype)
                    flat[off + numel // 3: off + numel // 2] = 0
                    if numel == 2048:  # what the fast way leaves to the other one
                        flat[off + 5], flat[off + 1500], flat[off + 1900] = float("nan"), float("inf"), 3e38
                    x = flat.cuda()
                    want = torch.from_numpy(quant_allreduce_oracle([flat[off:off + numel].float().numpy()], block)).to(dtype)
                    for out_off in (off, None, (off + 1) % 8):  # in the same place of a line, in place, in another one
                        y = x.clone() if out_off is None else torch.full((numel + 16,), 7.0, dtype=dtype, device="cuda")
                        o = off if out_off is None else out_off
                        before = y.cpu()
                        a, b = (y[o:o + numel], None) if out_off is None else (x[off:off + numel], y[o:o + numel])
                        job = ctx.all_reduce_async(a, b)
                        job.stream_wait()
                        job.release()
                        got = y.cpu()
                        same = got[o:o + numel].view(torch.int16 if dtype == torch.bfloat16 else torch.int32)
                        bits = want.view(torch.int16 if dtype == torch.bfloat16 else torch.int32)
                        assert torch.equal(same, bits), (dtype, off, numel, out_off)
                        assert torch.equal(got[:o].float(), before[:o].float()) and torch.equal(got[o + numel:].float(), before[o + numel:].float())
    finally:
        ctx.stop()
