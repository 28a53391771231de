"""The checked build of the library (``build.py --checked``, -DSWITCHML_CHECKED): the
aggregation kernels verify the geometry of every tile before touching it and report
STATUS_BOUNDS instead of dereferencing anything out of range. Stands in for a memory
checker on machines where none may be run. Runs in child processes because the library
to load is chosen by an environment variable before the package is imported."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKED = os.path.join(ROOT, "p4app-switchML_b200", "build-checked", "libswitchml_b200.so")

BODY = """
import sys
sys.path.insert(0, %r)
import numpy as np, torch
from switchml_b200._native import lib, NativeError
from switchml_b200.ops.emulation import emulated_allreduce, emulated_allreduce_with
from switchml_b200.ops.oracle import quant_allreduce_oracle, int_allreduce_oracle
assert lib().sml_checked_build() == 1, "not the checked build"
""" % ROOT


def _child(code, **env):
    e = dict(os.environ, SWITCHML_B200_LIBRARY=CHECKED, **env)
    r = subprocess.run([sys.executable, "-c", BODY + textwrap.dedent(code)], capture_output=True, text=True,
                       timeout=300, env=e)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]
    return r.stdout


@pytest.fixture(scope="module", autouse=True)
def built():
    if not os.path.exists(CHECKED):
        pytest.skip("build-checked/ is not there (python build.py --checked)")


def test_results_are_unchanged_and_no_check_fires():
    out = _child("""
        for n, numel, algo in ((2, 65, "staged"), (4, 40000, "staged"), (8, (1 << 20) + 1, "staged"),
                               (4, 4096, "oneshot"), (8, 255, "oneshot")):
            g = torch.Generator().manual_seed(numel)
            xs = [(torch.rand(numel, generator=g) * 2 - 1) * 10.0 ** (r % 3) for r in range(n)]
            outs = emulated_allreduce([x.cuda() for x in xs], mode="quant", algo=algo, block_numel=64,
                                      slot_bytes=32768)
            want = quant_allreduce_oracle([x.numpy() for x in xs], 64)
            assert all(np.array_equal(o.cpu().numpy(), want) for o in outs), (n, numel, algo)
            xi = [torch.randint(-2 ** 30, 2 ** 30, (numel,), generator=g, dtype=torch.int32) for r in range(n)]
            outs = emulated_allreduce([x.cuda() for x in xi], mode="sum", algo=algo)
            want = int_allreduce_oracle([x.numpy() for x in xi])
            assert all(np.array_equal(o.cpu().numpy(), want) for o in outs), (n, numel, algo)
        print("checked build ok")
    """)
    assert "checked build ok" in out


@pytest.mark.parametrize("algo", ["staged", "oneshot"])
def test_a_region_that_is_too_small_is_reported_not_touched(algo):
    """The kernels are told that the staging region is 4 KiB (the memory itself is as large
    as ever): every tile fails its check, the outputs stay as they were, status 3."""
    out = _child("""
        xs = [torch.ones(5000, device="cuda") * (r + 1) for r in range(4)]
        outs = [torch.full((5000,), -7.0, device="cuda") for _ in range(4)]
        try:
            emulated_allreduce(xs, mode="quant", algo=%r, block_numel=64, slot_bytes=32768, outputs=outs)
            raise SystemExit("the geometry check did not fire")
        except NativeError as e:
            msg = str(e)
        torch.cuda.synchronize()
        assert all(bool((o == -7.0).all()) for o in outs), "a refused tile was written"
        assert all(float(x[0]) == r + 1 for r, x in enumerate(xs))
        print("refused:", msg)
        # the device is fine afterwards
        y = torch.arange(10, device="cuda").sum().item()
        assert y == 45
    """ % algo, SWITCHML_CHECKED_PRETEND_STAGE_BYTES="4096")
    assert "refused:" in out and "kernel status" in out
    status = int(out.split("kernel status")[1].split()[0])
    assert status & 0xf == 3


@pytest.mark.parametrize("algo", ["staged", "push"])
def test_code_for_ranks_on_gpus_of_their_own(algo):
    """The checked build emulates with the code that ranks on several GPUs run over peer memory, which is not the one that
    the library emulates with: every element type and mode, ragged ends, tensors that are not vector aligned."""
    out = _child("""
        for n, numel, off in ((2, 70, 0), (2, 300001, 0), (3, 50001, 1), (4, 123457, 0), (8, (1 << 18) + 5, 2)):
            g = torch.Generator().manual_seed(numel)
            def place(t):
                frame = torch.zeros(numel + off, dtype=t.dtype, device="cuda")
                frame[off:].copy_(t)
                return frame[off:]
            opts = dict(algo=%r, block_numel=64, slot_bytes=32768)
            xs = [torch.randn(numel, generator=g) * 10.0 ** (r %% 3) for r in range(n)]
            for dtype in (torch.float32, torch.bfloat16):
                ys = [x.to(dtype) for x in xs]
                want = torch.from_numpy(quant_allreduce_oracle([y.float().numpy() for y in ys], 64)).to(dtype)
                for o in emulated_allreduce([place(y) for y in ys], mode="quant", **opts):
                    assert torch.equal(o.cpu(), want), (n, numel, dtype, "quant")
                # Sums in fp32 in some order of the ranks, and at most one rounding to bf16: one unit of 2^-8.
                want = sum(y.double() for y in ys)
                bound = 2.0 ** -20 * sum(y.double().abs() for y in ys) + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)
                for o in emulated_allreduce([place(y) for y in ys], mode="sum", **opts):
                    assert bool(((o.cpu().double() - want).abs() <= bound).all()), (n, numel, dtype, "sum")
            xi = [torch.randint(-2 ** 30, 2 ** 30, (numel,), generator=g, dtype=torch.int32) for r in range(n)]
            want = int_allreduce_oracle([x.numpy() for x in xi])
            for o in emulated_allreduce([place(x) for x in xi], mode="sum", **opts):
                assert np.array_equal(o.cpu().numpy(), want), (n, numel, "int")
        print("as on several GPUs")
    """ % algo)
    assert "as on several GPUs" in out


@pytest.mark.parametrize("algo", ["staged", "push"])
def test_every_access_of_ranks_that_share_a_gpu(algo):
    """The kernels for ranks that share a GPU look at each address here: none is out of place, whatever the geometry."""
    out = _child("""
        algo = %r
        cases = ((1, 256, 32768, 2), (2, 32, 131072, 1), (3, 1024, 12288, 3), (4, 64, 16384, 4), (5, 256, 65536, 5),
                 (7, 64, 32768, 2), (8, 1024, 32768, 1), (8, 256, 262144, 4))
        for n, block, slot_bytes, slots in cases[algo == "push":]:
            for numel, channels in ((1, 0), (1023, 3), (8192 * 40 - 1, 1), ((1 << 18) + 9 * 1024 + 5, 3), ((1 << 18) + 1, 0)):
                opts = dict(kernels="one_gpu", algo=algo, block_numel=block, slot_bytes=slot_bytes, slots_per_channel=slots, channels=channels)
                g = torch.Generator().manual_seed(numel + n)
                xs = [torch.randn(numel, generator=g) * 10.0 ** (r %% 3) for r in range(n)]
                for dtype in (torch.float32, torch.bfloat16):
                    ys = [x.to(dtype) for x in xs]
                    want = torch.from_numpy(quant_allreduce_oracle([y.float().numpy() for y in ys], block)).to(dtype)
                    for o in emulated_allreduce_with([y.cuda() for y in ys], mode="quant", **opts):
                        assert torch.equal(o.cpu(), want), (n, numel, dtype, "quant")
                    # n float32 additions and at most one rounding to bf16: 2^-24 and 2^-8 of what is added
                    want = sum(y.double() for y in ys)
                    bound = n * 2.0 ** -24 * sum(y.double().abs() for y in ys) + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)
                    for o in emulated_allreduce_with([y.cuda() for y in ys], mode="sum", **opts):
                        assert bool(((o.cpu().double() - want).abs() <= bound).all()), (n, numel, dtype, "sum")
                xi = [torch.randint(-2 ** 30, 2 ** 30, (numel,), generator=g, dtype=torch.int32) for r in range(n)]
                want = int_allreduce_oracle([x.numpy() for x in xi])
                for o in emulated_allreduce_with([x.cuda() for x in xi], mode="sum", **opts):
                    assert np.array_equal(o.cpu().numpy(), want), (n, numel, "int")
        print("all in place")
    """ % algo)
    assert "all in place" in out


@pytest.mark.parametrize("mode", ["quant", "sum"])
@pytest.mark.parametrize("algo", ["staged", "push"])
def test_outputs_that_are_too_small_are_reported_not_written(algo, mode):
    """The kernels are told that the outputs hold 4096 elements: no channel that goes beyond is written, status 3."""
    out = _child("""
        xs = [torch.ones(300000, device="cuda") * (r + 1) for r in range(4)]
        outs = [torch.full((300000,), -7.0, device="cuda") for _ in range(4)]
        try:
            emulated_allreduce_with(xs, kernels="one_gpu", mode=%r, algo=%r, block_numel=64, outputs=outs)
            raise SystemExit("no check fired")
        except NativeError as e:
            msg = str(e)
        torch.cuda.synchronize()
        assert all(bool((o[4096:] == -7.0).all()) for o in outs), "written beyond the end"
        print("refused:", msg)
    """ % (mode, algo), SWITCHML_CHECKED_PRETEND_OUTPUT_BYTES=str(4096 * 4))
    assert "refused:" in out and "kernel status" in out
    assert int(out.split("kernel status")[1].split()[0]) & 0xf == 3
