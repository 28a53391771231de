"""The streaming kernels (RunStaged, RunPush) on messages of 2^18 elements per rank and more. Ranks that share a GPU take
other kernels from there on, ranks on GPUs of their own do not, so they are asked for by name: in the library that
ships, and in the checked build, which runs the code for ranks on GPUs of their own."""
import os

import numpy as np
import pytest
import torch

from switchml_b200.ops.emulation import emulated_allreduce_with
from switchml_b200.ops.oracle import int_allreduce_oracle, quant_allreduce_oracle
from test_gpu_checked_build import CHECKED, _child

pytestmark = pytest.mark.gpu

LARGE = (1 << 20) + 1


def _inputs(n, numel, dtype=torch.float32, seed=0):
    g = torch.Generator().manual_seed(seed)
    if dtype == torch.int32:
        return [torch.randint(-2 ** 30, 2 ** 30, (numel,), generator=g, dtype=dtype) for _ in range(n)]
    return [((torch.rand(numel, generator=g) * 2 - 1) * 10.0 ** (r - 1)).to(dtype) for r in range(n)]


@pytest.mark.parametrize("algo", ["staged", "push"])
@pytest.mark.parametrize("n", [1, 2, 4, 8])
def test_exact(n, algo):
    if algo == "push" and n == 1:
        pytest.skip("pushing needs a peer")
    for dtype in (torch.float32, torch.bfloat16):
        xs = _inputs(n, LARGE, dtype)
        want = torch.from_numpy(quant_allreduce_oracle([x.float().numpy() for x in xs], 64)).to(dtype)
        for o in emulated_allreduce_with([x.cuda() for x in xs], kernels="streaming", mode="quant", algo=algo, block_numel=64, slot_bytes=32768):
            assert torch.equal(o.cpu(), want), dtype


@pytest.mark.parametrize("algo", ["staged", "push"])
@pytest.mark.parametrize("block", [32, 256, 1024])
def test_several_jobs_over_the_same_slots(block, algo):
    for lookahead in (-1, 2):
        xs = _inputs(4, 300001, seed=3)
        outs = emulated_allreduce_with([x.cuda() for x in xs], kernels="streaming", mode="quant", algo=algo, block_numel=block,
                                       slot_bytes=16 * 4 * block, slots_per_channel=4, repeats=3, channels=3, exponent_lookahead=lookahead)
        want = quant_allreduce_oracle([x.numpy() for x in xs], block)
        assert all(np.array_equal(o.cpu().numpy(), want) for o in outs)


@pytest.mark.parametrize("algo", ["staged", "push"])
@pytest.mark.parametrize("n", [2, 8])
def test_whole_numbers(n, algo):
    xs = _inputs(n, 777777, torch.int32)
    want = int_allreduce_oracle([x.numpy() for x in xs])
    for o in emulated_allreduce_with([x.cuda() for x in xs], kernels="streaming", mode="sum", algo=algo):
        assert np.array_equal(o.cpu().numpy(), want)


@pytest.mark.parametrize("algo", ["staged", "push"])
@pytest.mark.parametrize("dtype, eps", [(torch.float32, 2.0 ** -24), (torch.bfloat16, 2.0 ** -8)])
def test_plain_sums_in_place(dtype, eps, algo):
    xs = _inputs(4, 999999, dtype)
    ys = [x.cuda() for x in xs]
    outs = emulated_allreduce_with(ys, kernels="streaming", mode="sum", algo=algo, post_scale=0.25, outputs=ys)
    exact = sum(x.double() for x in xs) / 4
    # n - 1 float32 additions, each off by half an ulp (n for what they add to the last rounding), and the result's rounding
    bound = sum(x.double().abs() for x in xs) / 4 * (4 * 2.0 ** -24) + exact.abs() * eps + 1e-38
    assert bool(((outs[0].cpu().double() - exact).abs() <= bound).all())
    assert all(torch.equal(o, outs[0]) for o in outs[1:]), "all ranks hold the same bits"


def test_random_shapes_against_the_oracle():
    rng = np.random.default_rng(20261203)
    for case in range(16):
        n, block, algo = int(rng.integers(2, 9)), int(rng.choice([32, 64, 256, 1024])), ("staged", "push")[case % 2]
        numel = int(rng.integers(1 << 18, 1 << 19))
        options = {"block_numel": block, "slot_bytes": int(rng.choice([8, 16, 64])) * 4 * block,
                   "slots_per_channel": int(rng.choice([1, 2, 3, 4, 5])), "channels": int(rng.choice([0, 1, 3, 7]))}
        xs = [rng.standard_normal(numel).astype(np.float32) * np.float32(2.0 ** int(rng.integers(-30, 30))) for _ in range(n)]
        want = quant_allreduce_oracle(xs, block)
        for o in emulated_allreduce_with([torch.from_numpy(x).cuda() for x in xs], kernels="streaming", mode="quant", algo=algo, **options):
            assert np.array_equal(o.cpu().numpy().view(np.uint32), want.view(np.uint32)), (case, n, numel, algo, options)


needs_checked_build = pytest.mark.skipif(not os.path.exists(CHECKED), reason="build-checked/ is not there (python build.py --checked)")


@needs_checked_build
@pytest.mark.parametrize("algo", ["staged", "push"])
def test_long_streams_of_ranks_on_gpus_of_their_own(algo):
    out = _child("""
        for block in (32, 256, 1024):
            for channels, repeats, slots in ((3, 3, 2), (1, 2, 4), (0, 1, 3)):
                g = torch.Generator().manual_seed(block + channels)
                xs = [(torch.rand(300001, generator=g) * 2 - 1) * 10.0 ** (r - 1) for r in range(4)]
                for dtype in (torch.float32, torch.bfloat16):
                    ys = [x.to(dtype) for x in xs]
                    want = torch.from_numpy(quant_allreduce_oracle([y.float().numpy() for y in ys], block)).to(dtype)
                    outs = emulated_allreduce([y.cuda() for y in ys], mode="quant", algo=%r, block_numel=block, slot_bytes=16 * 4 * block,
                                              slots_per_channel=slots, repeats=repeats, channels=channels)
                    assert all(torch.equal(o.cpu(), want) for o in outs), (block, channels, dtype)
        print("long streams")
    """ % algo)
    assert "long streams" in out


@needs_checked_build
def test_one_barrier_between_ranks_on_gpus_of_their_own():
    """Everybody's input goes into everybody's memory there: every type and mode, aligned or not, in place or not, with
    nothing written beside the outputs."""
    out = _child("""
        for n, numel, off in ((2, 1, 0), (2, 4099, 1), (3, 255, 2), (4, 65537, 0), (8, 20003, 1), (8, 4096, 0)):
            for inplace in (False, True):
                def run(ts, want, check, **opts):
                    frames = [torch.full((numel + off + 8,), 7, dtype=t.dtype, device="cuda") for t in ts]
                    ins = []
                    for f, t in zip(frames, ts):
                        src = f if inplace else torch.empty_like(f)
                        src[off:off + numel].copy_(t)
                        ins.append(src[off:off + numel])
                    outs = [f[off:off + numel] for f in frames]
                    emulated_allreduce(ins, algo="oneshot", outputs=outs, **opts)
                    for f, o in zip(frames, outs):
                        assert check(o.cpu()), (n, numel, off, inplace, o.dtype, opts)
                        assert bool((f[:off] == 7).all()) and bool((f[off + numel:] == 7).all()), "beside the output"
                g = torch.Generator().manual_seed(numel + n)
                xs = [torch.randn(numel, generator=g) * 10.0 ** (r % 3) for r in range(n)]
                for dtype in (torch.float32, torch.bfloat16):
                    ys = [x.to(dtype) for x in xs]
                    for block in (32, 128, 256, 1024):
                        want = torch.from_numpy(quant_allreduce_oracle([y.float().numpy() for y in ys], block)).to(dtype)
                        run(ys, want, lambda o: torch.equal(o, want), mode="quant", block_numel=block)
                    # n float32 additions and at most one rounding to bf16
                    exact = sum(y.double() for y in ys)
                    bound = n * 2.0 ** -24 * sum(y.double().abs() for y in ys) + (2.0 ** -8 * exact.abs() if dtype == torch.bfloat16 else 0)
                    run(ys, exact, lambda o: bool(((o.double() - exact).abs() <= bound).all()), mode="sum")
                xi = [torch.randint(-2 ** 30, 2 ** 30, (numel,), generator=g, dtype=torch.int32) for r in range(n)]
                whole = torch.from_numpy(int_allreduce_oracle([x.numpy() for x in xi]))
                run(xi, whole, lambda o: torch.equal(o, whole), mode="sum")
        print("one barrier")
    """)
    assert "one barrier" in out
