"""The aggregation pipelines for ranks that share a GPU (csrc/kernels/one_gpu_allreduce.cu), which messages of 2^18
elements per rank and more take: against the CPU oracle, and with plain sums against float64."""
import numpy as np
import pytest
import torch

from switchml_b200._native import NativeError
from switchml_b200.ops.emulation import emulated_allreduce, emulated_allreduce_with
from switchml_b200.ops.oracle import int_allreduce_oracle, quant_allreduce_oracle

pytestmark = pytest.mark.gpu

SMALLEST = 1 << 18


def _inputs(n, numel, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    if dtype == torch.int32:
        return [torch.randint(-2 ** 30, 2 ** 30, (numel,), generator=g, dtype=dtype) for _ in range(n)]
    xs = [((torch.rand(numel, generator=g) * 2 - 1) * 10.0 ** (r % 4 - 2)) for r in range(n)]
    for x in xs:
        x[1000:5000] = 0.0  # blocks of zeros
        x[-3:] = 2.0 ** -100
    return [x.to(dtype) for x in xs]


# The last tile: full, one element, one short of a chunk, whole chunks and a ragged one; one channel: many more tiles than
# slots, stages and exponent slots.
@pytest.mark.parametrize("numel, channels", [(SMALLEST, 0), (SMALLEST + 1, 0), (8192 * 40 - 1, 1), (SMALLEST + 9 * 1024 + 5, 3)])
@pytest.mark.parametrize("n, block, slot_bytes, slots", [(1, 256, 32768, 2), (2, 32, 131072, 1), (3, 1024, 12288, 3), (4, 64, 16384, 4),
                                                        (5, 256, 65536, 5), (7, 64, 1, 2), (8, 1024, 32768, 1), (8, 256, 262144, 4)])
@pytest.mark.parametrize("algo", ["staged", "push"])
def test_exact(algo, n, block, slot_bytes, slots, numel, channels):
    if algo == "push" and n == 1:
        pytest.skip("pushing needs a peer")
    for dtype in (torch.float32, torch.bfloat16):
        xs = _inputs(n, numel, dtype, numel + n)
        want = torch.from_numpy(quant_allreduce_oracle([x.float().numpy() for x in xs], block)).to(dtype)
        for inplace in (False, True):
            ys = [x.cuda() for x in xs]
            outs = emulated_allreduce(ys, mode="quant", algo=algo, block_numel=block, slot_bytes=slot_bytes, slots_per_channel=slots,
                                      channels=channels, repeats=1 if inplace else 2, outputs=ys if inplace else None)
            for r, o in enumerate(outs):
                assert torch.equal(o.cpu(), want), (dtype, inplace, r)


@pytest.mark.parametrize("numel, channels", [(SMALLEST, 0), (SMALLEST + 1, 1), (SMALLEST + 16387, 3)])
@pytest.mark.parametrize("n, slot_bytes, slots", [(1, 65536, 2), (2, 65536, 1), (3, 1536, 2), (4, 16384, 4), (6, 131072, 3), (8, 262144, 4)])
@pytest.mark.parametrize("algo", ["staged", "push"])
def test_plain_sums(algo, n, slot_bytes, slots, numel, channels):
    if algo == "push" and n == 1:
        pytest.skip("pushing needs a peer")
    options = {"mode": "sum", "algo": algo, "slot_bytes": slot_bytes, "slots_per_channel": slots, "channels": channels}
    xs = _inputs(n, numel, torch.int32, n)
    for o in emulated_allreduce([x.cuda() for x in xs], **options):
        assert np.array_equal(o.cpu().numpy(), int_allreduce_oracle([x.numpy() for x in xs]))
    for dtype, eps in ((torch.float32, 2.0 ** -24), (torch.bfloat16, 2.0 ** -8)):  # half an ulp of 24 and of 8 bits
        xs = _inputs(n, numel, dtype, n)
        ys = [x.cuda() for x in xs]
        outs = emulated_allreduce(ys, post_scale=0.5, outputs=ys, **options)
        exact = sum(x.double() for x in xs) / 2
        # n - 1 float32 additions (n for what they add to the last rounding), each off by half an ulp, and the result's rounding
        bound = sum(x.double().abs() for x in xs) / 2 * (n * 2.0 ** -24) + exact.abs() * eps + 1e-38
        assert bool(((outs[0].cpu().double() - exact).abs() <= bound).all()), dtype
        for o in outs[1:]:
            assert torch.equal(o, outs[0]), "all ranks hold the same bits"


@pytest.mark.parametrize("algo", ["staged", "push"])
@pytest.mark.parametrize("n", [2, 3, 8])
def test_nothing_beside_the_outputs_is_written(n, algo):
    """Outputs in frames: aligned, with elements before and behind that stay as they are; the inputs stay, too."""
    for numel in (1, 5, 1023, 20 * 1024 + 9, SMALLEST + 4097):
        for mode, dtype in (("quant", torch.float32), ("quant", torch.bfloat16), ("sum", torch.float32), ("sum", torch.bfloat16), ("sum", torch.int32)):
            xs = _inputs(n, numel, dtype, numel + n)
            ins = [x.cuda() for x in xs]
            frames = [torch.full((numel + 48,), 7, dtype=dtype, device="cuda") for _ in range(n)]
            outs = [f[16:16 + numel] for f in frames]
            emulated_allreduce_with(ins, kernels="one_gpu", mode=mode, algo=algo, block_numel=64, slot_bytes=16384, channels=5, outputs=outs)
            for x, i, f, o in zip(xs, ins, frames, outs):
                assert bool((f[:16] == 7).all()) and bool((f[16 + numel:] == 7).all()), (numel, mode, dtype)
                assert torch.equal(i.cpu().view(torch.int16 if dtype == torch.bfloat16 else torch.int32), x.view(torch.int16 if dtype == torch.bfloat16 else torch.int32))
                assert torch.equal(o, outs[0])
            if mode == "quant":
                assert torch.equal(outs[0].cpu(), torch.from_numpy(quant_allreduce_oracle([x.float().numpy() for x in xs], 64)).to(dtype))
            elif dtype == torch.int32:
                assert np.array_equal(outs[0].cpu().numpy(), int_allreduce_oracle([x.numpy() for x in xs]))


def test_values_that_are_not_finite():
    """Infinities and NaN come out as between GPUs: as the same job in pieces below 2^18 elements gives them."""
    n, numel, block = 2, SMALLEST, 64
    xs = _inputs(n, numel, torch.float32, 5)
    xs[0][64] = float("inf")
    xs[1][128 * 64 + 3] = float("nan")
    xs[1][300 * 64] = -float("inf")
    xs[0][400 * 64] = 3.4e38
    for algo in ("staged", "push"):
        outs = emulated_allreduce([x.cuda() for x in xs], mode="quant", algo=algo, block_numel=block)
        for at in range(0, numel, numel // 4):
            part = emulated_allreduce([x[at:at + numel // 4].cuda() for x in xs], mode="quant", algo=algo, block_numel=block)
            for o, p in zip(outs, part):
                assert torch.equal(o[at:at + numel // 4].view(torch.int32), p.view(torch.int32)), (algo, at)


@pytest.mark.parametrize("n", [2, 3, 4, 8])
def test_sums_that_wrap(n):
    """Values that are not finite saturate, and sums of those wrap, as the oracle's do."""
    xs = _inputs(n, SMALLEST, torch.float32, n)
    for r, x in enumerate(xs):
        x[::64] = float("inf")
        x[1::64] = -float("inf") if r else 3e38
        x[2::64] = 3.4e38
    want = quant_allreduce_oracle([x.numpy() for x in xs], 64)
    for algo in ("staged", "push"):
        for o in emulated_allreduce([x.cuda() for x in xs], mode="quant", algo=algo, block_numel=64):
            assert np.array_equal(o.cpu().numpy().view(np.int32), want.view(np.int32)), algo


@pytest.mark.parametrize("block", [64, 128, 256, 512, 1024])
def test_the_largest_of_a_block_wherever_it_lies(block):
    """... with both signs, beside NaN, which never wins, and in blocks of nothing else than zeros of both signs."""
    for numel in (1 << 17, SMALLEST):  # the streaming kernels, and those for ranks that share a GPU
        xs = [x * 1e-3 for x in _inputs(2, numel, torch.float32, block)]
        blocks = numel // block
        at = torch.arange(blocks) * block + torch.arange(blocks) * 37 % block
        xs[0][at] = torch.where(torch.arange(blocks) % 2 == 0, 1.0, -1.0) * 2.0 ** (torch.arange(blocks) % 40 - 20)
        xs[1][at[::3] // block * block + (at[::3] + 5) % block] = float("nan")
        for x in xs:
            x.view(blocks, block)[::7] = 0.0
            x.view(blocks, block)[::7, ::3] = -0.0
        want = quant_allreduce_oracle([x.numpy() for x in xs], block)
        for algo in ("staged", "push"):
            for o in emulated_allreduce([x.cuda() for x in xs], mode="quant", algo=algo, block_numel=block):
                assert np.array_equal(o.cpu().numpy().view(np.int32), want.view(np.int32)), (algo, numel)


@pytest.mark.parametrize("block", [32, 64, 128, 256, 512, 1024])
def test_one_barrier_exact_at_the_ends_of_rows_and_blocks(block):
    for n in (1, 2, 3, 8):
        for numel in (1, 127, 129, 255, 256, 257, 1023, 1025, 2048 + 130, 20000 + 3):
            for dtype in (torch.float32, torch.bfloat16):
                xs = _inputs(n, numel, dtype, numel + n)
                want = torch.from_numpy(quant_allreduce_oracle([x.float().numpy() for x in xs], block)).to(dtype)
                outs = [torch.full((numel + 2,), 7.0, dtype=dtype, device="cuda") for _ in range(n)]
                views = [o[r % 2:r % 2 + numel] for r, o in enumerate(outs)]  # every other one begins beside a vector
                emulated_allreduce([x.cuda() for x in xs], mode="quant", algo="oneshot", block_numel=block, outputs=views)
                for r, o in enumerate(outs):
                    assert torch.equal(views[r].cpu(), want), (n, numel, dtype)
                    assert bool((o[:r % 2] == 7).all()) and bool((o[r % 2 + numel:] == 7).all())


@pytest.mark.parametrize("block", [1, 6, 16, 96, 100, 129, 384, 2048])
def test_one_barrier_exact_with_blocks_of_any_size(block):
    """... which no context has: not a power of two, or not from 32 to 1024. Over several channels, too."""
    for n in (2, 3, 8):
        for numel in (1, 95, 383, 385, 4096, 20000 + 3):
            for dtype in (torch.float32, torch.bfloat16):
                xs = _inputs(n, numel, dtype, numel + n)
                want = torch.from_numpy(quant_allreduce_oracle([x.float().numpy() for x in xs], block)).to(dtype)
                for o in emulated_allreduce([x.cuda() for x in xs], mode="quant", algo="oneshot", block_numel=block, slot_bytes=16384):
                    assert torch.equal(o.cpu(), want), (n, numel, dtype)


def test_a_rank_without_alignment_takes_the_streaming_kernels():
    numel = SMALLEST + 7
    xs = _inputs(2, numel + 1, torch.float32, 3)
    ys = [xs[0].cuda()[1:], xs[1].cuda()[:-1]]
    want = quant_allreduce_oracle([y.cpu().numpy() for y in ys], 64)
    for algo in ("staged", "push"):
        for o in emulated_allreduce(ys, mode="quant", algo=algo, block_numel=64):
            assert np.array_equal(o.cpu().numpy(), want)


@pytest.mark.parametrize("mode", ["quant", "sum"])
@pytest.mark.parametrize("n, algo", [(2, "push"), (2, "staged"), (3, "staged"), (8, "push")])
def test_a_rank_that_never_comes(n, algo, mode):
    """The waits for it run out: the call says so, whichever of them is the first, and the next one is as good as ever."""
    xs = _inputs(n, SMALLEST + 5, torch.float32, n)
    for timeout in (0.02, 0.001):
        with pytest.raises(NativeError, match="kernel status") as e:
            emulated_allreduce_with([x.cuda() for x in xs], present=n - 1, timeout=timeout, mode=mode, algo=algo)
        assert int(str(e.value).split("kernel status")[1].split()[0]) & 15 == 1  # timeout
    outs = emulated_allreduce([x.cuda() for x in xs], mode=mode, algo=algo)
    if mode == "quant":
        want = quant_allreduce_oracle([x.numpy() for x in xs], 256)
        assert all(np.array_equal(o.cpu().numpy(), want) for o in outs)
    else:
        assert torch.allclose(outs[0].cpu().double(), sum(x.double() for x in xs), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("mode", ["quant", "sum"])
@pytest.mark.parametrize("n", [1, 2, 4])
def test_waits_that_run_out_at_once(n, mode):
    """Limits in the range of what the waits take, so that any of them may be the first to run out: a call either fails or
    has the result."""
    xs = _inputs(n, (1 << 21) + 5, torch.int32 if mode == "sum" else torch.float32, n)
    want = int_allreduce_oracle([x.numpy() for x in xs]) if mode == "sum" else quant_allreduce_oracle([x.numpy() for x in xs], 256)
    ys = [x.cuda() for x in xs]
    for algo in ("staged",) if n == 1 else ("staged", "push"):
        for timeout in (1e-9, 1e-6, 4e-6, 8e-6, 12e-6, 16e-6, 20e-6, 30e-6):
            outs = [torch.zeros_like(y) for y in ys]
            try:
                emulated_allreduce_with(ys, timeout=timeout, mode=mode, algo=algo, outputs=outs)
            except NativeError as e:
                assert int(str(e).split("kernel status")[1].split()[0]) & 15 == 1
                continue
            assert all(np.array_equal(o.cpu().numpy(), want) for o in outs), (algo, timeout)


@pytest.mark.parametrize("kernels", ["one_gpu", "streaming"])
@pytest.mark.parametrize("algo", ["staged", "push"])
def test_epochs_that_start_over(algo, kernels):
    """The tags of exponent words have 24 bits: before they come round, words and flags are cleared and epochs start at 0
    again. Jobs of other lengths before and behind that, in the same staging memory, never take a word for another's."""
    rng = np.random.default_rng(7)
    for n in (2, 3, 8):
        for case in range(14):
            numel = int(rng.integers(1, 3 * SMALLEST if case % 2 else 5000))
            xs = _inputs(n, max(numel, 3), torch.float32, case)
            want = quant_allreduce_oracle([x.numpy() for x in xs], 64)
            outs = emulated_allreduce_with([x.cuda() for x in xs], kernels=kernels, epoch_limit=(1, 9, 30)[case % 3], mode="quant", algo=algo,
                                           block_numel=64, slot_bytes=16384, channels=3, repeats=1 + case % 3)
            assert all(np.array_equal(o.cpu().numpy(), want) for o in outs), (n, case)


@pytest.mark.parametrize("numel", [1000, SMALLEST])
def test_outputs_without_room_for_the_result(numel):
    xs = [torch.ones(numel, device="cuda") * r for r in range(2)]
    good = torch.empty(numel, device="cuda")
    for bad in (torch.empty(numel - 1, device="cuda"), torch.empty(2 * numel, device="cuda")[::2], torch.empty(numel, device="cuda", dtype=torch.bfloat16),
                torch.empty(numel, device="cuda", dtype=torch.float64), torch.empty(numel)):
        for outs in ([good, bad], (bad, good)):
            with pytest.raises(ValueError):
                emulated_allreduce(xs, mode="sum", outputs=outs)
    for outs in ([], [good], [good] * 3):
        with pytest.raises(ValueError):
            emulated_allreduce(xs, mode="sum", outputs=outs)
    # What has more room than that, and pinned memory.
    for outs in ([torch.zeros(numel + 5, device="cuda") for _ in xs], [torch.zeros(numel, pin_memory=True) for _ in xs]):
        for o in emulated_allreduce(xs, mode="sum", outputs=outs):
            assert bool((o[:numel] == 1).all()) and bool((o[numel:] == 0).all())


def test_arguments_that_python_looks_at():
    xs = [torch.ones(5000, device="cuda") * r for r in range(3)]
    for seq in (xs, tuple(xs)):  # with and without the native call
        for o in emulated_allreduce(seq, mode="sum"):
            assert torch.equal(o, torch.full_like(o, 3.0))
    with pytest.raises(AssertionError):
        emulated_allreduce([xs[0], xs[1][:100]], mode="sum")
    with pytest.raises(KeyError):
        emulated_allreduce([x.double() for x in xs], mode="sum")
    with pytest.raises(KeyError):
        emulated_allreduce(xs, mode="maximum")
