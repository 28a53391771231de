"""Edges of the kernels' dispatch and of the host path around them, each against the CPU oracle
or a plain PyTorch reference of the same operation."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import switchml_b200 as sml
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


@pytest.fixture
def ctx():
    c = sml.Context.get_instance()
    yield c
    if c.state() == sml.ContextState.RUNNING:
        c.stop()


@pytest.mark.parametrize("block", [32, 64, 256, 1024])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_worker_exact_pass_at_its_edges(ctx, dtype, block):
    """Every vector width (what the addresses allow), whole and partial last chunks, blocks of part of
    a row up to all rows; values of all scales, zero blocks, infinities' neighbours."""
    assert ctx.start(sml.make_config("cuda", packet_numel=block, mode="int32_quant", launch="inline"))
    gen = torch.Generator(device="cuda").manual_seed(block)
    for numel in (1, block - 1, 1023, 1024, 1025, 8192, 3 * 8192 + 1024 + block + 5):
        for off_in, off_out in ((0, 0), (1, 1), (2, 2), (4, 4), (0, 1), (3, 8)):
            base = torch.randn(numel + 16, device="cuda", generator=gen) * torch.logspace(-35, 35, numel + 16, device="cuda")
            base[numel // 2: numel // 2 + 2 * block] = 0.0
            x = base.to(dtype)[off_in:off_in + numel]
            frame = torch.full((numel + 16,), 7.0, dtype=dtype, device="cuda")
            y = frame[off_out:off_out + numel]
            ctx.all_reduce(x, y)
            want = torch.from_numpy(quant_allreduce_oracle([x.float().cpu().numpy()], block)).to(dtype)
            assert torch.equal(y.cpu(), want), (numel, off_in, off_out)
            assert bool((frame[:off_out] == 7).all()) and bool((frame[off_out + numel:] == 7).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int32, torch.uint8])
def test_one_worker_sum_copies_every_alignment(ctx, dtype):
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline"))
    for numel in (1, 7, 15, 16, 17, 8191, 65536 + 3):
        for off_in in (0, 1, 3):
            for off_out in (0, 1, 2, 5):
                x = torch.randint(1, 200, (numel + 8,), device="cuda").to(dtype)[off_in:off_in + numel]
                frame = torch.zeros(numel + 8, dtype=dtype, device="cuda")
                ctx.all_reduce(x, frame[off_out:off_out + numel])
                want = torch.zeros(numel + 8, dtype=dtype)
                want[off_out:off_out + numel] = x.cpu()
                assert torch.equal(frame.cpu(), want), (numel, off_in, off_out)


@pytest.mark.parametrize("launch", ["worker", "inline"])
def test_many_jobs_from_several_threads_and_streams(ctx, launch):
    """More jobs in flight than are enqueued directly, waited for by several threads at once, some by
    status alone; jobs on other streams than their predecessors."""
    assert ctx.start(sml.make_config("cuda", packet_numel=64, mode="int32_quant", launch=launch))
    numel, errors = 5000, []
    want = {}
    xs = [torch.randn(numel, device="cuda") * 2.0 ** i for i in range(4)]
    for i, x in enumerate(xs):
        want[i] = quant_allreduce_oracle([x.cpu().numpy()], 64)

    def walk(which):
        try:
            stream = torch.cuda.Stream()
            ys = [torch.zeros(numel, device="cuda") for _ in range(8)]
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                jobs = [ctx.all_reduce_async(xs[which], ys[k % 8]) for k in range(400)]
                jobs[-1].stream_wait()
                total = ys[0] + ys[7]
            stream.synchronize()
            assert np.array_equal(total.cpu().numpy(), 2 * want[which])
            for k, j in enumerate(jobs):
                if k % 50 == 7:
                    while j.status() not in (sml.JobStatus.FINISHED, sml.JobStatus.FAILED):
                        pass
                else:
                    assert j.wait(20000 if k % 2 else None) == sml.JobStatus.FINISHED, j.error()
                j.release()
        except BaseException as e:  # noqa: B902 - handed to the main thread
            errors.append(e)

    threads = [threading.Thread(target=walk, args=(w,)) for w in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    ctx.wait_for_all_jobs()
    st = ctx.get_stats()
    assert st["jobs_finished"] == 1600 and st["jobs_failed"] == 0


@pytest.mark.parametrize("launch", ["worker", "inline"])
def test_one_worker_counts_its_jobs(ctx, launch):
    """Jobs with a kernel and without one (a sum of one term, in place)."""
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch=launch))
    x = torch.zeros(1000, device="cuda")
    for out in (None, torch.empty_like(x), None):
        ctx.all_reduce(x, out)
    counted = ctx.get_stats()["backend"]
    assert counted["jobs_launched"] == 3 and counted["kernel_launches"] == 1


def test_a_brief_job_does_not_hold_up_its_producer(ctx):
    """launch = worker: jobs run beside what the producer's stream does. A short job behind long ones comes after
    them, but the stream that it was submitted on does not."""
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="worker"))
    x = torch.ones(1 << 28, device="cuda")
    y, z = torch.zeros_like(x), torch.zeros(1000, device="cuda")
    ctx.all_reduce(z, torch.empty_like(z))  # the first launch of a kernel loads it
    torch.cuda.synchronize()
    long_jobs = [ctx.all_reduce_async(x, y) for _ in range(20)]  # some 300 us each
    brief = ctx.all_reduce_async(y[:1000], z)
    here = torch.cuda.Event()
    here.record()
    here.synchronize()
    assert long_jobs[-1].status() != sml.JobStatus.FINISHED
    assert brief.wait() == sml.JobStatus.FINISHED and bool((z == 1).all())
    assert [j.wait() for j in long_jobs] == [sml.JobStatus.FINISHED] * 20


def test_a_stream_whose_handle_was_another_ones_waits(ctx):
    """A stream that is made after the job's own one was destroyed, and may have got its handle, comes after the
    job when it is told to."""
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline"))
    cudart = torch.cuda.cudart()

    def new_stream():
        handle = ctypes.c_void_p()
        assert int(cudart.cudaStreamCreate(ctypes.addressof(handle))) == 0
        return handle.value

    x = torch.ones(1 << 27, device="cuda")
    y, z = torch.zeros_like(x), torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    first, others = new_stream(), []
    jobs = [ctx.all_reduce_async(x, y, stream=first) for _ in range(10)]
    cudart.cudaStreamDestroy(first)
    while len(others) < 64 and (not others or others[-1] != first):
        others.append(new_stream())
    jobs[-1].stream_wait(others[-1])
    with torch.cuda.stream(torch.cuda.ExternalStream(others[-1])):
        z.copy_(y[-1000:])
    torch.cuda.synchronize()
    assert bool((z == 1).all())
    for j in jobs:
        assert j.wait() == sml.JobStatus.FINISHED
    for handle in others:
        cudart.cudaStreamDestroy(handle)


@pytest.mark.parametrize("mode", ["float_sum", "int32_quant"])
@pytest.mark.parametrize("numel,chunk", [(1, 1 << 24), (3, 2), ((1 << 18) + 1, 1 << 24), ((1 << 20) + 77, 1 << 18),
                                         (5_000_003, 1 << 24)])
def test_host_pipeline_chunks(ctx, mode, numel, chunk):
    """Chunks that divide the tensor and that do not; twice through the same buffers."""
    from switchml_b200.parallel.host_pipeline import HostAllReduce
    assert ctx.start(sml.make_config("cuda", packet_numel=64, mode=mode, launch="inline"))
    hx, hy = torch.empty(numel, pin_memory=True), torch.zeros(numel, pin_memory=True)
    pipe = HostAllReduce(ctx, numel, torch.float32, chunk_numel=chunk)
    for scale in (1.0, 1e-3):
        hx.copy_(torch.randn(numel) * scale)
        assert pipe.run(hx, hy) is hy
        if mode == "float_sum":
            assert torch.equal(hx, hy)
        else:
            want = np.concatenate([quant_allreduce_oracle([hx[lo:hi].numpy()], 64) for lo, hi in pipe.bounds])
            assert np.array_equal(hy.numpy(), want)
    pipe.close()


def test_host_pipeline_looks_at_its_tensors(ctx):
    """Tensors that are too short or of another shape are refused, longer, strided and converted ones are not."""
    from switchml_b200.parallel.host_pipeline import HostAllReduce
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline"))
    numel = 1000
    pipe = HostAllReduce(ctx, numel, torch.float32)
    x, y = torch.arange(2.0 * numel).pin_memory(), torch.zeros(numel).pin_memory()
    for bad in (x[:numel - 1], x[:numel].view(10, 100), x.view(2, numel)):
        with pytest.raises(RuntimeError):
            pipe.run(bad, y)
    for bad in (y[:numel - 1], y.view(10, 100)):
        with pytest.raises(RuntimeError):
            pipe.run(x, bad)
    for good in (x, x[::2], x.to(torch.int32), x.cuda()):
        out = torch.zeros(2 * numel)
        assert pipe.run(good, out[::2]) is not None
        assert torch.equal(out[::2], good[:numel].float().cpu()) and bool((out[1::2] == 0).all())


def test_host_pipeline_refuses_types_as_the_context_does(ctx):
    from switchml_b200.parallel.host_pipeline import HostAllReduce
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline"))
    x = torch.zeros(10, dtype=torch.float64).pin_memory()
    with pytest.raises(TypeError):
        HostAllReduce(ctx, 10, torch.float64).run(x, torch.empty_like(x))


def test_host_pipeline_of_nothing(ctx):
    from switchml_b200.parallel.host_pipeline import HostAllReduce
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline"))
    hx, hy = torch.empty(0, pin_memory=True), torch.empty(0, pin_memory=True)
    pipe = HostAllReduce(ctx, 0, torch.float32)
    assert pipe.bounds == [] and pipe.run(hx, hy) is hy


def test_host_pipeline_leaves_nothing_in_flight_when_it_fails(ctx):
    """A call that ends with an error, here because the context was stopped, has ended on the GPU too."""
    from switchml_b200.parallel.host_pipeline import HostAllReduce
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline"))
    numel = 1 << 26
    hx, hy = torch.ones(numel, pin_memory=True), torch.zeros(numel, pin_memory=True)
    pipe = HostAllReduce(ctx, numel, torch.float32)
    ctx.stop()
    with pytest.raises(RuntimeError):
        pipe.run(hx, hy)
    assert pipe.s_in.query() and pipe.s_comm.query() and pipe.s_out.query()


@pytest.mark.parametrize("K", [1, 15, 16, 63, 64, 65, 100, 128, 129])
@pytest.mark.parametrize("M,N", [(8, 8), (128, 128), (136, 264), (1000, 520)])
def test_wgrad_short_reductions(K, M, N):
    """The kernel for short reductions at the edges of its range: K around a step and a stage, tiles
    that stick out of the matrix on either side. Neighbouring memory stays as it is."""
    from switchml_b200.ops.wgrad import wgrad_gemm
    gen = torch.Generator(device="cuda").manual_seed(K + M)
    dy = torch.randn(K, M, device="cuda", generator=gen).bfloat16()
    x = torch.randn(K, N, device="cuda", generator=gen).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    frame = torch.full((M * N + 128,), 3.0, device="cuda")
    out = frame[64:64 + M * N].view(M, N)
    wgrad_gemm(dy, x, out=out, error_flag=err)
    assert int(err) == 0
    assert torch.allclose(out, dy.float().t() @ x.float(), rtol=1e-4, atol=1e-4 * K ** 0.5)
    assert bool((frame[:64] == 3).all()) and bool((frame[64 + M * N:] == 3).all())


@pytest.mark.parametrize("K", [256, 257, 300, 320, 448, 1000, 4096])
@pytest.mark.parametrize("M,N", [(8, 8), (136, 264), (1000, 520), (4000, 5000)])
def test_wgrad_one_cta_per_tile_and_long_reductions(K, M, N):
    """The kernel for short reductions beyond their range: whole boxes of 128 rows, last stages that K fills and that
    it does not, one tile and several per CTA."""
    from switchml_b200.ops.wgrad import wgrad_gemm
    gen = torch.Generator(device="cuda").manual_seed(K + M)
    dy = torch.randn(K, M, device="cuda", generator=gen).bfloat16()
    x = torch.randn(K, N, device="cuda", generator=gen).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    frame = torch.full((M * N + 128,), 3.0, device="cuda")
    out = wgrad_gemm(dy, x, out=frame[64:64 + M * N].view(M, N), error_flag=err, two_cta=False)
    assert int(err) == 0
    ref = dy.double().t() @ x.double()
    assert float((out - ref).norm() / ref.norm()) < 1e-5
    assert bool((frame[:64] == 3).all()) and bool((frame[64 + M * N:] == 3).all())


@pytest.mark.parametrize("K", [511, 512, 513, 576])
def test_wgrad_at_the_line_between_its_kernels(K):
    """Either kernel, and whichever is chosen, for more tiles than there are CTAs."""
    from switchml_b200.ops.wgrad import wgrad_gemm
    gen = torch.Generator(device="cuda").manual_seed(K)
    dy = torch.randn(K, 4104, device="cuda", generator=gen).bfloat16()
    x = torch.randn(K, 3000, device="cuda", generator=gen).bfloat16()
    ref = dy.double().t() @ x.double()
    for two_cta in (None, False, True):
        out = wgrad_gemm(dy, x, two_cta=two_cta)
        assert float((out - ref).norm() / ref.norm()) < 1e-5, two_cta


@pytest.mark.parametrize("K,M,N", [(8192, 512, 512), (8192, 1024, 1024), (4160, 264, 520), (2048, 1000, 1032), (300, 256, 128),
                                   (1000, 3000, 2000), (640, 2048, 4104), (65, 8, 8), (8192, 2304, 1024)])
def test_wgrad_pairs_of_ctas_with_every_split(K, M, N):
    """Two CTAs per tile, both tile widths, alone and two or four pairs to a tile; the same bits twice."""
    from switchml_b200.ops.wgrad import wgrad_gemm
    gen = torch.Generator(device="cuda").manual_seed(K + N)
    dy = torch.randn(K, M, device="cuda", generator=gen).bfloat16()
    x = torch.randn(K, N, device="cuda", generator=gen).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = wgrad_gemm(dy, x, error_flag=err, two_cta=True)
    assert int(err) == 0
    ref = dy.double().t() @ x.double()
    assert float((out - ref).norm() / ref.norm()) < 1e-5
    assert torch.allclose(out.double(), ref, rtol=1e-4, atol=2e-4 * K ** 0.5)
    assert torch.equal(wgrad_gemm(dy, x, two_cta=True), out)


@pytest.mark.parametrize("K,M,N", [(200, 5000, 9000), (64, 304, 20000), (1000, 8000, 4104)])
def test_wgrad_pairs_with_many_tiles(K, M, N):
    """More tiles than pairs of CTAs, whose epilogues run beside the next tile's multiplications but for the last."""
    from switchml_b200.ops.wgrad import wgrad_gemm
    gen = torch.Generator(device="cuda").manual_seed(K + N)
    dy = torch.randn(K, M, device="cuda", generator=gen).bfloat16()
    x = torch.randn(K, N, device="cuda", generator=gen).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = wgrad_gemm(dy, x, error_flag=err, two_cta=True)
    assert int(err) == 0
    assert torch.allclose(out, dy.float().t() @ x.float(), rtol=1e-4, atol=2e-4 * K ** 0.5)
    assert torch.equal(wgrad_gemm(dy, x, two_cta=True), out)


@pytest.mark.parametrize("K,M", [(1, 8), (3, 72), (255, 64), (256, 128), (257, 520), (4097, 1000), (8192, 4096)])
def test_column_sums(K, M):
    """Clusters of one to eight CTAs, ragged rows and columns; the same bits twice."""
    from switchml_b200.ops.wgrad import column_sums
    dy = torch.randn(K, M, device="cuda", generator=torch.Generator(device="cuda").manual_seed(K + M)).bfloat16()
    out = column_sums(dy)
    assert torch.allclose(out.double(), dy.double().sum(0), rtol=1e-5, atol=1e-5 * K ** 0.5)
    assert torch.equal(column_sums(dy), out)


@pytest.mark.parametrize("shape,features", [((256, 64), 128), ((3, 17, 72), 40), ((1, 8), 8)])
@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("x_dtype", [torch.float32, torch.bfloat16])
def test_fused_wgrad_linear_against_plain_linear(ctx, shape, features, bias, x_dtype):
    """Forward and all gradients of the layer under autocast, against nn.Linear."""
    from switchml_b200.ops.wgrad import FusedWgradLinear, wait_pending
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline", symm_heap_mb=16))
    torch.manual_seed(3)
    plain = torch.nn.Linear(shape[-1], features, bias=bias, device="cuda")
    layer = FusedWgradLinear(shape[-1], features, bias=bias, device="cuda")
    layer.load_state_dict(plain.state_dict())
    layer.attach(ctx)
    x = torch.randn(shape, device="cuda").to(x_dtype)
    results = []
    for module in (plain, layer):
        xi = x.clone().requires_grad_()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = module(xi)
        y.backward(torch.linspace(-1, 1, y.numel(), device="cuda").view(y.shape).to(y.dtype))
        wait_pending()
        assert xi.grad.dtype == x_dtype and module.weight.grad.dtype == torch.float32
        results.append([y.detach(), xi.grad, module.weight.grad] + ([module.bias.grad] if bias else []))
    for got, want in zip(results[1], results[0]):
        assert got.dtype == want.dtype and got.shape == want.shape
        assert float((got.float() - want.float()).norm()) <= 1e-2 * float(want.float().norm()) + 1e-6


@pytest.mark.parametrize("features", [64, 192])
def test_fused_wgrad_linear_with_another_weight(ctx, features):
    """A weight that the gradient's buffer does not fit is refused, and the buffer's neighbours stay as they are."""
    from switchml_b200.ops.wgrad import FusedWgradLinear
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline", symm_heap_mb=16))
    layer = FusedWgradLinear(64, 128, bias=False, device="cuda").attach(ctx)
    after = ctx.symmetric_empty(1 << 16, torch.float32).fill_(5.0)
    layer.weight = torch.nn.Parameter(torch.randn(features, 64, device="cuda"))
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = layer(torch.randn(32, 64, device="cuda"))
    with pytest.raises(RuntimeError):
        y.sum().backward()
    assert bool((after == 5).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_worker_exact_pass_of_odd_values(ctx, dtype):
    """Infinities, NaN, values whose integer saturates, denormals, negative zeros and halves of the grid:
    whatever the arithmetic, the bits are the oracle's."""
    block = 64
    assert ctx.start(sml.make_config("cuda", packet_numel=block, mode="int32_quant", launch="inline"))
    gen = torch.Generator().manual_seed(1)
    x = torch.randn(40 * 1024 + 13, generator=gen)
    x[0:3] = torch.tensor([float("inf"), -float("inf"), float("nan")])
    x[1024] = 3.0e38
    x[2048] = -2.0 ** 127
    x[3072:3072 + block] = torch.randn(block, generator=gen) * 1e-42   # denormals
    x[4096:4096 + block] = -0.0
    x[5120] = float("nan")
    # Halves of the grid of a block whose exponent is 1: multiples of 2^-31, ties to even.
    ties = torch.randint(-2 ** 20, 2 ** 20, (1024,), generator=gen).float() * 2.0 ** -31
    x[6144:7168] = ties
    x[6144:7168:block] = 1.5
    x[7168:8192] = torch.randn(1024, generator=gen) * 2.0 ** -119          # below the smallest exponent
    x[8192:9216] = torch.randn(1024, generator=gen).clamp(-1.9, 1.9) * 2.0 ** 126
    x = x.to(dtype)
    want = torch.from_numpy(quant_allreduce_oracle([x.float().numpy()], block)).to(dtype)
    for offset in (0, 1):
        frame = torch.empty(x.numel() + offset, dtype=dtype, device="cuda")
        d = frame[offset:]
        d.copy_(x)
        ctx.all_reduce(d)
        bits = torch.int32 if dtype == torch.float32 else torch.int16
        assert torch.equal(d.cpu().view(bits), want.view(bits)), offset


@pytest.mark.parametrize("K,M,N", [(16, 64, 64), (64, 1000, 2056), (2048, 512, 512), (1024, 2048, 4096)])
def test_kernels_launched_early_keep_the_order_of_the_stream(ctx, K, M, N):
    """Each kernel reads what the one before it wrote, and writes what the one before that read; also with an
    ordinary kernel between, on a stream of its own and out of a graph."""
    from switchml_b200.ops.wgrad import column_sums, wgrad_gemm
    assert ctx.start(sml.make_config("cuda", mode="float_sum", launch="inline"))
    gen = torch.Generator(device="cuda").manual_seed(K)
    source = torch.randint(-2, 3, (6, K, M), device="cuda", generator=gen).bfloat16()
    x = torch.randint(-2, 3, (K, N), device="cuda", generator=gen).bfloat16()
    a, b = torch.empty_like(source[0]), torch.empty_like(source[0])
    dw, kept = torch.empty(M, N, device="cuda"), torch.empty(6, M, N, device="cuda")
    sums = []

    def walk(i):
        j = [ctx.all_reduce_async(source[i].view(-1), a.view(-1)), ctx.all_reduce_async(a.view(-1), b.view(-1))]
        wgrad_gemm(b, x, out=dw)
        j.append(ctx.all_reduce_async(dw.view(-1), kept[i].view(-1)))
        sums.append(column_sums(b))
        if i % 2:
            b.zero_()
        return j

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        jobs = [j for i in range(6) for j in walk(i)]
    stream.synchronize()
    for j in jobs:
        assert j.wait() == sml.JobStatus.FINISHED
        j.release()
    for i in range(6):  # whole numbers: exact in any order
        assert torch.equal(kept[i], source[i].float().t() @ x.float()), i
        assert torch.equal(sums[i], source[i].float().sum(0)), i

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        wgrad_gemm(a, x, out=dw)
        kept[0].copy_(dw)
        wgrad_gemm(b, x, out=dw)
        wgrad_gemm(a, x, out=kept[1])
    for i in (2, 4):
        a.copy_(source[i])
        b.copy_(source[i + 1])
        graph.replay()
        for out, d in ((kept[0], a), (kept[1], a), (dw, b)):
            assert torch.equal(out, d.float().t() @ x.float())
