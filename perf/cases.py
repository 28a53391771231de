"""What a program that uses this library on one GPU has it do, as cases that can be timed.

Five kinds of work, each through the public Python interface:

``allreduce``  a job of the context (``Context.all_reduce_async`` / ``all_reduce``) with one worker:
               the exact mode's round trip through the block fixed point, or the plain sum
``aggregate``  the aggregation of several workers, all of them on this GPU
               (``ops.emulation.emulated_allreduce``)
``wgrad``      the weight-gradient GEMM (``ops.wgrad.wgrad_gemm``)
``layer``      forward and backward of ``FusedWgradLinear`` under bf16 autocast
``host``       a tensor in pinned host memory through ``HostAllReduce``

Sizes come from the size sweep (2^10 .. 2^28 elements), from 25 MB gradient buckets, from the
layers of the models in ``models/`` and from the tests.
"""
import torch

import switchml_b200 as sml
from switchml_b200.ops.emulation import emulated_allreduce
from switchml_b200.ops.wgrad import FusedWgradLinear, wait_pending, wgrad_gemm
from switchml_b200.parallel.host_pipeline import HostAllReduce

_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "int32": torch.int32, "uint8": torch.uint8}
_BYTES = {"float32": 4, "bfloat16": 2, "int32": 4, "uint8": 1}

_BUCKET = 25 * (1 << 20)  # bytes of a gradient bucket


def listed():
    return [
        # The shortest message of the size sweep, in stream order: nothing but latency.
        _allreduce("allreduce_1Ki_exact", 1 << 10, "float32", "int32_quant"),
        # A small tensor (a bias, a normalisation layer) through the call that waits for its result,
        # with the default launcher thread, as a program written for the original library makes it.
        _allreduce("allreduce_64Ki_blocking", (1 << 16) + 3, "float32", "int32_quant", call="blocking", block=1024),
        # A 25 MB gradient bucket, in place, exact mode: what the DDP hook submits during backward.
        _allreduce("allreduce_bucket_exact", _BUCKET // 4, "float32", "int32_quant", inplace=True),
        # The same for bf16 gradients.
        _allreduce("allreduce_bucket_exact_bf16", _BUCKET // 2, "bfloat16", "int32_quant", inplace=True),
        # A slice of a flat gradient buffer: an odd length that starts at an odd element.
        _allreduce("allreduce_ragged_exact", 1_000_003, "float32", "int32_quant", offset=1),
        # The headline message of 1 GiB, plain sum, out of place: the largest of the sweep.
        _allreduce("allreduce_1GiB_sum", 1 << 28, "float32", "float_sum"),
        # Aggregation of two workers in the exact mode (peer memory: shards are pushed to their owners).
        {"name": "aggregate_2_push_exact", "kind": "aggregate", "ranks": 2, "numel": 1 << 22, "dtype": "float32",
         "mode": "quant", "algo": "push", "block": 256},
        # Aggregation of four workers, plain sum, streamed through the slots.
        {"name": "aggregate_4_staged_sum", "kind": "aggregate", "ranks": 4, "numel": 1 << 24, "dtype": "float32",
         "mode": "sum", "algo": "staged", "block": 256},
        # Weight gradient of BERT-large's feed-forward layer at 16 x 512 tokens: bound by the tensor cores.
        {"name": "wgrad_bert_ffn", "kind": "wgrad", "k": 8192, "m": 4096, "n": 1024},
        # Weight gradient of VGG-19's fc6 at batch 32: bound by writing the gradient.
        {"name": "wgrad_vgg_fc6", "kind": "wgrad", "k": 32, "m": 4096, "n": 25088},
        # One feed-forward layer of BERT-large in training: forward, and backward with all its gradients.
        {"name": "layer_bert_ffn", "kind": "layer", "tokens": 8192, "out": 4096, "in": 1024},
        # A gradient bucket of a program that keeps its tensors in pinned host memory.
        {"name": "host_bucket_sum", "kind": "host", "numel": _BUCKET // 4},
    ]


def _allreduce(name, numel, dtype, mode, call="stream", inplace=False, offset=0, block=256):
    case = {"kind": "allreduce", "numel": numel, "dtype": dtype, "mode": mode, "call": call, "inplace": inplace,
            "offset": offset, "block": block}
    return dict(case, name=name) if name else case


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["allreduce"] * 5 + ["aggregate"] * 3 + ["wgrad"] * 2 + ["layer", "host"])
    if kind == "allreduce":
        mode = rng.choice(["int32_quant", "int32_quant", "float_sum"])
        exact = mode == "int32_quant"
        dtype = rng.choice(["float32", "float32", "bfloat16"] if exact else ["float32", "bfloat16", "int32", "uint8"])
        numel = _log_uniform(rng, 1 << 10, 1 << 28)
        if rng.random() < 0.5:
            numel = max(1 << 10, numel // 256 * 256)
        # A plain sum of one worker in place has nothing to do, so sums are out of place.
        return _allreduce("", numel, dtype, mode, call=rng.choice(["stream", "stream", "blocking"]),
                          inplace=exact and rng.random() < 0.5, offset=rng.choice([0, 0, 0, 1, 2]),
                          block=rng.choice([64, 256, 1024]))
    if kind == "aggregate":
        ranks = rng.choice([2, 4, 8])
        mode = rng.choice(["quant", "sum"])
        dtype = rng.choice(["float32", "float32", "bfloat16"] if mode == "quant" else ["float32", "bfloat16", "int32"])
        numel = _log_uniform(rng, 1 << 12, (1 << 26) // ranks)
        # Short messages take the one-barrier kernel, as in the cuda backend.
        algo = "oneshot" if numel < (1 << 18) else rng.choice(["push", "staged"])
        return {"kind": "aggregate", "ranks": ranks, "numel": numel, "dtype": dtype, "mode": mode, "algo": algo,
                "block": rng.choice([64, 256])}
    if kind == "wgrad":
        while True:
            # Either a batch of samples or a batch of tokens; features in multiples of 8.
            k = _log_uniform(rng, 8, 128) if rng.random() < 0.4 else _log_uniform(rng, 256, 8192)
            m, n = (8 * _log_uniform(rng, 64, 25088 // 8) for _ in range(2))
            if m * n <= 4096 * 25088 and 2 * k * m * n <= 2.5e11:
                return {"kind": "wgrad", "k": k, "m": m, "n": n}
    if kind == "layer":
        return {"kind": "layer", "tokens": _log_uniform(rng, 256, 8192), "out": 8 * _log_uniform(rng, 64, 512),
                "in": 8 * _log_uniform(rng, 64, 256)}
    return {"kind": "host", "numel": _log_uniform(rng, 1 << 16, 1 << 25)}


def _gradients(numel, dtype, gen):
    """Values like those of gradients: normal, of scales that vary along the tensor, with stretches
    that are zero (dead units, embedding rows that no token used)."""
    if dtype == torch.uint8:
        return torch.randint(0, 256, (numel,), device="cuda", dtype=dtype, generator=gen)
    if dtype == torch.int32:
        return torch.randint(-(1 << 20), 1 << 20, (numel,), device="cuda", dtype=dtype, generator=gen)
    x = torch.randn(numel, device="cuda", generator=gen)
    for part, scale in zip(x.chunk(8), (1e-3, 3e-2, 1e-4, 1.0, 2e-3, 1e-5, 1e-2, 5e-3)):
        part.mul_(scale)
    x[numel // 3: numel // 3 + numel // 16].zero_()
    return x.to(dtype)


_running = None  # configuration of the running context: it is a singleton of the process


def _context(backend_options, block=256):
    """The context with this configuration: started, or restarted when another one runs."""
    global _running
    text = sml.make_config("cuda", packet_numel=block, **backend_options)
    ctx = sml.Context.get_instance()
    if text != _running:
        torch.cuda.synchronize()
        if ctx.state() == sml.ContextState.RUNNING:
            ctx.stop()
        _running = None
        if not ctx.start(text):
            raise RuntimeError("the context did not start")
        _running = text
    return ctx, text


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "allreduce":
        ctx, text = _context({"mode": case["mode"], "launch": "inline" if case["call"] == "stream" else "worker"},
                             case["block"])
        numel, off, dtype = case["numel"], case["offset"], _DTYPES[case["dtype"]]
        flat = _gradients(numel + off, dtype, gen)
        x = flat[off:]
        y = None if case["inplace"] else torch.empty_like(flat)[off:]
        return {"kind": kind, "ctx": ctx, "config": text, "x": x, "y": y, "blocking": case["call"] == "blocking"}
    if kind == "aggregate":
        xs = [_gradients(case["numel"], _DTYPES[case["dtype"]], gen) for _ in range(case["ranks"])]
        options = {"mode": case["mode"], "algo": case["algo"], "block_numel": case["block"], "slot_bytes": 262144,
                   "slots_per_channel": 4, "outputs": [torch.empty_like(x) for x in xs]}
        return {"kind": kind, "xs": xs, "options": options}
    if kind == "wgrad":
        dy = torch.randn(case["k"], case["m"], device="cuda", generator=gen).mul_(1e-2).bfloat16()
        x = torch.randn(case["k"], case["n"], device="cuda", generator=gen).bfloat16()
        return {"kind": kind, "dy": dy, "x": x, "out": torch.empty(case["m"], case["n"], device="cuda")}
    if kind == "layer":
        # Gradients live in the context's symmetric heap, which is given back only as a whole: room for
        # the layers of many states.
        heap_mb = 64 + 48 * (case["out"] * case["in"] * 4 + (1 << 20)) // (1 << 20)
        ctx, text = _context({"mode": "float_sum", "launch": "inline", "symm_heap_mb": heap_mb})
        layer = FusedWgradLinear(case["in"], case["out"], device="cuda")
        with torch.no_grad():
            layer.weight.copy_(torch.randn(layer.weight.shape, device="cuda", generator=gen) * case["in"] ** -0.5)
            layer.bias.copy_(torch.randn(layer.bias.shape, device="cuda", generator=gen) * 1e-2)
        layer.attach(ctx)
        x = torch.randn(case["tokens"], case["in"], device="cuda", generator=gen).bfloat16().requires_grad_()
        dy = torch.randn(case["tokens"], case["out"], device="cuda", generator=gen).mul_(1e-2).bfloat16()
        return {"kind": kind, "config": text, "layer": layer, "x": x, "dy": dy}
    ctx, text = _context({"mode": "float_sum", "launch": "inline"})
    numel = case["numel"]
    hx = torch.empty(numel, pin_memory=True)
    hx.copy_(_gradients(numel, torch.float32, gen))
    return {"kind": kind, "config": text, "pipe": HostAllReduce(ctx, numel, torch.float32), "x": hx,
            "y": torch.empty(numel, pin_memory=True)}


def run(state):
    kind = state["kind"]
    if state.get("config", _running) != _running:
        raise RuntimeError("the context of this state has been stopped")
    if kind == "allreduce":
        ctx, x, y = state["ctx"], state["x"], state["y"]
        if state["blocking"]:
            ctx.all_reduce(x, y)
        else:
            job = ctx.all_reduce_async(x, y)
            job.stream_wait()
            job.release()
        return x if y is None else y
    if kind == "aggregate":
        return emulated_allreduce(state["xs"], **state["options"])
    if kind == "wgrad":
        return wgrad_gemm(state["dy"], state["x"], out=state["out"])
    if kind == "layer":
        layer, x = state["layer"], state["x"]
        x.grad = layer.bias.grad = None
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = layer(x)
        y.backward(state["dy"])
        wait_pending()
        return {"y": y.detach(), "dx": x.grad, "dw": layer.weight.grad, "db": layer.bias.grad}
    return state["pipe"].run(state["x"], state["y"])


def work(case):
    kind = case["kind"]
    if kind == "allreduce":
        return {"bytes": 2 * case["numel"] * _BYTES[case["dtype"]], "flops": 0}
    if kind == "aggregate":
        return {"bytes": 2 * case["ranks"] * case["numel"] * _BYTES[case["dtype"]], "flops": case["ranks"] * case["numel"]}
    if kind == "wgrad":
        k, m, n = case["k"], case["m"], case["n"]
        return {"bytes": 2 * k * (m + n) + 4 * m * n, "flops": 2 * k * m * n}
    if kind == "layer":
        t, o, i = case["tokens"], case["out"], case["in"]
        # x, dy read; y, dx written (bf16); the weight read, its gradient written (fp32); the bias and its gradient
        return {"bytes": 4 * t * (o + i) + 8 * o * i + 8 * o, "flops": 6 * t * o * i}
    return {"bytes": 2 * 4 * case["numel"], "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "aggregate" and case["mode"] == "sum" and case["dtype"] != "int32":
        return {"rel": 1e-2} if case["dtype"] == "bfloat16" else {"rel": 1e-6, "max": 1e-4}
    if kind == "wgrad":
        return {"rel": 2e-5}  # exact products of bf16 values, summed in fp32 in some order
    if kind == "layer":
        return {"rel": 1e-2}  # bf16 activations and gradients
    return "exact"
