"""Run the multi-rank aggregation kernels on ONE GPU.

Kernels of different ranks wait for each other, so they cannot be tested as separate
launches on a single device. Instead one cooperative launch plays all ranks: its
``blockIdx.y`` is the rank and every rank's staging memory lives on the same device
(csrc/kernels/allreduce_kernels.cu, ``AllReduceEmuKernel``). The code is that of ranks on GPUs of
their own, but for what only links ask for: the one-barrier kernel parks an input once and has
the others read it there, reducers keep more loads in flight, flags have GPU scope. The checked
build of the library runs the code between GPUs as it is. Messages of 2^18 elements per rank and
more ("staged" and "push") take pipelines made for ranks that share a GPU instead, whose results go
straight into all outputs (csrc/kernels/one_gpu_allreduce.cu), unless a tensor is off its 16-byte
boundary or in pinned memory; the checked build does not, unless it is asked to
(``emulated_allreduce_with``). Used by the GPU tests and for kernel profiling on one device.
"""
import ctypes

from .._native import lib, last_error, NativeError
from ..parallel.context import _emulate

ELEM = {"float32": 0, "int32": 1, "bfloat16": 2}
MODE = {"sum": 0, "quant": 1}
_ARRAYS = {}  # pointer array types by length
ALGO = {"staged": 0, "oneshot": 1, "push": 3}


def emulated_allreduce(inputs, mode="quant", algo="staged", block_numel=256, slot_bytes=131072,
                       slots_per_channel=2, channels=0, post_scale=1.0, repeats=1, outputs=None,
                       exponent_lookahead=-1):
    """Allreduce `inputs` (a list of equally sized 1-D CUDA tensors, one per virtual rank,
    all on the current device). Returns the list of per-rank outputs. `block_numel`: with "staged" and "push" a power of two
    from 32 to 1024 in the exact mode. `exponent_lookahead`: tiles by which the exact mode's exponents run ahead of their data
    (-1: the library's default) below 2^18 elements per rank; the pipelines above always run two ahead.

    `slot_bytes` and `slots_per_channel` are taken as they are (rounded to whole units of a tile) below 2^18 elements per rank. Above
    they are upper bounds: tiles and rings are cut to what stays in L2 and in shared memory. The results do not depend on either, but
    for the order in which plain sums add ("push": the owner of a shard first)."""
    if _emulate is not None and mode in MODE and algo in ALGO:
        try:
            done = _emulate(inputs, outputs, MODE[mode], ALGO[algo], block_numel, slot_bytes, slots_per_channel, channels, post_scale,
                            repeats, exponent_lookahead)
        except TypeError:  # a number of another type: below it is converted, or refused
            done = None
        if done is not None:
            return done
    return _through_ctypes(None, inputs, mode, algo, block_numel, slot_bytes, slots_per_channel, channels, post_scale, repeats, outputs,
                           exponent_lookahead)


class _Options(ctypes.Structure):
    _fields_ = [("kernels", ctypes.c_int), ("present", ctypes.c_int), ("timeout_ns", ctypes.c_uint64), ("epoch_limit", ctypes.c_uint64)]


_KERNELS = {None: 0, "streaming": 1, "one_gpu": 2}


def emulated_allreduce_with(inputs, kernels=None, present=0, timeout=0.0, epoch_limit=0, mode="quant", algo="staged", block_numel=256,
                            slot_bytes=131072, slots_per_channel=2, channels=0, post_scale=1.0, repeats=1, outputs=None, exponent_lookahead=-1):
    """The same for tests. `kernels`: "streaming" or "one_gpu", for "staged" and "push" of any size and in any build of the library
    (an error where those of ranks that share a GPU cannot). `present`: only the first `present` ranks come, so that the others' waits for the rest run out;
    `timeout`: seconds until any wait does (0: the library's 2 s). `epoch_limit`: epochs after which the flags and exponent words of
    the staging memory are cleared (0: 2^23)."""
    options = _Options(_KERNELS[kernels], present, int(timeout * 1e9), epoch_limit)
    return _through_ctypes(options, inputs, mode, algo, block_numel, slot_bytes, slots_per_channel, channels, post_scale, repeats, outputs,
                           exponent_lookahead)


def _through_ctypes(options, inputs, mode, algo, block_numel, slot_bytes, slots_per_channel, channels, post_scale, repeats, outputs,
                    exponent_lookahead):
    import torch
    n = len(inputs)
    x0 = inputs[0]
    dtype, numel = x0.dtype, x0.numel()
    elem = {torch.float32: 0, torch.int32: 1, torch.bfloat16: 2}[dtype]
    for x in inputs:
        assert x.is_cuda and x.is_contiguous() and x.dtype == dtype and x.numel() == numel
    if outputs is None:
        outputs = [torch.empty_like(x) for x in inputs]
    if len(outputs) != n:
        raise ValueError("%d outputs for %d inputs" % (len(outputs), n))
    for o in outputs:
        if torch.is_tensor(o) and (not o.is_contiguous() or o.dtype != dtype or o.numel() < numel or not (o.is_cuda or o.is_pinned())):
            raise ValueError("an output must be contiguous device (or pinned) memory of the inputs' type, with room for the result")
    esz_unit = n * max(block_numel, 128) * 4
    slot_bytes = max(esz_unit, slot_bytes // esz_unit * esz_unit)
    if algo == "push":  # a slot holds n-1 receive areas and n-1 result areas of one shard each
        slot_bytes = max(slot_bytes, 2 * esz_unit)
    array = _ARRAYS.get(n) or _ARRAYS.setdefault(n, ctypes.c_void_p * n)
    ins = array(*[x.data_ptr() for x in inputs])
    outs = array(*[o.data_ptr() for o in outputs])
    rc = lib().sml_emu_allreduce_with(ctypes.byref(_Options() if options is None else options), n, ins, outs, numel, elem, MODE[mode], ALGO[algo], block_numel,
                                      slot_bytes, slots_per_channel, channels, float(post_scale), repeats,
                                      int(exponent_lookahead))
    if rc != 0:
        raise NativeError("emulated allreduce failed (%d): %s" % (rc, last_error()))
    return outputs
