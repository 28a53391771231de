"""Weight-gradient GEMM on the tcgen05 tensor cores (csrc/kernels/wgrad_gemm.cu).

    dW = wgrad_gemm(dY, X)          # dY [tokens, out], X [tokens, in], bf16 -> dW [out, in] fp32

``FusedWgrad`` additionally sums dW over all workers inside the same kernel: the output
lives in the symmetric heap, every finished tile is reduced through the NVSwitch while
later tiles are still being computed.
"""
import ctypes
import os
import warnings
import weakref

import torch

from .._native import library_path, NativeError
from ..parallel.context import _current_stream

_LIB = None


class _FusedArgs(ctypes.Structure):
    _fields_ = [("rank", ctypes.c_int), ("nranks", ctypes.c_int),
                ("flags_peer", ctypes.c_void_p * 8), ("out_mc", ctypes.c_void_p),
                ("epoch", ctypes.c_ulonglong), ("timeout_ns", ctypes.c_ulonglong),
                ("scale", ctypes.c_float), ("work_counter", ctypes.c_void_p),
                ("mode", ctypes.c_int), ("gather_local", ctypes.c_void_p), ("gather_mc", ctypes.c_void_p),
                ("gather_counter", ctypes.c_void_p)]


def _lib():
    global _LIB
    if _LIB is None:
        path = library_path("libswitchml_gemm.so")
        if not os.path.exists(path):
            raise ImportError("libswitchml_gemm.so is not built (run build.py)")
        l = ctypes.CDLL(path)
        l.switchml_wgrad_gemm.restype = ctypes.c_int
        l.switchml_wgrad_gemm.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                          ctypes.c_int, ctypes.c_int, ctypes.POINTER(_FusedArgs),
                                          ctypes.c_void_p, ctypes.c_void_p]
        l.switchml_wgrad_gemm_2cta.restype = ctypes.c_int
        l.switchml_wgrad_gemm_2cta.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                               ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
        l.switchml_wgrad_gemm_auto.restype = ctypes.c_int
        l.switchml_wgrad_gemm_auto.argtypes = l.switchml_wgrad_gemm_2cta.argtypes
        l.switchml_column_sums.restype = ctypes.c_int
        l.switchml_column_sums.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
        l.switchml_wgrad_flag_words.restype = ctypes.c_int
        l.switchml_wgrad_flag_words.argtypes = [ctypes.c_int, ctypes.c_int]
        _LIB = l
    return _LIB


_ERRORS = {-1: "bad argument", -2: "M and N must be multiples of 8 and all tensors 16-byte aligned",
           -3: "cannot build the TMA tensor maps", -4: "kernel launch failed"}


def wgrad_gemm(dy, x, out=None, error_flag=None, two_cta=None):
    """dW[out_features, in_features] (fp32) = dY^T @ X for bf16 dY [K, M] and X [K, N].

    `two_cta`: use the kernel in which two CTAs share a tile (tcgen05 cta_group::2); default: by
    size (switchml_wgrad_gemm_auto)."""
    assert dy.is_cuda and x.is_cuda and dy.dtype == torch.bfloat16 and x.dtype == torch.bfloat16
    assert dy.dim() == 2 and x.dim() == 2
    K, M = dy.shape
    rows, N = x.shape
    assert rows == K
    if not dy.is_contiguous():
        dy = dy.contiguous()
    if not x.is_contiguous():
        x = x.contiguous()
    if out is None:
        out = torch.empty(M, N, dtype=torch.float32, device=dy.device)
    assert out.is_contiguous() and out.dtype == torch.float32 and out.numel() == M * N
    stream = _current_stream(dy.get_device())
    err_ptr = error_flag.data_ptr() if error_flag is not None else None
    l = _LIB or _lib()
    if two_cta is None:
        rc = l.switchml_wgrad_gemm_auto(dy.data_ptr(), x.data_ptr(), out.data_ptr(), M, N, K, err_ptr, stream)
    elif two_cta:
        rc = l.switchml_wgrad_gemm_2cta(dy.data_ptr(), x.data_ptr(), out.data_ptr(), M, N, K, err_ptr, stream)
    else:
        rc = l.switchml_wgrad_gemm(dy.data_ptr(), x.data_ptr(), out.data_ptr(), M, N, K, None, err_ptr, stream)
    if rc != 0:
        raise NativeError("wgrad_gemm: " + _ERRORS.get(rc, str(rc)))
    return out if out.shape == (M, N) else out.view(M, N)


def flag_words(M, N):
    return _lib().switchml_wgrad_flag_words(M, N)


class FusedWgrad:
    """Weight-gradient GEMM whose result is summed over all workers inside the kernel.

    One instance per weight matrix [M, N]. The gradient buffer and the tile flags live in
    the context's symmetric heap (every rank must create its instances in the same order).
    ``run(dy, x)`` leaves the reduced (scaled) gradient in ``self.grad`` on every rank; the
    kernel is enqueued on the current stream and needs no separate allreduce.
    """

    def __init__(self, ctx, M, N, scale=1.0, timeout_ms=20000.0, policy="auto"):
        self.ctx, self.M, self.N, self.scale = ctx, M, N, scale
        self.grad = ctx.symmetric_empty(M * N, torch.float32).view(M, N)
        words = flag_words(M, N)
        self.flags = ctx.symmetric_empty(words * 2, torch.int32)   # 64-bit words
        self.flags.zero_()
        self.error = torch.zeros(1, dtype=torch.int32, device=self.grad.device)
        local, peers, mc, _ = ctx.symmetric_info()
        self.nranks = sum(1 for p in peers if p)
        self.rank = peers.index(local)
        self.args = _FusedArgs()
        self.args.rank, self.args.nranks = self.rank, self.nranks
        flag_off = self.flags.data_ptr() - local
        for r in range(self.nranks):
            self.args.flags_peer[r] = peers[r] + flag_off
        self.args.out_mc = (mc + (self.grad.data_ptr() - local)) if mc else None
        self.args.epoch = 0
        self.args.timeout_ns = int(timeout_ms * 1e6)
        self.args.scale = scale
        self.counter = torch.zeros(1, dtype=torch.int32, device=self.grad.device)
        self.args.work_counter = self.counter.data_ptr()
        self.fused = self.nranks > 1 and bool(mc)
        self._symm = (local, mc)
        self.gather_buf = None     # [nranks * K * (M + N)] bf16 in the symmetric heap, made on first use
        self.gather_k = 0
        self.gather_counter = torch.zeros(1, dtype=torch.int32, device=self.grad.device)
        self.args.gather_counter = self.gather_counter.data_ptr()
        # "gather": the ranks exchange their (small) operands, every rank computes the tiles it
        # owns over all of them and broadcasts them: the gradient crosses the link once;
        # "fused": every rank multiplies its own operands and finished tiles are reduced through
        # the switch inside the GEMM kernel; "split": GEMM, then the in-place reduction as a
        # second kernel; "auto": gather when the operands of all ranks are less than a quarter of
        # the gradient (VGG's fully connected layers, K = batch), else split, which measured
        # faster than the fused reduction for long K.
        self.policy = policy
        torch.cuda.synchronize()

    def run(self, dy, x, side_stream=None):
        """Compute (and reduce) the gradient. With `side_stream` the kernel runs there,
        ordered after the current stream; call ``wait_pending()`` before using the result.
        Nothing later in backward needs dW, so this keeps the reduction off the critical path."""
        assert dy.dtype == torch.bfloat16 and x.dtype == torch.bfloat16
        dy, x = dy.contiguous(), x.contiguous()
        if side_stream is not None:
            side_stream.wait_stream(torch.cuda.current_stream(dy.device))
            dy.record_stream(side_stream)
            x.record_stream(side_stream)
            with torch.cuda.stream(side_stream):
                out = self.run(dy, x)
                ev = torch.cuda.Event()
                ev.record(side_stream)
            _PENDING.append(ev)
            return out
        if self.nranks == 1:
            return wgrad_gemm(dy, x, out=self.grad, error_flag=self.error)
        K = dy.shape[0]
        operand_bytes = self.nranks * K * (self.M + self.N) * 2
        gather = self.fused and (self.policy == "gather" or
                                 (self.policy == "auto" and 4 * operand_bytes <= self.M * self.N * 4))
        in_kernel = gather or (self.fused and self.policy == "fused")
        if gather and (self.gather_buf is None or self.gather_k != K):
            # every rank gets here with the same shapes in the same order, so the symmetric
            # allocations stay in step
            try:
                self.gather_buf = self.ctx.symmetric_empty(self.nranks * K * (self.M + self.N), torch.bfloat16)
            except MemoryError:
                # the heap is used up (it is never freed piecemeal); every rank sees the same heap,
                # so every rank falls back to the two-kernel path for this shape
                self.gather_buf, gather, in_kernel = None, False, self.fused and self.policy == "fused"
            else:
                self.gather_k = K
                local, mc = self._symm
                self.args.gather_local = self.gather_buf.data_ptr()
                self.args.gather_mc = mc + (self.gather_buf.data_ptr() - local)
        self.args.mode = 1 if gather else 0
        if in_kernel:
            self.args.epoch += 1
            self.counter.zero_()  # work queue of the in-kernel reduction starts at zero
            stream = torch.cuda.current_stream(dy.device).cuda_stream
            rc = _lib().switchml_wgrad_gemm(dy.data_ptr(), x.data_ptr(), self.grad.data_ptr(), self.M, self.N, K,
                                            ctypes.byref(self.args), self.error.data_ptr(), ctypes.c_void_p(stream))
            if rc != 0:
                raise NativeError("wgrad_gemm: " + _ERRORS.get(rc, str(rc)))
        else:
            wgrad_gemm(dy, x, out=self.grad, error_flag=self.error)
        if not in_kernel and self.nranks > 1:
            # No multicast mapping: reduce the finished gradient with the zero-copy kernel.
            job = self.ctx.all_reduce_async(self.grad.view(-1))
            job.stream_wait()
            job.release()
            if self.scale != 1.0:
                self.grad.mul_(self.scale)
        return self.grad


_PENDING = []
_SIDE_STREAMS = {}


def wait_pending(stream=None):
    """Order `stream` (default: current) after every weight-gradient kernel that was sent to
    a side stream since the last call."""
    if not _PENDING:
        return
    s = stream or torch.cuda.current_stream()
    while _PENDING:
        s.wait_event(_PENDING.pop())


def _side_stream(device):
    if device not in _SIDE_STREAMS:
        _SIDE_STREAMS[device] = torch.cuda.Stream(device=device, priority=-1)
    return _SIDE_STREAMS[device]


def column_sums(dy):
    """Sum over the rows of a bf16 matrix [K, M], in fp32 (M a multiple of 8, contiguous)."""
    assert dy.is_cuda and dy.dtype == torch.bfloat16 and dy.dim() == 2 and dy.is_contiguous()
    K, M = dy.shape
    out = torch.empty(M, dtype=torch.float32, device=dy.device)
    rc = (_LIB or _lib()).switchml_column_sums(dy.data_ptr(), out.data_ptr(), K, M, _current_stream(dy.get_device()))
    if rc != 0:
        raise NativeError("column_sums: " + _ERRORS.get(rc, str(rc)))
    return out


class _FusedLinearFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, plan):
        ctx.plan = plan
        ctx.save_for_backward(x, weight)
        ctx.bias_dtype = None if bias is None else bias.dtype
        return torch.nn.functional.linear(x, weight, bias)

    @staticmethod
    def backward(ctx, dy):
        x, weight = ctx.saved_tensors
        x2 = x.reshape(-1, x.shape[-1])
        dy2 = dy.reshape(-1, dy.shape[-1])
        dx = (dy2 @ weight.to(dy2.dtype)).reshape(x.shape) if ctx.needs_input_grad[0] else None
        with torch.no_grad():
            ctx.plan.run(dy2.to(torch.bfloat16), x2.to(torch.bfloat16))
        return dx, None, dy2.sum(0).to(ctx.bias_dtype) if ctx.bias_dtype is not None else None, None


class _PythonNode:
    """What lib/torch_switchml_linear.so offers, in Python: 150 instead of 20 us on the host for forward and backward
    of a small layer."""

    class Plan:
        def __init__(self, grad, error, run):
            self.run = run or (lambda dy, x: wgrad_gemm(dy, x, out=grad, error_flag=error))

    @staticmethod
    def fused_linear(x, weight, bias, plan):
        if torch.is_autocast_enabled():
            dt = torch.get_autocast_dtype("cuda")
            x, weight, bias = x.to(dt), weight.to(dt), bias.to(dt) if bias is not None else None
        return _FusedLinearFn.apply(x, weight, bias, plan)


_NODE = None


def _node():
    """lib/torch_switchml_linear.so, the layer's autograd node (csrc/torch/fused_linear.cc); built when it is
    missing, like the main library. Where it cannot be built or loaded (no headers of this PyTorch, no compiler) the
    node in Python does its work."""
    global _NODE
    if _NODE is None:
        import importlib.util
        _lib()
        path = library_path("torch_switchml_linear.so")
        try:
            if not os.path.exists(path):
                here = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
                spec = importlib.util.spec_from_file_location("_switchml_build", os.path.join(here, "build.py"))
                build = importlib.util.module_from_spec(spec)
                spec.loader.exec_module(build)
                build.build_torch_extension()
            spec = importlib.util.spec_from_file_location("torch_switchml_linear", path)
            module = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(module)
            _NODE = module
        except (ImportError, OSError, RuntimeError) as e:
            warnings.warn("FusedWgradLinear runs without lib/torch_switchml_linear.so: %s" % e)
            _NODE = _PythonNode
    return _NODE


class FusedWgradLinear(torch.nn.Linear):
    """``nn.Linear`` whose weight gradient is computed by ``FusedWgrad`` (fp32 weights,
    bf16 activations). Call ``attach(ctx)`` once after the context has started; the weight's
    ``.grad`` then aliases the symmetric gradient buffer and arrives already reduced."""

    wgrad = None
    overlap = True  # with several workers: run the weight-gradient kernel on a side stream
    _plan = None

    def attach(self, ctx, scale=1.0):
        self.wgrad = FusedWgrad(ctx, self.out_features, self.in_features, scale)
        self.weight.grad = self.wgrad.grad
        self.weight._sml_reduced_in_backward = True
        # The node keeps no reference to the layer: it would be one in a circle.
        wgrad, layer = self.wgrad, weakref.ref(self)

        def reduce_over_workers(dy, x):
            alive = layer()
            wgrad.run(dy, x, side_stream=_side_stream(dy.device) if alive is None or alive.overlap else None)

        # The side stream hides the sum over the workers; one worker has none, and nothing to do in Python.
        self._plan = _node().Plan(wgrad.grad, wgrad.error, reduce_over_workers if wgrad.nranks > 1 else None)
        return self

    def forward(self, x):
        if self._plan is None or not torch.is_grad_enabled():
            return super().forward(x)
        return _node().fused_linear(x, self.weight, self.bias, self._plan)
