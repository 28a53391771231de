"""Allreduce for callers whose tensors live in (pinned) host memory.

The reference's PyTorch integration always works this way: a CUDA tensor is copied to
pinned host memory, reduced by the CPU library and copied back, one step after the other
(pytorch_plugin/ProcessGroupSML.cpp:117-163). Here the direction is reversed — host data
is brought to the GPU, reduced over NVLink and returned. Three ways of doing it:

* pipelined copies (default): the tensor is cut into chunks; host→device copy, reduction (in
  place) and device→host copy of different chunks overlap on three streams. A native loop
  enqueues the chunks (csrc/backends/cuda/host_allreduce.cc).
* ``direct="out"``: chunks are copied host→device as above, but every chunk's reduction writes
  its result straight into the pinned output (the kernel's storer warps store over PCIe), so
  the device→host copy, its stream and the device copy of the result disappear.
* ``direct=True``: one job on the pinned buffers themselves. The aggregation kernel's loader
  warps read the input over PCIe while its storer warps write finished tiles back, so both
  directions and the NVLink phase overlap tile by tile inside a single launch, and no device
  copy of the tensor exists at all. (The cuda backend accepts any memory the GPU can reach:
  device, managed, or pinned host memory.)
"""
import math

import torch

from .._native import last_error, lib
from .context import _describe


def _chunk_bytes(nbytes):
    """Chunk of the copy pipeline for a message of this size. What the copies of the two directions do
    not overlap is one chunk, and a chunk costs some 10 us to start: at 55 GB/s the sum is least at
    sqrt(nbytes * 550 kB). A power of two, because copies of odd sizes ran a fifth slower (128 MiB:
    2.97 ms in 8 MiB chunks, 3.56 ms in 10.7 MiB chunks, 3.77 ms unchunked)."""
    return 1 << max(0, round(math.log2(math.sqrt(max(nbytes, 1) * 550e3))))


class HostAllReduce:
    """`chunk_numel`: the largest chunk; messages that it would leave in a few chunks are cut finer."""

    def __init__(self, ctx, numel, dtype, chunk_numel=1 << 24, device=None, direct=False):
        self.ctx = ctx
        self.numel = numel
        self.direct = direct
        dev = torch.device("cuda", torch.cuda.current_device() if device is None else device)
        self.s_comm = torch.cuda.Stream(device=dev)
        if direct is True:
            self.launches_per_run = 1
            return
        self.chunk = max(1, min(chunk_numel, numel))
        if not direct:
            esz = torch.empty((), dtype=dtype).element_size()
            self.chunk = max(1, min(self.chunk, _chunk_bytes(numel * esz) // esz))
        self.dx = torch.empty(numel, dtype=dtype, device=dev)
        self.s_in = torch.cuda.Stream(device=dev)
        self.s_out = torch.cuda.Stream(device=dev)
        self.bounds = [(o, min(o + self.chunk, numel)) for o in range(0, numel, self.chunk)]
        self.launches_per_run = len(self.bounds)

    def run(self, host_in, host_out):
        """Reduce `host_in` across workers into `host_out` (both pinned, 1-D). Blocks
        until `host_out` is complete."""
        if self.direct is True:
            job = self.ctx.all_reduce_async(host_in, host_out, stream=self.s_comm)
            status = job.wait()
            if status != 3:
                raise RuntimeError("allreduce on pinned memory failed: " + job.error())
            job.release()
            return host_out
        if self.direct == "out":
            jobs = []
            for lo, hi in self.bounds:
                with torch.cuda.stream(self.s_in):
                    self.dx[lo:hi].copy_(host_in[lo:hi], non_blocking=True)
                self.s_comm.wait_stream(self.s_in)
                jobs.append(self.ctx.all_reduce_async(self.dx[lo:hi], host_out[lo:hi], stream=self.s_comm))
            for j in jobs:
                if j.wait() != 3:
                    raise RuntimeError("allreduce into pinned memory failed: " + j.error())
                j.release()
            return host_out
        _, _, code, _, _ = _describe(self.dx)  # a type that the context does not take is refused here
        src, dst = host_in, host_out
        if not self._plain(src):
            # (an input of another shape is refused here)
            src = torch.empty(self.numel, dtype=self.dx.dtype, pin_memory=True).copy_(host_in[:self.numel])
        if not self._plain(dst):
            dst = torch.empty(self.numel, dtype=self.dx.dtype, pin_memory=True)
        with torch.cuda.device(self.dx.device):
            rc = lib().sml_host_allreduce(src.data_ptr(), dst.data_ptr(), self.dx.data_ptr(), self.numel,
                                          code, self.chunk, self.s_in.cuda_stream,
                                          self.s_comm.cuda_stream, self.s_out.cuda_stream)
        if rc != 0:
            raise RuntimeError("allreduce of host memory failed: " + last_error())
        if dst is not host_out:
            host_out[:self.numel].copy_(dst)
        return host_out

    def _plain(self, t):
        return (t.device.type == "cpu" and t.dtype == self.dx.dtype and t.dim() == 1 and t.is_contiguous()
                and t.numel() >= self.numel)

    def close(self):
        self.dx = None
