"""Quantize a tensor that lives in (pinned) host memory, overlapping PCIe copies with the kernel.

Rows are independent once `global_scale_inv` is known, so the input is cut into row chunks that are a
multiple of 128 rows (one chunk's scales are then a contiguous slab of the tiled scale buffer).  Chunk i is
copied host->device on one stream, quantized on a second, and its codes and scales are copied back on a
third, with events ordering the three; chunk i+1's upload runs while chunk i is quantized and chunk i-1
is downloaded.  The result is byte-identical to quantizing the whole tensor in one launch.

The link bounds it: the upload takes 1.21 of the 1.28 ms of a [4096, 4096] fp32 matrix.  What is left beside it is
the last chunk's kernel and download, which is why the chunks get smaller towards the end, and the host time
of the calls, which is why one compiled call issues them all.
"""
from __future__ import annotations

import torch

from . import _lib
from .kernels import _launch
from .sharding import round_up


def chunk_plan(rows: int, chunk_rows: int) -> list[tuple[int, int]]:
    """[start, stop) row ranges; every start is a multiple of 128."""
    if chunk_rows < 128 or chunk_rows % 128:
        raise ValueError("chunk_rows must be a positive multiple of 128")
    return [(a, min(a + chunk_rows, rows)) for a in range(0, rows, chunk_rows)]


# Upload per chunk: every copy costs the link ~4 us beside its bytes, and a large last chunk leaves its kernel and download
# uncovered.  [4096, 4096] fp32 / bf16, us: 2 MB 1455 / 765, 4 MB 1339 / 718, 8 MB 1297 / 698, 16 MB 1284 / 701 (the link alone:
# 1211 / 608).  The halving ends at 4 MB, small chunks cost more than they uncover ([1888, 2304] bf16 with 1 / 4 / 6 MB 229 / 219 /
# 221, [1024, 4096] bf16 222 / 213 / 222).  Up to ONE_CHUNK_BYTES one chunk on the caller's stream beats the round trips between
# streams (3.2 MB: 100 against 109 us).
CHUNK_BYTES = 16 << 20
LAST_CHUNK_BYTES = 4 << 20
ONE_CHUNK_BYTES = 4 << 20


def tapered_plan(rows: int, row_bytes: int, chunk_rows: int) -> list[tuple[int, int]]:
    """chunk_plan with chunks of about CHUNK_BYTES (at most chunk_rows), the last ones halved down to LAST_CHUNK_BYTES:
    nothing overlaps the last chunk's kernel and download.  A tensor of up to ONE_CHUNK_BYTES is one chunk."""
    chunk_plan(rows, chunk_rows)      # checks chunk_rows
    if rows * row_bytes <= ONE_CHUNK_BYTES and rows <= chunk_rows:
        return [(0, rows)]
    def rows_of(size: int) -> int:
        return max(128, size // max(row_bytes, 1) // 128 * 128)

    step, least = min(chunk_rows, rows_of(CHUNK_BYTES)), rows_of(LAST_CHUNK_BYTES)
    plan, a = [], 0
    while a < rows:
        left = rows - a
        take = step if left > 2 * step else min(step, max(least, round_up((left + 1) // 2, 128)))
        plan.append((a, min(a + take, rows)))
        a += take
    return plan


class HostQuantizer:
    """Reusable staging buffers, streams and events for one (rows, dim, dtype, variant) shape."""

    def __init__(self, rows: int, dim: int, dtype=torch.bfloat16, device="cuda", chunk_rows: int = 1024,
                 variant: int = _lib.VARIANT_MSE, lower: int = -3, upper: int = 7, depth: int = 3):
        if dim % 16:
            raise ValueError("dim must be divisible by 16")
        self.rows, self.dim, self.dtype, self.device = rows, dim, dtype, torch.device(device)
        self.variant, self.lower, self.upper = variant, lower, upper
        self.blocks = dim // 16
        self.k_pad = round_up(self.blocks, 4)
        self.plan = tapered_plan(rows, dim * torch.empty((), dtype=dtype).element_size(), chunk_rows)
        cr = max((b - a for a, b in self.plan), default=0)
        self.depth = min(depth, max(len(self.plan), 1))
        self.stage_in = [torch.empty((cr, dim), dtype=dtype, device=self.device) for _ in range(self.depth)]
        self.stage_codes = [torch.empty((cr, dim // 2), dtype=torch.uint8, device=self.device) for _ in range(self.depth)]
        self.stage_scales = [torch.empty(round_up(cr, 128) * self.k_pad, dtype=torch.uint8, device=self.device)
                             for _ in range(self.depth)]
        self.s_up, self.s_run, self.s_down = (torch.cuda.Stream(self.device) for _ in range(3))
        _lib.lib()
        self._pipe = _lib.fast.make_host_pipe(
            self.s_up.device_index, _lib.dtype_code(dtype), variant, lower, upper, rows, dim, tuple(r for ab in self.plan for r in ab),
            *(tuple(t.data_ptr() for t in ts) for ts in (self.stage_in, self.stage_codes, self.stage_scales)),
            self.s_up.cuda_stream, self.s_run.cuda_stream, self.s_down.cuda_stream)

    def __call__(self, x_host: torch.Tensor, gs_inv: torch.Tensor, codes_host: torch.Tensor,
                 scales_host: torch.Tensor, importance: torch.Tensor | None = None) -> None:
        """x_host [rows, dim] (pinned for real overlap); codes_host uint8 [rows, dim/2]; scales_host uint8
        [round_up(rows,128) * round_up(dim/16,4)] (tiled layout).  Returns once everything has been enqueued;
        the caller synchronises (e.g. torch.cuda.synchronize()) before reading the host outputs.  Calls from several threads,
        each on a stream of its own, go one after the other."""
        if tuple(x_host.shape) != (self.rows, self.dim) or x_host.dtype != self.dtype:
            raise ValueError("input does not match the shape this quantizer was built for")
        if self.rows == 0 or self.dim == 0:
            return
        if self.variant != _lib.VARIANT_WEIGHTED:
            importance = None
        elif importance is None:
            raise ValueError("the weighted variant needs an importance vector")
        else:
            if importance.numel() < self.dim or importance.device != self.stage_in[0].device:
                raise ValueError(f"importance must hold {self.dim} values on {self.stage_in[0].device}")
            importance = importance.float().contiguous()
            if importance.numel() > self.dim:
                importance = importance.reshape(-1)[:self.dim]
        if _lib.fast.host_pipe_call(self._pipe, x_host, gs_inv, codes_host, scales_host, importance):
            return
        # something about the operands: name it, or bring it into the form the call takes
        _launch._check_common(self.stage_in[0], gs_inv)
        if codes_host.ndim != 2 or codes_host.shape[0] < self.rows or codes_host.shape[1] != self.dim // 2:
            raise ValueError(f"codes_host must be [{self.rows}, {self.dim // 2}]")
        need = round_up(self.rows, 128) * self.k_pad
        if not scales_host.is_contiguous() or scales_host.numel() * scales_host.element_size() < need:
            raise ValueError(f"scales_host must be a contiguous buffer of {need} bytes")

        def plain(t):
            return t.detach().as_subclass(torch.Tensor)

        target = plain(codes_host)[:self.rows]
        direct = target.dtype == torch.uint8 and target.is_contiguous()
        codes = target if direct else torch.empty((self.rows, self.dim // 2), dtype=torch.uint8)
        if importance is not None:
            importance = plain(importance)
            if importance.data_ptr() & 15:
                importance = importance.clone()
        if not _lib.fast.host_pipe_call(self._pipe, plain(x_host).contiguous(), plain(gs_inv), codes, plain(scales_host), importance):
            raise ValueError("operands the host pipeline does not take")
        if not direct:      # strided, or of another type
            torch.cuda.current_stream(self.device).synchronize()
            target.copy_(codes)
