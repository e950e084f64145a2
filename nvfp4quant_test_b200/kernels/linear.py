"""Preallocated building blocks for a decode loop that is launched eagerly (no CUDA graph).

`nvfp4_scaled_mm_grouped` and the quantizer entry points allocate their outputs, check their arguments and build
their argument arrays on every call; that is tens of microseconds of Python per call, several times what the GPU
needs for a decode-sized launch.  The classes here do that work once: buffers are allocated and arguments are
checked at construction, a call is one call into the library.  Outputs are reused from call to call (copy what must be kept), and
an instance serves one stream at a time.  Bits equal the allocating entry points'.
"""
from __future__ import annotations

import ctypes

import torch

from .. import _lib
from .. import helper as _helper
from . import kernel_ScaleSweep_MSE as _mse
from .kernel_fused import scalesweep_nvfp4_quant_with_global_scales
from .kernel_gemm import PreparedWeight, _scale_bytes, nvfp4_scaled_mm_multi
from .kernel_vllm import create_fp4_output_tensors


class ActivationQuantizer:
    """global scale -> ScaleSweep_MSE quantization of an activation [tokens, k] with one host call
    (nvfp4_quant_chain_multi_launch: two dependent launches, one up to 64 KiB).  Its buffers are an activation's: a PreparedWeight on
    them would be read while a later call rewrites them."""

    def __init__(self, tokens: int, k: int, device, fp8_max: float = _helper.FP8_E4M3_MAX_4OVER6,
                 dtype: torch.dtype = torch.bfloat16):
        if tokens < 1 or k < 16 or k % 16:
            raise ValueError("tokens >= 1 and k a positive multiple of 16 are required")
        self.tokens, self.k, self.dtype, self.fp8_max = tokens, k, dtype, float(fp8_max)
        self.device = torch.device(device)
        if self.device.type == "cuda" and self.device.index is None:
            self.device = torch.device("cuda", torch.cuda.current_device())   # tensors report an explicit index
        self._dtype_code = _lib.dtype_code(dtype)
        self.codes, scales = create_fp4_output_tensors(tokens, k, self.device, True)
        self.scales = scales.view(torch.float8_e4m3fn)
        self.global_scale = torch.zeros(2, dtype=torch.float32, device=self.device)   # (scale, 1 / scale)
        self._scratch = torch.zeros(2, dtype=torch.int32, device=self.device)
        self._args = (self.global_scale.data_ptr(), self._scratch.data_ptr(), self.codes.data_ptr(), scales.data_ptr(),
                      tokens, k, k, _mse.LOWER_BOUND, _mse.UPPER_BOUND, 1)
        self._scales_storage = scales
        self._result = (self.codes, self.scales, self.global_scale[0:1])
        self._chain = None
        if self.device.type == "cuda":
            self._chain = _lib.fast.make_chain(
                self._dtype_code, _lib.VARIANT_MSE, self.device.index, self.fp8_max, self.global_scale.data_ptr(),
                self._scratch.data_ptr(), self.codes.data_ptr(), scales.data_ptr(), tokens, k, _mse.LOWER_BOUND, _mse.UPPER_BOUND)

    def __call__(self, x: torch.Tensor):
        """Returns (codes, scales, global_scale[0:1]); the three tensors are this object's buffers."""
        if _lib.fast.chain_call(self._chain, x):
            return self._result
        if x.shape != (self.tokens, self.k) or x.dtype != self.dtype or x.device != self.device or not x.is_contiguous():
            raise ValueError(f"x must be a contiguous {self.dtype} [{self.tokens}, {self.k}] tensor on {self.device}")
        if x.data_ptr() & 15:
            raise ValueError("x must be 16-byte aligned")
        with _lib.device_guard(self.device):
            st = _lib.lib().nvfp4_quant_chain_launch(_lib.VARIANT_MSE, x.data_ptr(), self._dtype_code, None, self.fp8_max,
                                                     *self._args, _lib.current_stream_ptr(self.device))
        _lib.check(st, "nvfp4_quant_chain_launch")
        return self._result


class LinearGroup:
    """y_i = (alpha_a * weight_scale_i) * dq(a) @ dq(weight_i).T for prepared weights that read the same activation
    (q / k / v, gate / up), `tokens` rows at a time, into preallocated bf16 outputs: one nvfp4_gemm_launch_grouped call."""

    def __init__(self, weights: list[PreparedWeight], weight_scales: list[torch.Tensor], tokens: int):
        if not weights or len(weights) != len(weight_scales) or len(weights) > 64:
            raise ValueError("between 1 and 64 weights, one scale tensor per weight")
        self.weights, self.weight_scales, self.tokens = list(weights), list(weight_scales), tokens
        self.device, self.k = weights[0].device, weights[0].k
        for w, s in zip(weights, weight_scales):
            if w.device != self.device or w.k != self.k or not w._handle:
                raise ValueError("the weights of a group share the device and K, and must be open")
            if s.dtype != torch.float32 or s.device != self.device or s.numel() < 1:
                raise ValueError("weight scales must be float32 tensors on the weights' device")
        n = len(weights)
        self.outs = [torch.empty((tokens, w.n), dtype=torch.bfloat16, device=self.device) for w in weights]
        self._handles = (ctypes.c_void_p * n)(*[w._handle.value for w in weights])
        self._alphas = (ctypes.c_void_p * n)(*[s.data_ptr() for s in weight_scales])
        self._outs = (ctypes.c_void_p * n)(*[o.data_ptr() for o in self.outs])
        self._n = n
        self._min_scale_bytes = _scale_bytes(tokens, self.k)
        self._group = None
        if self.device.type == "cuda":
            self._group = _lib.fast.make_group(self.device.index, tokens, self.k, tuple(w._handle.value for w in weights),
                                               tuple(s.data_ptr() for s in weight_scales), tuple(o.data_ptr() for o in self.outs))

    def __call__(self, codes: torch.Tensor, scales: torch.Tensor, alpha_a: torch.Tensor | None):
        """codes / scales: the quantized activation [tokens, K/2] and its tiled scales; alpha_a: its global scale (one
        float32 on the device) or None.  Returns this object's output tensors."""
        if _lib.fast.group_call(self._group, codes, scales, alpha_a):
            return self.outs
        if (codes.shape != (self.tokens, self.k // 2) or codes.dtype != torch.uint8 or codes.device != self.device
                or not codes.is_contiguous()):
            raise ValueError(f"codes must be a contiguous uint8 [{self.tokens}, {self.k // 2}] tensor on {self.device}")
        if scales.numel() * scales.element_size() < self._min_scale_bytes or not scales.is_contiguous():
            raise ValueError("scales are smaller than the tiled layout of the activation needs")
        if scales.device != self.device:
            raise ValueError(f"scales must be on {self.device}")
        if alpha_a is not None and (alpha_a.dtype != torch.float32 or alpha_a.device != self.device or alpha_a.numel() < 1):
            raise ValueError(f"alpha_a must be a float32 tensor on {self.device}")
        with _lib.device_guard(self.device):
            st = _lib.lib().nvfp4_gemm_launch_grouped(self._handles, self._n, codes.data_ptr(), scales.data_ptr(),
                                                      None if alpha_a is None else alpha_a.data_ptr(), self._alphas,
                                                      self._outs, self.tokens, _lib.current_stream_ptr(self.device))
        _lib.check(st, "nvfp4_gemm_launch_grouped")
        return self.outs


class DecodeStep:
    """Everything a layer computes from activations that are all at hand, in one host call: the quantization of each
    activation (ActivationQuantizer) and the products that read it (LinearGroup).  One or two launches quantize the
    activations together, one multiplies (nvfp4_quant_chain_multi_launch, nvfp4_gemm_launch_multi).  Outputs are the
    groups' own; bits equal calling quantizers and groups one by one, up to the order of the fp32 sums."""

    def __init__(self, quantizers: list[ActivationQuantizer], groups: list[tuple[int, LinearGroup]]):
        """groups: (index of the quantizer whose output it reads, group)."""
        for i, group in groups:
            q = quantizers[i]
            if q.k != group.k or q.tokens != group.tokens or q.device != group.device:
                raise ValueError("a group and the quantizer it reads must agree on device, tokens and K")
        self.quantizers, self.groups = list(quantizers), list(groups)
        self._program = None
        if all(q._chain is not None for q in quantizers) and all(g._group is not None for _, g in groups):
            self._program = _lib.fast.make_program(tuple(q._chain for q in quantizers), tuple(i for i, _ in groups),
                                                   tuple(g._group for _, g in groups))

    def __call__(self, *acts: torch.Tensor) -> list[list[torch.Tensor]]:
        """One activation per quantizer; returns each group's outputs."""
        if not _lib.fast.program_call(self._program, *acts):
            if len(acts) != len(self.quantizers):
                raise ValueError(f"{len(self.quantizers)} activations are needed, got {len(acts)}")
            quantized = [q(x) for q, x in zip(self.quantizers, acts)]
            for i, group in self.groups:
                group(*quantized[i])
        return [group.outs for _, group in self.groups]


def nvfp4_linear_multi(acts: list[torch.Tensor], index: list[int], weights: list[PreparedWeight], scale_vecs: list[torch.Tensor],
                       slots: list[int], fp8_max: float = _helper.FP8_E4M3_MAX_4OVER6) -> list[torch.Tensor]:
    """[acts[index[i]] @ weights[i].T for i], in bf16: every activation [M, K] is quantized with its own global scale
    (ScaleSweep_MSE), the weights' global scales are scale_vecs[i][slots[i]].  One host call and three to four launches for
    a layer's matrices; the quantized activations are not returned.  Bits as scalesweep_nvfp4_quant_with_global_scale and
    nvfp4_scaled_mm_multi."""
    got = _lib.fast.linear_multi(_lib.VARIANT_MSE, acts, fp8_max, _mse.LOWER_BOUND, _mse.UPPER_BOUND, index,
                                 [w._fast for w in weights], scale_vecs, slots)
    if got is not None:
        return got
    quantized = scalesweep_nvfp4_quant_with_global_scales(acts, fp8_max)
    return nvfp4_scaled_mm_multi([quantized[i][0] for i in index], [quantized[i][1] for i in index],
                                 [quantized[i][2] for i in index], weights,
                                 [vec[s:s + 1] for vec, s in zip(scale_vecs, slots)])
