"""Global scale + ScaleSweep quantization as one call.

The reference computes the tensor-wide scale first (`get_nvfp4_global_scale`, helper.py:96-100 of
efsotr/nvfp4quant_test) and hands its reciprocal to the quantizer (bench.py:57-67): two passes over the tensor
and two launches from two host calls.  Here it is one host call: two dependent launches, or one for a tensor of up to 128 KiB,
whose CTAs each take the scale themselves.  (One cooperative launch that keeps the tensor in registers across a grid-wide wait
is in the C ABI, nvfp4_quant_fused_launch, for tensors that fit the resident grid; it takes longer than two launches, 1 x
4096: 5.6 against 5.1 us, 16 x 8192: 7.3 against 6.3.)
"""
from __future__ import annotations

import torch

from .. import _lib
from .. import helper as _helper
from ._launch import BLOCK_SIZE, check_importance, quant_out
from .kernel_vllm import create_fp4_output_tensors
from . import kernel_ScaleSweep as _weighted
from . import kernel_ScaleSweep_MSE as _mse


def scalesweep_nvfp4_quant_with_global_scale(
    input: torch.Tensor,
    fp8_max: float = _helper.FP8_E4M3_MAX_4OVER6,
    importance: torch.Tensor | None = None,
    is_sf_swizzled_layout: bool = True,
    padded_n: int | None = None,
    *,
    lower_bound: int | None = None,
    upper_bound: int | None = None,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """(codes, scales, global_scale, global_scale_inv).  Without `importance` this is ScaleSweep_MSE (window
    -3..+7), with it the importance-weighted ScaleSweep (window -8..+7 unless given); the two scale tensors are
    0-dim float32 views, as `get_nvfp4_global_scale` returns them."""
    if importance is None:
        got = _lib.fast.quant_dynamic(_lib.VARIANT_MSE, input, None, fp8_max, is_sf_swizzled_layout, padded_n,
                                      _mse.LOWER_BOUND if lower_bound is None else lower_bound,
                                      _mse.UPPER_BOUND if upper_bound is None else upper_bound)
    else:
        got = _lib.fast.quant_dynamic(_lib.VARIANT_WEIGHTED, input, importance, fp8_max, is_sf_swizzled_layout, padded_n,
                                      _weighted.LOWER_BOUND if lower_bound is None else lower_bound,
                                      _weighted.UPPER_BOUND if upper_bound is None else upper_bound)
    if got is not None:
        return got
    if input.ndim != 2:
        raise ValueError(f"input must be 2D [num_row, dim], got {tuple(input.shape)}")
    if importance is None:
        variant, mod = _lib.VARIANT_MSE, _mse
    else:
        check_importance(input, importance)
        variant, mod = _lib.VARIANT_WEIGHTED, _weighted
    lower = mod.LOWER_BOUND if lower_bound is None else lower_bound
    upper = mod.UPPER_BOUND if upper_bound is None else upper_bound
    m, n = input.shape
    if n % BLOCK_SIZE != 0:
        raise ValueError(f"input.shape[-1] must be divisible by {BLOCK_SIZE}")
    if not input.is_cuda:
        raise ValueError("input must be a CUDA tensor: these kernels have no CPU path")
    if m == 0 or n == 0:
        raise ValueError("the global scale of an empty tensor is undefined")
    if not float(fp8_max) > 0.0:
        raise ValueError(f"fp8_max must be positive, got {fp8_max}")
    output, output_scale = create_fp4_output_tensors(m, n, input.device, is_sf_swizzled_layout, padded_n=padded_n)
    g, g_inv = _helper.get_nvfp4_global_scale(input, fp8_max)
    quant_out(variant, input, importance, g_inv, is_sf_swizzled_layout, output, output_scale, lower, upper)
    return output, output_scale.view(torch.float8_e4m3fn), g, g_inv


def scalesweep_nvfp4_quant_with_global_scales(inputs: list[torch.Tensor], fp8_max: float = _helper.FP8_E4M3_MAX_4OVER6):
    """[scalesweep_nvfp4_quant_with_global_scale(x, fp8_max) for x in inputs], sharing launches: a layer's activations."""
    got = _lib.fast.quant_dynamic_multi(_lib.VARIANT_MSE, inputs, fp8_max, _mse.LOWER_BOUND, _mse.UPPER_BOUND)
    if got is not None:
        return got
    return [scalesweep_nvfp4_quant_with_global_scale(x, fp8_max) for x in inputs]
