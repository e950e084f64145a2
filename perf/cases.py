"""The work a user of this package has it do, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what a program holds before the call, `run` is one pass through the
public entry points, `work` is what one pass cannot do without, `tolerance` how far another correct implementation at the
same precision may be off.  `listed` names one case of each kind of work, `draw` gives more of the same ranges.
"""
from __future__ import annotations

import torch

from nvfp4quant_test_b200 import _lib, host_pipeline, llama_stack
from nvfp4quant_test_b200 import helper as H
from nvfp4quant_test_b200 import kernels as K

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
DEVICE = "cuda"
DECODE_TOKENS = 64   # layers of up to this many tokens go through the preallocated decode blocks


def listed():
    return [
        # One decoded token whose activation scale was calibrated before: the smallest call there is, all launch latency
        # and host time (bsz 1 of the reference's latency table).
        {"name": "act_1x8192", "kind": "act", "variant": "mse", "m": 1, "n": 8192, "dtype": "bf16", "padded_n": 0, "tiled": True},
        # The headline workload: 8192 prefill tokens of width 8192, unweighted sweep, scale given.
        {"name": "act_8192x8192", "kind": "act", "variant": "mse", "m": 8192, "n": 8192, "dtype": "bf16", "padded_n": 0, "tiled": True},
        # The amax baseline (drop-in for vllm's scaled_fp4_quant) on a prefill chunk: a pass over memory, no sweep.
        {"name": "amax_2048x8192", "kind": "act", "variant": "amax", "m": 2048, "n": 8192, "dtype": "bf16", "padded_n": 0, "tiled": True},
        # A few dozen tokens with the scale taken from the tensor itself (dynamic activation quantization), fp16, a width
        # that is no multiple of 64 and is padded for the GEMM.
        {"name": "dynamic_77x5104_f16", "kind": "dynamic", "m": 77, "n": 5104, "dtype": "f16", "padded_n": 5120},
        # Offline weight quantization: importance from a calibration batch, global scale, weighted sweep (Laplace data,
        # the shapes of the importance-weighted configuration).
        {"name": "weight_8192x8192", "kind": "weight", "m": 8192, "n": 8192, "calib": 4096, "dtype": "bf16"},
        # A checkpoint's fp32 matrix in pinned host memory, quantized chunk by chunk on its way through the GPU.
        {"name": "host_4096x4096_f32", "kind": "host", "m": 4096, "n": 4096, "dtype": "f32"},
        # The bare GEMM as a drop-in for cutlass_scaled_fp4_mm (raw operands): a decode batch against a large weight ...
        {"name": "gemm_16x14336x8192", "kind": "gemm", "m": 16, "n": 14336, "k": 8192},
        # ... and a ragged one: neither tokens, outputs nor K fill a tile.
        {"name": "gemm_333x5000x2880", "kind": "gemm", "m": 333, "n": 5000, "k": 2880},
        # One linear layer at prefill, from bf16 activations to bf16 outputs: scale, sweep, GEMM on a prepared weight.
        # The largest case.
        {"name": "linear_2048x28672x8192", "kind": "linear", "m": 2048, "n": 28672, "k": 8192, "dtype": "bf16"},
        # The seven matrices of a decoder layer (Llama-3-8B shapes) for one decoded token, preallocated, launched eagerly.
        {"name": "decode_layer_1", "kind": "layer", "m": 1, "hidden": 4096, "kv": 1024, "ffn": 14336},
        # The same layer for a short prompt, through the allocating entry points on side streams.
        {"name": "prefill_layer_256", "kind": "layer", "m": 256, "hidden": 4096, "kv": 1024, "ffn": 14336},
        # The way back: tiled scales to row-major and codes to fp32, what every error measurement of a quantizer does.
        {"name": "dequant_4096x14336", "kind": "dequant", "m": 4096, "n": 14336},
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], even over the logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def _mult(rng, lo, hi, step):
    return max(lo, _log(rng, lo, hi) // step * step)


def draw(rng):
    kind = rng.choice(["act", "act", "act", "dynamic", "weight", "host", "gemm", "gemm", "linear", "layer", "layer", "dequant"])
    if kind == "act":
        n = _mult(rng, 1024, 14336, 16)
        m = _log(rng, 1, min(8192, 8192 * 8192 // n))
        pad = (n + 63) // 64 * 64 if rng.random() < 0.3 else 0
        return {"kind": kind, "variant": rng.choice(["mse", "mse", "amax"]), "m": m, "n": n,
                "dtype": rng.choice(["bf16", "bf16", "f16", "f32"]), "padded_n": pad if pad != n else 0, "tiled": rng.random() < 0.85}
    if kind == "dynamic":
        n = _mult(rng, 1024, 14336, 16)
        pad = (n + 63) // 64 * 64
        return {"kind": kind, "m": _log(rng, 1, 4096 * 4096 // n), "n": n,
                "dtype": rng.choice(["bf16", "bf16", "f16", "f32"]), "padded_n": pad if pad != n else 0}
    if kind == "weight":
        n = _mult(rng, 1024, 14336, 16)
        return {"kind": kind, "m": _log(rng, 256, min(28672, 8192 * 8192 // n)), "n": n, "calib": _log(rng, 256, 4096),
                "dtype": rng.choice(["bf16", "bf16", "f16", "f32"])}
    if kind == "host":
        n = _mult(rng, 1024, 8192, 16)
        return {"kind": kind, "m": _log(rng, 256, 4096 * 4096 // n), "n": n, "dtype": rng.choice(["bf16", "f16", "f32"])}
    if kind == "gemm":
        k = _mult(rng, 1024, 14336, 64)
        n = _log(rng, 512, 28672)
        n = n // 64 * 64 if rng.random() < 0.7 else n
        m = _log(rng, 1, min(8192, 2048 * 28672 * 8192 // (n * k)))
        return {"kind": kind, "m": m, "n": n, "k": k}
    if kind == "linear":
        k = _mult(rng, 1024, 14336, 64)
        n = _mult(rng, 512, 28672, 64)
        m = _log(rng, 1, min(8192, 2048 * 28672 * 8192 // (n * k)))
        return {"kind": kind, "m": m, "n": n, "k": k, "dtype": rng.choice(["bf16", "bf16", "f16"])}
    if kind == "layer":
        hidden = _mult(rng, 1024, 5120, 256)
        ffn = _mult(rng, 2 * hidden, 14336, 256)
        return {"kind": kind, "m": rng.choice([_log(rng, 1, 64), _log(rng, 65, 1024)]), "hidden": hidden,
                "kv": max(256, hidden // rng.choice([1, 4, 8]) // 64 * 64), "ffn": ffn}
    n = _mult(rng, 1024, 14336, 16)
    return {"kind": kind, "m": _log(rng, 16, min(8192, 4096 * 14336 // n)), "n": n}


# ---- inputs ---------------------------------------------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _normal(g, shape, dtype=torch.bfloat16, std=1.0):
    return torch.empty(shape, dtype=torch.float32, device=DEVICE).normal_(0.0, std, generator=g).to(dtype)


def _laplace(g, shape, dtype=torch.bfloat16):
    """Laplace(0, 1): an exponential magnitude with a random sign."""
    mag = torch.empty(shape, dtype=torch.float32, device=DEVICE).exponential_(1.0, generator=g)
    sign = torch.empty(shape, dtype=torch.float32, device=DEVICE).random_(0, 2, generator=g).mul_(2.0).sub_(1.0)
    return mag.mul_(sign).to(dtype)


def _quantized(x):
    """(codes, tiled scales, global scale) of a matrix, by the unweighted sweep."""
    gs, gs_inv = H.get_nvfp4_global_scale(x, H.FP8_E4M3_MAX_4OVER6)
    codes, scales = K.scalesweep_mse_nvfp4_quant_impl(x, gs_inv)
    return codes, scales, gs


def _layer_state(case, g):
    shapes = {"q": (case["hidden"], case["hidden"]), "k": (case["kv"], case["hidden"]), "v": (case["kv"], case["hidden"]),
              "o": (case["hidden"], case["hidden"]), "gate": (case["ffn"], case["hidden"]), "up": (case["ffn"], case["hidden"]),
              "down": (case["hidden"], case["ffn"])}
    weights = {name: _normal(g, shape, std=0.02) for name, shape in shapes.items()}
    importance = {k: H.channel_square_norm(_normal(g, (256, k))) for k in (case["hidden"], case["ffn"])}
    qlayer = llama_stack.quantize_layer(weights, importance)
    scales = llama_stack.stack_weight_scales(qlayer)
    prepared = llama_stack.prepare_layer(qlayer)
    acts = {k: _normal(g, (case["m"], k)) for k in (case["hidden"], case["ffn"])}
    state = {"acts": acts, "qlayer": qlayer, "scales": scales, "prepared": prepared}
    if case["m"] <= DECODE_TOKENS:
        state["decode"] = llama_stack.DecodeLayer(qlayer, scales, prepared, case["m"], torch.device(DEVICE, torch.cuda.current_device()))
    else:
        state["side"] = [torch.cuda.Stream() for _ in range(4)]
    return state


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    state = {"case": case}
    if kind == "act":
        x = _normal(g, (case["m"], case["n"]), DTYPES[case["dtype"]])
        fp8_max = H.FP8_E4M3_MAX_NVFP4 if case["variant"] == "amax" else H.FP8_E4M3_MAX_4OVER6
        state.update(x=x, gs_inv=H.get_nvfp4_global_scale(x, fp8_max)[1], padded_n=case["padded_n"] or None)
    elif kind == "dynamic":
        state.update(x=_normal(g, (case["m"], case["n"]), DTYPES[case["dtype"]]), padded_n=case["padded_n"] or None)
    elif kind == "weight":
        state.update(w=_laplace(g, (case["m"], case["n"]), DTYPES[case["dtype"]]), calib=_laplace(g, (case["calib"], case["n"])))
    elif kind == "host":
        dtype = DTYPES[case["dtype"]]
        w = _normal(g, (case["m"], case["n"]), dtype, std=0.02)
        importance = H.channel_square_norm(_normal(g, (256, case["n"])))
        gs_inv = H.get_nvfp4_global_scale(w, H.FP8_E4M3_MAX_4OVER6)[1]
        x = torch.empty((case["m"], case["n"]), dtype=dtype, pin_memory=True)
        x.copy_(w)
        codes = torch.empty((case["m"], case["n"] // 2), dtype=torch.uint8, pin_memory=True)
        scales = torch.zeros((case["m"] + 127) // 128 * 128 * ((case["n"] // 16 + 3) // 4 * 4), dtype=torch.uint8, pin_memory=True)
        hq = host_pipeline.HostQuantizer(case["m"], case["n"], dtype, variant=_lib.VARIANT_WEIGHTED, lower=-8, upper=7)
        state.update(x=x, importance=importance, gs_inv=gs_inv, codes=codes, scales=scales, quantizer=hq)
    elif kind == "gemm":
        qa, sa, ga = _quantized(_laplace(g, (case["m"], case["k"])))
        qb, sb, gb = _quantized(_laplace(g, (case["n"], case["k"])))
        state.update(qa=qa, sa=sa, qb=qb, sb=sb, alpha=(ga * gb).reshape(1))
    elif kind == "linear":
        x = _laplace(g, (case["m"], case["k"]), DTYPES[case["dtype"]])
        qb, sb, gb = _quantized(_laplace(g, (case["n"], case["k"])))
        state.update(x=x, weight=K.PreparedWeight(qb, sb), gs_w=gb.reshape(1).clone())
    elif kind == "layer":
        state.update(_layer_state(case, g))
    elif kind == "dequant":
        codes, scales, gs = _quantized(_normal(g, (case["m"], case["n"])))
        state.update(codes=codes, scales=scales, gs=gs)
    else:
        raise ValueError(f"unknown kind: {kind}")
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "act":
        quant = K.amax_nvfp4_quant_impl if case["variant"] == "amax" else K.scalesweep_mse_nvfp4_quant_impl
        return quant(s["x"], s["gs_inv"], case["tiled"], s["padded_n"])
    if kind == "dynamic":
        return K.scalesweep_nvfp4_quant_with_global_scale(s["x"], H.FP8_E4M3_MAX_4OVER6, padded_n=s["padded_n"])
    if kind == "weight":
        importance = H.channel_square_norm(s["calib"])
        gs, gs_inv = H.get_nvfp4_global_scale(s["w"], H.FP8_E4M3_MAX_4OVER6)
        codes, scales = K.scalesweep_weighted_mse_nvfp4_quant_impl(s["w"], importance, gs_inv)
        return codes, scales, gs, importance
    if kind == "host":
        s["quantizer"](s["x"], s["gs_inv"], s["codes"], s["scales"], s["importance"])
        return s["codes"], s["scales"]
    if kind == "gemm":
        return K.nvfp4_scaled_mm(s["qa"], s["qb"], s["sa"], s["sb"], s["alpha"], torch.bfloat16)
    if kind == "linear":
        gs, gs_inv = H.get_nvfp4_global_scale(s["x"], H.FP8_E4M3_MAX_4OVER6)
        codes, scales = K.scalesweep_mse_nvfp4_quant_impl(s["x"], gs_inv)
        return K.nvfp4_scaled_mm_prepared(codes, scales, gs * s["gs_w"], s["weight"])
    if kind == "layer":
        if "decode" in s:
            return s["decode"](s["acts"])
        return llama_stack.layer_gemms(s["qlayer"], s["acts"], {}, s["scales"], s["side"], s["prepared"])
    linear = K.unswizzle_vllm_fp4_scale(s["scales"], case["m"], case["n"])
    return H.dequantize("base", s["codes"], linear, s["gs"])


# ---- what a pass cannot do without ----------------------------------------------------------------------------------


def _size(case):
    return DTYPES[case["dtype"]].itemsize


def _packed(m, k):
    """Bytes of a quantized [m, k] matrix: half a byte per element and one scale byte per block of 16."""
    return m * k // 2 + m * k // 16


def _gemm_work(m, n, k):
    return {"bytes": _packed(m, k) + _packed(n, k) + 2 * m * n, "flops": 2 * m * n * k}


def work(case):
    kind, m = case["kind"], case["m"]
    if kind in ("act", "dynamic"):
        return {"bytes": m * case["n"] * _size(case) + _packed(m, case["padded_n"] or case["n"]), "flops": 0}
    if kind == "weight":
        n = case["n"]
        return {"bytes": case["calib"] * n * 2 + m * n * _size(case) + _packed(m, n) + 4 * n, "flops": 2 * case["calib"] * n}
    if kind == "host":
        n = case["n"]
        return {"bytes": m * n * _size(case) + _packed(m, n) + 4 * n, "flops": 0}
    if kind == "gemm":
        return _gemm_work(m, case["n"], case["k"])
    if kind == "linear":
        w = _gemm_work(m, case["n"], case["k"])
        return {"bytes": w["bytes"] + m * case["k"] * _size(case) - _packed(m, case["k"]), "flops": w["flops"]}
    if kind == "layer":
        h, kv, ffn = case["hidden"], case["kv"], case["ffn"]
        weights = h * (2 * h + 2 * kv + 3 * ffn)
        outputs = m * (3 * h + 2 * kv + 2 * ffn)
        return {"bytes": _packed(1, weights) + 2 * outputs + 2 * m * (h + ffn), "flops": 2 * m * weights}
    n = case["n"]
    return {"bytes": _packed(m, n) + 4 * m * n, "flops": 0}


def tolerance(case):
    if case["kind"] in ("gemm", "linear", "layer"):
        # fp32 accumulation in any order, one rounding to bf16: two correct results differ by a bf16 ulp here and there
        return {"rel": 4e-3, "max": 1.6e-2}
    if case["kind"] == "weight":
        # the importance is a fp32 sum over the calibration rows; its last bits decide a tie between two scales now and then
        return {"rel": 1e-5, "differ": 1e-4}
    # codes, scale bytes, global scales and dequantized values are fixed bit for bit
    return "exact"
