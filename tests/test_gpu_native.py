"""GPU: the compiled half of the entry points gives what the Python path gives, and hands over what it does not cover."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def python_path(cuda_lib, monkeypatch):
    """Switches the compiled functions off for the calls made inside `with`."""
    import contextlib

    from nvfp4quant_test_b200 import _lib

    @contextlib.contextmanager
    def off():
        with monkeypatch.context() as mp:
            mp.setattr(_lib, "fast", types.SimpleNamespace(**{k: _lib._not_common for k in vars(_lib.fast)}))
            yield

    return off


def _flat(v):
    return [t for x in v for t in _flat(x)] if isinstance(v, (tuple, list)) else [v]


def _same(got, want):
    got, want = _flat(got), _flat(want)
    assert len(got) == len(want)
    for g, w in zip(got, want):
        assert g.shape == w.shape and g.dtype == w.dtype and g.device == w.device and g.is_contiguous() == w.is_contiguous()
        assert torch.equal(g.contiguous().reshape(-1).view(torch.uint8), w.contiguous().reshape(-1).view(torch.uint8))


def _calls(m, n, dtype, tiled, padded_n):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H

    g = torch.Generator(device="cuda").manual_seed(m * 31 + n)
    x = torch.randn((m, n), generator=g, device="cuda").to(dtype)
    imp = torch.rand((1, n), generator=g, device="cuda")
    gs_inv = H.get_nvfp4_global_scale(x, 256.0)[1]
    wide = torch.randn((m, n + 16), generator=g, device="cuda").to(dtype)
    yield lambda: H.get_nvfp4_global_scale(x, 448.0)
    yield lambda: H.channel_square_norm(x)
    yield lambda: H.channel_square_norm(wide[:, 16:])
    yield lambda: K.scalesweep_mse_nvfp4_quant_impl(x, gs_inv, tiled, padded_n)
    yield lambda: K.scalesweep_weighted_mse_nvfp4_quant_impl(x, imp, gs_inv, tiled, padded_n)
    yield lambda: K.scalesweep_weighted_mse_nvfp4_quant_impl(x, imp.half(), gs_inv, tiled, padded_n)      # converted in Python
    yield lambda: K.amax_nvfp4_quant_impl(x, gs_inv, tiled, padded_n)
    yield lambda: K.scalesweep_nvfp4_quant_with_global_scale(x, 256.0, None, tiled, padded_n)
    yield lambda: K.scalesweep_nvfp4_quant_with_global_scale(x, 256.0, imp, tiled, padded_n, lower_bound=-2, upper_bound=3)
    yield lambda: K.scalesweep_mse_nvfp4_quant_impl(wide[:, :n], gs_inv, tiled, padded_n)                 # strided
    yield lambda: K.scalesweep_mse_nvfp4_quant_impl(torch.nn.Parameter(x), gs_inv, tiled, padded_n)


@pytest.mark.parametrize("m,n,dtype,tiled,padded_n", [
    (1, 16, torch.bfloat16, True, None), (3, 8192, torch.bfloat16, True, None), (129, 208, torch.float16, True, 256),
    (5, 48, torch.float32, False, None), (77, 4096, torch.bfloat16, False, 4160)])
def test_compiled_calls_equal_the_python_path(python_path, m, n, dtype, tiled, padded_n):
    for call in _calls(m, n, dtype, tiled, padded_n):
        got = call()
        with python_path():
            want = call()
        _same(got, want)


@pytest.mark.parametrize("m,n,k", [(1, 128, 64), (16, 72, 320), (130, 257, 512)])
def test_compiled_gemm_calls_equal_the_python_path(python_path, m, n, k):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn((m, k), generator=g, device="cuda").bfloat16()
    w = torch.randn((n, k), generator=g, device="cuda").bfloat16()
    (gx, ix), (gw, iw) = H.get_nvfp4_global_scale(x), H.get_nvfp4_global_scale(w)
    qx, sx = K.scalesweep_mse_nvfp4_quant_impl(x, ix)
    qw, sw = K.scalesweep_mse_nvfp4_quant_impl(w, iw)
    pw, alpha = K.PreparedWeight(qw, sw), (gx * gw).reshape(1)
    out = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    calls = [lambda: K.nvfp4_scaled_mm(qx, qw, sx, sw, alpha, torch.bfloat16),
             lambda: K.nvfp4_scaled_mm(qx, qw, sx, sw, alpha, torch.bfloat16, out),
             lambda: K.nvfp4_scaled_mm_prepared(qx, sx, alpha, pw),
             lambda: K.nvfp4_scaled_mm_grouped(qx, sx, gx.reshape(1), [pw, pw], [gw.reshape(1), gw.reshape(1)]),
             lambda: K.LinearGroup([pw], [gw.reshape(1)], m)(qx, sx, gx.reshape(1)),
             lambda: K.ActivationQuantizer(m, k, "cuda")(x)]
    for call in calls:
        got = [t.clone() for t in _flat(call())]
        with python_path():
            want = call()
        _same(got, want)
    assert K.nvfp4_scaled_mm(qx, qw, sx, sw, alpha, torch.bfloat16, out) is out
    pw.close()
    with pytest.raises(ValueError, match="closed"):
        K.nvfp4_scaled_mm_prepared(qx, sx, alpha, pw)
    with pytest.raises(ValueError, match="disagree on K"):
        K.nvfp4_scaled_mm(qx[:, : k // 2 - 32].contiguous(), qw, sx, sw, alpha, torch.bfloat16)


def test_compiled_calls_use_the_current_stream_and_record_into_a_graph(cuda_lib):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H

    x = torch.randn((64, 4096), device="cuda").bfloat16()
    want = K.scalesweep_nvfp4_quant_with_global_scale(x, 256.0)
    streams = [torch.cuda.Stream() for _ in range(40)]      # more than scratch words are kept for
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            got = K.scalesweep_nvfp4_quant_with_global_scale(x, 256.0)
        s.synchronize()
        _same(got, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        gs, gs_inv = H.get_nvfp4_global_scale(x, 256.0)
        q = K.scalesweep_mse_nvfp4_quant_impl(x, gs_inv)
    graph.replay()
    torch.cuda.synchronize()
    _same(q, want[:2])


@pytest.mark.parametrize("m,n", [(1, 16), (31, 208), (128, 64), (129, 4096), (300, 80)])
@pytest.mark.parametrize("dtype", [torch.uint8, torch.float8_e4m3fn])
def test_scale_layouts_and_dequantization_equal_torch(cuda_lib, m, n, dtype):
    """Every code, scale byte (NaN included) and edge of a tile, against the same functions on CPU tensors (plain torch)."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import _lib
    from nvfp4quant_test_b200 import helper as H

    g = torch.Generator().manual_seed(m * 7 + n)
    codes = torch.randint(0, 256, (m, n // 2), dtype=torch.uint8, generator=g)
    linear = torch.randint(0, 256, (m, n // 16), dtype=torch.uint8, generator=g)
    gs = torch.tensor(0.0123)
    tiled = K.swizzle_vllm_fp4_scale(linear.view(dtype), m, n)
    got = K.swizzle_vllm_fp4_scale(linear.view(dtype).cuda(), m, n)
    assert got.dtype == tiled.dtype and torch.equal(got.view(torch.uint8).cpu(), tiled.view(torch.uint8))
    back = K.unswizzle_vllm_fp4_scale(got, m, n)
    assert back.shape == (m, n // 16) and torch.equal(back.view(torch.uint8).cpu(), linear)
    assert torch.equal(H.unpack_fp4_e2m1(codes.cuda()).cpu().view(torch.int32), H.unpack_fp4_e2m1(codes).view(torch.int32))
    fp8 = linear.view(torch.float8_e4m3fn)
    want = H.dequantize("base", codes, fp8, gs)
    for g1 in (gs.cuda(), gs.reshape(1).cuda()):
        have = H.dequantize("base", codes.cuda(), fp8.cuda(), g1).cpu()
        assert have.shape == want.shape and torch.equal(have.isnan(), want.isnan())
        assert torch.equal(have[~want.isnan()].view(torch.int32), want[~want.isnan()].view(torch.int32))
    assert _lib.fast.dequant(codes.cuda(), fp8.cuda(), gs.cuda()) is not None and _lib.fast.scale_layout(got, m, n // 16, False) is not None


@pytest.mark.parametrize("m,n,padded_n,tiled", [(129, 16, None, False), (300, 32, None, True), (77, 48, None, False), (3, 112, 176, True),
                                                (127, 2048, None, True), (129, 2048, 4096, True), (1, 6144, None, True),
                                                (200, 2064, None, True), (45, 6128, 6144, False), (900, 1968, None, True), (900, 1952, 1968, False),
                                                (401, 9200, None, False)])
def test_quantizer_grids_equal_the_scalar_body(cuda_lib, m, n, padded_n, tiled):
    """Every grid (slots numbered through in two CTA sizes, rows of CTAs with and without idle threads and padding) against the scalar
    transcription, at widths where the division by the row length and the padding can go wrong."""
    from nvfp4quant_test_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn((m, n), generator=g, device="cuda").bfloat16()
    imp = torch.rand((1, n), generator=g, device="cuda")
    gs_inv = torch.tensor([37.5], device="cuda")
    p = padded_n or n
    size = (m + 127) // 128 * 128 * ((p // 16 + 3) // 4 * 4) if tiled else m * p // 16
    for variant, lower, upper in ((0, -3, 7), (0, -2, 5), (1, -8, 7), (1, -1, 1), (2, 0, 0)):
        want = None
        for impl in (3, 0, 7, 8, 9) if variant == 2 else (1, 0, 3, 7, 8, 9):
            codes = torch.full((m, p // 2), 0xA5, dtype=torch.uint8, device="cuda")
            scales = torch.full((size,), 0xA5, dtype=torch.uint8, device="cuda")
            _lib.check(cuda_lib.nvfp4_quant_launch_impl(impl, variant, x.data_ptr(), 0, imp.data_ptr(), gs_inv.data_ptr(), codes.data_ptr(),
                                                        scales.data_ptr(), m, n, p, lower, upper, int(tiled), None), "launch")
            torch.cuda.synchronize()
            want = want or (codes, scales)
            assert torch.equal(codes, want[0]) and torch.equal(scales, want[1]), (impl, variant, lower)


@pytest.mark.parametrize("shapes", [[(1, 64)], [(1, 4096), (1, 14336)], [(3, 4096), (3, 16384), (200, 320)],
                                    [(64, 4096), (64, 14336)], [(256, 4096), (256, 14336)], [(1100, 8192), (9, 48)],
                                    [(2, 128)] * 6])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_chains_over_several_tensors_equal_single_calls(cuda_lib, shapes, dtype):
    """Global scale inside the quantizer, two launches shared by the tensors, or launches of their own: same bytes."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H

    xs = [torch.randn(s, device="cuda").to(dtype) * (i + 1) for i, s in enumerate(shapes)]
    for _ in range(2):      # scratch words come back zeroed
        got = K.scalesweep_nvfp4_quant_with_global_scales(xs, 256.0)
        for x, g in zip(xs, got):
            gs, gs_inv = H.get_nvfp4_global_scale(x, 256.0)
            _same(g, [*K.scalesweep_mse_nvfp4_quant_impl(x, gs_inv), gs, gs_inv])
            imp = torch.rand((1, x.shape[1]), device="cuda")
            _same(K.scalesweep_nvfp4_quant_with_global_scale(x, 256.0, imp),
                  [*K.scalesweep_weighted_mse_nvfp4_quant_impl(x, imp, gs_inv), gs, gs_inv])


@pytest.mark.parametrize("tokens", [1, 16, 33, 64])
def test_decode_step_equals_quantizers_and_groups_one_by_one(python_path, tokens):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    def weight(n, k):
        c, s, gs, _ = K.scalesweep_nvfp4_quant_with_global_scale(torch.randn((n, k), device="cuda").bfloat16(), 256.0)
        return K.PreparedWeight(c, s), gs.reshape(1)

    sets = [[weight(512, 1024), weight(200, 1024)], [weight(512, 1024)], [weight(1024, 2752)]]
    quantizers = [K.ActivationQuantizer(tokens, 1024, "cuda"), K.ActivationQuantizer(tokens, 2752, "cuda")]
    groups = [(i, K.LinearGroup([w for w, _ in ws], [s for _, s in ws], tokens)) for i, ws in zip((0, 0, 1), sets)]
    step = K.DecodeStep(quantizers, groups)
    acts = [torch.randn((tokens, k), device="cuda").bfloat16() for k in (1024, 2752)]
    got = [o.clone() for o in _flat(step(*acts))]
    assert gemm_last_status() == 0
    with python_path():
        want = _flat(step(*acts))
    for g, w in zip(got, want):
        assert torch.allclose(g.float(), w.float(), rtol=2.0 ** -7, atol=float(w.abs().max()) * 2.0 ** -12)
    with pytest.raises(ValueError, match="activations are needed"):
        step(acts[0])
    with pytest.raises(ValueError, match="agree"):
        K.DecodeStep(quantizers, [(1, groups[0][1])])


@pytest.mark.parametrize("rows,dim,dtype,chunk", [(1, 16, torch.bfloat16, 128), (300, 48, torch.float16, 128), (1000, 4096, torch.float32, 256),
                                                  (700, 8192, torch.bfloat16, 1024)])
def test_host_pipeline_forms(cuda_lib, rows, dim, dtype, chunk):
    """One chunk and many, weighted, pageable and strided operands, calls back to back from two streams."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import _lib
    from nvfp4quant_test_b200.host_pipeline import HostQuantizer

    g = torch.Generator().manual_seed(rows)
    x = torch.randn((rows, dim), generator=g).to(dtype)
    imp = torch.rand((1, dim), generator=g).cuda()
    gs_inv = torch.tensor([41.0], device="cuda")
    codes, scales = (t.cpu() for t in K.scalesweep_weighted_mse_nvfp4_quant_impl(x.cuda(), imp, gs_inv))
    scales = scales.view(torch.uint8).reshape(-1)
    hq = HostQuantizer(rows, dim, dtype, "cuda", chunk_rows=chunk, variant=_lib.VARIANT_WEIGHTED, lower=-8, upper=7)
    wide = torch.zeros((rows, dim), dtype=torch.uint8)
    for xs, out in ((x.pin_memory(), torch.zeros_like(codes).pin_memory()), (x, torch.zeros_like(codes)),
                    (x.t().contiguous().t(), wide[:, : dim // 2])):
        sc = torch.zeros_like(scales).pin_memory()
        for s in (torch.cuda.current_stream(), torch.cuda.Stream()):
            out.zero_()
            with torch.cuda.stream(s):
                hq(xs, gs_inv, out, sc, imp)
                hq(xs, gs_inv, out, sc, imp)
            torch.cuda.synchronize()
            assert torch.equal(out, codes) and torch.equal(sc, scales)
    with pytest.raises(ValueError, match="importance"):
        hq(x, gs_inv, torch.zeros_like(codes), scales)
    with pytest.raises(ValueError, match="scales_host"):
        hq(x, gs_inv, torch.zeros_like(codes), scales[:-1], imp)
    with pytest.raises(ValueError, match="does not match"):
        hq(x[:, :0], gs_inv, codes, scales, imp)


@pytest.mark.parametrize("m", [3, 65, 300])
def test_linear_multi_equals_its_steps(python_path, m):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    def weight(n, k):
        c, s, gs, _ = K.scalesweep_nvfp4_quant_with_global_scale(torch.randn((n, k), device="cuda").bfloat16(), 256.0)
        return K.PreparedWeight(c, s), gs

    ks = (512, 1024, 512, 512)
    made = [weight(n, k) for n, k in zip((256, 1000, 72, 512), ks)]
    acts = [torch.randn((m, k), device="cuda").bfloat16() * (k / 100) for k in (512, 1024)]
    vecs = {512: torch.stack([made[i][1] for i in (0, 2, 3)]), 1024: made[1][1].reshape(1)}
    args = (acts, [0, 1, 0, 0], [w for w, _ in made], [vecs[k] for k in ks], [0, 0, 1, 2])
    got = K.nvfp4_linear_multi(*args)
    assert gemm_last_status() == 0
    with python_path():
        want = K.nvfp4_linear_multi(*args)
    if m > 64:
        _same(got, want)
    for g, w in zip(got, want):
        assert torch.allclose(g.float(), w.float(), rtol=2.0 ** -7, atol=float(w.abs().max()) * 2.0 ** -12)
    with pytest.raises(ValueError, match="disagree on K"):
        K.nvfp4_linear_multi(acts, [1, 1, 0, 0], *args[2:])
