"""GPU: forms of calls at the edges of what the entry points take, and their order on a stream."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 256])
def test_a_weight_is_complete_before_a_product_reads_it(cuda_lib, tokens):
    """A weight whose quantizer runs for hundreds of microseconds, then a short quantization and the product with it in dependent
    launches, nothing else between: the product must wait for the weight, freshly made and requantized in place."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H

    n, k = 28672, 8192
    g = torch.Generator(device="cuda").manual_seed(tokens)
    ws = [torch.randn((n, k), generator=g, device="cuda").bfloat16() * f for f in (1.0, 2.0, 0.5)]
    pairs = [H.get_nvfp4_global_scale(w, 256.0) for w in ws]
    vecs = [gs.reshape(1) for gs, _ in pairs]
    x = torch.randn((tokens, k), generator=g, device="cuda").bfloat16()
    used = torch.full((n, k // 2), 0x77, dtype=torch.uint8, device="cuda")   # the block the first codes are likely to get
    K.scalesweep_mse_nvfp4_quant_impl(x, pairs[0][1])                        # modules loaded
    torch.cuda.synchronize()
    del used
    codes, scales = K.scalesweep_mse_nvfp4_quant_impl(ws[0], pairs[0][1])
    weight = K.PreparedWeight(codes, scales)
    got = [K.nvfp4_linear_multi([x], [0], [weight], [vecs[0]], [0])[0]]
    for i in (1, 2, 0):
        K.scalesweep_mse_nvfp4_quant_out(ws[i], pairs[i][1], True, output=codes, output_scale=scales)
        got.append(K.nvfp4_linear_multi([x], [0], [weight], [vecs[i]], [0])[0])
    torch.cuda.synchronize()
    for i, have in zip((0, 1, 2, 0), got):
        K.scalesweep_mse_nvfp4_quant_out(ws[i], pairs[i][1], True, output=codes, output_scale=scales)
        torch.cuda.synchronize()
        assert torch.equal(have, K.nvfp4_linear_multi([x], [0], [weight], [vecs[i]], [0])[0])
        torch.cuda.synchronize()


@pytest.mark.parametrize("path,n", [(6, 131072), (6, 262144), (6, 262208), (1, 524288)])
def test_products_with_thousands_of_column_tiles(cuda_lib, path, n):
    """Counts of column tiles at which (m-tiles of a band) x (column tiles) used to leave the int range, against 256-wide tiles."""
    import nvfp4quant_test_b200.kernels as K

    m, k = 130, 64
    g = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.randint(0, 256, (rows, k // 2), dtype=torch.uint8, device="cuda", generator=g) for rows in (m, n))
    sa, sb = (torch.randint(0x30, 0x40, ((rows + 127) // 128 * 128, 4), dtype=torch.uint8, device="cuda", generator=g) for rows in (m, n))
    one = torch.ones(1, device="cuda")
    got = []
    try:
        for p in (path, 2):
            assert cuda_lib.nvfp4_gemm_force_path(p) == 0
            got.append(K.nvfp4_scaled_mm(a, b, sa, sb, one, torch.bfloat16))
            torch.cuda.synchronize()
    finally:
        cuda_lib.nvfp4_gemm_force_path(0)
    assert torch.equal(*got)


def _quantized(m=32, n=256):
    g = torch.Generator(device="cuda").manual_seed(3)
    codes = torch.randint(0, 256, (m, n // 2), dtype=torch.uint8, device="cuda", generator=g)
    scales = torch.randint(0x20, 0x70, (m, n // 16), dtype=torch.uint8, device="cuda", generator=g).view(torch.float8_e4m3fn)
    return codes, scales, torch.tensor(0.5, device="cuda")


def test_dequantization_stays_differentiable_in_the_global_scale(cuda_lib):
    import torch.autograd.forward_ad as fwd

    from nvfp4quant_test_b200 import helper as H

    q, s, gs = _quantized()
    unit = H.dequantize_base(q, s, torch.ones((), device="cuda"))
    g = gs.clone().requires_grad_()
    y = H.dequantize_base(q, s, g)
    assert torch.equal(y.detach(), H.dequantize_base(q, s, gs))
    (grad,) = torch.autograd.grad(y.sum(), g)
    # two fp32 sums of the same n values in any order: n * 2^-24 of the sum of their magnitudes apart
    assert abs(grad - unit.sum()) <= unit.abs().sum() * unit.numel() * 2.0 ** -24
    with torch.no_grad():
        assert not H.dequantize_base(q, s, g).requires_grad
    with fwd.dual_level():
        tangent = fwd.unpack_dual(H.dequantize_base(q, s, fwd.make_dual(gs, torch.ones_like(gs)))).tangent
        assert tangent is not None and torch.equal(tangent, unit)
    assert torch.equal(torch.func.grad(lambda v: H.dequantize_base(q, s, v).sum())(gs), grad)
    both = torch.func.vmap(lambda v: H.dequantize_base(q, s, v))(torch.stack([gs, gs * 2]))
    assert torch.equal(both[1], H.dequantize_base(q, s, gs * 2))
    assert torch.equal(H.dequantize_base(q, s, torch._neg_view(gs)), -H.dequantize_base(q, s, gs))


@pytest.mark.parametrize("trace", ["make_fx", "compile"])
def test_dequantization_and_scale_layouts_can_be_traced(cuda_lib, trace):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H

    q, s, gs = _quantized()

    def f(q, s, gs):
        tiled = K.swizzle_vllm_fp4_scale(s, 32, 256)
        return H.dequantize_base(q, K.unswizzle_vllm_fp4_scale(tiled, 32, 256), gs), H.unpack_fp4_e2m1(q)

    if trace == "make_fx":
        from torch.fx.experimental.proxy_tensor import make_fx

        traced = make_fx(f)(q, s, gs)
    else:
        traced = torch.compile(f, backend="eager", fullgraph=True)
    other = (q.flip(0).contiguous(), s.view(torch.uint8).flip(0).contiguous().view(torch.float8_e4m3fn), gs * 2)
    for got, want in zip(traced(*other), f(*other)):
        assert torch.equal(got, want)


@pytest.mark.parametrize("streams", [0, 2])
@pytest.mark.parametrize("rows", [(0, 0), (3, 0)])
def test_a_layer_of_prepared_weights_takes_an_activation_without_rows(cuda_lib, streams, rows):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import llama_stack as S

    qlayer = {name: K.scalesweep_nvfp4_quant_with_global_scale(torch.randn(shape, device="cuda").bfloat16(), 256.0)[:3]
              for name, shape in {"a": (64, 128), "b": (72, 256)}.items()}
    acts = {k: torch.randn((m, k), device="cuda").bfloat16() for m, k in zip(rows, (128, 256))}
    side = [torch.cuda.Stream() for _ in range(streams)] or None
    scales = S.stack_weight_scales(qlayer)
    got = S.layer_gemms(qlayer, acts, {}, scales, side, S.prepare_layer(qlayer))
    want = S.layer_gemms(qlayer, acts, {}, scales)
    assert {k: tuple(v.shape) for k, v in got.items()} == {"a": (rows[0], 64), "b": (rows[1], 72)}
    assert all(torch.equal(got[k], want[k]) for k in got)


@pytest.mark.parametrize("fp8_max", [0.0, -448.0, float("nan")])
def test_a_maximum_that_is_not_positive_is_refused(cuda_lib, fp8_max):
    import nvfp4quant_test_b200.kernels as K

    x = torch.randn((4, 64), device="cuda").bfloat16()
    for importance in (None, torch.ones((1, 64), device="cuda")):
        with pytest.raises(ValueError, match="positive"):
            K.scalesweep_nvfp4_quant_with_global_scale(x, fp8_max, importance)
    with pytest.raises(ValueError, match="positive"):
        K.scalesweep_nvfp4_quant_with_global_scales([x, x], fp8_max)


def _host_operands(m=200, n=96):
    g = torch.Generator().manual_seed(1)
    return torch.randn((m, n), generator=g).bfloat16(), torch.rand((1, n), generator=g).cuda(), torch.tensor([40.0], device="cuda")


@pytest.mark.parametrize("form", ["flat importance", "longer importance", "importance of no use", "more rows", "int16 codes", "subclass"])
def test_host_pipeline_takes_what_it_took(cuda_lib, form):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import _lib
    from nvfp4quant_test_b200.host_pipeline import HostQuantizer

    class Sub(torch.Tensor):
        pass

    x, imp, gs = _host_operands()
    m, n = x.shape
    if form == "importance of no use":
        want, variant, window = K.scalesweep_mse_nvfp4_quant_impl(x.cuda(), gs), _lib.VARIANT_MSE, (-3, 7)
    else:
        want, variant, window = K.scalesweep_weighted_mse_nvfp4_quant_impl(x.cuda(), imp, gs), _lib.VARIANT_WEIGHTED, (-8, 7)
    hq = HostQuantizer(m, n, torch.bfloat16, "cuda", chunk_rows=128, variant=variant, lower=window[0], upper=window[1])
    codes = torch.zeros((m + 7 if form == "more rows" else m, n // 2), dtype=torch.int16 if form == "int16 codes" else torch.uint8)
    scales = torch.zeros(want[1].numel(), dtype=torch.uint8)
    imp = {"flat importance": imp[0], "longer importance": torch.cat([imp, imp], 1), "importance of no use": torch.ones(3)}.get(form, imp)
    args = (x, gs, codes, scales, imp)
    hq(*(t.as_subclass(Sub) for t in args) if form == "subclass" else args)
    torch.cuda.synchronize()
    assert torch.equal(codes[:m].to(torch.uint8), want[0].cpu()) and not codes[m:].any()
    assert torch.equal(scales, want[1].view(torch.uint8).reshape(-1).cpu())


def test_host_pipeline_refuses_codes_of_another_shape(cuda_lib):
    from nvfp4quant_test_b200.host_pipeline import HostQuantizer

    x, imp, gs = _host_operands()
    m, n = x.shape
    hq = HostQuantizer(m, n, torch.bfloat16, "cuda", chunk_rows=128)
    scales = torch.zeros(256 * 8, dtype=torch.uint8)
    for shape in ((m * n // 2,), (n // 2, m), (m - 1, n // 2)):
        with pytest.raises(ValueError, match="codes_host"):
            hq(x, gs, torch.zeros(shape, dtype=torch.uint8), scales)
    with pytest.raises(ValueError, match="importance"):
        HostQuantizer(m, n, torch.bfloat16, "cuda", variant=1, lower=-8, upper=7)(x, gs, torch.zeros((m, n // 2), dtype=torch.uint8), scales, imp[:, :-1])


@pytest.mark.parametrize("rows,chunk", [(2000, 256), (300, 512)])     # several chunks, one chunk
def test_host_pipeline_is_shared_by_threads(cuda_lib, rows, chunk):
    import threading

    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200.host_pipeline import HostQuantizer

    g = torch.Generator().manual_seed(rows)
    gs = torch.tensor([40.0], device="cuda")
    hq = HostQuantizer(rows, 4096, torch.bfloat16, "cuda", chunk_rows=chunk)
    wrong = []

    def work(x, want, stream):
        codes, scales = torch.zeros_like(want[0]).pin_memory(), torch.zeros_like(want[1]).pin_memory()
        with torch.cuda.stream(stream):
            for _ in range(20):
                codes.zero_(), scales.zero_()
                hq(x, gs, codes, scales)
                stream.synchronize()
                if not (torch.equal(codes, want[0]) and torch.equal(scales, want[1])):
                    wrong.append(1)

    xs = [torch.randn((rows, 4096), generator=g).bfloat16().pin_memory() for _ in range(3)]
    wants = []
    for x in xs:
        codes, scales = K.scalesweep_mse_nvfp4_quant_impl(x.cuda(), gs)
        wants.append((codes.cpu(), scales.view(torch.uint8).reshape(-1).cpu()))
    threads = [threading.Thread(target=work, args=(x, w, torch.cuda.Stream())) for x, w in zip(xs, wants)]
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("ranges", [3, 6, 7, 8])
@pytest.mark.parametrize("stages", [(25, 24), (24, 25), (49, 13, 24), (9, 8)])
def test_forced_k_ranges_of_products_of_different_k(cuda_lib, ranges, stages):
    """A number of ranges that leaves none of any product empty: an empty one would add uninitialised TMEM."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    def operand(rows, k):
        return K.scalesweep_nvfp4_quant_with_global_scale(torch.randn((rows, k), device="cuda").bfloat16(), 256.0)[:3]

    acts, weights = [operand(16, 256 * s) for s in stages], [operand(200, 256 * s) for s in stages]
    prepared = [K.PreparedWeight(c, s) for c, s, _ in weights]
    try:
        assert cuda_lib.nvfp4_gemm_force_path(5) == 0 and cuda_lib.nvfp4_gemm_tune(ranges, -1) == 0
        got = K.nvfp4_scaled_mm_multi(*[list(c) for c in zip(*acts)], prepared, [w[2].reshape(1) for w in weights])
        torch.cuda.synchronize()
    finally:
        cuda_lib.nvfp4_gemm_force_path(0)
        cuda_lib.nvfp4_gemm_tune(0, -1)
    assert gemm_last_status() == 0
    for s, a, w, x in zip(stages, acts, weights, got):
        full = [H.dequantize("base", q, K.unswizzle_vllm_fp4_scale(sc, q.shape[0], 256 * s), gs).double() for q, sc, gs in (a, w)]
        want = full[0] @ full[1].T
        assert ((x.double() - want).abs() <= want.abs() * 2.0 ** -7 + want.abs().max() * 2.0 ** -16).all()


def test_channel_norms_of_one_strided_row(cuda_lib):
    from nvfp4quant_test_b200 import helper as H

    x = torch.randn((1, 128), device="cuda").bfloat16()
    assert torch.equal(H.channel_square_norm(x[:, ::2]), H.channel_square_norm(x[:, ::2].contiguous()))
    column = torch.randn((64, 4), device="cuda").bfloat16()
    assert torch.equal(H.channel_square_norm(column.t()[1:2]), column.float().square().t()[1:2])


@pytest.mark.parametrize("lower", [-(1 << 70), (1 << 32) - 3])
def test_window_bounds_beyond_an_int_go_the_way_of_ctypes(cuda_lib, lower):
    """ctypes keeps the low 32 bits of an int argument: 0 and -3 here."""
    import nvfp4quant_test_b200.kernels as K

    x, imp = torch.randn((4, 64), device="cuda").bfloat16(), torch.rand((1, 64), device="cuda")
    gs_inv = torch.ones(1, device="cuda")
    same = 0 if lower < 0 else -3
    for call in (lambda b: K.scalesweep_weighted_mse_nvfp4_quant_impl(x, imp, gs_inv, lower_bound=b, upper_bound=7),
                 lambda b: K.scalesweep_nvfp4_quant_with_global_scale(x, 256.0, imp, lower_bound=b, upper_bound=7)):
        for got, want in zip(call(lower), call(same)):
            assert torch.equal(got.reshape(-1).view(torch.uint8), want.reshape(-1).view(torch.uint8))


def test_products_refuse_operands_in_host_memory(cuda_lib):
    """Every operand of every form: what is not on the weight's device is an error of the call, not of the GPU."""
    import nvfp4quant_test_b200.kernels as K

    x, w = (torch.randn((rows, 128), device="cuda").bfloat16() for rows in (4, 64))
    (a, sa, ga, _), (b, sb, gb, _) = (K.scalesweep_nvfp4_quant_with_global_scale(t) for t in (x, w))
    ga, gb, out = ga.reshape(1), gb.reshape(1), torch.empty((4, 64), dtype=torch.bfloat16, device="cuda")
    weight = K.PreparedWeight(b, sb)
    group, quantizer = K.LinearGroup([weight], [gb], 4), K.ActivationQuantizer(4, 128, "cuda")
    forms = [(K.nvfp4_scaled_mm, [a, b, sa, sb, ga, torch.bfloat16, out]), (K.nvfp4_scaled_mm_prepared, [a, sa, ga, weight, out]),
             (K.nvfp4_scaled_mm_grouped, [a, sa, ga, [weight], [gb], [out]]), (K.nvfp4_scaled_mm_multi, [[a], [sa], [ga], [weight], [gb]]),
             (K.nvfp4_linear_multi, [[x], [0], [weight], [gb], [0]]), (group, [a, sa, ga]), (quantizer, [x])]
    for call, args in forms:
        for i, arg in enumerate(args):
            if isinstance(arg, torch.Tensor):
                moved = arg.cpu()
            elif isinstance(arg, list) and isinstance(arg[0], torch.Tensor):
                moved = [arg[0].cpu()]
            else:
                continue
            with pytest.raises(ValueError):
                call(*args[:i], moved, *args[i + 1:])
        call(*args)
    torch.cuda.synchronize()


def test_scratch_words_of_many_streams_and_threads(cuda_lib):
    """More streams than scratch words are kept for, used by several threads at once."""
    import threading

    from nvfp4quant_test_b200 import helper as H

    x = torch.randn((300, 8192), device="cuda").bfloat16()
    xs = [x * (i + 1) for i in range(8)]
    want = [H.get_nvfp4_global_scale(t)[0].item() for t in xs]
    wrong = []

    def work(i):
        streams = [torch.cuda.Stream() for _ in range(6)]
        for _ in range(30):
            got = []
            for s in streams:
                with torch.cuda.stream(s):
                    got.append(H.get_nvfp4_global_scale(xs[i])[0])
            torch.cuda.synchronize()
            wrong.extend(1 for g in got if g.item() != want[i])

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("m,n,padded_n,tiled", [(129, 16, None, True), (3, 112, 176, True), (300, 48, None, False), (77, 4096, None, True), (130, 4096, 8192, True),
                                                (129, 8192, None, False), (401, 7216, 7232, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_quantizer_bodies_by_size_equal_the_plain_ones(cuda_lib, m, n, padded_n, tiled, dtype):
    """Slots in large CTAs with the loop rolled (5), warps of rows (6), amax on rows of whole chunks (8): padding rows, padding columns,
    rows longer and shorter than a CTA."""
    from nvfp4quant_test_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn((m, n), generator=g, device="cuda").to(dtype)
    gs_inv, p = torch.tensor([37.5], device="cuda"), padded_n or n
    size = (m + 127) // 128 * 128 * ((p // 16 + 3) // 4 * 4) if tiled else m * p // 16
    for variant, lower, upper, plain, bodies in ((0, -3, 7, 1, (5, 6)), (0, -2, 5, 1, (5, 6)), (2, 0, 0, 3, (5, 6, 7, 8))):
        want = None
        for impl in (plain, *bodies):
            codes, scales = (torch.full(s, 0xA5, dtype=torch.uint8, device="cuda") for s in ((m, p // 2), (size,)))
            _lib.check(cuda_lib.nvfp4_quant_launch_impl(impl, variant, x.data_ptr(), _lib.dtype_code(dtype), None, gs_inv.data_ptr(), codes.data_ptr(),
                                                        scales.data_ptr(), m, n, p, lower, upper, int(tiled), None), "launch")
            torch.cuda.synchronize()
            want = want or (codes, scales)
            assert torch.equal(codes, want[0]) and torch.equal(scales, want[1]), (impl, variant, lower)


@pytest.mark.parametrize("variant,dtype,blocks", [(0, torch.bfloat16, 393216), (0, torch.float16, 393216), (2, torch.float32, 131072), (2, torch.bfloat16, 524288)])
def test_quantizer_choice_by_size_equals_the_plain_body(cuda_lib, variant, dtype, blocks):
    """Either side of the sizes at which the default changes: whole chunks and three kinds of ragged rows."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import _lib

    gs_inv = torch.tensor([37.5], device="cuda")
    call = K.amax_nvfp4_quant_impl if variant == 2 else K.scalesweep_mse_nvfp4_quant_impl
    for n in (4096, 4176, 7216, 13328):
        for m in (blocks * 16 // n, -(-blocks * 16 // n)):
            x = torch.randn((m, n), device="cuda").to(dtype)
            got = call(x, gs_inv)
            codes, scales = torch.empty_like(got[0]), torch.empty_like(got[1])
            _lib.check(cuda_lib.nvfp4_quant_launch_impl(1 if variant == 0 else 3, variant, x.data_ptr(), _lib.dtype_code(dtype), None, gs_inv.data_ptr(),
                                                        codes.data_ptr(), scales.data_ptr(), m, n, n, -3, 7, 1, None), "launch")
            assert torch.equal(codes, got[0]) and torch.equal(scales.view(torch.uint8), got[1].view(torch.uint8)), (n, m)


@pytest.mark.parametrize("dtype,n", [(torch.bfloat16, 4096), (torch.float32, 2048)])
@pytest.mark.parametrize("m", [8, 9, 16, 17])
def test_scale_inside_the_quantizer_up_to_its_limit(cuda_lib, dtype, n, m):
    """64 and 128 KiB and one row more: one launch and two, same bytes."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H

    x = torch.randn((m, n), device="cuda").to(dtype)
    codes, scales, gs, gs_inv = K.scalesweep_nvfp4_quant_with_global_scale(x, 256.0)
    want = H.get_nvfp4_global_scale(x, 256.0)
    plain = K.scalesweep_mse_nvfp4_quant_impl(x, want[1])
    assert gs == want[0] and gs_inv == want[1] and torch.equal(codes, plain[0])
    assert torch.equal(scales.view(torch.uint8), plain[1].view(torch.uint8))
    codes, scales, gs = K.ActivationQuantizer(m, n, "cuda", dtype=dtype)(x)
    assert gs[0] == want[0] and torch.equal(codes, plain[0]) and torch.equal(scales.view(torch.uint8), plain[1].view(torch.uint8))
