"""GPU: one launch over several products gives the bits of the products launched one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operand(rows, k, seed):
    import nvfp4quant_test_b200.kernels as K

    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((rows, k), generator=g, device="cuda").bfloat16()
    codes, scales, gs, _ = K.scalesweep_nvfp4_quant_with_global_scale(x, 256.0)
    return codes, scales, gs


@pytest.mark.parametrize("path", [0, 1, 3, 4, 7])
@pytest.mark.parametrize("m,shapes", [
    (65, [(64, 64)] * 3),                                                        # tiles of one K stage, mostly padding
    (129, [(257, 320), (1000, 1024), (128, 320), (72, 2560)]),                   # ragged N, three K classes
    (300, [(4096, 4096), (1024, 4096), (1024, 4096), (4096, 4096), (2048, 4096), (4096, 14336)]),
    (700, [(512, 256)] * 9 + [(4100, 1984), (256, 512)]),                        # more than one launch takes
    (16, [(512, 1024), (256, 1024), (512, 320)]),                                # decode-sized: grouped by activation
])
def test_list_of_products_equals_one_by_one(cuda_lib, path, m, shapes):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    if m <= 64 and path:
        pytest.skip("the decode-sized kernel takes these")
    acts = {k: _operand(m, k, m + k) for k in {k for _, k in shapes}}
    weights = [_operand(n, k, 7 * i + n) for i, (n, k) in enumerate(shapes)]
    prepared = [K.PreparedWeight(c, s) for c, s, _ in weights]
    scale = [w[2].reshape(1) for w in weights]
    use = [acts[k] for _, k in shapes]
    want = [K.nvfp4_scaled_mm_grouped(a[0], a[1], a[2], [p], [s])[0] for a, p, s in zip(use, prepared, scale)]
    try:
        assert cuda_lib.nvfp4_gemm_force_path(path) == 0
        got = K.nvfp4_scaled_mm_multi([a[0] for a in use], [a[1] for a in use], [a[2] for a in use], prepared, scale)
        first = [i for i, (_, k) in enumerate(shapes) if k == shapes[0][1]]
        grouped = K.nvfp4_scaled_mm_grouped(use[0][0], use[0][1], use[0][2], [prepared[i] for i in first], [scale[i] for i in first])
        torch.cuda.synchronize()
    finally:
        cuda_lib.nvfp4_gemm_force_path(0)
    assert gemm_last_status() == 0
    if m > 64:      # K ranges per tile of the decode-sized kernel depend on the group
        for g, w in zip(got, want):
            assert torch.equal(g, w)
        for g, i in zip(grouped, first):
            assert torch.equal(g, want[i])
    else:
        for g, w in zip(got, want):
            assert torch.allclose(g.float(), w.float(), rtol=2.0 ** -7, atol=float(w.abs().max()) * 2.0 ** -12)


@pytest.mark.parametrize("m", [1, 15, 32, 33])
@pytest.mark.parametrize("shapes", [
    [(643, 10240), (384, 1344), (72, 128), (768, 1280)],       # 4, 2, 1 and 2 K ranges; clusters with tiles missing
    [(2000, 4096), (12800, 512), (12800, 512), (12800, 576)],  # so many tiles that only the longest K is cut
])
def test_products_of_different_k_in_one_decode_launch(cuda_lib, m, shapes):
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    acts = [_operand(m, k, i) for i, (_, k) in enumerate(shapes)]
    weights = [_operand(n, k, 50 + i) for i, (n, k) in enumerate(shapes)]
    prepared = [K.PreparedWeight(c, s) for c, s, _ in weights]
    scale = [w[2].reshape(1) for w in weights]
    columns = [list(c) for c in zip(*acts)]
    got = K.nvfp4_scaled_mm_multi(*columns, prepared, scale)
    again = K.nvfp4_scaled_mm_multi(*columns, prepared, scale)
    for (_, k), a, w, x, y in zip(shapes, acts, weights, got, again):
        full = [H.dequantize("base", q, K.unswizzle_vllm_fp4_scale(s, q.shape[0], k), gs).double() for q, s, gs in (a, w)]
        want = (full[0] @ full[1].T).float()
        assert torch.allclose(x.float(), want, rtol=2.0 ** -7, atol=float(want.abs().max()) * 2.0 ** -12)
        assert torch.equal(x, y)
    assert gemm_last_status() == 0


def test_list_arguments_are_checked(cuda_lib):
    import nvfp4quant_test_b200.kernels as K

    a, s, gs = _operand(80, 128, 1)
    c, sw, gw = _operand(64, 128, 2)
    w = K.PreparedWeight(c, sw)
    with pytest.raises(ValueError, match="same length"):
        K.nvfp4_scaled_mm_multi([a, a], [s], [gs], [w], [gw])
    with pytest.raises(ValueError, match="disagree on K"):
        K.nvfp4_scaled_mm_multi([a[:, :32].contiguous()], [s], [gs], [w], [gw])
    assert cuda_lib.nvfp4_gemm_launch_multi(None, 1, 8, None) == -1
    assert cuda_lib.nvfp4_gemm_launch_multi(None, 65, 8, None) == -5
    w.close()
    with pytest.raises(ValueError, match="closed"):
        K.nvfp4_scaled_mm_multi([a], [s], [gs], [w], [gw])


@pytest.mark.parametrize("path", [1, 2, 3, 4, 6, 7])
@pytest.mark.parametrize("m,n", [(33, 8), (129, 63), (130, 66), (257, 100), (300, 191), (128, 193), (100, 255), (257, 260), (65, 768)])
def test_every_row_alignment_and_edge_of_the_epilogue(cuda_lib, path, m, n):
    """Rows of whole 16 bytes, of 4 bytes and of 2, pieces cut by both edges of the matrix, nothing written beside it."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200 import helper as H

    k = 320
    a, sa, ga = _operand(m, k, m)
    b, sb, gb = _operand(n, k, n)
    alpha = (ga * gb).reshape(1)
    guard = torch.full((m * n + 256,), 7.0, dtype=torch.bfloat16, device="cuda")
    out = guard[128:128 + m * n].view(m, n)
    try:
        assert cuda_lib.nvfp4_gemm_force_path(path) == 0
        K.nvfp4_scaled_mm(a, b, sa, sb, alpha, torch.bfloat16, out)
        torch.cuda.synchronize()
    finally:
        cuda_lib.nvfp4_gemm_force_path(0)
    one = torch.ones((), device="cuda")
    da = H.dequantize("base", a, K.unswizzle_vllm_fp4_scale(sa, m, k), one).double()
    db = H.dequantize("base", b, K.unswizzle_vllm_fp4_scale(sb, n, k), one).double()
    want = (da @ db.T) * alpha.double()
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -7 + want.abs().max() * 2.0 ** -16).all()
    assert (guard[:128] == 7.0).all() and (guard[128 + m * n:] == 7.0).all()
