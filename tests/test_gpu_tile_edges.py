"""GPU: the GEMM kernels at the edges of their boxes and rings, the decode-sized kernel's exchange of partials, and every form of the channel square norm at the ends of its batches."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TILES = (1, 2, 6)      # copy boxes that end with the matrix
PAIRS = (3, 4, 7)      # zero-filled boxes
RANGES_OF_ONE = 1


def _operand(rows, k, g):
    codes = torch.randint(0, 256, (rows, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    scales = torch.randint(0x28, 0x48, ((rows + 127) // 128 * 128, k // 16), dtype=torch.uint8, device="cuda", generator=g)
    return codes, scales


# K: below one 256-wide stage, one, around the four to eight stages of the rings, and once more round them; M and N: one row, one less and
# one more than a tile of 64 / 128 / 256, a whole tile
@pytest.mark.parametrize("k", [64, 256, 1024, 1344, 2048, 3136])
@pytest.mark.parametrize("m,n", [(1, 8), (17, 127 * 8), (64, 264), (65, 64), (127, 65 * 8), (128, 128), (129, 136), (255, 200), (257, 392)])
def test_boxes_and_rings_at_their_ends(cuda_lib, m, n, k):
    """Exact: all tile and pair kernels accumulate in one K order, from a raw and from a prepared weight, whatever the boxes;
    the rows behind the output stay as they were.  The decode-sized kernel with one K range keeps that order too."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    g = torch.Generator(device="cuda")
    g.manual_seed(m * 7919 + n * 31 + k)
    (a, sa), (b, sb) = _operand(m, k, g), _operand(n, k, g)
    alpha = torch.full((1,), 0.011, dtype=torch.float32, device="cuda")
    pw = K.PreparedWeight(b, sb)
    want = None
    try:
        for path in (*PAIRS, *TILES, 5):
            if path in PAIRS and n <= 128 or path == 5 and m > 128:
                continue
            assert cuda_lib.nvfp4_gemm_force_path(path) == 0
            cuda_lib.nvfp4_gemm_tune(RANGES_OF_ONE if path == 5 else 0, -1)
            for prepared in (False, True):
                whole = torch.full((m + 4, n), float("nan"), dtype=torch.bfloat16, device="cuda")
                if prepared:
                    K.nvfp4_scaled_mm_prepared(a, sa, alpha, pw, out=whole[:m])
                else:
                    K.nvfp4_scaled_mm(a, b, sa, sb, alpha, torch.bfloat16, out=whole[:m])
                assert gemm_last_status() == 0, (path, prepared)
                assert torch.isnan(whole[m:]).all() and not torch.isnan(whole[:m]).any(), (path, prepared)
                want = whole[:m] if want is None else want
                assert torch.equal(whole[:m], want), (path, prepared)
    finally:
        cuda_lib.nvfp4_gemm_force_path(0)
        cuda_lib.nvfp4_gemm_tune(0, -1)
        pw.close()


E2M1 = (0, .5, 1, 1.5, 2, 3, 4, 6, -0., -.5, -1, -1.5, -2, -3, -4, -6)


def _values(codes, scales, rows):
    """What `rows` rows of codes and tiled scales stand for, in fp64."""
    low_first = torch.stack([codes & 15, codes >> 4], 2).reshape(rows, -1).long()
    v = torch.tensor(E2M1, dtype=torch.float64, device="cuda")[low_first]
    s = scales.reshape(scales.shape[0] // 128, -1, 32, 4, 4).permute(0, 3, 2, 1, 4).reshape(scales.shape[0], -1)[:rows]
    return v * s.view(torch.float8_e4m3fn).double().repeat_interleave(16, 1)


# N: one tile, 32 (partials behind the ring), 34 (31 and 17 tokens in four ranges: two CTAs on an SM, partials in the ring), 150 (in two
# ranges of many stages: three CTAs on an SM)
@pytest.mark.parametrize("n", [128, 32 * 128, 34 * 128 - 8, 150 * 128])
@pytest.mark.parametrize("m,ranks", [(1, 8), (2, 3), (5, 4), (9, 8), (16, 2), (17, 4), (31, 4), (33, 2), (63, 4), (65, 2), (100, 3)])
def test_partials_meet_whatever_the_tokens_of_a_rank(cuda_lib, m, n, ranks):
    """Token counts that the K ranges do not divide, ranks without a token, and both places of the exchange.  |sum of the fp32 sums'
    roundings| <= K 2^-24 sum |a b|, and one rounding to bf16."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    k = 4096
    g = torch.Generator(device="cuda")
    g.manual_seed(m * 31 + n + ranks)
    (a, sa), (b, sb) = _operand(m, k, g), _operand(n, k, g)
    alpha = torch.full((1,), 0.0078125, dtype=torch.float32, device="cuda")
    va, vb = _values(a, sa, m), _values(b, sb, n)
    want = va @ vb.T * 0.0078125
    bound = (va.abs() @ vb.abs().T) * 0.0078125 * (k * 2.0 ** -24) + want.abs() * 2.0 ** -8
    pw = K.PreparedWeight(b, sb)
    try:
        assert cuda_lib.nvfp4_gemm_force_path(5) == 0 and cuda_lib.nvfp4_gemm_tune(ranks, -1) == 0
        raw = K.nvfp4_scaled_mm(a, b, sa, sb, alpha, torch.bfloat16)
        prepared = K.nvfp4_scaled_mm_prepared(a, sa, alpha, pw)
        assert gemm_last_status() == 0
    finally:
        cuda_lib.nvfp4_gemm_force_path(0)
        cuda_lib.nvfp4_gemm_tune(0, -1)
        pw.close()
    assert torch.equal(raw, prepared)
    assert bool(((raw.double() - want).abs() <= bound).all())


# q / k / v of a small layer (a list of tiles from the first token on), gate / up of one (decode-sized at few tokens, then tiles), few tiles
# and a long K (decode-sized throughout)
@pytest.mark.parametrize("k,ns", [(1024, (1024, 256, 256)), (2048, (8192, 8192)), (8192, (512, 264, 128))])
@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65, 128, 129])
def test_groups_on_either_side_of_the_choice(cuda_lib, m, k, ns):
    """Grouped products by whichever kernel is chosen.  |sum of the fp32 sums' roundings| <= K 2^-24 sum |a b|, and one rounding to bf16."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    g = torch.Generator(device="cuda")
    g.manual_seed(m * 31 + k)
    a, sa = _operand(m, k, g)
    va, alpha = _values(a, sa, m), torch.full((1,), 0.0078125, device="cuda")
    operands = [_operand(n, k, g) for n in ns]
    pws = [K.PreparedWeight(*o) for o in operands]
    one = torch.ones(1, device="cuda")
    got = K.nvfp4_scaled_mm_multi([a] * len(ns), [sa] * len(ns), [one] * len(ns), pws, [alpha] * len(ns))
    assert gemm_last_status() == 0
    for out, (b, sb), n in zip(got, operands, ns):
        vb = _values(b, sb, n)
        want = va @ vb.T * 0.0078125
        bound = (va.abs() @ vb.abs().T) * 0.0078125 * (k * 2.0 ** -24) + want.abs() * 2.0 ** -8
        assert bool(((out.double() - want).abs() <= bound).all()), n


@pytest.mark.parametrize("m", [33, 80, 129, 300])
def test_lists_in_every_tile(cuda_lib, m):
    """Products of different K and N in one launch of each tile kernel equal the one-by-one calls bit for bit."""
    import nvfp4quant_test_b200.kernels as K
    from nvfp4quant_test_b200.kernels.kernel_gemm import gemm_last_status

    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    shapes = [(512, 1024), (136, 1024), (1000, 320), (264, 2752), (2048, 1024), (72, 64), (3000, 320)]
    acts = {k: _operand(m, k, g) for _, k in shapes}
    pws = [K.PreparedWeight(*_operand(n, k, g)) for n, k in shapes]
    alphas = [torch.rand(1, device="cuda", generator=g) * 0.01 + 0.01 for _ in shapes]
    one = torch.ones(1, device="cuda")
    try:
        cuda_lib.nvfp4_gemm_force_path(1)
        single = [K.nvfp4_scaled_mm_prepared(*acts[k], al, pw) for (_, k), al, pw in zip(shapes, alphas, pws)]
        for path in (0, 1, 2, 6):
            assert cuda_lib.nvfp4_gemm_force_path(path) == 0
            got = K.nvfp4_scaled_mm_multi([acts[k][0] for _, k in shapes], [acts[k][1] for _, k in shapes], [one] * len(shapes), pws, alphas)
            assert gemm_last_status() == 0, path
            for i, (x, y) in enumerate(zip(got, single)):
                assert torch.equal(x, y), (path, i)
    finally:
        cuda_lib.nvfp4_gemm_force_path(0)


# columns: one CTA, at most one / two / three / four and five / more an SM; rows: none of a group's, one, around the batches of 4, 8, 16, 32
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n", [4, 1072, 4736, 7104, 9488, 12288])
def test_square_norm_batches(cuda_lib, n, dtype):
    """All terms are positive, so that a sum over ceil(m / 64) rows and six levels of a tree is within that many roundings (one more for
    the square) of the exact one.  The rows behind the matrix and the columns beside it are NaN: nothing of them gets into a sum.
    Slices of 1072 columns take another form than the whole and give the same bits."""
    from nvfp4quant_test_b200 import helper as H

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    for m in (1, 63, 65, 256, 257, 64 * 7 + 3, 64 * 8, 64 * 9 + 1, 64 * 15 + 63, 64 * 31 + 1, 64 * 32, 64 * 33 + 5, 64 * 47 + 2):
        whole = torch.full((m + 3, n + 8), float("nan"), dtype=dtype, device="cuda")
        whole[:m, :n] = torch.randn((m, n), device="cuda", generator=g).to(dtype)
        x = whole[:m, :n]
        got = H.channel_square_norm(x)
        want = (x.double() ** 2).sum(0, keepdim=True)
        bound = ((m + 63) // 64 + 7) * 2.0 ** -24
        assert bool(((got.double() - want).abs() <= bound * want).all()), (m, n)
        if n > 1072:
            assert torch.equal(H.channel_square_norm(x[:, 16:1088]), got[:, 16:1088]), (m, n)
