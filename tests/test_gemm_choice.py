"""CPU: the kernel choice between the rows of the measured table."""
import ctypes
import pathlib
import re

import pytest

TABLE = pathlib.Path(__file__).resolve().parents[1] / "nvfp4quant_test_b200" / "csrc" / "gemm_plan_table.inc"


@pytest.fixture(scope="module")
def plan():
    from nvfp4quant_test_b200 import _lib, build

    build.build()
    L = _lib.lib()

    def call(m, n, k, sms=148):
        path, ranges = ctypes.c_int(-1), ctypes.c_int(-1)
        assert L.nvfp4_gemm_plan(m, n, k, sms, ctypes.byref(path), ctypes.byref(ranges)) == 0
        return path.value

    return call


@pytest.mark.parametrize("m,n,k,fastest", [(600, 7168, 8192, 2), (1100, 4096, 14336, 2), (1450, 3584, 8192, 4),
                                           (745, 7168, 8192, 4)])
def test_a_row_gives_way_where_its_kernel_needs_another_wave(plan, m, n, k, fastest):
    """Measured 14 to 56 % faster than the kernel of the row above."""
    assert plan(m, n, k) == fastest


def test_rows_hold_at_their_own_sizes(plan):
    rows = [tuple(map(int, r)) for r in re.findall(r"^\{(\d+), (\d+), (\d+), (\d+)\}", TABLE.read_text(), re.M)]
    assert all(plan(m, n, k) in (path, 5) for m, n, k, path in rows)


@pytest.mark.parametrize("m,tiles,k,decode", [(33, 48, 7168, False), (48, 48, 4096, False), (48, 56, 7168, False), (40, 64, 8192, False),
                                              (48, 32, 2048, False), (48, 32, 14336, True), (48, 112, 2048, False), (48, 112, 4608, False),
                                              (46, 112, 8192, False), (48, 148, 2048, False), (33, 224, 4096, False), (33, 47, 7168, False),
                                              (40, 65, 8192, False), (48, 111, 4608, False)])
def test_decode_sized_kernel_at_33_to_48_tokens(plan, m, tiles, k, decode):
    """Measured at least 3 % apart, in this order, us, decode-sized / best tile kernel: 33 x 48 tiles x 7168 9.6 / 8.6, 48 x 48 x 4096 7.8 /
    6.2, 48 x 56 x 7168 10.1 / 8.8, 40 x 64 x 8192 11.6 / 10.4, 48 x 32 x 2048 5.8 / 3.7, x 14336 10.5 / 13.7, 48 x 112 x 2048 6.8 / 5.3, x 4608 10.2 /
    9.0, 46 x 112 x 8192 14.7 / 13.2, 48 x 148 x 2048 7.7 / 6.1, 33 x 224 x 4096 14.0 / 13.5; the last three are one tile off one of these."""
    assert (plan(m, tiles * 128, k) == 5) == decode


@pytest.mark.parametrize("m,n,k,fastest", [(1, 512, 1024, 6), (16, 128, 64, 6), (1, 4096, 4096, 5), (16, 8192, 8192, 5), (16, 4096, 14336, 5),
                                           (16, 14336, 8192, 1), (32, 28672, 8192, 5), (24, 6144, 4096, 6), (28, 14336, 8192, 1)])
def test_small_launches_take_what_is_fastest(plan, m, n, k, fastest):
    """us, decode-sized / best tile kernel: 1 x 512 x 1024 3.0 / 2.6, 16 x 128 x 64 2.3 / 2.0, 1 x 4096 x 4096 4.5 / 5.4, 16 x 8192 x 8192 9.5 / 10.3,
    16 x 4096 x 14336 9.5 / 13.8, 16 x 14336 x 8192 14.0 / 13.1 (raw 14.4 / 13.5), 32 x 28672 x 8192 23.5 / 24.1, 24 x 6144 x 4096 6.2 / 6.4 (32 tokens 6.6 /
    6.2), 28 x 14336 x 8192 14.0 / 13.3."""
    assert plan(m, n, k) == fastest


def test_rows_of_output_that_no_copy_can_store_cost_tile_kernels_more(plan):
    """N that is no multiple of 8: us, decode-sized / best tile kernel, 30 x 12797 x 1024 4.3 / 5.6; 30 x 12800 x 1024 4.2 / 3.9."""
    assert plan(30, 12797, 1024) == 5 and plan(30, 12800, 1024) != 5
