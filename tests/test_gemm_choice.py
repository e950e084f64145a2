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


@pytest.mark.parametrize("m,tiles,k,decode", [(33, 48, 7168, True), (48, 48, 4096, False), (48, 56, 7168, True), (40, 64, 8192, True),
                                              (48, 32, 2048, False), (48, 32, 14336, True), (48, 112, 2048, False), (48, 112, 4608, True),
                                              (46, 112, 8192, False), (48, 148, 2048, False), (33, 224, 4096, True)])
def test_decode_sized_kernel_at_33_to_48_tokens(plan, m, tiles, k, decode):
    """Measured at least 1 % apart, in this order (33 x 224 tiles x 4096: 6 %; 48 x 32 x 2048: 23 %)."""
    assert (plan(m, tiles * 128, k) == 5) == decode
