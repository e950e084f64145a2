"""CPU: the C ABI library loads and exports what include/nvfp4_b200.h declares; argument
validation answers without touching a GPU."""
import ctypes
import pathlib
import re

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def L():
    from nvfp4quant_test_b200 import _lib, build

    build.build()
    return _lib.lib()


def declared_functions():
    text = (ROOT / "include" / "nvfp4_b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(nvfp4_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(L):
    from nvfp4quant_test_b200 import _lib

    names = declared_functions()
    assert len(names) >= 10
    for n in names:
        assert hasattr(L, n), f"{n} declared in the header but not exported"
    assert set(_lib.EXPORTS) <= set(names)


def test_abi_version_and_status_strings(L):
    from nvfp4quant_test_b200 import _lib

    assert L.nvfp4_abi_version() >= 1
    assert _lib.status_string(0) == "ok"
    for code in range(-9, 0):
        s = _lib.status_string(code)
        assert s and s != "unknown status"
    assert _lib.status_string(-99) == "unknown status"


def test_quant_launch_rejects_bad_arguments_before_launching(L):
    q = L.nvfp4_quant_launch
    P = 0x1000  # fake, aligned, never dereferenced: validation fails first
    assert q(7, P, 0, None, P, P, P, 4, 64, 64, -3, 7, 1, None) == -3          # variant
    assert q(0, P, 9, None, P, P, P, 4, 64, 64, -3, 7, 1, None) == -3          # dtype
    assert q(0, P, 0, None, P, P, P, 4, 60, 64, -3, 7, 1, None) == -2          # n % 16
    assert q(0, P, 0, None, P, P, P, 4, 64, 48, -3, 7, 1, None) == -2          # padded_n < n
    assert q(0, P, 0, None, P, P, P, 4, 64, 72, -3, 7, 1, None) == -2          # padded_n % 16
    assert q(0, P, 0, None, P, P, P, -1, 64, 64, -3, 7, 1, None) == -2
    assert q(0, P, 0, None, P, P, P, 4, 64, 64, 3, 2, 1, None) == -5           # empty window
    assert q(0, P, 0, None, P, P, P, 4, 64, 64, -40, 40, 1, None) == -5        # > 64 candidates
    assert q(0, None, 0, None, P, P, P, 4, 64, 64, -3, 7, 1, None) == -1       # null x
    assert q(1, P, 0, None, P, P, P, 4, 64, 64, -8, 7, 1, None) == -1          # weighted without importance
    assert q(0, P + 2, 0, None, P, P, P, 4, 64, 64, -3, 7, 1, None) == -4      # misaligned x
    assert q(0, P, 0, None, P, P + 1, P, 4, 64, 64, -3, 7, 1, None) == -4      # misaligned codes
    assert q(0, P, 0, None, P, P, P, 0, 64, 64, -3, 7, 1, None) == 0           # empty input: nothing to do
    assert L.nvfp4_quant_launch_impl(12, 0, P, 0, None, P, P, P, 4, 64, 64, -3, 7, 1, None) == -3


def test_gemm_launch_rejects_bad_arguments_before_launching(L):
    g = L.nvfp4_gemm_launch
    P = 0x1000
    assert g(P, P, P, P, P, P, 128, 128, 96, None, 0, None) == -2    # K % 64
    assert g(P, P, P, P, P, P, -1, 128, 64, None, 0, None) == -2
    assert g(None, P, P, P, P, P, 128, 128, 64, None, 0, None) == -1
    assert g(P + 4, P, P, P, P, P, 128, 128, 64, None, 0, None) == -4
    assert g(P, P, P, P, P, P, 0, 128, 64, None, 0, None) == 0       # empty output
    assert L.nvfp4_gemm_workspace_bytes(8192, 8192, 8192) == 0
    assert L.nvfp4_gemm_workspace_bytes(16, 8192, 8192) == 0
    try:                                                          # K ranges need fp32 partial tiles
        assert L.nvfp4_gemm_tune(4, 0) == 0
        need = L.nvfp4_gemm_workspace_bytes(16, 8192, 8192)
        assert need == 4 * 16 * 8192 * 4
        assert g(P, P, P, P, P, P, 16, 8192, 8192, None, 0, None) == -6      # workspace missing
        assert g(P, P, P, P, P, P, 16, 8192, 8192, P, need - 1, None) == -6  # workspace too small
    finally:
        L.nvfp4_gemm_tune(0, -1)
    assert L.nvfp4_gemm_tune(99, 0) == -3


def test_global_scale_rejects_bad_arguments(L):
    f = L.nvfp4_global_scale_launch
    P = 0x1000
    assert f(P, 5, 16, 448.0, P, P, None) == -3
    assert f(P, 0, -1, 448.0, P, P, None) == -2
    assert f(P, 0, 16, 448.0, None, P, None) == -1
    assert f(P + 2, 0, 16, 448.0, P, P, None) == -4


def test_fused_launch_rejects_bad_arguments_before_launching(L):
    f = L.nvfp4_quant_fused_launch
    P = 0x1000  # fake, aligned, never dereferenced: validation fails first
    ok = [0, P, 0, None, 256.0, P, P, P, P, 4, 64, 64, -3, 7, 1, None]

    def call(**kw):
        a = list(ok)
        for i, v in kw.items():
            a[int(i[1:])] = v
        return f(*a)

    assert call(a0=2) == -3            # the amax variant has no fused form
    assert call(a2=5) == -3            # dtype
    assert call(a10=60) == -2          # n not a multiple of 16
    assert call(a11=48) == -2          # padded_n < n
    assert call(a12=7, a13=-3) == -5   # empty window
    assert call(a4=0.0) == -5          # fp8_max must be positive
    assert call(a9=0) == -2            # an empty tensor has no maximum
    assert call(a5=None) == -1         # null outputs
    assert call(a0=1) == -1            # weighted without importance
    assert call(a1=P + 2) == -4        # misaligned input


def test_gemm_kernel_choice_by_shape(L):
    """nvfp4_gemm_plan answers on the host which kernel a shape takes on a 148-SM GPU: the decode-sized kernel (5)
    with its K ranges where few tokens, few weight tiles or a long K make it the fastest, up to 128 tokens; tile and pair kernels else."""
    def plan(M, N, K, sms=148):
        path, ranges = ctypes.c_int(-1), ctypes.c_int(-1)
        assert L.nvfp4_gemm_plan(M, N, K, sms, ctypes.byref(path), ctypes.byref(ranges)) == 0
        return path.value, ranges.value

    assert plan(1, 4096, 4096) == (5, 4)             # 32 weight tiles x 4 ranges = 128 CTAs
    assert plan(16, 8192, 8192) == (5, 4)            # 64 tiles: 2 ranges fill the SMs, one more cut pays (two CTAs / SM)
    assert plan(32, 8192, 8192) == (6, 1)            # level (10.0 to 10.8 and 10.2 to 10.3 us)
    assert plan(16, 4096, 14336) == (5, 8)
    assert plan(16, 14336, 4096) == (1, 1)           # 112 tiles cover most SMs: 8.6 to 8.8 and 8.3 to 8.5 us
    assert plan(16, 28672, 8192) == (5, 1)
    assert plan(1, 512, 2048) == (5, 4)              # at least two K stages per range
    assert plan(16, 128, 64) == (6, 1)
    assert plan(64, 4096, 14336) == (5, 4)           # few tiles, long K: still the decode-sized kernel
    assert plan(128, 4096, 14336) == (5, 4)
    # shapes outside the measured table: the cost model (128x64 tiles for one or two token tiles and few weight tiles,
    # CTA pairs for large shapes)
    assert plan(64, 2048, 2048) == (6, 1)
    assert plan(8192, 16384, 4096) == (4, 1)
    assert plan(20000, 8192, 8192) == (4, 1)         # beyond the largest tabulated M
    assert plan(256, 8192, 8192, sms=132) == plan(256, 8192, 8192, sms=131) == (1, 1)   # another SM count: the table does not apply, the model does
    # shapes of the measured table take the kernel that was fastest when it was generated
    table = ROOT / "nvfp4quant_test_b200" / "csrc" / "gemm_plan_table.inc"
    rows = [tuple(int(v) for v in m.groups()) for m in re.finditer(r"^\{(\d+), (\d+), (\d+), (\d+)\}", table.read_text(), re.M)]
    assert len(rows) >= 40
    for M, N, K, path in rows:
        got = plan(M, N, K)
        assert got == (path, 1) or (M <= 128 and got[0] == 5), (M, N, K, path, got)   # up to 128 tokens the decode kernel may take it
        if M > 128:
            assert plan(M - 60, N, K) == (path, 1)    # a launch uses the row with the smallest tabulated M >= its own
    # forcing a kernel / K ranges is honoured, larger M than the skinny kernel takes falls back
    try:
        assert L.nvfp4_gemm_force_path(5) == 0 and L.nvfp4_gemm_tune(8, -1) == 0
        assert plan(100, 1024, 8192) == (5, 8)
        assert plan(300, 1024, 8192)[0] != 5
        assert L.nvfp4_gemm_force_path(2) == 0 and L.nvfp4_gemm_tune(0, -1) == 0
        assert plan(1, 4096, 4096) == (2, 1)
    finally:
        L.nvfp4_gemm_force_path(0)
        L.nvfp4_gemm_tune(0, -1)
    assert L.nvfp4_gemm_plan(1, 4096, 100, 148, None, None) < 0
    p_, r_ = ctypes.c_int(), ctypes.c_int()
    assert L.nvfp4_gemm_plan(1, 4096, 100, 148, ctypes.byref(p_), ctypes.byref(r_)) == -2


def test_quant_chain_launch_rejects_bad_arguments_before_launching(L):
    P = 0x1000
    f = L.nvfp4_quant_chain_launch
    assert f(0, P, 0, None, 256.0, P, P, P, P, 0, 64, 64, -3, 7, 1, None) == -2      # empty tensor: no maximum
    assert f(0, P, 0, None, 0.0, P, P, P, P, 4, 64, 64, -3, 7, 1, None) == -5        # fp8_max must be positive
    assert f(0, P, 0, None, 256.0, None, P, P, P, 4, 64, 64, -3, 7, 1, None) == -1   # no place for the scale
    assert f(0, P, 7, None, 256.0, P, P, P, P, 4, 64, 64, -3, 7, 1, None) == -3      # dtype (refused by the first launch)
    assert f(0, P + 2, 0, None, 256.0, P, P, P, P, 4, 64, 64, -3, 7, 1, None) == -4  # misaligned input


def test_gemm_prepare_rejects_bad_arguments_and_release_is_safe(L):
    h = ctypes.c_void_p()
    P = 0x1000   # fake, aligned, never dereferenced: tensor maps only record the address
    assert L.nvfp4_gemm_prepare(P, P, 256, 100, ctypes.byref(h)) == -2 and not h.value       # K % 64
    assert L.nvfp4_gemm_prepare(None, P, 256, 128, ctypes.byref(h)) == -1
    assert L.nvfp4_gemm_prepare(P + 8, P, 256, 128, ctypes.byref(h)) == -4
    assert L.nvfp4_gemm_prepare(P, P, 256, 128, None) == -1
    assert L.nvfp4_gemm_release(None) == 0
    assert L.nvfp4_gemm_launch_prepared(None, P, P, P, P, 16, None, 0, None) == -1
    bogus = (ctypes.c_uint32 * 64)()
    assert L.nvfp4_gemm_launch_prepared(ctypes.addressof(bogus), P, P, P, P, 16, None, 0, None) == -3   # not a handle
    assert L.nvfp4_gemm_set_wait_limit_ns(1) == -5 and L.nvfp4_quant_fused_set_wait_limit_ns(1) == -5
    # grouped launch: count, NULL arrays, NULL entries and things that are not handles are refused before any GPU call
    one = (ctypes.c_void_p * 1)(ctypes.addressof(bogus))
    ptr = (ctypes.c_void_p * 1)(P)
    null = (ctypes.c_void_p * 1)(None)
    assert L.nvfp4_gemm_launch_grouped(None, 0, P, P, None, None, None, 16, None) == 0
    assert L.nvfp4_gemm_launch_grouped(one, -1, P, P, None, ptr, ptr, 16, None) == -5
    assert L.nvfp4_gemm_launch_grouped(one, 65, P, P, None, ptr, ptr, 16, None) == -5
    assert L.nvfp4_gemm_launch_grouped(None, 1, P, P, None, ptr, ptr, 16, None) == -1
    assert L.nvfp4_gemm_launch_grouped(null, 1, P, P, None, ptr, ptr, 16, None) == -1
    assert L.nvfp4_gemm_launch_grouped(one, 1, P, P, None, null, ptr, 16, None) == -1
    assert L.nvfp4_gemm_launch_grouped(one, 1, P, P, None, ptr, ptr, 16, None) == -3
