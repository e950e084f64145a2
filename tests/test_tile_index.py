"""CPU: the numbering of output tiles and the copy boxes of operands, compiled for the host, for column counts at which a product of
ints used to overflow and for tiles at and behind the end of a matrix."""
import ctypes
import pathlib
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "nvfp4quant_test_b200" / "csrc"


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("tile_index")
    (d / "shim.cpp").write_text('#include "tile_index.cuh"\nextern "C" void locate(int tile, int m_tiles, int n_tiles, int wish, int* out) '
                                "{ nvfp4::gemm::tile_to_mn(tile, m_tiles, n_tiles, nvfp4::gemm::band_rows(wish, m_tiles), out[0], out[1]); }\n"
                                'extern "C" int box_rows(int rows, int tile, int height) { return nvfp4::gemm::box_rows(rows, tile, height); }\n'
                                'extern "C" int box_map(int box_rows, int height) { return nvfp4::gemm::box_map(box_rows, height); }\n'
                                'extern "C" int has_map(int rows, int height, int map) { return nvfp4::gemm::has_map(rows, height, nvfp4::gemm::BoxMap(map)); }\n')
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-fsanitize=signed-integer-overflow,integer-divide-by-zero",
                    "-fsanitize-undefined-trap-on-error", f"-I{CSRC}", str(d / "shim.cpp"), "-o", str(d / "shim.so")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


@pytest.fixture
def locate(shim):
    def call(tile, m_tiles, n_tiles, wish):
        out = (ctypes.c_int * 2)()
        shim.locate(tile, m_tiles, n_tiles, wish, out)
        return tuple(out)

    return call


@pytest.mark.parametrize("n_tiles", [1, 3, 2047, 2048, 4096, 4097, 262144, 1 << 24])
@pytest.mark.parametrize("wish", [1, 2, 16, 1 << 20])     # the last is the default
@pytest.mark.parametrize("m_tiles", [1, 2, 5, 16, 127])
def test_tiles_are_numbered_in_bands(locate, m_tiles, n_tiles, wish):
    total = m_tiles * n_tiles
    if total > 0x7fff0000:
        pytest.skip("more tiles than a launch takes")
    for tile in {t for t in (0, 1, 2, m_tiles - 1, m_tiles, total // 3, total // 2, total - n_tiles, total - 2, total - 1) if 0 <= t < total}:
        band, rest = divmod(tile, min(wish, m_tiles) * n_tiles)
        rows = min(wish, m_tiles - band * min(wish, m_tiles))
        assert locate(tile, m_tiles, n_tiles, wish) == (band * min(wish, m_tiles) + rest % rows, rest // rows)
    if total <= 5000:
        assert len({locate(t, m_tiles, n_tiles, wish) for t in range(total)}) == total


@pytest.mark.parametrize("height", [64, 96, 128, 256])
@pytest.mark.parametrize("rows", [1, 63, 64, 96, 127, 128, 129, 192, 256, 257, 1000, 1280, 4096])
def test_tiles_take_the_maps_that_are_encoded_and_no_others(shim, rows, height):
    """A matrix of whole boxes has no map of a last one that is not whole, one shorter than a box no other.  A tile behind the last
    one, of which launches of several products in clusters of up to eight have some, copies nothing and takes no map."""
    no_map, whole, rest = range(3)
    tiles = -(-rows // height)
    taken = set()
    for tile in range(tiles + 8):
        n = shim.box_rows(rows, tile, height)
        assert n == max(0, min(height, rows - tile * height))
        took = shim.box_map(n, height)
        assert took == (no_map if tile >= tiles else rest if tile == tiles - 1 and rows % height else whole)
        taken.add(took)
    assert taken - {no_map} == {m for m in (whole, rest) if shim.has_map(rows, height, m)}
