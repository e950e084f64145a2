// Numbering of output tiles: plain index arithmetic, for the kernels and the host.
#pragma once

#ifdef __CUDACC__
#define NVFP4_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define NVFP4_HOST_DEVICE inline
#endif

namespace nvfp4 {
namespace gemm {

// Most tiles of a launch: numbers of tiles, and the next tile of any worker, stay within an int.
constexpr long long kMaxTiles = 0x7fff0000LL;

// m-tiles per band for a wish of `group` (see tile_to_mn).  More than there are would be the same numbering, but group * n_tiles
// must not leave the int range.
NVFP4_HOST_DEVICE int band_rows(int group, int m_tiles) { return group < m_tiles ? group : m_tiles; }

// Tile index -> (m tile, n tile).  Tiles are numbered in bands of `group` m-tiles (1 .. m_tiles): inside a band the m index runs
// fastest, then n.  The CTAs that run at the same time then cover a roughly square patch of the output, so every A
// tile and every B tile is being fetched by a moderate number of CTAs at once instead of one B tile by all of them.
NVFP4_HOST_DEVICE void tile_to_mn(int tile, int m_tiles, int n_tiles, int group, int& mt, int& nt) {
    const int band = tile / (group * n_tiles);
    const int first_m = band * group;
    const int rows = group < m_tiles - first_m ? group : m_tiles - first_m;
    const int in_band = tile - band * group * n_tiles;
    nt = in_band / rows;
    mt = first_m + in_band - nt * rows;
}

// Rows of the copy box of tile `tile` in a matrix of `rows` rows: `height`, fewer in a last tile that is not whole, none behind
// the last tile (a CTA of a launch of several products may lie there).
NVFP4_HOST_DEVICE int box_rows(int rows, int tile, int height) {
    const int left = rows - tile * height;
    return left < 0 ? 0 : left < height ? left : height;
}

// The tensor map that copies a box of so many rows.  A map that no box of the matrix needs is not encoded (see make_operand_maps),
// and nothing may be read from it.
enum BoxMap : int { kNoMap, kWholeMap, kRestMap };
NVFP4_HOST_DEVICE BoxMap box_map(int box_rows, int height) { return box_rows == height ? kWholeMap : box_rows > 0 ? kRestMap : kNoMap; }
// Whether some box of a matrix of `rows` rows needs the map.
NVFP4_HOST_DEVICE bool has_map(long long rows, int height, BoxMap map) { return map == kWholeMap ? rows >= height : rows % height != 0; }

}  // namespace gemm
}  // namespace nvfp4
