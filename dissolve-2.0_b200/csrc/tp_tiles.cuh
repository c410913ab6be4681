// tp_tiles.cuh -- row tiles of a mesh, as the tiled kernels see them.
//
// A tile is a group of R nearby rows (vertices).  Its cells are the distinct cells the
// rows touch, ascending.  Every CSR value of a P1 operator is an ordered sum over cells:
// the diagonal (r, r) over the cells of r, an off-diagonal (r, v) over the cells holding
// the edge r-v.  Within a cell the entries are symmetric bit for bit, so (r, v) and (v, r)
// are the same sum: each edge is summed once, by the tile that owns it (the tile of its
// lower endpoint), and written to both positions.  The tables list, per tile row, its
// cells as (position in the tile's cell list, upper-triangle index of the row's local
// vertex), and per owned
// edge its cells as (position, upper-triangle index of the edge in the cell's 4x4 block),
// in ascending cell order; each row's and each edge's terms are contiguous and padded to
// a multiple of 8 with terms of an all-zero slot past the tile's cells, so a thread reads 8
// terms with one 16-byte load and adds them without a branch (a sum that starts at +0 never
// is -0, so adding +0 changes no bit), and a warp's loads of consecutive rows or edges are
// one contiguous range.
#pragma once
#include "tp_common.cuh"

namespace tp {

constexpr int TILE_LOC_BITS = 12;  // cell position in the tile: < 4096
constexpr uint32_t TILE_LOC_MASK = (1u << TILE_LOC_BITS) - 1;

// Where a tile's tables are: one 32-byte load starts every other load of the tile.
struct __align__(32) TileHead {
  int32_t c0, m;    // first cell, number of cells
  int32_t d0, KD;   // diagonal terms: first, per row (a multiple of 8)
  int32_t e0, ne;   // owned edges: first, number
  int32_t t0, KE;   // edge terms: first, per edge (a multiple of 8)
};

struct TileView {
  int R, n_tiles, max_cells, max_edges;
  const TileHead* head;      // (n_tiles)
  const int32_t* rows;       // (n_tiles * R) row ids, -1 where a tile has fewer rows
  const int32_t* diag_pos;   // (n_tiles * R) CSR position of (r, r), -1 for an empty row
  const int32_t* cells;      // distinct cells of each tile, ascending
  const uint16_t* dterms;    // [row][k]: loc | tri_index << 12 (padding: loc = m)
  const int2* edge_pos;      // CSR positions of (r, v) and (v, r), r the lower endpoint
  const int2* edge_rv;       // (r, v)
  const uint16_t* eterms;    // [edge][k]: loc | tri_index << 12 (padding: loc = m)
};

// one 32-byte load
__device__ __forceinline__ TileHead tile_head(const TileView& tv, int t) {
  TileHead h;
  const int4* p = reinterpret_cast<const int4*>(tv.head + t);
  const int4 a = __ldg(p), b = __ldg(p + 1);
  h.c0 = a.x, h.m = a.y, h.d0 = a.z, h.KD = a.w;
  h.e0 = b.x, h.ne = b.y, h.t0 = b.z, h.KE = b.w;
  return h;
}

}  // namespace tp

struct tp_tiles {
  tp::TileView v;
  void* dmem = nullptr;
  size_t bytes = 0;
  int64_t n_terms = 0;
  ~tp_tiles() {
    if (dmem) cudaFree(dmem);
  }
};
