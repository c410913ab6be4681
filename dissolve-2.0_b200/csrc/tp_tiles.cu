// tp_tiles.cu -- row tiles for the tiled assembly and operator kernels (built once, on the GPU).
//
// The row-owned kernels (one thread per CSR row, summing the row's cells in ascending
// order) read each cell record once per incident row: four times, each a 64-byte gather
// of its own.  A tile of R nearby rows touches far fewer distinct cells than it visits
// (2.1x fewer for R = 64 on a jittered Kuhn cube), so a tiled kernel loads the tile's
// distinct cells once, coalesced, computes their element entries into shared memory and
// sums the diagonal of each row and each owned edge from there (tp_tiles.cuh).
//
// Rows are grouped by recursive coordinate bisection (split the longest axis of the
// bounding box at a multiple of R, depth first), which keeps tiles compact on
// unstructured and jittered meshes alike; the depth-first order puts neighbouring tiles
// next to each other in the launch, so cell records shared by them stay in L2.
//
// The bisection keeps the vertices sorted along each axis (a radix sort of coordinates
// quantised to 24 bits of the bounding box, ties in vertex order): a segment's extent is
// then its first and last vertex, a split marks one side by position in the split axis'
// order, and a stable partition carries all three orders to the next level.  Segment
// boundaries do not depend on the coordinates, so every level is four launches over all
// segments.  One block per tile then sorts the tile's cell visits, twice (sizes, tables).
// On a 64^3 Kuhn cube the kernels take 1.4 ms (the two table passes 0.8, bound by their
// shared-memory sorts; the rest about 70 short launches) and the call 3.8 ms with its
// allocations and size readback, against 160-190 ms when 16 host threads built the tables.
#include <algorithm>
#include <vector>

#include "tp_tiles.cuh"

using namespace tp;

namespace {

constexpr int RS_T = 256, RS_I = 8, RS_B = RS_T * RS_I;  // threads, items, block of the sorts
constexpr int KEY_BITS = 24;

// ----------------------------------------------------------------- keys
// FP64 as an unsigned integer of the same order
__device__ __forceinline__ unsigned long long ordered(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return (u >> 63) ? ~u : u | 0x8000000000000000ull;
}
__device__ __forceinline__ double from_ordered(unsigned long long u) {
  return __longlong_as_double((long long)((u >> 63) ? u & 0x7fffffffffffffffull : ~u));
}

// bounding box of the finite coordinates: box[a] minima, box[3 + a] maxima (ordered)
__global__ void k_box(int64_t nv, const double* __restrict__ xyz4,
                      unsigned long long* __restrict__ box) {
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nv;
       i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const double x = xyz4[4 * i + a];
      if (isfinite(x)) {
        lo[a] = fmin(lo[a], x);
        hi[a] = fmax(hi[a], x);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[a] = fmin(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmax(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMin(box + a, ordered(lo[a]));
      atomicMax(box + 3 + a, ordered(hi[a]));
    }
  }
}

__global__ void k_keys(int64_t nv, const double* __restrict__ xyz4,
                       const unsigned long long* __restrict__ box, uint32_t* __restrict__ key,
                       int32_t* __restrict__ ord) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nv) return;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double lo = from_ordered(box[a]), ext = from_ordered(box[3 + a]) - lo;
    const double q = ext > 0.0 ? (xyz4[4 * i + a] - lo) / ext * (double)((1 << KEY_BITS) - 1) : 0.0;
    // non-finite coordinates (of vertices no cell uses) go to the ends
    key[a * nv + i] = q > 0.0 ? (uint32_t)fmin(q, (double)((1 << KEY_BITS) - 1)) : 0u;
    ord[a * nv + i] = (int32_t)i;
  }
}

// ----------------------------------------------------------------- radix sort
// One 8-bit pass of a stable LSD sort of the ids by key[axis][id] (blockIdx.y = axis).
__global__ void __launch_bounds__(RS_T) k_sort_hist(int64_t nv, int nb, int shift,
                                                    const uint32_t* __restrict__ key,
                                                    const int32_t* __restrict__ ord,
                                                    int32_t* __restrict__ hist) {
  __shared__ int32_t h[256];
  key += blockIdx.y * nv;
  ord += blockIdx.y * nv;
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * RS_B;
#pragma unroll
  for (int k = 0; k < RS_I; k++) {
    const int64_t i = base + k * RS_T + threadIdx.x;
    if (i < nv) atomicAdd(&h[(key[ord[i]] >> shift) & 255u], 1);
  }
  __syncthreads();
  hist[((int64_t)blockIdx.y * 256 + threadIdx.x) * nb + blockIdx.x] = h[threadIdx.x];
}

// exclusive scan of the (digit, block) counts of one axis in place (one block per axis)
__global__ void __launch_bounds__(1024) k_sort_scan(int64_t n, int32_t* __restrict__ hist) {
  __shared__ int32_t s[32];
  hist += blockIdx.x * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t per = (n + 1023) / 1024;
  const int64_t b = threadIdx.x * per, e = min(b + per, n);
  int32_t sum = 0;
  for (int64_t i = b; i < e; i++) sum += hist[i];
  int32_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int32_t v = s[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    s[lane] = v;
  }
  __syncthreads();
  int32_t run = inc - sum + (warp ? s[warp - 1] : 0);
  for (int64_t i = b; i < e; i++) {
    const int32_t v = hist[i];
    hist[i] = run;
    run += v;
  }
}

__global__ void __launch_bounds__(RS_T) k_sort_scatter(int64_t nv, int nb, int shift,
                                                       const uint32_t* __restrict__ key,
                                                       const int32_t* __restrict__ ord,
                                                       const int32_t* __restrict__ hist,
                                                       int32_t* __restrict__ out) {
  constexpr int W = RS_T / 32;
  __shared__ int32_t cnt[W][256];
  key += blockIdx.y * nv;
  ord += blockIdx.y * nv;
  out += blockIdx.y * nv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < W * 256; i += RS_T) (&cnt[0][0])[i] = 0;
  __syncthreads();
  // warp w owns items [w * 32 RS_I, (w + 1) * 32 RS_I) of the block, 32 consecutive a round
  const int64_t base = (int64_t)blockIdx.x * RS_B + warp * 32 * RS_I;
  int32_t id[RS_I];
  uint32_t dg[RS_I], mask[RS_I];
#pragma unroll
  for (int k = 0; k < RS_I; k++) {
    const int64_t i = base + k * 32 + lane;
    id[k] = i < nv ? ord[i] : -1;
    dg[k] = id[k] >= 0 ? (key[id[k]] >> shift) & 255u : 256u;  // 256: past the end
    mask[k] = __match_any_sync(0xffffffffu, dg[k]);
    if (id[k] >= 0 && lane == __ffs(mask[k]) - 1) cnt[warp][dg[k]] += __popc(mask[k]);
    __syncwarp();
  }
  __syncthreads();
  {
    int32_t run = hist[((int64_t)blockIdx.y * 256 + threadIdx.x) * nb + blockIdx.x];
#pragma unroll
    for (int w = 0; w < W; w++) {
      const int32_t v = cnt[w][threadIdx.x];
      cnt[w][threadIdx.x] = run;
      run += v;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < RS_I; k++) {
    if (id[k] >= 0) out[cnt[warp][dg[k]] + __popc(mask[k] & ((1u << lane) - 1u))] = id[k];
    __syncwarp();
    if (id[k] >= 0 && lane == __ffs(mask[k]) - 1) cnt[warp][dg[k]] += __popc(mask[k]);
    __syncwarp();
  }
}

// ----------------------------------------------------------------- bisection
// The segment of a level that holds position i (lo ascending, disjoint), or -1.
struct Seg {
  int32_t lo, left, hi, pad;  // split into [lo, lo + left) and [lo + left, hi)
};
__device__ __forceinline__ int find_seg(const Seg* __restrict__ seg, int ns, int64_t i) {
  int a = 0, b = ns;
  while (b - a > 1) {
    const int m = (a + b) >> 1;
    if (seg[m].lo <= i)
      a = m;
    else
      b = m;
  }
  return (ns > 0 && i >= seg[a].lo && i < seg[a].hi) ? a : -1;
}

// side[v] of every vertex in a segment of this level: by its position along the segment's
// longest axis
__global__ void k_rcb_mark(int64_t nv, int ns, const Seg* __restrict__ seg,
                           const unsigned long long* __restrict__ box,
                           const uint32_t* __restrict__ key, const int32_t* __restrict__ ord,
                           uint8_t* __restrict__ side) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const int s = find_seg(seg, ns, i);
  if (s < 0) return;
  const Seg g = seg[s];
  int ax = 0;
  double best = -1.0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int32_t* o = ord + a * nv;
    const double scale = from_ordered(box[3 + a]) - from_ordered(box[a]);
    const double ext = (double)(key[a * nv + o[g.hi - 1]] - key[a * nv + o[g.lo]]) * scale;
    if (ext > best) {
      best = ext;
      ax = a;
    }
  }
  side[ord[ax * nv + i]] = i - g.lo >= g.left;
}

// vertices of side 0 per block of RS_B positions (blockIdx.y = axis)
__global__ void __launch_bounds__(RS_T) k_rcb_count(int64_t nv, const int32_t* __restrict__ ord,
                                                    const uint8_t* __restrict__ side,
                                                    int32_t* __restrict__ cnt) {
  __shared__ int32_t s[RS_T / 32];
  ord += blockIdx.y * nv;
  int32_t c = 0;
#pragma unroll
  for (int k = 0; k < RS_I; k++) {
    const int64_t i = (int64_t)blockIdx.x * RS_B + k * RS_T + threadIdx.x;
    if (i < nv) c += side[ord[i]] == 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < RS_T / 32; w++) c += s[w];
    cnt[blockIdx.y * gridDim.x + blockIdx.x] = c;
  }
}

// zero[axis][i] = vertices of side 0 before position i
__global__ void __launch_bounds__(RS_T) k_rcb_prefix(int64_t nv, const int32_t* __restrict__ ord,
                                                     const uint8_t* __restrict__ side,
                                                     const int32_t* __restrict__ cnt,
                                                     int32_t* __restrict__ zero) {
  constexpr int W = RS_T / 32;
  __shared__ int32_t s[W + 1];
  ord += blockIdx.y * nv;
  zero += blockIdx.y * nv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t before = 0;  // side-0 vertices of the earlier blocks
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += RS_T) before += cnt[blockIdx.y * gridDim.x + b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (lane == 0) s[warp] = before;
  __syncthreads();
  before = 0;
  for (int w = 0; w < W; w++) before += s[w];
  __syncthreads();
  // warp w: 32 RS_I consecutive positions, 32 a round
  const int64_t base = (int64_t)blockIdx.x * RS_B + warp * 32 * RS_I;
  uint32_t m[RS_I];
  int32_t tot = 0;
#pragma unroll
  for (int k = 0; k < RS_I; k++) {
    const int64_t i = base + k * 32 + lane;
    m[k] = __ballot_sync(0xffffffffu, i < nv && side[ord[i < nv ? i : 0]] == 0);
    tot += __popc(m[k]);
  }
  if (lane == 0) s[warp] = tot;
  __syncthreads();
  int32_t run = before;
  for (int w = 0; w < warp; w++) run += s[w];
#pragma unroll
  for (int k = 0; k < RS_I; k++) {
    const int64_t i = base + k * 32 + lane;
    if (i < nv) zero[i] = run + __popc(m[k] & ((1u << lane) - 1u));
    run += __popc(m[k]);
  }
}

__global__ void k_rcb_scatter(int64_t nv, int ns, const Seg* __restrict__ seg,
                              const int32_t* __restrict__ ord, const uint8_t* __restrict__ side,
                              const int32_t* __restrict__ zero, int32_t* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nv) return;
  ord += blockIdx.y * nv;
  zero += blockIdx.y * nv;
  out += blockIdx.y * nv;
  const int32_t v = ord[i];
  const int s = find_seg(seg, ns, i);
  int64_t to = i;
  if (s >= 0) {
    const Seg g = seg[s];
    const int32_t z = zero[i] - zero[g.lo];
    to = side[v] ? g.lo + g.left + (i - g.lo - z) : g.lo + z;
  }
  out[to] = v;
}

// ----------------------------------------------------------------- tables
// What a tile builder found wrong first (code 0: nothing), for the host's message.
struct TileError {
  int code, a, b;
};
enum { TE_CELLS = 1, TE_ROWLEN, TE_SLOT, TE_SYMMETRY };

__device__ __forceinline__ void tile_fail(TileError* err, int code, int a, int b) {
  if (atomicCAS(&err->code, 0, code) == 0) {
    err->a = a;
    err->b = b;
  }
}

__device__ __forceinline__ int lower_bound(const int32_t* __restrict__ v, int lo, int hi,
                                           int32_t x) {
  while (lo < hi) {
    const int m = (lo + hi) >> 1;
    if (v[m] < x)
      lo = m + 1;
    else
      hi = m;
  }
  return lo;
}

// ascending bitonic sort of n (a power of two) values in shared memory by the block
__device__ __forceinline__ void block_sort(int32_t* v, int n) {
  for (int k = 2; k <= n; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (int t = threadIdx.x; t < n / 2; t += blockDim.x) {
        const int i = 2 * t - (t & (j - 1));  // the lower index of pair t
        const int32_t x = v[i], y = v[i + j];
        if ((x > y) == ((i & k) == 0)) {
          v[i] = y;
          v[i + j] = x;
        }
      }
    }
  __syncthreads();
}

// cell visits (sum of degrees) and CSR entries per tile, their maxima over tiles
__global__ void k_tile_visits(int nt, const int32_t* __restrict__ start,
                              const int32_t* __restrict__ idx, const int32_t* __restrict__ vptr,
                              const int32_t* __restrict__ indptr, int32_t* __restrict__ most) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= nt) return;
  int32_t n = 0, e = 0;
  for (int i = start[t] + lane; i < start[t + 1]; i += 32) {
    const int32_t r = idx[i];
    n += vptr[r + 1] - vptr[r];
    e += indptr[r + 1] - indptr[r];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    n += __shfl_xor_sync(0xffffffffu, n, o);
    e += __shfl_xor_sync(0xffffffffu, e, o);
  }
  if (lane == 0) {
    atomicMax(most, n);
    atomicMax(most + 1, e);
  }
}

struct TileBuild {
  int R, cap, edge_cap;    // rows per tile; visits (a power of two) and edges a block holds
  const int32_t *start, *idx;
  const int32_t *vptr, *v2c, *indptr, *indices;
  const uint32_t* slots;
  uint16_t* cnt;           // edge_cap counters per tile, or NULL: in shared memory
  int4* sizes;             // cells, diagonal terms, edges, edge terms of each tile
  TileError* err;
  // FILL: the tables
  int32_t *rows, *diag_pos, *cells;
  uint16_t *dterms, *eterms;
  int2 *edge_pos, *edge_rv;
  const TileHead* head;
};

constexpr int TB_T = 256;
constexpr int TB_MAXR = 256;

// One block per tile.  FILL = false: the table sizes; FILL = true: the tables.
template <bool FILL>
__global__ void __launch_bounds__(TB_T) k_tile_build(TileBuild b) {
  extern __shared__ int32_t s_sort[];  // cap visits, then up to 4096 distinct cells ...
  int32_t* s_tc = s_sort + b.cap;
  // ... then (FILL) the local index of every visit and the terms of every owned edge so far
  uint16_t* s_loc = reinterpret_cast<uint16_t*>(s_tc + (1 << TILE_LOC_BITS));
  uint16_t* s_cnt = b.cnt ? b.cnt + (int64_t)blockIdx.x * b.edge_cap : s_loc + b.cap;
  __shared__ int32_t s_row[TB_MAXR], s_vis[TB_MAXR + 1], s_edge[TB_MAXR + 1], s_dl[TB_MAXR];
  __shared__ int32_t s_scan[TB_T], s_kmax, s_kemax, s_bad;
  const int t = blockIdx.x, tid = threadIdx.x;
  const int r0 = b.start[t], nr = b.start[t + 1] - r0;
  if (tid == 0) s_kmax = s_kemax = s_bad = 0;
  // rows of the tile ascending (writes then walk the CSR forward)
  int p2 = 32;
  while (p2 < nr) p2 <<= 1;
  for (int i = tid; i < p2; i += TB_T) s_row[i] = i < nr ? b.idx[r0 + i] : INT32_MAX;
  block_sort(s_row, p2);
  // per row: degree, diagonal position, owned edges (its CSR entries past the diagonal)
  if (tid < TB_MAXR) {
    int deg = 0, ne = 0;
    if (tid < nr) {
      const int32_t r = s_row[tid];
      deg = b.vptr[r + 1] - b.vptr[r];
      const int p0 = b.indptr[r], p1 = b.indptr[r + 1];
      if (p1 - p0 > 256) {
        tile_fail(b.err, TE_ROWLEN, r, p1 - p0);
        s_bad = 1;
      }
      const int at = lower_bound(b.indices, p0, p1, r);
      const bool has = at < p1 && b.indices[at] == r;
      s_dl[tid] = at - p0 - (has ? 0 : 1);  // entries past this one are owned edges
      ne = p1 - at - (has ? 1 : 0);
      atomicMax(&s_kmax, deg);
      if constexpr (FILL) {
        b.rows[(int64_t)t * b.R + tid] = r;
        b.diag_pos[(int64_t)t * b.R + tid] = has ? at : -1;
      }
    } else if (FILL && tid < b.R) {
      b.rows[(int64_t)t * b.R + tid] = -1;
      b.diag_pos[(int64_t)t * b.R + tid] = -1;
    }
    // prefix sums over the rows
    s_vis[tid + 1] = deg;
    s_edge[tid + 1] = ne;
  }
  __syncthreads();
  if (tid == 0) {
    s_vis[0] = s_edge[0] = 0;
    for (int i = 1; i <= nr; i++) {
      s_vis[i] += s_vis[i - 1];
      s_edge[i] += s_edge[i - 1];
    }
  }
  __syncthreads();
  const int nvis = s_vis[nr], nedge = s_edge[nr];
  if (nvis > b.cap || nedge > b.edge_cap || s_bad) {
    if (tid == 0) {
      if (!s_bad) tile_fail(b.err, TE_CELLS, t, nvis / 4);
      if (!FILL) b.sizes[t] = make_int4(0, 0, 0, 0);
    }
    return;
  }
  // the tile's visits, sorted, and their distinct cells
  int n2 = 32;
  while (n2 < nvis) n2 <<= 1;
  auto row_of = [&](int k) {  // the tile row of visit k
    int lo = 0, hi = nr;
    while (hi - lo > 1) {
      const int m = (lo + hi) >> 1;
      if (s_vis[m] <= k)
        lo = m;
      else
        hi = m;
    }
    return lo;
  };
  for (int k = tid; k < n2; k += TB_T) {
    int32_t c = INT32_MAX;
    if (k < nvis) {
      const int i = row_of(k);
      c = b.v2c[b.vptr[s_row[i]] + (k - s_vis[i])] >> 2;
    }
    s_sort[k] = c;
  }
  block_sort(s_sort, n2);
  const int per = (n2 + TB_T - 1) / TB_T;
  int nu = 0;
  for (int k = tid * per; k < min((tid + 1) * per, nvis); k++)
    nu += k == 0 || s_sort[k] != s_sort[k - 1];
  s_scan[tid] = nu;
  __syncthreads();
  for (int o = 1; o < TB_T; o <<= 1) {
    const int v = tid >= o ? s_scan[tid - o] : 0;
    __syncthreads();
    s_scan[tid] += v;
    __syncthreads();
  }
  const int m = s_scan[TB_T - 1];
  if (m >= (1 << TILE_LOC_BITS)) {
    if (tid == 0) {
      tile_fail(b.err, TE_CELLS, t, m);
      if (!FILL) b.sizes[t] = make_int4(0, 0, 0, 0);
    }
    return;
  }
  int at = s_scan[tid] - nu;
  for (int k = tid * per; k < min((tid + 1) * per, nvis); k++)
    if (k == 0 || s_sort[k] != s_sort[k - 1]) s_tc[at++] = s_sort[k];
  for (int e = tid; e < nedge; e += TB_T) s_cnt[e] = 0;
  __syncthreads();
  const int KD = (s_kmax + 7) & ~7;
  if constexpr (FILL) {
    const TileHead h = b.head[t];
    for (int i = tid; i < m; i += TB_T) b.cells[h.c0 + i] = s_tc[i];
    // local index of every visit and the diagonal terms [row][k]
    uint16_t* dt = b.dterms + h.d0;
    for (int k = tid; k < KD * b.R; k += TB_T) dt[k] = (uint16_t)m;
    for (int k = tid; k < h.KE * nedge; k += TB_T) b.eterms[h.t0 + k] = (uint16_t)m;
    __syncthreads();
    for (int k = tid; k < nvis; k += TB_T) {
      const int i = row_of(k);
      const int32_t e = b.v2c[b.vptr[s_row[i]] + (k - s_vis[i])];
      const int loc = lower_bound(s_tc, 0, m, e >> 2);
      s_loc[k] = (uint16_t)loc;
      const int li = e & 3;
      const int tri = li * (9 - li) / 2;  // 0, 4, 7, 9
      dt[(int64_t)i * KD + (k - s_vis[i])] = (uint16_t)(loc | (tri << TILE_LOC_BITS));
    }
    __syncthreads();
  }
  // edge terms: each row's thread walks its cells in ascending order
  const int t0 = FILL ? b.head[t].t0 : 0, KE = FILL ? b.head[t].KE : 0;
  if (tid < nr) {
    const int32_t r = s_row[tid];
    const int v0 = b.vptr[r], deg = b.vptr[r + 1] - v0, len = b.indptr[r + 1] - b.indptr[r];
    const int dl = s_dl[tid], e0 = s_edge[tid];
    int most = 0;
    for (int k = 0; k < deg; k++) {
      const int li = b.v2c[v0 + k] & 3;
      const uint32_t sv = b.slots[v0 + k];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (j == li) continue;
        const int sl = (sv >> (8 * j)) & 0xff;
        if (sl >= len) {
          tile_fail(b.err, TE_SLOT, sl, r);
          s_bad = 1;
          continue;
        }
        if (sl <= dl) continue;  // owned by the other endpoint's tile
        const int e = e0 + sl - dl - 1;
        const int q = s_cnt[e];
        s_cnt[e] = (uint16_t)(q + 1);
        most = max(most, q + 1);
        if constexpr (FILL) {
          const int a = li < j ? li : j, c = li < j ? j : li;
          const int tri = (a == 0 ? 0 : (a == 1 ? 4 : 7)) + (c - a);
          b.eterms[t0 + (int64_t)e * KE + q] =
              (uint16_t)(s_loc[s_vis[tid] + k] | (tri << TILE_LOC_BITS));
        }
      }
    }
    if (!FILL) atomicMax(&s_kemax, most);
  }
  __syncthreads();
  if constexpr (!FILL) {
    if (tid == 0)
      b.sizes[t] = s_bad ? make_int4(0, 0, 0, 0)
                         : make_int4(m, KD, nedge, nedge ? (s_kemax + 7) & ~7 : 0);
  } else {
    const int eb = b.head[t].e0;
    for (int e = tid; e < nedge; e += TB_T) {
      int lo = 0, hi = nr;  // the row that owns edge e
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s_edge[mid] <= e)
          lo = mid;
        else
          hi = mid;
      }
      const int32_t r = s_row[lo];
      const int p = b.indptr[r] + s_dl[lo] + 1 + (e - s_edge[lo]);
      const int32_t v = b.indices[p];
      const int h1 = b.indptr[v + 1];
      int q = lower_bound(b.indices, b.indptr[v], h1, r);
      const bool pair = q < h1 && b.indices[q] == r;
      // an entry that no cell touches needs no partner: its zero is written twice, to row r
      if (!pair && s_cnt[e]) tile_fail(b.err, TE_SYMMETRY, r, v);
      b.edge_pos[eb + e] = make_int2(p, pair ? q : p);
      b.edge_rv[eb + e] = make_int2(r, pair ? v : r);
    }
  }
}

struct DeviceBuffer {
  char* p = nullptr;
  ~DeviceBuffer() {
    if (p) cudaFree(p);
  }
};

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

extern "C" int tp_tiles_create(const tp_mesh* m, int rows_per_tile, void* stream,
                               tp_tiles** out) {
  TP_REQUIRE(m && out && m->coords4 && m->v2c_ptr && m->v2c && m->v2c_slots && m->indptr &&
                 m->indices,
             "tiles need coords4, incidence, slots and the CSR pattern");
  TP_REQUIRE(rows_per_tile >= 32 && rows_per_tile <= TB_MAXR && rows_per_tile % 32 == 0,
             "rows_per_tile must be a multiple of 32 in [32, 256]");
  TP_REQUIRE(m->n_verts >= 0 && m->n_verts < INT32_MAX, "bad vertex count");
  *out = nullptr;
  const int R = rows_per_tile;
  const int64_t nv = m->n_verts;
  cudaStream_t st = as_stream(stream);

  // segments of every level (they do not depend on the coordinates) and the tile starts
  std::vector<std::vector<Seg>> levels;
  std::vector<int32_t> start;
  {
    std::vector<std::pair<int64_t, int64_t>> cur, next;
    if (nv > 0) cur.push_back({0, nv});
    while (!cur.empty()) {
      std::vector<Seg> lv;
      next.clear();
      for (const auto& c : cur) {
        const int64_t n = c.second - c.first;
        if (n <= R) {
          start.push_back((int32_t)c.first);
          continue;
        }
        const int64_t left = ((n + R - 1) / R / 2) * R;
        lv.push_back({(int32_t)c.first, (int32_t)left, (int32_t)c.second, 0});
        next.push_back({c.first, c.first + left});
        next.push_back({c.first + left, c.second});
      }
      if (!lv.empty()) levels.push_back(std::move(lv));
      cur.swap(next);
    }
    std::sort(start.begin(), start.end());
  }
  const int nt = (int)start.size();
  start.push_back((int32_t)nv);
  std::vector<Seg> segs;
  for (const auto& lv : levels) segs.insert(segs.end(), lv.begin(), lv.end());

  const int nb = (int)((nv + RS_B - 1) / RS_B);
  const size_t nv1 = (size_t)std::max<int64_t>(nv, 1), nb1 = (size_t)std::max(nb, 1);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off += a256(std::max<size_t>(bytes, 1));
    return at;
  };
  const size_t o_box = take(6 * 8), o_err = take(sizeof(TileError)), o_most = take(8),
               o_key = take(3 * nv1 * 4), o_ord0 = take(3 * nv1 * 4), o_ord1 = take(3 * nv1 * 4),
               o_hist = take(3 * 256 * nb1 * 4), o_side = take(nv1), o_zero = take(3 * nv1 * 4),
               o_cnt = take(3 * nb1 * 4), o_seg = take(sizeof(Seg) * segs.size()),
               o_start = take(4 * start.size()), o_size = take(sizeof(int4) * (size_t)nt);
  DeviceBuffer tmp;
  TP_CUDA_TRY(cudaMalloc(&tmp.p, off));
  auto* box = reinterpret_cast<unsigned long long*>(tmp.p + o_box);
  auto* err = reinterpret_cast<TileError*>(tmp.p + o_err);
  auto* most = reinterpret_cast<int32_t*>(tmp.p + o_most);
  auto* key = reinterpret_cast<uint32_t*>(tmp.p + o_key);
  int32_t* ord = reinterpret_cast<int32_t*>(tmp.p + o_ord0);
  int32_t* alt = reinterpret_cast<int32_t*>(tmp.p + o_ord1);
  auto* hist = reinterpret_cast<int32_t*>(tmp.p + o_hist);
  auto* side = reinterpret_cast<uint8_t*>(tmp.p + o_side);
  auto* zero = reinterpret_cast<int32_t*>(tmp.p + o_zero);
  auto* cnt = reinterpret_cast<int32_t*>(tmp.p + o_cnt);
  auto* seg = reinterpret_cast<Seg*>(tmp.p + o_seg);
  auto* d_start = reinterpret_cast<int32_t*>(tmp.p + o_start);
  auto* sizes = reinterpret_cast<int4*>(tmp.p + o_size);
  // minima start at the largest ordered value, maxima at the smallest
  TP_CUDA_TRY(cudaMemsetAsync(box, 0xff, 3 * 8, st));
  TP_CUDA_TRY(cudaMemsetAsync(box + 3, 0, 3 * 8, st));
  TP_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(TileError), st));
  TP_CUDA_TRY(cudaMemsetAsync(most, 0, 8, st));
  if (!segs.empty())
    TP_CUDA_TRY(cudaMemcpyAsync(seg, segs.data(), sizeof(Seg) * segs.size(),
                                cudaMemcpyHostToDevice, st));
  TP_CUDA_TRY(cudaMemcpyAsync(d_start, start.data(), 4 * start.size(), cudaMemcpyHostToDevice, st));
  if (nv > 0) {
    const int g = grid_for(nv, RS_T);
    const dim3 gb(nb, 3), gs(g, 3);
    k_box<<<grid_for(nv, RS_T, 4 * sm_count()), RS_T, 0, st>>>(nv, m->coords4, box);
    k_keys<<<g, RS_T, 0, st>>>(nv, m->coords4, box, key, ord);
    TP_LAUNCH_CHECK();
    for (int shift = 0; shift < KEY_BITS; shift += 8) {
      k_sort_hist<<<gb, RS_T, 0, st>>>(nv, nb, shift, key, ord, hist);
      k_sort_scan<<<3, 1024, 0, st>>>((int64_t)256 * nb, hist);
      k_sort_scatter<<<gb, RS_T, 0, st>>>(nv, nb, shift, key, ord, hist, alt);
      std::swap(ord, alt);
    }
    TP_LAUNCH_CHECK();
    const Seg* sl = seg;
    for (const auto& lv : levels) {
      const int ns = (int)lv.size();
      k_rcb_mark<<<g, RS_T, 0, st>>>(nv, ns, sl, box, key, ord, side);
      k_rcb_count<<<gb, RS_T, 0, st>>>(nv, ord, side, cnt);
      k_rcb_prefix<<<gb, RS_T, 0, st>>>(nv, ord, side, cnt, zero);
      k_rcb_scatter<<<gs, RS_T, 0, st>>>(nv, ns, sl, ord, side, zero, alt);
      std::swap(ord, alt);
      sl += ns;
    }
    TP_LAUNCH_CHECK();
    k_tile_visits<<<grid_for(nt, 8), 256, 0, st>>>(nt, d_start, ord, m->v2c_ptr, m->indptr,
                                                     most);
    TP_LAUNCH_CHECK();
  }
  int32_t h_most[2] = {0, 0};
  TP_CUDA_TRY(cudaMemcpyAsync(h_most, most, 8, cudaMemcpyDeviceToHost, st));
  TP_CUDA_TRY(cudaStreamSynchronize(st));
  // fewer than 4096 distinct cells are visited fewer than 16384 times
  TileBuild b = {};
  b.R = R;
  b.cap = 32;
  while (b.cap < h_most[0] && b.cap < (4 << TILE_LOC_BITS)) b.cap <<= 1;
  b.start = d_start;
  b.idx = ord;
  b.vptr = m->v2c_ptr;
  b.v2c = m->v2c;
  b.indptr = m->indptr;
  b.indices = m->indices;
  b.slots = m->v2c_slots;
  b.sizes = sizes;
  b.err = err;
  b.edge_cap = h_most[1];
  // the edges' counters: in shared memory up to six edges per cell and some spare (all that
  // the pattern of a mesh asks for), else (a pattern with more entries) in device memory
  const bool wide = b.edge_cap > (7 << TILE_LOC_BITS);
  const size_t smem = sizeof(int32_t) * ((size_t)b.cap + (1 << TILE_LOC_BITS)) +
                      sizeof(uint16_t) * ((size_t)b.cap + (wide ? 0 : (size_t)b.edge_cap));
  DeviceBuffer counters;
  if (wide) {
    TP_CUDA_TRY(cudaMalloc(&counters.p, sizeof(uint16_t) * (size_t)b.edge_cap * (size_t)nt));
    b.cnt = reinterpret_cast<uint16_t*>(counters.p);
  }
  std::vector<int4> h_sizes(nt);
  auto check = [&]() -> int {
    TileError e;
    TP_CUDA_TRY(cudaMemcpyAsync(&e, err, sizeof(e), cudaMemcpyDeviceToHost, st));
    if (nt)
      TP_CUDA_TRY(cudaMemcpyAsync(h_sizes.data(), sizes, sizeof(int4) * nt,
                                  cudaMemcpyDeviceToHost, st));
    TP_CUDA_TRY(cudaStreamSynchronize(st));
    switch (e.code) {
      case 0:
        return TP_OK;
      case TE_CELLS:
        set_error("tile %d touches %d cells or more (at most %d)", e.a, e.b,
                  (1 << TILE_LOC_BITS) - 1);
        return TP_ERR_CAPACITY;
      case TE_ROWLEN:
        set_error("row %d has %d entries (tiles support 256)", e.a, e.b);
        return TP_ERR_CAPACITY;
      case TE_SLOT:
        set_error("incidence slot %d outside row %d", e.a, e.b);
        return TP_ERR_INDEX;
      default:
        set_error("pattern is not symmetric at (%d, %d)", e.a, e.b);
        return TP_ERR_INDEX;
    }
  };
  if (nt) {
    if (smem > 40 * 1024) {  // with the static arrays, past the 48 KB default
      TP_CUDA_TRY(cudaFuncSetAttribute(k_tile_build<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      TP_CUDA_TRY(cudaFuncSetAttribute(k_tile_build<true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    }
    k_tile_build<false><<<nt, TB_T, smem, st>>>(b);
    TP_LAUNCH_CHECK();
  }
  int rc = check();
  if (rc) return rc;
  std::vector<TileHead> head(nt);
  int64_t tc = 0, td = 0, te = 0, tt = 0;
  int max_cells = 0, max_edges = 0;
  for (int t = 0; t < nt; t++) {
    const int4 z = h_sizes[t];
    head[t] = {(int32_t)tc, z.x, (int32_t)td, z.y, (int32_t)te, z.z, (int32_t)tt, z.w};
    tc += z.x;
    td += (int64_t)z.y * R;
    te += z.z;
    tt += (int64_t)z.w * z.z;
    if (tc > INT32_MAX || td > INT32_MAX || te > INT32_MAX || tt > INT32_MAX) {
      set_error("tile terms exceed int32 offsets");
      return TP_ERR_CAPACITY;
    }
    max_cells = std::max(max_cells, z.x);
    max_edges = std::max(max_edges, z.z);
  }

  tp_tiles* h = new tp_tiles();
  struct Guard {
    tp_tiles* h;
    ~Guard() { delete h; }
  } guard{h};
  off = 0;
  const size_t o_head = take(sizeof(TileHead) * (size_t)nt), o_rows = take(4 * (size_t)nt * R),
               o_dpos = take(4 * (size_t)nt * R), o_cells = take(4 * (size_t)tc),
               o_dterms = take(2 * (size_t)td), o_epos = take(8 * (size_t)te),
               o_erv = take(8 * (size_t)te), o_eterms = take(2 * (size_t)tt);
  h->bytes = off;
  cudaError_t ce = cudaMalloc(&h->dmem, h->bytes);
  if (ce != cudaSuccess) {
    h->dmem = nullptr;
    set_error("tiles: cudaMalloc of %zu bytes failed: %s", h->bytes, cudaGetErrorString(ce));
    return TP_ERR_CUDA;
  }
  char* p = static_cast<char*>(h->dmem);
  TileView& v = h->v;
  v.R = R;
  v.n_tiles = nt;
  v.max_cells = max_cells;
  v.max_edges = max_edges;
  b.rows = reinterpret_cast<int32_t*>(p + o_rows);
  b.diag_pos = reinterpret_cast<int32_t*>(p + o_dpos);
  b.cells = reinterpret_cast<int32_t*>(p + o_cells);
  b.dterms = reinterpret_cast<uint16_t*>(p + o_dterms);
  b.edge_pos = reinterpret_cast<int2*>(p + o_epos);
  b.edge_rv = reinterpret_cast<int2*>(p + o_erv);
  b.eterms = reinterpret_cast<uint16_t*>(p + o_eterms);
  v.rows = b.rows;
  v.diag_pos = b.diag_pos;
  v.cells = b.cells;
  v.dterms = b.dterms;
  v.edge_pos = b.edge_pos;
  v.edge_rv = b.edge_rv;
  v.eterms = b.eterms;
  v.head = b.head = reinterpret_cast<TileHead*>(p + o_head);
  if (nt)
    TP_CUDA_TRY(cudaMemcpyAsync(p + o_head, head.data(), sizeof(TileHead) * (size_t)nt,
                                cudaMemcpyHostToDevice, st));
  if (nt) {
    k_tile_build<true><<<nt, TB_T, smem, st>>>(b);
    TP_LAUNCH_CHECK();
  }
  rc = check();
  if (rc) return rc;
  h->n_terms = td + tt;
  guard.h = nullptr;
  *out = h;
  return TP_OK;
}

extern "C" int tp_tiles_info(const tp_tiles* t, int32_t* n_tiles, int32_t* rows_per_tile,
                             int32_t* max_cells, int64_t* n_entries, size_t* device_bytes) {
  TP_REQUIRE(t, "null tiles");
  if (n_tiles) *n_tiles = t->v.n_tiles;
  if (rows_per_tile) *rows_per_tile = t->v.R;
  if (max_cells) *max_cells = t->v.max_cells;
  if (n_entries) *n_entries = t->n_terms;
  if (device_bytes) *device_bytes = t->bytes;
  return TP_OK;
}

extern "C" int tp_tiles_destroy(tp_tiles* t) {
  delete t;
  return TP_OK;
}
