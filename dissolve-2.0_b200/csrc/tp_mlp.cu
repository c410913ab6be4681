// tp_mlp.cu -- per-vertex MLP that predicts the next backward-Euler state (the Krylov
// initial guess), BF16 on the tensor cores with FP32 accumulation.
//
// Network: 16 inputs (10 used) -> 64 -> ReLU -> 64 -> ReLU -> 1, one network shared by
// all species; a row is one (vertex, species) pair.  Features (normalised by per-input
// affine maps fixed at training time):
//   0 phi, 1 |grad phi|, 2 u^n, 3 u^{n-1}, 4 u^n - u^{n-1}, 5 log D_s, 6 k_s, 7 1,
//   8 (D_s K u^n)_v, 9 (D_s K (u^n - u^{n-1}))_v -- the stiffness images give the
//   network the local curvature that decides how fast each part of the change decays
// The output y predicts (u^{n+1} - B) / sigma and the guess is B + sigma y, with the base
// B = u^n or the linear extrapolation 2 u^n - u^{n-1} (the network learns the correction
// to the extrapolation: with zero output the guess is the extrapolation itself).
//
// Inference (k_mlp_predict) runs layers 1 and 2 as tcgen05.mma on 256-row tiles with the
// accumulators in tensor memory.  Training uses mma.sync.m16n8k16 fragments (row.col,
// bf16 x bf16 -> f32): a warp owns 16 rows; layer outputs stay in registers and are
// re-packed from the accumulator layout into the next layer's A layout.  Backward: the
// weight gradients
// are GEMMs over the row dimension (dW2 = dZ2^T H1, dW1 = dZ1^T X) fed from transposed
// tiles staged in shared memory; every CTA writes its partial gradient, and the AdamW
// kernel sums the partials in CTA order (training is deterministic for a given grid).
#include <cuda_bf16.h>

#include <algorithm>

#include <atomic>

#include "tp_common.cuh"

namespace tp {

constexpr int MLP_IN = 16, MLP_H = 64;
// shared-memory row strides (bf16 elements) of the weight and staging tiles: 24 and 72
// put the 8 rows a B-fragment load touches into 8 different bank groups (16 and 64
// would hit the same banks 2 and 8 times)
constexpr int W1S = 24, W2S = 72, GS = 72;
// FP32 master parameter vector layout
constexpr int OFF_W1 = 0;                      // [64][16]
constexpr int OFF_B1 = OFF_W1 + MLP_H * MLP_IN;  // [64]
constexpr int OFF_W2 = OFF_B1 + MLP_H;           // [64][64]
constexpr int OFF_B2 = OFF_W2 + MLP_H * MLP_H;   // [64]
constexpr int OFF_W3 = OFF_B2 + MLP_H;           // [64]
constexpr int OFF_B3 = OFF_W3 + MLP_H;           // [1]
constexpr int MLP_P = OFF_B3 + 1;

constexpr int NFEAT = 10;  // used inputs: 0..6 fields, 7 bias, 8..9 operator images

struct MlpFeat {
  const double* U;      // (V, ld) u^n
  const double* Up;     // (V, ld) u^{n-1}
  const double* phi;    // (V) or NULL
  const double* ngphi;  // (V) or NULL
  const double* opU;    // (V, ld) D_s K u^n or NULL
  const double* opDU;   // (V, ld) D_s K (u^n - u^{n-1}) or NULL
  int S, ld;
  int base;  // the guess the output corrects: 0 u^n, 1 2 u^n - u^{n-1}, 2 none
  float logD[4], k[4];
  float mean[NFEAT], istd[NFEAT];
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ void mma_bf16(float c[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the fields row r = v * S + s reads (r < number of rows)
struct RowFields {
  double u, up, phi, ngphi, opu, opdu;
};

__device__ __forceinline__ RowFields row_fields(const MlpFeat& F, int64_t v, int s) {
  const int64_t i = v * F.ld + s;
  RowFields x;
  x.u = F.U[i];
  x.up = F.Up[i];
  x.phi = F.phi ? F.phi[v] : 0.0;
  x.ngphi = F.ngphi ? F.ngphi[v] : 0.0;
  x.opu = F.opU ? F.opU[i] : 0.0;
  x.opdu = F.opDU ? F.opDU[i] : 0.0;
  return x;
}

// all NFEAT normalised features of a row from its fields, branch-free
__device__ __forceinline__ void fields_features(const MlpFeat& F, const RowFields& r, int s,
                                                float f[NFEAT]) {
  float x[NFEAT];
  x[0] = (float)r.phi;
  x[1] = (float)r.ngphi;
  x[2] = (float)r.u;
  x[3] = (float)r.up;
  x[4] = (float)(r.u - r.up);
  x[5] = F.logD[s];
  x[6] = F.k[s];
  x[7] = 0.0f;
  x[8] = (float)r.opu;
  x[9] = (float)r.opdu;
#pragma unroll
  for (int k = 0; k < NFEAT; k++) f[k] = (k == 7) ? 1.0f : (x[k] - F.mean[k]) * F.istd[k];
}

__device__ __forceinline__ void row_features(const MlpFeat& F, int64_t v, int s,
                                             float f[NFEAT]) {
  fields_features(F, row_fields(F, v, s), s, f);
}

// shared-memory copy of the BF16 weights
struct MlpSmem {
  __nv_bfloat16 W1[MLP_H][W1S];
  __nv_bfloat16 W2[MLP_H][W2S];
  float w3[MLP_H];
  float b1[MLP_H], b2[MLP_H];
  float b3;
};

// W2T (the backward pass): W2 transposed, [in][out]
__device__ void load_weights(MlpSmem& sm, const float* __restrict__ P,
                             __nv_bfloat16 (*W2T)[W2S]) {
  // every load of a thread in flight before its first conversion
  constexpr int T = 128, N1 = MLP_H * MLP_IN / T, N2 = MLP_H * MLP_H / T;
  float w1[N1], w2[N2];
#pragma unroll
  for (int k = 0; k < N1; k++) w1[k] = __ldg(P + OFF_W1 + k * T + threadIdx.x);
#pragma unroll
  for (int k = 0; k < N2; k++) w2[k] = __ldg(P + OFF_W2 + k * T + threadIdx.x);
  for (int i = threadIdx.x; i < MLP_H; i += T) {
    sm.w3[i] = __bfloat162float(__float2bfloat16_rn(P[OFF_W3 + i]));
    sm.b1[i] = P[OFF_B1 + i];
    sm.b2[i] = P[OFF_B2 + i];
  }
  if (threadIdx.x == 0) sm.b3 = P[OFF_B3];
#pragma unroll
  for (int k = 0; k < N1; k++) {
    const int i = k * T + threadIdx.x;
    sm.W1[i / MLP_IN][i % MLP_IN] = __float2bfloat16_rn(w1[k]);
  }
#pragma unroll
  for (int k = 0; k < N2; k++) {
    const int i = k * T + threadIdx.x;
    const __nv_bfloat16 w = __float2bfloat16_rn(w2[k]);
    sm.W2[i / MLP_H][i % MLP_H] = w;
    W2T[i % MLP_H][i / MLP_H] = w;
  }
  __syncthreads();
}

// four 8x8 matrices of a row-major BF16 array, lane l giving the address of row l % 8 of
// matrix l / 8: fragments (row g, columns 2t, 2t + 1) into registers ...
__device__ __forceinline__ void ldm4(uint32_t r[4], const __nv_bfloat16* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
// ... and fragments stored transposed (row g of the fragment becomes column g)
__device__ __forceinline__ void stm4t(__nv_bfloat16* p, const uint32_t r[4]) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(a),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}

// C[n-tile n] += A (4 k-steps of fragments) B, B[k][j] = W[j][k] for W [64][ldk] row-major
__device__ __forceinline__ void mma_64x64(float c[8][4], const uint32_t a[4][4],
                                          const __nv_bfloat16* W, int ldk, int lane) {
#pragma unroll
  for (int n = 0; n < 8; n++) {
    uint32_t b[8];  // k = 0..31, 32..63 of the tile's 8 columns
    ldm4(b, W + (n * 8 + (lane & 7)) * ldk + (lane >> 3) * 8);
    ldm4(b + 4, W + (n * 8 + (lane & 7)) * ldk + 32 + (lane >> 3) * 8);
#pragma unroll
    for (int kk = 0; kk < 4; kk++)
      mma_bf16(c[n], a[kk][0], a[kk][1], a[kk][2], a[kk][3], b[2 * kk], b[2 * kk + 1]);
  }
}

// BF16 A fragments of max(z, 0) for the 8 n-tiles of a 16 x 64 accumulator
__device__ __forceinline__ void relu_fragments(const float z[8][4], uint32_t a[4][4]) {
#pragma unroll
  for (int kk = 0; kk < 4; kk++) {
    const float* lo = z[2 * kk];
    const float* hi = z[2 * kk + 1];
    a[kk][0] = pack_bf16(fmaxf(lo[0], 0.f), fmaxf(lo[1], 0.f));
    a[kk][1] = pack_bf16(fmaxf(lo[2], 0.f), fmaxf(lo[3], 0.f));
    a[kk][2] = pack_bf16(fmaxf(hi[0], 0.f), fmaxf(hi[1], 0.f));
    a[kk][3] = pack_bf16(fmaxf(hi[2], 0.f), fmaxf(hi[3], 0.f));
  }
}

// ----------------------------------------------------------------- inference
// 5th-generation tensor cores: 256-row tiles, two rows (128 apart) per thread of a 128-thread
// CTA.  Layer 1 (128 x 64, K = 16) and layer 2 (128 x 64, K = 64 as four K = 16 steps) of
// each half are tcgen05.mma from shared-memory operands into tensor memory (64 columns a
// half; z2 takes z1's columns once every thread has read them), issued by one thread and
// completed through an mbarrier (tcgen05.commit); every thread reads its own rows back with
// tcgen05.ld (warp w owns TMEM lanes 32w..32w+31).  Operands are K-major without swizzle: 8-row x 16-byte
// core matrices, the two 8-element K halves 128 bytes apart, 8-row groups 256 bytes apart.
// Every mbarrier wait is bounded; a wait that runs out sets the call's status word and
// g_mlp_tc_timeout, ends the CTA's tiles and still releases its tensor memory.
constexpr int TC_M = 128;           // rows of an MMA, threads of a CTA
constexpr int TC_R = 2;             // rows of a thread: a tile is TC_R MMAs
constexpr int TC_ROWS = TC_R * TC_M;
constexpr int TC_COLS = TC_R * MLP_H;  // tensor-memory columns: z1, then z2, of each row
constexpr int TC_CTAS = 3;          // CTAs of an SM (tensor memory and registers would hold 4)
constexpr uint32_t TC_WAIT_LIMIT = 1u << 24;  // default polls of one mbarrier phase (~0.1 s)

__device__ int g_mlp_tc_timeout;

// wait bound and failure-path test switch of the next launches (tp_mlp_set_wait_limit)
struct TcWait {
  uint32_t polls;
  int skip_issue;
  int32_t* status;
};

struct TcSmem {
  // of each 128-row part: h1, one 4 KB block per K step.  The features lie in the first
  // block: layer 1 has read them before h1 is written, layer 2 has read h1 before the next
  // tile's features (43 KB in all: no opt-in per launch).
  __nv_bfloat16 A2[TC_R][4][TC_M * 16];
  __nv_bfloat16 W1[MLP_H * 16];    // 2 KB
  __nv_bfloat16 W2[4][MLP_H * 16]; // 8 KB
  alignas(16) float b1[MLP_H], b2[MLP_H], w3[MLP_H];
  float b3;
  uint64_t bar;
  uint32_t taddr;
};

// element offset of (row, k) in a K-major no-swizzle block of 16 K columns
__device__ __forceinline__ int tc_off(int row, int k) {
  return (row >> 3) * 128 + (k >> 3) * 64 + (row & 7) * 8 + (k & 7);
}

__device__ __forceinline__ uint64_t tc_desc(const void* smem) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
  uint64_t d = (uint64_t)((a >> 4) & 0x3FFFu);  // start address
  d |= (uint64_t)(128 >> 4) << 16;              // leading byte offset: the K halves
  d |= (uint64_t)(256 >> 4) << 32;              // stride byte offset: 8-row groups
  d |= (uint64_t)1 << 46;                       // descriptor version of sm_100
  return d;                                     // base offset 0, no swizzle
}

// kind::f16 instruction descriptor: F32 accumulate, BF16 A and B (K-major), N = 64, M = 128
constexpr uint32_t TC_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MLP_H >> 3) << 17) |
                              ((uint32_t)(TC_M >> 4) << 24);

__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a, uint64_t b, int accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(TC_IDESC), "r"(accumulate));
}

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  const uint32_t ba = (uint32_t)__cvta_generic_to_shared(bar);
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ba)
               : "memory");
}

// bounded wait for the given phase of the mbarrier; false when the limit ran out
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t phase, uint32_t polls) {
  const uint32_t ba = (uint32_t)__cvta_generic_to_shared(bar);
  for (uint32_t it = 0; it < polls; it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}"
        : "=r"(done)
        : "r"(ba), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void tc_timed_out(const TcWait& tw) {
  atomicExch(&g_mlp_tc_timeout, 1);
  if (tw.status) atomicExch(tw.status, 1);
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void proxy_fence() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane (tc_ld_wait before their use)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t r[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
template <int N>
__device__ __forceinline__ void tc_ld_wait(uint32_t (&r)[N][16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < N; k++)
#pragma unroll
    for (int i = 0; i < 16; i++) asm volatile("" : "+r"(r[k][i]));
}

// Two FP32 values in one 64-bit register: packed add and multiply-add (each half rounded on
// its own, as the scalar operations).
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
// BF16 pair of max(z + b, 0): rounding is monotonic and keeps 0, so the maximum may follow it
__device__ __forceinline__ uint32_t bias_relu_bf16(uint32_t z0, uint32_t z1, uint64_t b) {
  const float2 v = f2_unpack(f2_add(f2_pack(__uint_as_float(z0), __uint_as_float(z1)), b));
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
  asm("max.bf16x2 %0, %0, %1;" : "+r"(r) : "r"(0u));
  return r;
}

// x_out[v, s] = B[v, s] + sigma * y(v, s)  (or y_out[r] = y when x_out is NULL).
// Every thread gathers all features of its row (no divergent per-feature branches).
//
// Bound by the serial chain of a CTA (features, MMA, wait, epilogue, MMA, wait, epilogue): with
// three CTAs an SM half of the issue slots stay empty and the tensor pipe runs a quarter of the
// time; DRAM is at 18 %.  What shortens the chain are fewer instructions and shared-memory
// reads in it.  So: bias, BF16 rounding and maximum on packed pairs; the biases and w3
// (16 bytes a read, the same for every lane) read once for two rows; the weights read with
// every load in flight; one barrier less per tile.  823,875 rows: 50 us with one row per
// thread and scalar epilogues, 45.7 with packed ones, 36.7 with the weights' loads batched,
// 32.7 with two rows per thread and 3 CTAs per SM.  (4 CTAs, the most that tensor memory
// holds: 32.1, but 18.5 instead of 16.6 at 300,000 rows, with more prologues for fewer
// tiles; one row per thread 20.6 there, and 8.7 instead of 8.3 at 30,000.)
__global__ void __launch_bounds__(TC_M, TC_CTAS) k_mlp_predict(MlpFeat F, int64_t nrows,
                                                      const float* __restrict__ P, float sigma,
                                                      double* __restrict__ x_out,
                                                      float* __restrict__ y_out, TcWait tw) {
  __shared__ __align__(128) TcSmem sm;
  const int tid = threadIdx.x, warp = tid >> 5;
  // weights in the operand layout (BF16), biases and w3 (w3 rounded to BF16 as in training)
  // (every load of a thread in flight before its first conversion)
  constexpr int N1 = MLP_H * 16 / TC_M, N2 = MLP_H * MLP_H / TC_M;
  float w1[N1], w2[N2];
#pragma unroll
  for (int k = 0; k < N1; k++) w1[k] = __ldg(P + OFF_W1 + k * TC_M + tid);
#pragma unroll
  for (int k = 0; k < N2; k++) w2[k] = __ldg(P + OFF_W2 + k * TC_M + tid);
  for (int i = tid; i < MLP_H; i += blockDim.x) {
    sm.b1[i] = P[OFF_B1 + i];
    sm.b2[i] = P[OFF_B2 + i];
    sm.w3[i] = __bfloat162float(__float2bfloat16_rn(P[OFF_W3 + i]));
  }
  if (tid == 0) sm.b3 = P[OFF_B3];
#pragma unroll
  for (int k = 0; k < N1; k++) {
    const int i = k * TC_M + tid;
    sm.W1[tc_off(i >> 4, i & 15)] = __float2bfloat16_rn(w1[k]);
  }
#pragma unroll
  for (int k = 0; k < N2; k++) {
    const int i = k * TC_M + tid, c = i & 63;
    sm.W2[c >> 4][tc_off(i >> 6, c & 15)] = __float2bfloat16_rn(w2[k]);
  }
  if (warp == 0) {
    const uint32_t slot = (uint32_t)__cvta_generic_to_shared(&sm.taddr);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
                 "r"(TC_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    const uint32_t ba = (uint32_t)__cvta_generic_to_shared(&sm.bar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ba), "r"(1));
  }
  proxy_fence();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t taddr = sm.taddr;
  const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
  uint32_t phase = 0;
  constexpr int R = TC_R;
  const int64_t ntiles = (nrows + TC_ROWS - 1) / TC_ROWS;
  // (vertex, species) of this thread's first row, advanced by a grid of rows from tile to
  // tile; row k of the thread is 128 k rows on
  const int64_t step = (int64_t)gridDim.x * TC_ROWS, dv = step / F.S;
  const int ds = (int)(step - dv * F.S), dvk = TC_M / F.S, dsk = TC_M - dvk * F.S;
  int64_t r = (int64_t)blockIdx.x * TC_ROWS + tid, v = r / F.S;
  int s = (int)(r - v * F.S);
  auto advance = [&](int64_t& vv, int& ss, int64_t a, int b) {
    vv += a;
    ss += b;
    if (ss >= F.S) {
      ss -= F.S;
      vv++;
    }
  };
  RowFields cur[R];
  auto load_rows = [&]() {
    int64_t vk = v;
    int sk = s;
#pragma unroll
    for (int k = 0; k < R; k++) {
      cur[k] = RowFields{};
      if (r + k * TC_M < nrows) cur[k] = row_fields(F, vk, sk);
      advance(vk, sk, dvk, dsk);
    }
  };
  // the fields of the CTA's first tile; every tile's MMAs overlap the next tile's loads
  load_rows();
  bool ok = true;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    bool in[R];
    double base[R];
    int64_t out[R];
    {
      int64_t vk = v;
      int sk = s;
#pragma unroll
      for (int q = 0; q < R; q++) {
        in[q] = r + q * TC_M < nrows;
        float f[NFEAT];
        fields_features(F, cur[q], sk, f);
        uint32_t w[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const float lo = (in[q] && 2 * k < NFEAT) ? f[2 * k] : 0.f;
          const float hi = (in[q] && 2 * k + 1 < NFEAT) ? f[2 * k + 1] : 0.f;
          w[k] = pack_bf16(lo, hi);
        }
        __nv_bfloat16* A = sm.A2[q][0];
        *reinterpret_cast<uint4*>(A + tc_off(tid, 0)) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(A + tc_off(tid, 8)) = make_uint4(w[4], w[5], w[6], w[7]);
        base[q] = F.base == 1 ? 2.0 * cur[q].u - cur[q].up : (F.base == 0 ? cur[q].u : 0.0);
        out[q] = x_out ? vk * F.ld + sk : r + q * TC_M;
        advance(vk, sk, dvk, dsk);
      }
    }
    proxy_fence();
    tc_fence_before();
    // also: every thread's reads of the last tile's z2 are done
    if (__syncthreads_or(!ok)) break;
    tc_fence_after();
    if (tid == 0 && !tw.skip_issue) {
#pragma unroll
      for (int q = 0; q < R; q++)
        tc_mma(taddr + q * MLP_H, tc_desc(sm.A2[q][0]), tc_desc(sm.W1), 0);
      tc_commit(&sm.bar);
    }
    r += step;
    advance(v, s, dv, ds);
    load_rows();
    ok = tc_wait(&sm.bar, phase, tw.polls);
    phase ^= 1u;
    tc_fence_after();
    // h1 = relu(z1 + b1), BF16, into the layer-2 operand: 16 columns at a time
#pragma unroll
    for (int j = 0; j < 4; j++) {
      uint32_t z[R][16];
#pragma unroll
      for (int q = 0; q < R; q++) tc_ld16(taddr + lane_base + q * MLP_H + 16 * j, z[q]);
      tc_ld_wait(z);
      uint32_t w[R][8];
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        const ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(&sm.b1[16 * j + 2 * k]);
#pragma unroll
        for (int q = 0; q < R; q++) {
          w[q][k] = bias_relu_bf16(z[q][2 * k], z[q][2 * k + 1], bb.x);
          w[q][k + 1] = bias_relu_bf16(z[q][2 * k + 2], z[q][2 * k + 3], bb.y);
        }
      }
#pragma unroll
      for (int q = 0; q < R; q++) {
        __nv_bfloat16* A = sm.A2[q][j];
        *reinterpret_cast<uint4*>(A + tc_off(tid, 0)) =
            make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
        *reinterpret_cast<uint4*>(A + tc_off(tid, 8)) =
            make_uint4(w[q][4], w[q][5], w[q][6], w[q][7]);
      }
    }
    proxy_fence();
    tc_fence_before();
    if (__syncthreads_or(!ok)) break;
    tc_fence_after();
    if (tid == 0 && !tw.skip_issue) {  // every thread has read z1: z2 takes its columns
#pragma unroll
      for (int q = 0; q < R; q++)
#pragma unroll
        for (int j = 0; j < 4; j++)
          tc_mma(taddr + q * MLP_H, tc_desc(sm.A2[q][j]), tc_desc(sm.W2[j]), j > 0);
      tc_commit(&sm.bar);
    }
    ok = tc_wait(&sm.bar, phase, tw.polls);
    phase ^= 1u;
    tc_fence_after();
    // layer 3 on the CUDA cores: BF16-rounded h2 . w3 + b3
    uint64_t acc[R][2];
#pragma unroll
    for (int q = 0; q < R; q++) acc[q][0] = acc[q][1] = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      uint32_t z[R][16];
#pragma unroll
      for (int q = 0; q < R; q++) tc_ld16(taddr + lane_base + q * MLP_H + 16 * j, z[q]);
      tc_ld_wait(z);
#pragma unroll
      for (int k = 0; k < 16; k += 4) {
        const ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(&sm.b2[16 * j + k]);
        const ulonglong2 ww = *reinterpret_cast<const ulonglong2*>(&sm.w3[16 * j + k]);
        auto h2 = [](uint32_t p) {
          return f2_pack(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
        };
#pragma unroll
        for (int q = 0; q < R; q++) {
          acc[q][0] = f2_fma(h2(bias_relu_bf16(z[q][k], z[q][k + 1], bb.x)), ww.x, acc[q][0]);
          acc[q][1] = f2_fma(h2(bias_relu_bf16(z[q][k + 2], z[q][k + 3], bb.y)), ww.y, acc[q][1]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < R; q++) {
      const float2 p = f2_unpack(f2_add(acc[q][0], acc[q][1]));
      const float y = p.x + p.y + sm.b3;
      if (in[q] && ok) {
        if (x_out)
          x_out[out[q]] = base[q] + (double)sigma * (double)y;
        else
          y_out[out[q]] = y;
      }
    }
  }
  if (!ok) tc_timed_out(tw);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr),
                 "r"(TC_COLS));
}

// features of every row, materialised (training set), BF16 (nrows, 16): one thread per
// row, one 32-byte store
__global__ void k_mlp_features(MlpFeat F, int64_t nrows, __nv_bfloat16* __restrict__ X) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrows;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = r / F.S;
    const int s = (int)(r - v * F.S);
    float f[NFEAT];
    row_features(F, v, s, f);
    uint32_t w[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const float lo = (2 * k < NFEAT) ? f[2 * k] : 0.f;
      const float hi = (2 * k + 1 < NFEAT) ? f[2 * k + 1] : 0.f;
      w[k] = pack_bf16(lo, hi);
    }
    uint4* dst = reinterpret_cast<uint4*>(X + r * MLP_IN);
    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// training target (u^{n+1} - u^n) / sigma per row
__global__ void k_mlp_target(int64_t nrows, int S, int ld, const double* __restrict__ Un,
                             const double* __restrict__ Uprev,
                             const double* __restrict__ Unext, float inv_sigma,
                             float* __restrict__ T) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrows;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = r / S;
    const int s = (int)(r - v * S);
    const int64_t i = v * ld + s;
    const double b = Uprev ? 2.0 * Un[i] - Uprev[i] : Un[i];
    T[r] = (float)((Unext[i] - b) * inv_sigma);
  }
}

// ----------------------------------------------------------------- training
struct GradSmem {
  __nv_bfloat16 dz2T[MLP_H][GS];  // [out unit][chunk row]
  __nv_bfloat16 h1T[MLP_H][GS];   // [hidden unit][chunk row]
  __nv_bfloat16 dz1T[MLP_H][GS];
  __nv_bfloat16 xT[MLP_IN][GS];
  __nv_bfloat16 W2T[MLP_H][W2S];  // W2 transposed: B operand of dH1 = dZ2 W2
  float dw3[4][MLP_H];  // per warp
  float db3[4];
  float loss[4];
};

// One CTA = 4 warps = 64-row chunks.  Partial gradients (MLP_P floats) and the loss
// partial (sum of squared errors) per CTA.  wscale = 2 / (rows in the batch).
//
// Bound by instruction issue, not by the tensor cores: operands move between the fragment
// layouts with ldmatrix and (transposed) stmatrix, four 8x8 matrices at a time, the bias
// gradients are one more product with ones, and the sums of layer 3 and of the loss stay in
// each thread until the last chunk.  65,536 rows, cold caches: 25.8 us with 2-byte stores
// and a scalar loop for the bias sums, 17.2 us in this form (1,024 chunks on 296 CTAs: the
// fourth turn is half empty).
__global__ void __launch_bounds__(128) k_mlp_grad(const __nv_bfloat16* __restrict__ X,
                                                  const float* __restrict__ T, int64_t row0,
                                                  int64_t nrows, const float* __restrict__ P,
                                                  float wscale, float* __restrict__ part,
                                                  float* __restrict__ loss_part) {
  __shared__ __align__(16) MlpSmem sm;
  extern __shared__ __align__(16) unsigned char grad_dyn[];  // GradSmem (> 48 KB static)
  GradSmem& gs = *reinterpret_cast<GradSmem*>(grad_dyn);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  // inputs and targets of rows g, g + 8 of this warp's 16 rows of a chunk
  auto load_rows = [&](int64_t ch, uint32_t xa[4], float& ta, float& tb) {
    const int64_t ra = ch * 64 + warp * 16 + g, rb = ra + 8;
    const uint32_t* Xa = reinterpret_cast<const uint32_t*>(X + (row0 + ra) * MLP_IN);
    const uint32_t* Xb = reinterpret_cast<const uint32_t*>(X + (row0 + rb) * MLP_IN);
    xa[0] = ra < nrows ? __ldg(Xa + t) : 0u;
    xa[1] = rb < nrows ? __ldg(Xb + t) : 0u;
    xa[2] = ra < nrows ? __ldg(Xa + t + 4) : 0u;
    xa[3] = rb < nrows ? __ldg(Xb + t + 4) : 0u;
    ta = ra < nrows ? __ldg(T + row0 + ra) : 0.f;
    tb = rb < nrows ? __ldg(T + row0 + rb) : 0.f;
  };
  const int64_t nchunks = (nrows + 63) / 64;
  uint32_t xn[4] = {0u, 0u, 0u, 0u};
  float tn0 = 0.f, tn1 = 0.f;
  if (blockIdx.x < nchunks) load_rows(blockIdx.x, xn, tn0, tn1);
  load_weights(sm, P, gs.W2T);
  // dW2 rows [16 warp, 16 warp + 16) x 64 cols; dW1 rows [16 warp, +16) x 16 cols; db2 and
  // db1 of the same rows (every column of the product with ones)
  float dW2[8][4], dW1[2][4], db2[4], db1[4];
#pragma unroll
  for (int n = 0; n < 8; n++) dW2[n][0] = dW2[n][1] = dW2[n][2] = dW2[n][3] = 0.f;
#pragma unroll
  for (int n = 0; n < 2; n++) dW1[n][0] = dW1[n][1] = dW1[n][2] = dW1[n][3] = 0.f;
#pragma unroll
  for (int e = 0; e < 4; e++) db2[e] = db1[e] = 0.f;
  float dw3[8][2], ls = 0.f, bs = 0.f;  // this thread's rows: units 8 n + 2 t + e
#pragma unroll
  for (int n = 0; n < 8; n++) dw3[n][0] = dw3[n][1] = 0.f;
  for (int64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    uint32_t xa[4] = {xn[0], xn[1], xn[2], xn[3]};
    const float ta = tn0, tb = tn1;
    if (ch + gridDim.x < nchunks) load_rows(ch + gridDim.x, xn, tn0, tn1);
    // ---- forward: z1 -> h1 (fragments) and the signs of z1, z2
    uint32_t ha[4][4], m1 = 0;
    {
      float z1[8][4];
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        uint32_t b[4];  // two n-tiles, K = 16
        ldm4(b, &sm.W1[(n + (lane >> 4)) * 8 + (lane & 7)][((lane >> 3) & 1) * 8]);
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const float2 bb = *reinterpret_cast<const float2*>(&sm.b1[(n + q) * 8 + 2 * t]);
          z1[n + q][0] = z1[n + q][2] = bb.x;
          z1[n + q][1] = z1[n + q][3] = bb.y;
          mma_bf16(z1[n + q], xa[0], xa[1], xa[2], xa[3], b[2 * q], b[2 * q + 1]);
        }
      }
      relu_fragments(z1, ha);
#pragma unroll
      for (int n = 0; n < 8; n++)
#pragma unroll
        for (int e = 0; e < 4; e++) m1 |= (z1[n][e] > 0.f ? 1u : 0u) << (4 * n + e);
    }
    float z2[8][4];
#pragma unroll
    for (int n = 0; n < 8; n++) {
      const float2 bb = *reinterpret_cast<const float2*>(&sm.b2[n * 8 + 2 * t]);
      z2[n][0] = z2[n][2] = bb.x;
      z2[n][1] = z2[n][3] = bb.y;
    }
    mma_64x64(z2, ha, &sm.W2[0][0], W2S, lane);
    // layer 3 (64 -> 1) on the CUDA cores: BF16-rounded h2 . w3, reduced over the quad
    float s0 = 0.f, s1 = 0.f;
    float h2[8][4];
#pragma unroll
    for (int n = 0; n < 8; n++) {
      const float2 w = *reinterpret_cast<const float2*>(&sm.w3[n * 8 + 2 * t]);
#pragma unroll
      for (int e = 0; e < 4; e++)
        h2[n][e] = __bfloat162float(__float2bfloat16_rn(fmaxf(z2[n][e], 0.f)));
      s0 += h2[n][0] * w.x;
      s0 += h2[n][1] * w.y;
      s1 += h2[n][2] * w.x;
      s1 += h2[n][3] * w.y;
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    const int64_t ra = ch * 64 + warp * 16 + g;
    const float e0 = ra < nrows ? s0 + sm.b3 - ta : 0.f;
    const float e1 = ra + 8 < nrows ? s1 + sm.b3 - tb : 0.f;
    const float d0 = wscale * e0, d1 = wscale * e1;  // dL/dy
    ls += e0 * e0 + e1 * e1;
    bs += d0 + d1;
    // ---- dw3 and dZ2 = dy w3 [z2 > 0], as fragments
    uint32_t da[4][4];
    {
#pragma unroll
      for (int n = 0; n < 8; n++) {
        const float2 w = *reinterpret_cast<const float2*>(&sm.w3[n * 8 + 2 * t]);
        dw3[n][0] += d0 * h2[n][0] + d1 * h2[n][2];
        dw3[n][1] += d0 * h2[n][1] + d1 * h2[n][3];
        const float a0 = z2[n][0] > 0.f ? d0 * w.x : 0.f, a1 = z2[n][1] > 0.f ? d0 * w.y : 0.f;
        const float a2 = z2[n][2] > 0.f ? d1 * w.x : 0.f, a3 = z2[n][3] > 0.f ? d1 * w.y : 0.f;
        da[n >> 1][(n & 1) * 2] = pack_bf16(a0, a1);
        da[n >> 1][(n & 1) * 2 + 1] = pack_bf16(a2, a3);
      }
    }
    // ---- dH1 = dZ2 W2, dZ1 = dH1 [z1 > 0]
    uint32_t d1a[4][4];
    {
      float dz1[8][4];
#pragma unroll
      for (int n = 0; n < 8; n++) dz1[n][0] = dz1[n][1] = dz1[n][2] = dz1[n][3] = 0.f;
      mma_64x64(dz1, da, &gs.W2T[0][0], W2S, lane);
#pragma unroll
      for (int n = 0; n < 8; n++) {
#pragma unroll
        for (int e = 0; e < 4; e++) dz1[n][e] = (m1 >> (4 * n + e)) & 1u ? dz1[n][e] : 0.f;
        d1a[n >> 1][(n & 1) * 2] = pack_bf16(dz1[n][0], dz1[n][1]);
        d1a[n >> 1][(n & 1) * 2 + 1] = pack_bf16(dz1[n][2], dz1[n][3]);
      }
    }
    // ---- stage the transposed tiles (columns = this chunk's 64 rows)
    const int su = (lane & 7) + ((lane >> 4) & 1) * 8;         // unit of this lane's address
    const int sc = warp * 16 + ((lane >> 3) & 1) * 8;          // first chunk row of its matrix
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
      stm4t(&gs.dz2T[kk * 16 + su][sc], da[kk]);
      stm4t(&gs.dz1T[kk * 16 + su][sc], d1a[kk]);
      stm4t(&gs.h1T[kk * 16 + su][sc], ha[kk]);
    }
    stm4t(&gs.xT[su][sc], xa);
    __syncthreads();
    // ---- dW2[i][j] += sum_r dZ2T[i][r] H1T[j][r];  dW1[i][j] += sum_r dZ1T[i][r] XT[j][r]
    const int i0 = warp * 16;
    uint32_t a2[4][4], a1[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
      const int ar = i0 + (lane & 7) + ((lane >> 3) & 1) * 8, ac = kk * 16 + (lane >> 4) * 8;
      ldm4(a2[kk], &gs.dz2T[ar][ac]);
      ldm4(a1[kk], &gs.dz1T[ar][ac]);
      constexpr uint32_t ONES = 0x3F803F80u;
      mma_bf16(db2, a2[kk][0], a2[kk][1], a2[kk][2], a2[kk][3], ONES, ONES);
      mma_bf16(db1, a1[kk][0], a1[kk][1], a1[kk][2], a1[kk][3], ONES, ONES);
    }
    mma_64x64(dW2, a2, &gs.h1T[0][0], GS, lane);
#pragma unroll
    for (int n = 0; n < 2; n++) {
      uint32_t b[8];
      ldm4(b, &gs.xT[n * 8 + (lane & 7)][(lane >> 3) * 8]);
      ldm4(b + 4, &gs.xT[n * 8 + (lane & 7)][32 + (lane >> 3) * 8]);
#pragma unroll
      for (int kk = 0; kk < 4; kk++)
        mma_bf16(dW1[n], a1[kk][0], a1[kk][1], a1[kk][2], a1[kk][3], b[2 * kk], b[2 * kk + 1]);
    }
    __syncthreads();
  }
  // write this CTA's partial gradient
  float* out = part + (int64_t)blockIdx.x * MLP_P;
  const int i0 = warp * 16;
#pragma unroll
  for (int n = 0; n < 8; n++) {
    const int j = n * 8 + 2 * t;
    out[OFF_W2 + (i0 + g) * MLP_H + j] = dW2[n][0];
    out[OFF_W2 + (i0 + g) * MLP_H + j + 1] = dW2[n][1];
    out[OFF_W2 + (i0 + g + 8) * MLP_H + j] = dW2[n][2];
    out[OFF_W2 + (i0 + g + 8) * MLP_H + j + 1] = dW2[n][3];
  }
#pragma unroll
  for (int n = 0; n < 2; n++) {
    const int j = n * 8 + 2 * t;
    out[OFF_W1 + (i0 + g) * MLP_IN + j] = dW1[n][0];
    out[OFF_W1 + (i0 + g) * MLP_IN + j + 1] = dW1[n][1];
    out[OFF_W1 + (i0 + g + 8) * MLP_IN + j] = dW1[n][2];
    out[OFF_W1 + (i0 + g + 8) * MLP_IN + j + 1] = dW1[n][3];
  }
  if (t == 0) {
    out[OFF_B2 + i0 + g] = db2[0];
    out[OFF_B2 + i0 + g + 8] = db2[2];
    out[OFF_B1 + i0 + g] = db1[0];
    out[OFF_B1 + i0 + g + 8] = db1[2];
  }
  // layer 3 and the loss: over the 8 quads of the warp, then over the warps
#pragma unroll
  for (int n = 0; n < 8; n++) {
#pragma unroll
    for (int e = 0; e < 2; e++) {
      float pw = dw3[n][e];
      pw += __shfl_xor_sync(0xffffffffu, pw, 4);
      pw += __shfl_xor_sync(0xffffffffu, pw, 8);
      pw += __shfl_xor_sync(0xffffffffu, pw, 16);
      if (g == 0) gs.dw3[warp][n * 8 + 2 * t + e] = pw;
    }
  }
  ls += __shfl_xor_sync(0xffffffffu, ls, 4);
  ls += __shfl_xor_sync(0xffffffffu, ls, 8);
  ls += __shfl_xor_sync(0xffffffffu, ls, 16);
  bs += __shfl_xor_sync(0xffffffffu, bs, 4);
  bs += __shfl_xor_sync(0xffffffffu, bs, 8);
  bs += __shfl_xor_sync(0xffffffffu, bs, 16);
  if (lane == 0) {
    gs.loss[warp] = ls;
    gs.db3[warp] = bs;
  }
  __syncthreads();
  if (threadIdx.x < MLP_H)
    out[OFF_W3 + threadIdx.x] = ((gs.dw3[0][threadIdx.x] + gs.dw3[1][threadIdx.x]) +
                                 gs.dw3[2][threadIdx.x]) + gs.dw3[3][threadIdx.x];
  if (threadIdx.x == 0) {
    out[OFF_B3] = ((gs.db3[0] + gs.db3[1]) + gs.db3[2]) + gs.db3[3];
    loss_part[blockIdx.x] = ((gs.loss[0] + gs.loss[1]) + gs.loss[2]) + gs.loss[3];
  }
}

// Sum the CTA partials, AdamW on the FP32 master parameters.  A block takes 32 parameters
// (the last block the loss), one per lane; warp w adds the partials w, w + 8, ... and the
// warps' sums are added in order: a fixed order whatever the schedule, and 8 independent
// chains of loads per parameter where one thread per parameter walked all of them (bound by
// the latency of those chains: 296 partials, cold caches, 31 us in that form, 9.5 in this).
__global__ void __launch_bounds__(256) k_mlp_adamw(
    const float* __restrict__ part, int nparts, const float* __restrict__ loss_part,
    float* __restrict__ P, float* __restrict__ m, float* __restrict__ v, float lr, float b1,
    float b2, float eps, float wd, float bc1, float bc2, float* __restrict__ grad_out,
    float* __restrict__ loss_out) {
  __shared__ float s[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool loss = blockIdx.x == gridDim.x - 1;
  const int p = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (loss) {
    for (int c = threadIdx.x; c < nparts; c += 256) acc += loss_part[c];
  } else if (p < MLP_P) {
#pragma unroll 8
    for (int c = warp; c < nparts; c += 8) acc += __ldg(part + (int64_t)c * MLP_P + p);
  }
  s[warp][lane] = acc;
  __syncthreads();
  if (warp != 0) return;
  float gsum = 0.f;
#pragma unroll
  for (int w = 0; w < 8; w++) gsum += s[w][lane];
  if (loss) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gsum += __shfl_xor_sync(0xffffffffu, gsum, o);
    if (lane == 0 && loss_out) *loss_out = gsum;
    return;
  }
  if (p >= MLP_P) return;
  if (grad_out) grad_out[p] = gsum;
  if (lr > 0.f) {
    const float mm = b1 * m[p] + (1.f - b1) * gsum;
    const float vv = b2 * v[p] + (1.f - b2) * gsum * gsum;
    m[p] = mm;
    v[p] = vv;
    const bool decay = !((p >= OFF_B1 && p < OFF_W2) || (p >= OFF_B2 && p < OFF_W3) ||
                         p == OFF_B3);
    P[p] -= lr * ((mm / bc1) / (sqrtf(vv / bc2) + eps) + (decay ? wd * P[p] : 0.f));
  }
}

}  // namespace tp

using namespace tp;

static MlpFeat make_feat(const tp_mlp_inputs* in) {
  MlpFeat F;
  F.U = in->U;
  F.Up = in->U_prev;
  F.phi = in->phi;
  F.ngphi = in->normgradphi;
  F.opU = in->opU;
  F.opDU = in->opDU;
  F.S = in->S;
  F.ld = in->ld;
  F.base = in->base;
  for (int s = 0; s < 4; s++) {
    F.logD[s] = (float)in->logD[s];
    F.k[s] = (float)in->k[s];
  }
  for (int f = 0; f < NFEAT; f++) {
    F.mean[f] = (float)in->mean[f];
    F.istd[f] = (float)in->istd[f];
  }
  return F;
}

static std::atomic<uint32_t> g_tc_polls{TC_WAIT_LIMIT};
static std::atomic<int> g_tc_skip{0};

extern "C" int tp_mlp_param_count(void) { return MLP_P; }

extern "C" int tp_mlp_predict(const tp_mlp_inputs* in, const float* params, float sigma,
                              double* x_out, float* y_out, void* stream) {
  TP_REQUIRE(in && in->U && in->U_prev && params && (x_out || y_out), "null pointer");
  TP_REQUIRE(in->S >= 1 && in->S <= 4 && in->ld >= in->S, "bad S/ld");
  TP_REQUIRE(in->base >= 0 && in->base <= 2, "base must be 0 (u^n), 1 (2 u^n - u^{n-1}) or 2 (none)");
  const int64_t nrows = in->n_verts * in->S;
  if (nrows == 0) return TP_OK;
  cudaStream_t st = as_stream(stream);
  TcWait tw{g_tc_polls.load(), g_tc_skip.load(), in->tc_status};
  if (tw.status) TP_CUDA_TRY(cudaMemsetAsync(tw.status, 0, sizeof(int32_t), st));
  const int64_t ntiles = (nrows + TC_ROWS - 1) / TC_ROWS;
  const int grid = (int)std::min<int64_t>(ntiles, (int64_t)sm_count() * TC_CTAS);
  k_mlp_predict<<<grid, TC_M, 0, st>>>(make_feat(in), nrows, params, sigma, x_out, y_out, tw);
  TP_LAUNCH_CHECK();
  return TP_OK;
}

extern "C" int tp_mlp_set_wait_limit(unsigned int polls, int skip_issue) {
  g_tc_polls.store(polls ? polls : TC_WAIT_LIMIT);
  g_tc_skip.store(skip_issue ? 1 : 0);
  return TP_OK;
}

extern "C" int tp_mlp_tensor_status(int* timed_out, void* stream) {
  TP_REQUIRE(timed_out, "null pointer");
  cudaStream_t st = as_stream(stream);
  TP_CUDA_TRY(cudaMemcpyFromSymbolAsync(timed_out, g_mlp_tc_timeout, sizeof(int), 0,
                                        cudaMemcpyDeviceToHost, st));
  TP_CUDA_TRY(cudaStreamSynchronize(st));
  return TP_OK;
}

extern "C" int tp_mlp_features(const tp_mlp_inputs* in, void* X, void* stream) {
  TP_REQUIRE(in && in->U && in->U_prev && X, "null pointer");
  const int64_t nrows = in->n_verts * in->S;
  if (nrows == 0) return TP_OK;
  k_mlp_features<<<grid_for(nrows * MLP_IN, 256, 65535), 256, 0, as_stream(stream)>>>(
      make_feat(in), nrows, static_cast<__nv_bfloat16*>(X));
  TP_LAUNCH_CHECK();
  return TP_OK;
}

extern "C" int tp_mlp_target(int64_t n_verts, int S, int ld, const double* U_n,
                             const double* U_prev, const double* U_next, double sigma, float* T,
                             void* stream) {
  TP_REQUIRE(U_n && U_next && T && sigma > 0, "bad argument");
  const int64_t nrows = n_verts * S;
  if (nrows == 0) return TP_OK;
  k_mlp_target<<<grid_for(nrows, 256, 65535), 256, 0, as_stream(stream)>>>(
      nrows, S, ld, U_n, U_prev, U_next, (float)(1.0 / sigma), T);
  TP_LAUNCH_CHECK();
  return TP_OK;
}

extern "C" size_t tp_mlp_grad_workspace_floats(int grid) { return (size_t)grid * (MLP_P + 1); }

extern "C" int tp_mlp_train_step(const void* X, const float* T, int64_t row0, int64_t nrows,
                                 float* params, float* adam_m, float* adam_v, int step,
                                 float lr, float beta1, float beta2, float eps,
                                 float weight_decay, int grid, float* workspace,
                                 float* grad_out, float* loss_out, void* stream) {
  TP_REQUIRE(X && T && params && workspace && grid >= 1, "bad argument");
  TP_REQUIRE(lr <= 0.f || (adam_m && adam_v && step >= 1), "AdamW state required");
  cudaStream_t st = as_stream(stream);
  float* part = workspace;
  float* loss_part = workspace + (size_t)grid * MLP_P;
  const float wscale = nrows > 0 ? 2.0f / (float)nrows : 0.f;
  TP_CUDA_TRY(cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(GradSmem)));
  k_mlp_grad<<<grid, 128, sizeof(GradSmem), st>>>(static_cast<const __nv_bfloat16*>(X), T, row0,
                                                  nrows, params, wscale, part, loss_part);
  TP_LAUNCH_CHECK();
  const float bc1 = 1.f - powf(beta1, (float)std::max(step, 1));
  const float bc2 = 1.f - powf(beta2, (float)std::max(step, 1));
  k_mlp_adamw<<<(MLP_P + 31) / 32 + 1, 256, 0, st>>>(part, grid, loss_part, params, adam_m, adam_v,
                                                   lr, beta1, beta2, eps, weight_decay, bc1,
                                                   bc2, grad_out, loss_out);
  TP_LAUNCH_CHECK();
  return TP_OK;
}
