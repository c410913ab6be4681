// tp_ccg.cu -- Jacobi-PCG with one thread-block cluster per system.
//
// A solve of a few thousand to a few ten thousand rows is bound by the latency of its two
// synchronisations per iteration, not by its arithmetic: over the whole chip each costs a
// grid barrier and an L2 round trip for the partial sums.  A system that fits 8 or 16 SMs
// is solved here by one cluster: partial sums and the halo of the shared vector travel
// through distributed shared memory, and several systems run side by side, one per cluster,
// the largest first.
//
// Chronopoulos-Gear form, the recurrences of k_cgw (tp_pcg.cu):
//
//   loop  p = u + beta p, s = w + beta s, xi += alpha p, r -= alpha s, u = D^-1 r
//         u into the CTA's window and pushed into the windows that hold it as halo
//                                                            | the halo's bytes have come
//         w = A u;  r.u, r.r, w.u to every CTA of the cluster | the sums' bytes have come
//         totals, lane decisions, alpha, beta (one warp of every CTA, same bits)
//   when a lane asks (FP32 inner: its recurrence residual fell by delta; both: it reached
//   the tolerance and no lane still runs): x += xi, r = b - A x in FP64, and the loop goes
//   on from there.  Convergence is declared on that FP64 residual only.
//
// Synchronisation.  No barrier is needed per iteration: the halo values and the partial sums
// are sent with st.async, whose bytes complete an mbarrier of the receiving CTA, so each of
// the two exchanges costs one distributed-shared-memory latency.  A CTA may overwrite its
// window because its neighbours send the next values only after they hold every CTA's
// sums, which it sends after its product; the sums alternate between two buffers.  Before
// an FP64 sweep the CTAs meet at an mbarrier where each arrives once at every other's.
// Waits are bounded in time (tp_pcg_set_wait_limit).  A CTA that gives up ends its solve with
// TP_ERR_TIMEOUT and takes part in no later exchange, so the others complete at most the
// passes that it has sent its data for and then give up as well (or end converged).  The
// closing cluster barrier is the only one after the start: a CTA leaves it, and frees its
// shared memory, when none of the others starts another send.
//
// Layout.  The rows of a system are split into equal ranges of 32-row slices over the
// cluster's CTAs.  r, p, s, xi and D^-1 of a row live in its thread's registers (thread =
// lane of the row's slice); the inner values of the slices in tensor memory (8 FP32 or 4
// FP64 slices of at most 16 entries per warp), past those in shared memory or L2; the
// window of u (own rows, then the halo in row order), w and the 16-bit window-local columns
// in shared memory (as byte offsets).  Entry k of a slice's row sits at base + 128 (k / 4) +
// 4 lane + k % 4: four columns per 8-byte load; slices are at least 16 entries wide, so
// that those in tensor memory have fixed addresses.  Dot products are FP64 partials summed in CTA order:
// results depend on the cluster size only, which is fixed at create.
// A system past one cluster runs the same passes on every SM (GRID): the exchanges then go
// through L2, and again no barrier is needed per iteration, because the data carries its own
// flag.  Every row of u is published in 16-byte units that hold values and the pass number
// (a unit is written and read in one access), and a CTA polls the units of its halo and the
// partial sums of the others until their number is this pass': one store and one load of
// latency per exchange, where a grid barrier costs an arrival, a poll and then the load.
// The buffers are cleared before a solve, so an old number is never taken for a new one; a
// unit is rewritten only after its readers have sent the sums that the writer waits for.
// Past two rows a thread, three or four FP32 columns are laid out for it in another way
// (cc_planes): planes in shared memory, the vectors in tensor memory.  The product is bound
// by shared-memory bandwidth there: 274,625 rows of three columns, us per iteration: 10.0
// with rows padded to 16 bytes and vectors spilled past the registers, 8.6 with planes, 6.5
// once one column is left (columns of larger diffusion take half as many passes more).
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "tp_ccg.cuh"
#include "tp_ops.cuh"

namespace tp {

constexpr int CC_T = 512, CC_W = CC_T / 32;
constexpr unsigned long long CC_WAIT_NS = 2000000000ull;  // default bound of a wait: 2 s
// how long a CTA whose wait ran out stays after the closing cluster barrier: no send starts
// after it, and one in flight lands within about a microsecond
constexpr unsigned long long CC_DRAIN_NS = 200000ull;
constexpr int CC_SLOT_BITS = 14, CC_SRC_BITS = 13;  // push entry: rank | window slot | source row

struct CcgPart {
  int32_t row0, nrows;     // rows of this CTA's range (global id of the first)
  int32_t nslices, slice_off;  // slice offsets (nslices + 1) at slice_off of the table
  int32_t nhalo, npush, push_off, entries;
  int32_t val_slice, pad;  // slices from here on keep their values outside tensor memory
  int64_t entry_off;
};

struct CcgOut {
  int32_t iterations, n_reliable, status, pad;
  int32_t lane_iters[4], lane_status[4];
  double lane_rtrue[4], lane_bb[4];
};

template <typename VT>
struct CcgArgs {
  const CcgPart* parts;  // C per cluster
  const int32_t* order;  // system of each cluster, largest first
  int S, max_it;
  double delta2;
  const int32_t* slices;
  const uint16_t* loc_col;
  const uint32_t* push;
  VT* packed;  // inner values in slice order (parts whose values are not in shared memory)
  const VT* inK;               // CSR values, or
  const VT* sK;                // SELL-32 values of the single system
  const int32_t* sell_slice;
  CsrView<double> A64;
  const VT* diag;  // (n, LD) or NULL
  const double* b;
  double* x;
  const double* rtol;
  CcgOut* out;
  int win_cap, dyn_bytes;
  // GRID: halo rows of every part, published rows (16-byte units), partial sums (units of
  // two buffers x CTA x 16), arrivals of the grid barrier around the FP64 sweeps
  const int32_t* halo;
  ulonglong2* ubuf;
  ulonglong2* sums;
  unsigned int* bar;
  unsigned long long wait_limit_ns;
  unsigned int wait_missing;  // > 0 (tests): every wait expects that many bytes too many
};

// ----------------------------------------------------------------- cluster primitives
__device__ __forceinline__ uint32_t cl_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cl_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cl_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cl_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cl_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cl_sync() {
  cl_arrive();
  cl_wait();
}
__device__ __forceinline__ uint32_t cl_map(const void* smem, uint32_t rank) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(sa), "r"(rank));
  return r;
}
// one arrival at another CTA's mbarrier; publishes this CTA's writes before it to the cluster
__device__ __forceinline__ void cl_mb_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mbar)
               : "memory");
}
// asynchronous stores to another CTA's shared memory; the bytes complete its mbarrier
__device__ __forceinline__ void cl_send(uint32_t dst, double v, uint32_t mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(
                   dst),
               "d"(v), "r"(mbar)
               : "memory");
}
// NB bytes (4, 8 or a multiple of 16) of this CTA's shared memory
template <int NB>
__device__ __forceinline__ void cl_send_row(uint32_t dst, const void* src, uint32_t mbar) {
  if constexpr (NB == 4) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(src);
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(
                     dst),
                 "r"(v), "r"(mbar)
                 : "memory");
  } else if constexpr (NB == 8) {
    const uint2 v = *reinterpret_cast<const uint2*>(src);
    asm volatile(
        "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(
            dst),
        "r"(v.x), "r"(v.y), "r"(mbar)
        : "memory");
  } else {
#pragma unroll
    for (int k = 0; k < NB / 16; k++) {
      const uint4 v = reinterpret_cast<const uint4*>(src)[k];
      asm volatile(
          "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, "
          "[%5];" ::"r"(dst + 16 * k),
          "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(mbar)
          : "memory");
    }
  }
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mb_init(uint64_t* mb, uint32_t arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(mb)), "r"(arrivals)
               : "memory");
}
__device__ __forceinline__ void mb_expect(uint64_t* mb, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(mb)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mb_try(uint64_t* mb, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(mb)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long cc_time() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// false when the phase did not complete within limit_ns
__device__ __forceinline__ bool mb_wait(uint64_t* mb, uint32_t parity,
                                        unsigned long long limit_ns) {
  if (mb_try(mb, parity)) return true;
  const unsigned long long t0 = cc_time();
  while (!mb_try(mb, parity))
    if (cc_time() - t0 > limit_ns) return false;
  return true;
}

// 16 bytes in one access (GRID exchanges)
__device__ __forceinline__ void st_unit(ulonglong2* p, unsigned long long lo,
                                        unsigned long long hi) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"(lo), "l"(hi)
      : "memory");
}
__device__ __forceinline__ ulonglong2 ld_unit(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\t"
      "mov.b128 {%0, %1}, t;\n\t}"
      : "=l"(v.x), "=l"(v.y)
      : "l"(p)
      : "memory");
  return v;
}
// a unit whose number is not `want` yet: polled until it is, false after limit_ns or once
// another thread of the CTA gave up
template <int SHIFT>
__device__ __forceinline__ bool poll_unit(const ulonglong2* p, ulonglong2& v, uint32_t want,
                                          unsigned long long limit_ns, const volatile int* gave_up) {
  if ((uint32_t)(v.y >> SHIFT) == want) return true;
  unsigned long long t0 = 0;
  for (unsigned n = 0;; n++) {
    v = ld_unit(p);
    if ((uint32_t)(v.y >> SHIFT) == want) return true;
    if ((n & 15u) == 15u) {
      if (*gave_up) return false;
      const unsigned long long t = cc_time();
      if (t0 == 0)
        t0 = t;
      else if (t - t0 > limit_ns)
        return false;
    }
  }
}

// tensor memory: 16 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void cc_tm_alloc(uint32_t* slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
      smem_addr(slot)));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
}
__device__ __forceinline__ void cc_tm_st16(uint32_t t, const uint32_t v[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
      "%13,%14,%15,%16};" ::"r"(t),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
      "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void cc_tm_ld16(uint32_t t, uint32_t r[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(t)
      : "memory");
}
__device__ __forceinline__ void cc_tm_st4(uint32_t t, const uint32_t v[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(t), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void cc_tm_ld4(uint32_t t, uint32_t r[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(t)
               : "memory");
}
__device__ __forceinline__ void cc_tm_ld1(uint32_t t, uint32_t& r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(t) : "memory");
}
__device__ __forceinline__ void cc_tm_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void cc_tm_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Sum NV values over the lanes of a warp by halving: at each step a lane keeps half of
// its values and hands the other half to its partner, so NV values cost about NV + 4
// shuffles instead of 5 NV.  Value v ends in lane lane_of_value<NV>(v) (and, for the
// steps past the last halving, in its partners); fixed order.
template <int NV>
struct WarpReduce {
  // values left after each halving: NV, ceil(NV/2), ...
  static __device__ __forceinline__ double run(double* v, int lane) {
    step<NV, 16>(v, lane);
    return v[0];
  }
  template <int N, int O>
  static __device__ __forceinline__ void step(double* v, int lane) {
    constexpr int H = (N + 1) / 2;
    const bool up = (lane & O) != 0;
    if constexpr (N > 1) {
#pragma unroll
      for (int k = 0; k < H; k++) {
        const double hi = (k + H < N) ? v[k + H] : 0.0;
        const double send = up ? v[k] : hi;
        const double keep = up ? hi : v[k];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, send, O);
      }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
    }
    if constexpr (O > 1) step<H, O / 2>(v, lane);
  }
  // the value whose sum lane `lane` holds after run (-1: none)
  static __device__ __forceinline__ int value_of(int lane) {
    return descend<NV, 16>(lane);
  }
  template <int N, int O>
  static __device__ __forceinline__ int descend(int lane) {
    constexpr int H = (N + 1) / 2;
    int base = 0, n = N;
    if constexpr (N > 1) {
      if (lane & O) base = H;
      n = H;
    }
    (void)n;
    if constexpr (O > 1) {
      const int sub = descend<H, O / 2>(lane);
      if (sub < 0) return -1;
      const int v = base + sub;
      return v < N ? v : -1;
    } else {
      return base < N ? base : -1;
    }
  }
};

// LD values of entry i of a shared-memory array
template <typename VT, int LD>
__device__ __forceinline__ void lds_row(const VT* w, int i, VT v[LD]) {
  constexpr int NB = LD * (int)sizeof(VT);
  if constexpr (NB <= 8) {
#pragma unroll
    for (int s = 0; s < LD; s++) v[s] = w[i * LD + s];
  } else {
    VT t[LD];
#pragma unroll
    for (int k = 0; k < NB / 16; k++) {
      const uint4 u = reinterpret_cast<const uint4*>(w + (size_t)i * LD)[k];
      memcpy(reinterpret_cast<char*>(t) + 16 * k, &u, 16);
    }
#pragma unroll
    for (int s = 0; s < LD; s++) v[s] = t[s];
  }
}
template <typename VT, int LD>
__device__ __forceinline__ void sts_row(VT* w, int i, const VT v[LD]) {
  constexpr int NB = LD * (int)sizeof(VT);
  if constexpr (NB <= 8) {
#pragma unroll
    for (int s = 0; s < LD; s++) w[i * LD + s] = v[s];
  } else {
#pragma unroll
    for (int k = 0; k < NB / 16; k++) {
      uint4 u;
      memcpy(&u, reinterpret_cast<const char*>(v) + 16 * k, 16);
      reinterpret_cast<uint4*>(w + (size_t)i * LD)[k] = u;
    }
  }
}
// y += v u; pairs of FP32 columns as one packed FMA
template <typename VT, int LD>
__device__ __forceinline__ void axpy_row(VT v, const VT u[LD], VT y[LD]) {
  if constexpr (sizeof(VT) == 4 && LD >= 2) {
    unsigned long long vv;
    asm("mov.b64 %0, {%1, %1};" : "=l"(vv) : "f"(v));
#pragma unroll
    for (int s = 0; s < LD; s += 2) {
      unsigned long long uu, yy;
      asm("mov.b64 %0, {%1, %2};" : "=l"(uu) : "f"(u[s]), "f"(u[s + 1]));
      asm("mov.b64 %0, {%1, %2};" : "=l"(yy) : "f"(y[s]), "f"(y[s + 1]));
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(yy) : "l"(vv), "l"(uu));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(y[s]), "=f"(y[s + 1]) : "l"(yy));
    }
  } else {
#pragma unroll
    for (int s = 0; s < LD; s++) y[s] += v * u[s];
  }
}

// Whether a system over all SMs keeps its rows in planes and its vectors in tensor memory
// (k_ccg): three or four FP32 columns and more than two rows a thread, whose vectors do not
// fit the registers (three columns, us per iteration at 274,625 rows: 10.1 with 16-byte
// rows and spilled vectors, 8.7 with planes; at 117,649, two rows a thread: 6.1 and 6.4).
template <typename VT>
constexpr bool cc_planes(int NC, int RPT, bool grid) {
  return grid && sizeof(VT) == 4 && NC >= 3 && RPT > 2;
}

// RPT: slices per warp (rows per thread).  Dynamic shared memory: two buffers of partial
// sums (16 CTAs x 16), the window (win_cap rows), w, then this part's slice offsets, push
// list, diagonal, columns and values, each where it still fits.
// NC: columns computed (S <= NC <= LD).
template <typename VT, int LD, int NC, int RPT, bool GRID>
__global__ void __launch_bounds__(CC_T, 1) k_ccg(CcgArgs<VT> a) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  double* const s_part = reinterpret_cast<double*>(s_dyn);  // [2][rank][quantity * 4 + column]
  VT* const s_win = reinterpret_cast<VT*>(s_dyn + 2 * 16 * 16 * sizeof(double));
  __shared__ double s_red[CC_W][16];
  __shared__ __align__(8) uint64_t s_mb[GRID ? 3 : 4];  // partial sums (two), halo, meeting
  __shared__ uint32_t s_taddr;
  // Waits that ran out: set between two CTA barriers and read after the second.  A thread past
  // that barrier may set it again in its next wait, so the two places that read it each ask for
  // their own value, which all threads then read alike.
  enum : int { GAVE_UP = 1, GAVE_UP_SUMS = 2 };  // the meeting or the halo; the sums
  __shared__ volatile int s_gave_up;
  // what warp 0 decided for the next pass (Ctl bits, refreshed columns) and its coefficients
  __shared__ int s_ctl, s_mask, s_run;
  __shared__ VT s_al[4], s_be[4];
  enum : int { CTL_REFRESH = 1, CTL_FIN = 2, CTL_EXIT = 4 };
  // PL: the window, w and the diagonal in planes, 32 values of a column side by side (row i,
  // column s at (i / 32) 32 NC + 32 s + i % 32): a column of 32 neighbouring rows is one
  // 128-byte access, and no room or bandwidth goes to a padding column.  The vectors of a
  // row are then kept in tensor memory, 16 words per slice next to the values: word 4 s
  // + 0..3 r, p, q, xi of column s, word 12 + s D^-1 (four columns: D^-1 in registers).
  constexpr bool PL = cc_planes<VT>(NC, RPT, GRID);
  // ONE: once a single column still runs, a pass computes and exchanges that column only
  // (three columns at 274,625 rows: 6.5 us a pass instead of 8.7; with 16-byte rows, where
  // such a pass reads as much shared memory as a full one, it gains less than the second
  // code path costs the full passes: 4 % at 117,649 rows)
  constexpr bool ONE = PL;
  static_assert(!PL || RPT <= 4, "tensor memory: 16 words of values and 16 of vectors a slice");
  constexpr int RB = PL ? NC * (int)sizeof(VT) : LD * (int)sizeof(VT);
  auto padded = [](int n) { return PL ? (n + 31) & ~31 : n; };
  auto w_ld = [](const VT* w, int i, VT v[LD]) {
    if constexpr (PL) {
      const VT* q = w + (i >> 5) * 32 * NC + (i & 31);
#pragma unroll
      for (int s = 0; s < LD; s++) v[s] = s < NC ? q[32 * (s < NC ? s : 0)] : VT(0);
    } else {
      lds_row<VT, LD>(w, i, v);
    }
  };
  auto w_st = [](VT* w, int i, const VT v[LD]) {
    if constexpr (PL) {
      VT* q = w + (i >> 5) * 32 * NC + (i & 31);
#pragma unroll
      for (int s = 0; s < NC; s++) q[32 * s] = v[s];
    } else {
      sts_row<VT, LD>(w, i, v);
    }
  };
  auto w_at = [](int i, int s) {  // where column s of row i is
    return PL ? (i >> 5) * 32 * NC + 32 * s + (i & 31) : i * LD + s;
  };
  constexpr int VW = (int)sizeof(VT) / 4;             // 32-bit words of a value
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = GRID ? blockIdx.x : cl_rank(), C = GRID ? gridDim.x : cl_size();
  const int S = a.S;
  // GRID: 16-byte units of a published row, and where a unit keeps its pass number
  constexpr int UW = sizeof(VT) == 8 ? NC : (NC + 2) / 3;
  constexpr int TAG = sizeof(VT) == 8 ? 0 : 32;
  uint32_t epoch = 1, arrivals = 0, ph_x = 0;
  // x written by every CTA of the system is visible to all.  A wait that runs out is acted on
  // by this pass' check after the halo.
  auto x_sync = [&]() {
    if constexpr (!GRID) {
      __syncthreads();
      if (tid < (int)C) cl_mb_arrive(cl_map(&s_mb[3], (uint32_t)tid));
      if (!mb_wait(&s_mb[3], ph_x, a.wait_limit_ns)) s_gave_up = GAVE_UP;
      ph_x ^= 1u;
    } else {
      __syncthreads();
      if (tid == 0) {
        arrivals += C + a.wait_missing;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        const unsigned long long t0 = cc_time();
        for (;;) {
          uint32_t v;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
          if ((int)(v - arrivals) >= 0) break;
          if (cc_time() - t0 > a.wait_limit_ns) {
            s_gave_up = GAVE_UP;
            break;
          }
        }
      }
      __syncthreads();
    }
  };
  // GRID: this pass' u of a row for the CTAs that hold it as halo
  auto publish = [&](int64_t row, const VT* uv) {
    if constexpr (GRID) {
#pragma unroll
      for (int k = 0; k < UW; k++) {
        if constexpr (sizeof(VT) == 8) {
          st_unit(a.ubuf + row * UW + k, (unsigned long long)__double_as_longlong(uv[k]), epoch);
        } else {
          auto w = [&](int s) {
            return (unsigned long long)(s < NC ? __float_as_uint(uv[s < NC ? s : 0]) : 0u);
          };
          st_unit(a.ubuf + row * UW + k, w(3 * k) | w(3 * k + 1) << 32,
                  w(3 * k + 2) | (unsigned long long)epoch << 32);
        }
      }
    }
  };
  if (warp == 0) cc_tm_alloc(&s_taddr);
  if (tid == 0) {
    s_gave_up = 0;
    for (int k = 0; k < 3; k++) mb_init(&s_mb[k], 1);
    if constexpr (!GRID) mb_init(&s_mb[3], C + (a.wait_missing ? 1u : 0u));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if constexpr (GRID)
    __syncthreads();
  else
    cl_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tm = s_taddr + ((uint32_t)(32 * (warp & 3)) << 16) + 128u * (uint32_t)(warp >> 2);
  uint32_t ph_part = 0, ph_halo = 0;  // mbarrier phases: bit b of ph_part for buffer b
  uint32_t buf = 0;
  bool alive = true;
  {
    const int sys = GRID ? 0 : a.order[cl_id()];
    const CcgPart part = a.parts[GRID ? (int64_t)rank : (int64_t)cl_id() * C + rank];
    const int nrows = part.nrows;
    const int64_t row0 = part.row0;
    // ---- this part's tables: byte offsets into s_dyn, 16-byte granules; -1: no room (the
    // data stays in L2)
    int top = 2 * 16 * 16 * (int)sizeof(double) + a.win_cap * RB;
    auto carve = [&](int bytes) -> int {
      bytes = (bytes + 15) & ~15;
      if (top + bytes > a.dyn_bytes) return -1;
      const int at = top;
      top += bytes;
      return at;
    };
    VT* const s_w = reinterpret_cast<VT*>(s_dyn + carve(padded(nrows) * RB));
    int32_t* const s_sl = reinterpret_cast<int32_t*>(s_dyn + carve(4 * (part.nslices + 1)));
    // the rows to push (GRID: the halo rows to poll)
    uint32_t* const s_push = reinterpret_cast<uint32_t*>(s_dyn + carve(4 * part.npush));
    const int o_diag = a.diag ? carve(padded(nrows) * RB) : -1;
    const int o_col = carve(2 * part.entries);
    const uint16_t* const g_col = a.loc_col + part.entry_off;
    for (int i = tid; i <= part.nslices; i += CC_T) s_sl[i] = a.slices[part.slice_off + i];
    for (int i = tid; i < part.npush; i += CC_T)
      s_push[i] = GRID ? (uint32_t)a.halo[part.push_off + i] : a.push[part.push_off + i];
    if (o_col >= 0)
      for (int i = tid; i < part.entries / 8; i += CC_T)
        reinterpret_cast<uint4*>(s_dyn + o_col)[i] = reinterpret_cast<const uint4*>(g_col)[i];
    if (o_diag >= 0) {
      VT* const d = reinterpret_cast<VT*>(s_dyn + o_diag);
      if constexpr (PL) {
        for (int i = tid; i < nrows; i += CC_T) {
          VT t[LD];
          ldv<VT, LD>(a.diag, row0 + i, t);
          w_st(d, i, t);
        }
      } else {
        for (int i = tid; i < nrows * LD; i += CC_T) d[i] = a.diag[row0 * LD + i];
      }
    }
    __syncthreads();
    const int v0 = s_sl[part.val_slice];  // first entry whose value is not in tensor memory
    const int o_val = o_col >= 0 ? carve((int)sizeof(VT) * (part.entries - v0)) : -1;
    VT* const s_val = reinterpret_cast<VT*>(s_dyn + o_val);
    VT* const g_val = a.packed + part.entry_off;  // used only where o_val < 0

    // ---- inner values into place (a Dirichlet row's values are 0: its u is 0)
    for (int i = 0, sl = warp; sl < part.nslices; i++, sl += CC_W) {
      const int base = s_sl[sl], nk = (s_sl[sl + 1] - base) >> 5;
      const int lr = sl * 32 + lane;
      const int64_t row = row0 + lr;
      int p0 = 0, len = 0;
      if (lr < nrows && !(a.A64.bc && a.A64.bc[row])) {
        p0 = a.A64.indptr[row];
        len = a.A64.indptr[row + 1] - p0;
      }
      const int g0 = a.sK ? a.sell_slice[(row0 >> 5) + sl] + lane : 0;
      auto value = [&](int k) -> VT {
        if (k >= len) return VT(0);
        return a.sK ? a.sK[g0 + k * 32] : a.inK[p0 + k];
      };
      if (sl < part.val_slice) {
        constexpr int NV16 = 16 / VW;  // values of one 16-column store
#pragma unroll
        for (int h = 0; h < VW; h++) {
          uint32_t v[16];
#pragma unroll
          for (int k = 0; k < NV16; k++) {
            const VT t = value(h * NV16 + k);
            memcpy(&v[k * VW], &t, sizeof(VT));
          }
          cc_tm_st16(tm + 16u * (uint32_t)(VW * i + h), v);
        }
      } else {
        for (int k = 0; k < nk; k++) {
          const int e = base + 128 * (k >> 2) + 4 * lane + (k & 3);
          const VT t = value(k);
          if (o_val >= 0)
            s_val[e - v0] = t;
          else
            g_val[e] = t;
        }
      }
    }
    cc_tm_wait_st();

    // rows of this thread: slice warp + 16 i, lane.  In registers, or (PL) in tensor memory:
    // loads (all lanes, then vec_wait) and stores are copies, a register form's cost nothing.
    struct Vec {
      VT r[NC], p[NC], q[NC], xi[NC], dv[NC];
    };
    constexpr bool DV = PL && NC <= 3;  // D^-1 in tensor memory
    Vec vec[PL ? 1 : RPT] = {};
    VT dvr[PL && !DV ? RPT : 1][NC];
    const uint32_t tv0 = tm + 64u;
    auto vec_ld = [&](int i, uint32_t t[16]) {
      if constexpr (PL) cc_tm_ld16(tv0 + 16u * (uint32_t)i, t);
    };
    auto vec_get = [&](int i, const uint32_t t[16], Vec& v) {
      if constexpr (PL) {
#pragma unroll
        for (int s = 0; s < NC; s++) {
          v.r[s] = __uint_as_float(t[4 * s]);
          v.p[s] = __uint_as_float(t[4 * s + 1]);
          v.q[s] = __uint_as_float(t[4 * s + 2]);
          v.xi[s] = __uint_as_float(t[4 * s + 3]);
          if constexpr (DV)
            v.dv[s] = __uint_as_float(t[(12 + s) & 15]);
          else
            v.dv[s] = dvr[i][s];
        }
      } else {
        v = vec[i];
      }
    };
    auto vec_put = [&](int i, const Vec& v) {
      if constexpr (PL) {
        uint32_t t[16];
        t[15] = 0u;
#pragma unroll
        for (int s = 0; s < NC; s++) {
          t[4 * s] = __float_as_uint(v.r[s]);
          t[4 * s + 1] = __float_as_uint(v.p[s]);
          t[4 * s + 2] = __float_as_uint(v.q[s]);
          t[4 * s + 3] = __float_as_uint(v.xi[s]);
          if constexpr (DV) t[(12 + s) & 15] = __float_as_uint(v.dv[s]);
        }
        cc_tm_st16(tv0 + 16u * (uint32_t)i, t);
      } else {
        vec[i] = v;
      }
    };
    auto vec_wait = [&]() {
      if constexpr (PL) cc_tm_wait_ld();
    };
    // ---- Jacobi diagonal (FP64 values) through s_w; Dirichlet values into x
    for (int sl = warp; sl < part.nslices; sl += CC_W) {
      const int lr = sl * 32 + lane;
      if (lr < nrows) {
        const int64_t row = row0 + lr;
        VT d[LD];
        const bool bcr = a.A64.bc && a.A64.bc[row];
        double kd = 0.0;
        if (!bcr)
          for (int e = a.A64.indptr[row]; e < a.A64.indptr[row + 1]; e++)
            if (a.A64.indices[e] == row) kd = a.A64.K[e];
#pragma unroll
        for (int s = 0; s < LD; s++) {
          double t = a.A64.dscale[s] * kd;
          if (a.A64.diag) t += a.A64.diag[row * LD + s];
          d[s] = (s < S && !bcr && t != 0.0) ? VT(1.0 / t) : VT(0);
          if (bcr) a.x[row * LD + s] = a.b[row * LD + s];
        }
        w_st(s_w, lr, d);
        VT z[LD];
#pragma unroll
        for (int s = 0; s < LD; s++) z[s] = VT(0);
        w_st(s_win, lr, z);
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      const int lr = (warp + i * CC_W) * 32 + lane;
      VT t[LD];
#pragma unroll
      for (int s = 0; s < LD; s++) t[s] = VT(0);
      if (lr < nrows) w_ld(s_w, lr, t);
      Vec v;
#pragma unroll
      for (int s = 0; s < NC; s++) {
        v.r[s] = v.p[s] = v.q[s] = v.xi[s] = VT(0);
        v.dv[s] = t[s];
        if constexpr (PL && !DV) dvr[i][s] = t[s];
      }
      vec_put(i, v);
    }
    if constexpr (PL) cc_tm_wait_st();

    // lane state: lane s < S of warp 0 holds column s (the same bits in every CTA)
    const int col = lane & 3;
    const bool is_col = lane < 4 && col < S;
    double st_alpha = 0.0, st_beta = 0.0, st_rmax2 = 0.0, st_tol2 = 0.0,
           st_bb = 0.0, st_rtrue = 0.0;
    // 1 / rz and 1 / alpha of the last step (0: none yet); their product would leave the FP64
    // range for r.D^-1 r below 1e-154 or above 1e154
    double inv_rz = 0.0, inv_al = 0.0;
    // STILL: at the tolerance, until a sweep confirms it
    enum : int { DONE = 0, RUNS = 1, STILL = 2 };
    int st_act = DONE, st_status = TP_OK, st_iters = 0;
    unsigned tr_mask = (1u << S) - 1;  // columns refreshed by the next FP64 sweep
    bool refresh = true, first = true, fin = false;
    int one = -1;  // ONE: the only column that still runs (the others stand still), or -1
    int it = 0, n_rel = 0;

    for (;;) {
      double acc[2 * NC];  // r.u | r.r
#pragma unroll
      for (int k = 0; k < 2 * NC; k++) acc[k] = 0.0;
      if (refresh) {
        // ---- x += xi, then r = b - A x in FP64 (r through s_w)
#pragma unroll
        for (int i = 0; i < RPT; i++) {
          const int lr = (warp + i * CC_W) * 32 + lane;
          uint32_t tw[16];
          Vec v;
          vec_ld(i, tw);
          vec_wait();
          vec_get(i, tw, v);
          if (lr < nrows) {
            const int64_t row = row0 + lr;
            VT t[LD];
#pragma unroll
            for (int s = 0; s < LD; s++) t[s] = s < NC ? v.r[s < NC ? s : 0] : VT(0);
            w_st(s_w, lr, t);
#pragma unroll
            for (int s = 0; s < NC; s++) {
              if (((tr_mask >> s) & 1) && !first) a.x[row * LD + s] += (double)v.xi[s];
              if ((tr_mask >> s) & 1) v.xi[s] = VT(0);
            }
          }
          vec_put(i, v);
        }
        if constexpr (PL) cc_tm_wait_st();
        x_sync();
        // a slice at a time: 8 lanes walk a row (coalesced index and value loads, 4 rows per
        // step, the steps' loads in flight together), the sums go to the rows' own lanes
        double rr[NC], bb[NC];
#pragma unroll
        for (int s = 0; s < NC; s++) rr[s] = bb[s] = 0.0;
#pragma unroll 1
        for (int sl = warp; sl < part.nslices; sl += CC_W) {
          const int lr = sl * 32 + lane;
          const bool in = lr < nrows;
          const int64_t row = row0 + min(lr, nrows - 1);
          const bool bcr = in && a.A64.bc && a.A64.bc[row];
          int p0 = a.A64.indptr[row], p1 = a.A64.indptr[row + 1];
          if (!in || bcr) p1 = p0;
          double xr[LD], ax[NC];
          ldv_cg<double, LD>(a.x, row, xr);
#pragma unroll
          for (int s = 0; s < NC; s++) ax[s] = 0.0;
          constexpr int UG = LD == 1 ? 4 : (LD == 2 ? 2 : 1);
#pragma unroll UG
          for (int g = 0; g < 8; g++) {
            const int src = 4 * g + (lane >> 3);
            const int q0 = __shfl_sync(0xffffffffu, p0, src), q1 = __shfl_sync(0xffffffffu, p1, src);
            double t[NC];
#pragma unroll
            for (int s = 0; s < NC; s++) t[s] = 0.0;
            const int e = q0 + (lane & 7);
            // two entries per lane (rows of up to 16), past the row's end with value 0
            const bool i0 = e < q1, i1 = e + 8 < q1;
            const int j0 = i0 ? __ldg(a.A64.indices + e) : (int)row0;
            const int j1 = i1 ? __ldg(a.A64.indices + e + 8) : (int)row0;
            const double k0 = i0 ? __ldg(a.A64.K + e) : 0.0;
            const double k1 = i1 ? __ldg(a.A64.K + e + 8) : 0.0;
            double x0[LD], x1[LD];
            ldv_cg<double, LD>(a.x, j0, x0);
            ldv_cg<double, LD>(a.x, j1, x1);
#pragma unroll
            for (int s = 0; s < NC; s++) {
              if (i0) t[s] = k0 * x0[s];
              if (i1) t[s] += k1 * x1[s];
            }
            for (int f = e + 16; f < q1; f += 8) {
              const double kv = __ldg(a.A64.K + f);
              ldv_cg<double, LD>(a.x, __ldg(a.A64.indices + f), x0);
#pragma unroll
              for (int s = 0; s < NC; s++) t[s] += kv * x0[s];
            }
#pragma unroll
            for (int s = 0; s < NC; s++) {
#pragma unroll
              for (int o = 4; o > 0; o >>= 1) t[s] += __shfl_xor_sync(0xffffffffu, t[s], o);
              const double v = __shfl_sync(0xffffffffu, t[s], (lane & 3) * 8);
              if ((lane >> 2) == g) ax[s] = v;
            }
          }
          if (in) {
            VT rv[LD];
            w_ld(s_w, lr, rv);
#pragma unroll
            for (int s = 0; s < NC; s++) {
              const double dd = (a.A64.diag && !bcr) ? a.A64.diag[row * LD + s] : 0.0;
              const double av = bcr ? xr[s] : a.A64.dscale[s] * ax[s] + dd * xr[s];
              const double bv = (s < S) ? a.b[row * LD + s] : 0.0;
              const double r64 = (s < S) ? bv - av : 0.0;
              bb[s] += bv * bv;
              if (fin || ((tr_mask >> s) & 1)) rr[s] += r64 * r64;
              if (!fin && ((tr_mask >> s) & 1)) rv[s] = (VT)r64;
            }
            w_st(s_w, lr, rv);
          }
        }
        if (first) {
#pragma unroll
          for (int s = 0; s < NC; s++) {
            const double t = warp_sum(bb[s]);
            if (lane == 0) s_red[warp][12 + s] = t;
          }
        }
#pragma unroll
        for (int s = 0; s < NC; s++) acc[NC + s] = rr[s];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < RPT; i++) {
          const int lr = (warp + i * CC_W) * 32 + lane;
          uint32_t tw[16];
          Vec v;
          vec_ld(i, tw);
          vec_wait();
          vec_get(i, tw, v);
          if (lr < nrows) {
            VT uv[LD], rv[LD];
            w_ld(s_win, lr, uv);
            w_ld(s_w, lr, rv);
#pragma unroll
            for (int s = 0; s < NC; s++) {
              v.r[s] = rv[s];
              if (!fin && ((tr_mask >> s) & 1)) uv[s] = v.dv[s] * v.r[s];
              acc[s] += (double)v.r[s] * (double)uv[s];
            }
            w_st(s_win, lr, uv);
            publish(row0 + lr, uv);
          }
          vec_put(i, v);
        }
        if constexpr (PL) cc_tm_wait_st();
      } else if (ONE && one >= 0) {
        // ---- the same for the one column that still runs
        if constexpr (ONE) {
          uint32_t tw[RPT][4], td[RPT];
#pragma unroll
          for (int i = 0; i < RPT; i++) {
            cc_tm_ld4(tv0 + 16u * (uint32_t)i + 4u * (uint32_t)one, tw[i]);
            if constexpr (DV) cc_tm_ld1(tv0 + 16u * (uint32_t)i + 12u + (uint32_t)one, td[i]);
          }
          const float al = s_al[one], be = s_be[one];
          cc_tm_wait_ld();
          // D^-1 of a register form
          auto sel = [&](const VT* v) {
            VT t = v[0];
#pragma unroll
            for (int s = 1; s < NC; s++) t = one == s ? v[s] : t;
            return t;
          };
#pragma unroll
          for (int i = 0; i < RPT; i++) {
            const int sl = warp + i * CC_W, lr = sl * 32 + lane;
            const int at = w_at(lr, one);
            float r = __uint_as_float(tw[i][0]), p = __uint_as_float(tw[i][1]),
                  q = __uint_as_float(tw[i][2]), xi = __uint_as_float(tw[i][3]);
            const float dv = DV ? __uint_as_float(td[i]) : sel(dvr[DV ? 0 : i]);
            if (lr < nrows) {
              p = s_win[at] + be * p;
              q = s_w[at] + be * q;
              xi += al * p;
              r -= al * q;
              const float u = dv * r;
              acc[0] += (double)r * (double)u;
              acc[1] += (double)r * (double)r;
              s_win[at] = u;
              st_unit(a.ubuf + (row0 + lr) * UW, (unsigned long long)__float_as_uint(u),
                      (unsigned long long)epoch << 32);
            }
            const uint32_t t[4] = {__float_as_uint(r), __float_as_uint(p), __float_as_uint(q),
                                   __float_as_uint(xi)};
            cc_tm_st4(tv0 + 16u * (uint32_t)i + 4u * (uint32_t)one, t);
          }
          cc_tm_wait_st();
        }
      } else {
        // ---- vector update with this iteration's alpha and beta
        VT al[NC], be[NC];
#pragma unroll
        for (int s = 0; s < NC; s++) {
          al[s] = s_al[s];
          be[s] = s_be[s];
        }
        uint32_t tw[PL ? RPT : 1][16];
        if constexpr (PL) {
#pragma unroll
          for (int i = 0; i < RPT; i++) vec_ld(i, tw[i]);
          vec_wait();
        }
#pragma unroll
        for (int i = 0; i < RPT; i++) {
          const int lr = (warp + i * CC_W) * 32 + lane;
          Vec v;
          vec_get(i, tw[PL ? i : 0], v);
          if (lr < nrows) {
            VT uv[LD], wv[LD];
            w_ld(s_win, lr, uv);
            w_ld(s_w, lr, wv);
#pragma unroll
            for (int s = 0; s < NC; s++) {
              v.p[s] = uv[s] + be[s] * v.p[s];
              v.q[s] = wv[s] + be[s] * v.q[s];
              v.xi[s] += al[s] * v.p[s];
              v.r[s] -= al[s] * v.q[s];
              uv[s] = v.dv[s] * v.r[s];
              acc[s] += (double)v.r[s] * (double)uv[s];
              acc[NC + s] += (double)v.r[s] * (double)v.r[s];
            }
            w_st(s_win, lr, uv);
            publish(row0 + lr, uv);
          }
          vec_put(i, v);
        }
        if constexpr (PL) cc_tm_wait_st();
      }
      // ---- the rows other CTAs hold as halo, then (while they travel) this warp's r.u, r.r
      __syncthreads();
      if constexpr (!GRID) {
        if (tid == 0) mb_expect(&s_mb[2], (uint32_t)(part.nhalo * RB) + a.wait_missing);
        for (int i = tid; i < part.npush; i += CC_T) {
          const uint32_t e = s_push[i];
          const uint32_t src = e & ((1u << CC_SRC_BITS) - 1);
          const uint32_t slot = (e >> CC_SRC_BITS) & ((1u << CC_SLOT_BITS) - 1);
          const uint32_t dst = e >> (CC_SRC_BITS + CC_SLOT_BITS);
          cl_send_row<RB>(cl_map(s_win + (size_t)slot * LD, dst), s_win + (size_t)src * LD,
                          cl_map(&s_mb[2], dst));
        }
      }
      if (ONE && one >= 0) {
        const double v = WarpReduce<2>::run(acc, lane);
        const int id = WarpReduce<2>::value_of(lane);
        if (id >= 0) s_red[warp][4 * id + one] = v;
      } else {
        const double v = WarpReduce<2 * NC>::run(acc, lane);
        const int id = WarpReduce<2 * NC>::value_of(lane);
        if (id >= 0) s_red[warp][(id / NC) * 4 + id % NC] = v;
      }
      // a wait that runs out is acted on after a CTA barrier, by every thread
      if constexpr (GRID) {
        const uint32_t want = epoch + a.wait_missing;
        constexpr int U = UW == 1 ? 8 : (UW == 2 ? 4 : 2);
        if (ONE && one >= 0) {
          for (int i0 = tid; i0 < part.nhalo; i0 += 8 * CC_T) {
            ulonglong2 v[8];
            const ulonglong2* src[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
              src[k] = a.ubuf + (int64_t)s_push[min(i0 + k * CC_T, part.nhalo - 1)] * UW;
              v[k] = ld_unit(src[k]);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
              if (i0 + k * CC_T < part.nhalo) {
                if (!poll_unit<TAG>(src[k], v[k], want, a.wait_limit_ns, &s_gave_up)) s_gave_up = GAVE_UP;
                const int i = nrows + i0 + k * CC_T;
                const uint32_t w = (uint32_t)v[k].x;
                memcpy(s_win + w_at(i, one), &w, 4);
              }
            }
          }
        } else
        for (int i0 = tid; i0 < part.nhalo; i0 += U * CC_T) {
          ulonglong2 v[U][UW];
          const ulonglong2* src[U];
#pragma unroll
          for (int k = 0; k < U; k++) {
            const int i = min(i0 + k * CC_T, part.nhalo - 1);
            src[k] = a.ubuf + (int64_t)s_push[i] * UW;
#pragma unroll
            for (int j = 0; j < UW; j++) v[k][j] = ld_unit(src[k] + j);
          }
#pragma unroll
          for (int k = 0; k < U; k++) {
            if (i0 + k * CC_T < part.nhalo) {
              VT uv[LD];
#pragma unroll
              for (int s = 0; s < LD; s++) uv[s] = VT(0);
#pragma unroll
              for (int j = 0; j < UW; j++) {
                if (!poll_unit<TAG>(src[k] + j, v[k][j], want, a.wait_limit_ns, &s_gave_up))
                  s_gave_up = GAVE_UP;
                if constexpr (sizeof(VT) == 8) {
                  uv[j] = __longlong_as_double((long long)v[k][j].x);
                } else {
                  const uint32_t w[3] = {(uint32_t)v[k][j].x, (uint32_t)(v[k][j].x >> 32),
                                         (uint32_t)v[k][j].y};
#pragma unroll
                  for (int s = 0; s < 3; s++)
                    if (3 * j + s < LD) uv[3 * j + s] = __uint_as_float(w[s]);
                }
              }
              w_st(s_win, nrows + i0 + k * CC_T, uv);
            }
          }
        }
        __syncthreads();
      } else {
        if (!mb_wait(&s_mb[2], ph_halo, a.wait_limit_ns)) s_gave_up = GAVE_UP;
        ph_halo ^= 1u;
      }

      // ---- w = A u from the window; w.u
      double wu[NC];
#pragma unroll
      for (int s = 0; s < NC; s++) wu[s] = 0.0;
      // columns are byte offsets into the window (GRID: its entries; PL: its words).
      // N: columns computed, NC or (one column left) 1
      constexpr uint32_t CU = PL ? 4 : (GRID ? RB : 1);
      const unsigned char* const s_winb =
          reinterpret_cast<const unsigned char*>(s_win) + (ONE && one >= 0 ? 4 * w_at(0, one) : 0);
      auto gather4 = [&](auto N, uint2 c, const VT* v, VT* ak, VT* ak2) {
        const uint32_t cc[4] = {c.x & 0xffffu, c.x >> 16, c.y & 0xffffu, c.y >> 16};
        if constexpr (PL) {
          constexpr int n = decltype(N)::value;
          VT u[4][n];
#pragma unroll
          for (int k = 0; k < 4; k++)
#pragma unroll
            for (int s = 0; s < n; s++)
              u[k][s] = reinterpret_cast<const VT*>(s_winb + cc[k] * CU)[32 * s];
#pragma unroll
          for (int k = 0; k < 4; k++) {
            VT* const y = (k & 1) ? ak2 : ak;
            if constexpr (n >= 2) axpy_row<VT, 2>(v[k], u[k], y);
            if constexpr (n == 4) axpy_row<VT, 2>(v[k], u[k] + 2, y + 2);
            if constexpr (n & 1) y[n - 1] += v[k] * u[k][n - 1];
          }
        } else {
          VT u[4][LD];
#pragma unroll
          for (int k = 0; k < 4; k++)
            lds_row<VT, LD>(reinterpret_cast<const VT*>(s_winb + cc[k] * CU), 0, u[k]);
          axpy_row<VT, LD>(v[0], u[0], ak);
          axpy_row<VT, LD>(v[1], u[1], ak2);
          axpy_row<VT, LD>(v[2], u[2], ak);
          axpy_row<VT, LD>(v[3], u[3], ak2);
        }
      };
      auto row_done = [&](auto N, int sl, const VT* ak, const VT* ak2) {
        const int lr = sl * 32 + lane;
        if (lr >= nrows) return;
        if constexpr (ONE && decltype(N)::value == 1) {
          const int at = w_at(lr, one);
          const VT ur = s_win[at];
          VT dg = VT(0);
          if (o_diag >= 0)
            dg = reinterpret_cast<const VT*>(s_dyn + o_diag)[at];
          else if (a.diag)
            dg = a.diag[(row0 + lr) * LD + one];
          const VT wv = VT(a.A64.dscale[one]) * (ak[0] + ak2[0]) + dg * ur;
          wu[0] += (double)wv * (double)ur;
          s_w[at] = wv;
        } else {
          VT ur[LD], dg[LD], wv[LD];
          w_ld(s_win, lr, ur);
          if (o_diag >= 0) {
            w_ld(reinterpret_cast<const VT*>(s_dyn + o_diag), lr, dg);
          } else {
#pragma unroll
            for (int s = 0; s < LD; s++) dg[s] = VT(0);
            if (a.diag) ldv<VT, LD>(a.diag, row0 + lr, dg);
          }
#pragma unroll
          for (int s = 0; s < (PL ? NC : LD); s++) {
            wv[s] = VT(a.A64.dscale[s]) * (ak[s] + ak2[s]) + dg[s] * ur[s];
            if (s < NC) wu[s] += (double)wv[s] * (double)ur[s];
          }
          w_st(s_w, lr, wv);
        }
      };
      // slices in tensor memory: NS of the warp side by side (their loads and gathers
      // overlap); SC: columns in shared memory
      auto tm_slices = [&](auto N, auto NSC, auto SC, int i, int sl) {
        constexpr int n = PL ? decltype(N)::value : LD;
        constexpr int NS = decltype(NSC)::value;
        constexpr int NG = 4 / VW;  // chunks of 4 entries per 16 tensor-memory columns
        VT ak[NS][n], ak2[NS][n];
#pragma unroll
        for (int j = 0; j < NS; j++)
#pragma unroll
          for (int s = 0; s < n; s++) ak[j][s] = ak2[j][s] = VT(0);
#pragma unroll
        for (int h = 0; h < VW; h++) {
          uint32_t tv[NS][16];
          uint2 c[NS][NG];
#pragma unroll
          for (int j = 0; j < NS; j++)
            cc_tm_ld16(tm + 16u * (uint32_t)(VW * (i + j) + h), tv[j]);
#pragma unroll
          for (int j = 0; j < NS; j++)
#pragma unroll
            for (int g = 0; g < NG; g++) {
              const int e = (sl + j * CC_W) * 512 + 4 * lane + 128 * (h * NG + g);
              if constexpr (decltype(SC)::value)
                c[j][g] = *reinterpret_cast<const uint2*>(s_dyn + o_col + 2 * e);
              else
                c[j][g] = __ldg(reinterpret_cast<const uint2*>(g_col + e));
            }
          cc_tm_wait_ld();
#pragma unroll
          for (int j = 0; j < NS; j++) {
            VT v[4 * NG];
            memcpy(v, tv[j], sizeof(v));
#pragma unroll
            for (int g = 0; g < NG; g++) gather4(N, c[j][g], v + 4 * g, ak[j], ak2[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < NS; j++) row_done(N, sl + j * CC_W, ak[j], ak2[j]);
      };
      // two where the rows' vectors leave the registers
      constexpr int NS2 = (PL && NC == 3) || (RB <= 8 && RPT <= 2) ? 2 : 1;
      auto product = [&](auto N) {
        int i = 0, sl = warp;
        if (o_col >= 0) {
          if constexpr (NS2 > 1) {
#pragma unroll 1
            for (; sl + CC_W < part.val_slice; i += 2, sl += 2 * CC_W)
              tm_slices(N, std::integral_constant<int, NS2>{}, std::true_type{}, i, sl);
          }
#pragma unroll 1
          for (; sl < part.val_slice; i++, sl += CC_W)
            tm_slices(N, std::integral_constant<int, 1>{}, std::true_type{}, i, sl);
        } else {
#pragma unroll 1
          for (; sl < part.val_slice; i++, sl += CC_W)
            tm_slices(N, std::integral_constant<int, 1>{}, std::false_type{}, i, sl);
        }
#pragma unroll 1
        for (; sl < part.nslices; sl += CC_W) {
          const int base = s_sl[sl], nc = (s_sl[sl + 1] - base) >> 7;  // chunks of 4 entries
          constexpr int n = PL ? decltype(N)::value : LD;
          VT ak[n], ak2[n];
#pragma unroll
          for (int s = 0; s < n; s++) ak[s] = ak2[s] = VT(0);
#pragma unroll 4
          for (int g = 0; g < nc; g++) {
            const int e = base + 4 * lane + 128 * g;
            VT v[4];
            if (o_val >= 0) {
              memcpy(v, __builtin_assume_aligned(s_val + (e - v0), 16), sizeof(v));
            } else {
#pragma unroll
              for (int k = 0; k < VW; k++) {
                const uint4 t = __ldcg(reinterpret_cast<const uint4*>(g_val + e) + k);
                memcpy(reinterpret_cast<char*>(v) + 16 * k, &t, 16);
              }
            }
            const uint2 c = o_col >= 0 ? *reinterpret_cast<const uint2*>(s_dyn + o_col + 2 * e)
                                       : __ldg(reinterpret_cast<const uint2*>(g_col + e));
            gather4(N, c, v, ak, ak2);
          }
          row_done(N, sl, ak, ak2);
        }
      };
      if (ONE && one >= 0)
        product(std::integral_constant<int, 1>{});
      else
        product(std::integral_constant<int, NC>{});

      // ---- sums over the CTA, then to every CTA of the cluster
      {
        if (ONE && one >= 0) {
          const double v = warp_sum(wu[0]);
          if (lane == 0) s_red[warp][8 + one] = v;
        } else {
          const double v = WarpReduce<NC>::run(wu, lane);
          const int id = WarpReduce<NC>::value_of(lane);
          if (id >= 0) s_red[warp][8 + id] = v;
        }
        __syncthreads();
        // a CTA that gave up sends no sums, so no other completes this pass either
        if (s_gave_up == GAVE_UP) {
          alive = false;
          break;
        }
        const int slot = tid & 15;
        const uint32_t dst = (uint32_t)(tid >> 4);
        const bool used = ONE && one >= 0 ? (slot & 3) == one && slot < 12
                                         : (slot & 3) < NC && (slot < 12 || first);
        if (GRID ? (dst == 0 && used) : (dst < C && used)) {
          double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
          for (int g = 0; g < CC_W; g++) t[g & 3] += s_red[g][slot];
          const double v = (t[0] + t[1]) + (t[2] + t[3]);
          if constexpr (GRID)
            st_unit(a.sums + ((int64_t)buf * C + rank) * 16 + slot,
                    (unsigned long long)__double_as_longlong(v), epoch);
          else
            cl_send(cl_map(s_part + (buf * 16 + rank) * 16 + slot, dst), v,
                    cl_map(&s_mb[buf], dst));
        }
        if constexpr (!GRID) {
          if (tid == 0)
            mb_expect(&s_mb[buf], C * (uint32_t)((first ? 4 : 3) * NC * sizeof(double)) +
                                      a.wait_missing);
        } else {
          // group g of 32 adds the sums of CTAs g, g + 32, ... (up to 5 loads in flight)
          const int g = tid >> 4;
          double t2 = 0.0;
          if (used) {
            const ulonglong2* src = a.sums + ((int64_t)buf * C + g) * 16 + slot;
            for (int b0 = g; b0 < (int)C; b0 += 5 * 32, src += 5 * 32 * 16) {
              ulonglong2 u[5];
#pragma unroll
              for (int k = 0; k < 5; k++)
                if (b0 + 32 * k < (int)C) u[k] = ld_unit(src + 32 * 16 * k);
#pragma unroll
              for (int k = 0; k < 5; k++) {
                if (b0 + 32 * k < (int)C) {
                  if (!poll_unit<0>(src + 32 * 16 * k, u[k], epoch, a.wait_limit_ns, &s_gave_up))
                    s_gave_up = GAVE_UP_SUMS;
                  t2 += __longlong_as_double((long long)u[k].x);
                }
              }
            }
          }
          s_part[tid] = t2;
          __syncthreads();
        }
      }
      // ---- warp 0: totals (lanes l and l + 16 sum half of the CTAs each), lane decisions
      if (warp == 0) {
        if constexpr (!GRID)
          if (!mb_wait(&s_mb[buf], (ph_part >> buf) & 1u, a.wait_limit_ns))
            s_gave_up = GAVE_UP_SUMS;
        double tot;
        if constexpr (GRID) {
          const double* pp = s_part + (lane & 15) + (lane >> 4) * 16 * 16;
          double t[16];
#pragma unroll
          for (int g = 0; g < 16; g++) t[g] = pp[g * 16];
#pragma unroll
          for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int g = 0; g < o; g++) t[g] += t[g + o];
          tot = t[0] + __shfl_xor_sync(0xffffffffu, t[0], 16);
        } else {
          const double* pp = s_part + buf * 256 + (lane & 15) + ((lane >> 4) ? 8 * 16 : 0);
          const int nc = (lane >> 4) ? (int)C - 8 : min((int)C, 8);
          double t[8];
#pragma unroll
          for (int g = 0; g < 8; g++) t[g] = (g < nc) ? pp[g * 16] : 0.0;
          tot = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
          tot += __shfl_xor_sync(0xffffffffu, tot, 16);
        }
        const double gm = __shfl_sync(0xffffffffu, tot, col);
        const double rr = __shfl_sync(0xffffffffu, tot, 4 + col);
        const double dl = __shfl_sync(0xffffffffu, tot, 8 + col);
        // beta = gamma / gamma_old, alpha = gamma / (delta - beta gamma / alpha_old): the
        // rules of cg_coefficients (tp_pcg.cu) with the reciprocals of the last step's values
        auto coefficients = [&](double den, double beta) {
          st_beta = beta;
          const double inv = 1.0 / gm;
          st_alpha = gm / den;
          inv_rz = inv;
          inv_al = den * inv;
        };
        const double den0 = dl - (gm * inv_rz) * (gm * inv_al);
        // the common step: every running lane goes on, nothing to decide
        const bool runs = is_col && st_act == RUNS;
        const bool plain = rr > st_tol2 && !(rr < a.delta2 * st_rmax2) && rr < 1e300 &&
                           gm > 0.0 && gm < 1e300 && dl > 0.0 && den0 > 0.0 && den0 < 1e300;
        if (!refresh && it + 1 < a.max_it && !__any_sync(0xffffffffu, runs && !plain) &&
            __any_sync(0xffffffffu, runs)) {
          it++;
          if (runs) coefficients(den0, gm * inv_rz);
          if (lane < 4) {
            s_al[lane] = runs ? (VT)st_alpha : VT(0);
            s_be[lane] = runs ? (VT)st_beta : VT(0);
          }
          const unsigned run = __ballot_sync(0xffffffffu, runs);
          if (lane == 0) {
            s_ctl = 0;
            s_run = (int)run;
          }
        } else {
        const bool fine = isfinite(gm) && isfinite(rr) && isfinite(dl);
        bool coef = false;  // this lane takes new coefficients
        int ctl = 0;
        if (!refresh) {
          it++;
          bool trig = false;
          if (runs) {
            if (!fine) {
              st_act = 0;
              st_status = TP_ERR_NONFINITE;
              st_iters = it;
            } else if (rr <= st_tol2) {
              st_act = STILL;
            } else {
              trig = a.delta2 > 0.0 && rr < a.delta2 * st_rmax2;
            }
          }
          const unsigned run = __ballot_sync(0xffffffffu, is_col && st_act == RUNS);
          const unsigned act = __ballot_sync(0xffffffffu, is_col && st_act);
          if (__any_sync(0xffffffffu, trig) || (act && !run)) {
            ctl = CTL_REFRESH;
            tr_mask = act;
          } else {
            coef = is_col && st_act == RUNS;
          }
        } else if (first) {
          const double bb = __shfl_sync(0xffffffffu, tot, 12 + col);
          if (is_col) {
            const double rt = a.rtol[(int64_t)sys * S + col];
            st_bb = bb;
            st_tol2 = rt * rt * bb;
            st_rtrue = st_rmax2 = rr;
            const bool f = isfinite(rr) && isfinite(gm);
            st_act = f && rr > st_tol2 ? RUNS : DONE;
            st_status = !f ? TP_ERR_NONFINITE : (st_act ? -1 : TP_OK);
            if (st_act && !isfinite(dl)) {
              st_act = 0;
              st_status = TP_ERR_NONFINITE;
            }
            coef = st_act;
          }
        } else if (fin) {
          if (is_col) {
            st_rtrue = rr;
            if (st_status == -1) {
              st_status = rr <= st_tol2 ? TP_OK : TP_ERR_NOT_CONVERGED;
              st_iters = it;
            }
          }
          ctl = CTL_EXIT;
        } else {
          n_rel++;
          if (is_col && ((tr_mask >> col) & 1)) {
            st_rtrue = rr;
            if (!fine) {
              st_act = 0;
              st_status = TP_ERR_NONFINITE;
              st_iters = it;
            } else if (rr <= st_tol2) {
              st_act = 0;
              st_status = TP_OK;
              st_iters = it;
            } else {
              st_rmax2 = rr;
              coef = true;
            }
          }
        }
        if (coef) {
          if (!(dl > 0.0)) {
            st_act = 0;
            st_status = TP_ERR_BREAKDOWN;
            st_iters = it;
          } else if (den0 > 0.0 && st_act == RUNS) {
            coefficients(den0, gm * inv_rz);
          } else {
            // the direction restarts along u: rounding, or a column that stood still, whose p
            // and q are overwritten meanwhile
            coefficients(dl, 0.0);
            st_act = RUNS;
          }
        }
        const unsigned act = __ballot_sync(0xffffffffu, is_col && st_act);
        if (!(ctl & CTL_EXIT) && (!act || (it >= a.max_it && !(ctl & CTL_REFRESH)))) {
          // every lane confirmed by a sweep: x and the residuals are final; otherwise x +=
          // xi of every lane and one FP64 residual
          const unsigned bad =
              __ballot_sync(0xffffffffu, is_col && (st_act || st_status != TP_OK));
          ctl = bad ? CTL_REFRESH | CTL_FIN : CTL_EXIT;
          tr_mask = (1u << S) - 1;
        }
        const bool go = is_col && st_act == RUNS;
        if (lane < 4) {
          s_al[lane] = go ? (VT)st_alpha : VT(0);
          s_be[lane] = go ? (VT)st_beta : VT(0);
        }
        const unsigned run = __ballot_sync(0xffffffffu, go);
        if (lane == 0) {
          s_ctl = ctl;
          s_mask = (int)tr_mask;
          s_run = (int)run;
        }
        }
      }
      ph_part ^= 1u << buf;
      buf ^= 1u;
      epoch++;
      __syncthreads();
      if (s_gave_up == GAVE_UP_SUMS) {
        alive = false;
        break;
      }
      const int ctl = s_ctl;
      if (ctl & CTL_EXIT) break;
      first = false;
      refresh = (ctl & CTL_REFRESH) != 0;
      fin = (ctl & CTL_FIN) != 0;
      tr_mask = (unsigned)s_mask;
      if constexpr (ONE) one = !refresh && __popc(s_run) == 1 ? __ffs(s_run) - 1 : -1;
    }

    if (rank == 0 && warp == 0) {
      if (!alive) st_status = TP_ERR_TIMEOUT;
      const unsigned m = __ballot_sync(0xffffffffu, is_col && st_status != TP_OK);
      const int worst = __shfl_sync(0xffffffffu, st_status, m ? __ffs(m) - 1 : 0);
      CcgOut* o = a.out + sys;
      if (lane < 4) {
        o->lane_iters[col] = is_col ? st_iters : 0;
        o->lane_status[col] = is_col ? st_status : TP_OK;
        o->lane_rtrue[col] = is_col ? st_rtrue : 0.0;
        o->lane_bb[col] = is_col ? st_bb : 0.0;
      }
      if (lane == 0) {
        o->iterations = it;
        o->n_reliable = n_rel;
        o->status = m ? worst : TP_OK;
      }
    }
  }
  // Nothing is in flight towards a CTA that finished its solve: it has received all that the
  // others sent.  After a wait that ran out their last sends may be: the CTA stays until no
  // other starts one (the barrier) and those in flight have landed.
  if constexpr (GRID) {
    __syncthreads();
  } else {
    cl_sync();
    if (!alive) {
      const unsigned long long t0 = cc_time();
      while (cc_time() - t0 < CC_DRAIN_NS) {
      }
    }
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(s_taddr));
}

// ----------------------------------------------------------------- tables (once)
// entries of every slice of a part (32 x its longest row, at least 16, rounded up to 4)
// and their running offset
__global__ void k_ccg_slices(CcgPart* parts, const int32_t* __restrict__ indptr,
                             int32_t* __restrict__ slices, int tm_slices) {
  CcgPart& p = parts[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t* out = slices + p.slice_off;
  for (int sl = warp; sl < p.nslices; sl += blockDim.x >> 5) {
    const int lr = sl * 32 + lane;
    int len = 0;
    if (lr < p.nrows) len = indptr[p.row0 + lr + 1] - indptr[p.row0 + lr];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
    if (lane == 0) out[sl + 1] = max((len + 3) & ~3, 16) * 32;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0, most = 0;
    out[0] = 0;
    for (int sl = 0; sl < p.nslices; sl++) {
      most = max(most, out[sl + 1]);
      out[sl + 1] = (run += out[sl + 1]);
    }
    p.entries = run;
    // tensor memory holds 16 values per row; a part with a longer row keeps all values
    // outside it
    p.val_slice = most > 16 * 32 ? 0 : min(p.nslices, tm_slices);
  }
}

// One block per part.  The halo as a bitmap over the system's rows (shared memory), so its
// ascending order and every column's window slot come from popcounts.  FILL = false: the
// halo size and, per rank, the halo positions where that rank's rows begin; window-local
// columns (times rb; planes > 0: words of a window in that many planes).  FILL = true: the push entries (rank of this part, slot, source row)
// into the producers' lists at push_at (per producer and consumer), or, when halo is given
// (GRID), the halo's rows at the part's push_off.
template <bool FILL>
__global__ void k_ccg_halo(CcgPart* parts, int C, const int32_t* __restrict__ sys_row0,
                           const int32_t* __restrict__ sys_rows,
                           const int32_t* __restrict__ indptr,
                           const int32_t* __restrict__ indices,
                           const int32_t* __restrict__ slices, int rb, int planes,
                           uint16_t* __restrict__ loc_col,
                           int32_t* __restrict__ bounds, const int32_t* __restrict__ push_at,
                           uint32_t* __restrict__ push, int32_t* __restrict__ halo,
                           int32_t* __restrict__ flag) {
  extern __shared__ uint32_t s_bits[];
  const int sys = blockIdx.x / C, rank = blockIdx.x % C;
  const CcgPart p = parts[blockIdx.x];
  const int n = sys_rows[sys], base = sys_row0[sys];
  const int nw = (n + 31) / 32;
  uint32_t* s_pre = s_bits + nw;
  const int own0 = p.row0 - base, own1 = own0 + p.nrows;
  for (int i = threadIdx.x; i < nw; i += blockDim.x) s_bits[i] = 0u;
  __syncthreads();
  const int e0 = p.nrows ? indptr[p.row0] : 0, e1 = p.nrows ? indptr[p.row0 + p.nrows] : 0;
  for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
    const int j = indices[e] - base;
    if (j < 0 || j >= n)
      *flag = 1;  // a column outside the system: not block diagonal
    else if (j < own0 || j >= own1)
      atomicOr(&s_bits[j >> 5], 1u << (j & 31));
  }
  __syncthreads();
  // exclusive popcount prefix: every warp scans a contiguous chunk, then the chunk totals
  __shared__ int s_tot[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int per = ((nw + W - 1) / W + 31) & ~31;
  int run = 0;
  for (int i0 = warp * per; i0 < min(nw, (warp + 1) * per); i0 += 32) {
    const int i = i0 + lane;
    const int c = (i < nw) ? __popc(s_bits[i]) : 0;
    int s = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    if (i < nw) s_pre[i] = run + s - c;
    run += __shfl_sync(0xffffffffu, s, 31);
  }
  if (lane == 0) s_tot[warp + 1] = run;
  __syncthreads();
  if (threadIdx.x == 0) {
    s_tot[0] = 0;
    for (int k = 1; k <= W; k++) s_tot[k] += s_tot[k - 1];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nw; i += blockDim.x) s_pre[i] += s_tot[i / per];
  __syncthreads();
  auto halo_pos = [&](int j) {
    return (int)s_pre[j >> 5] + __popc(s_bits[j >> 5] & ((1u << (j & 31)) - 1u));
  };
  const CcgPart* sp = parts + (int64_t)sys * C;
  if constexpr (!FILL) {
    for (int k = threadIdx.x; bounds && k <= C; k += blockDim.x) {
      // halo entries with a row below rank k's first row (ranks in row order)
      const int j = (k < C) ? min(sp[k].row0 - base, n) : n;
      bounds[(int64_t)blockIdx.x * (C + 1) + k] = (j < n) ? halo_pos(j) : s_tot[W];
    }
    if (threadIdx.x == 0) parts[blockIdx.x].nhalo = s_tot[W];
    const int32_t* sl_off = slices + p.slice_off;
    for (int sl = warp; sl < p.nslices; sl += W) {
      const int b = sl_off[sl], w = (sl_off[sl + 1] - b) >> 5;
      const int lr = sl * 32 + lane;
      int p0 = 0, len = 0;
      if (lr < p.nrows) {
        p0 = indptr[p.row0 + lr];
        len = indptr[p.row0 + lr + 1] - p0;
      }
      for (int k = 0; k < w; k++) {
        int c = (lr < p.nrows) ? lr : 0;  // padding: value 0
        if (k < len) {
          const int j = indices[p0 + k] - base;
          if (j >= 0 && j < n)
            c = (j >= own0 && j < own1) ? j - own0 : p.nrows + halo_pos(j);
        }
        loc_col[p.entry_off + b + 128 * (k >> 2) + 4 * lane + (k & 3)] = 
            (uint16_t)(planes ? (c >> 5) * 32 * planes + (c & 31) : c * rb);
      }
    }
  } else {
    for (int i = threadIdx.x; i < nw; i += blockDim.x) {
      uint32_t m = s_bits[i];
      while (m) {
        const int j = 32 * i + __ffs(m) - 1;
        m &= m - 1;
        if (halo) {
          halo[p.push_off + halo_pos(j)] = base + j;
          continue;
        }
        int lo = 0, hi = C;  // the last rank whose first row is <= j owns it
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (sp[mid].row0 - base <= j)
            lo = mid;
          else
            hi = mid;
        }
        const int h = halo_pos(j);
        const int at = push_at[((int64_t)sys * C + lo) * C + rank] + h -
                       bounds[(int64_t)blockIdx.x * (C + 1) + lo];
        const uint32_t src = (uint32_t)(j - (sp[lo].row0 - base));
        push[at] = src | ((uint32_t)(p.nrows + h) << CC_SRC_BITS) |
                   ((uint32_t)rank << (CC_SRC_BITS + CC_SLOT_BITS));
      }
    }
  }
}

// ----------------------------------------------------------------- host side
// The systems of one cluster size.
struct CcgClass {
  int fp32, C, nsys;
  size_t dyn;
  void* fn = nullptr;
  CcgArgs<float> af;
  CcgArgs<double> ad;
  CcgPart* d_parts = nullptr;
  int32_t* d_order = nullptr;
  int32_t* d_slices = nullptr;
  uint16_t* d_cols = nullptr;
  uint32_t* d_push = nullptr;
  void* d_packed = nullptr;
  // all SMs on one system: halo rows; barrier, sums and published rows (cleared per solve)
  bool grid = false;
  int32_t* d_halo = nullptr;
  char* d_xch = nullptr;
  size_t xch_bytes = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t done = nullptr;
  ~CcgClass() {
    for (void* p : {(void*)d_parts, (void*)d_order, (void*)d_slices, (void*)d_cols, (void*)d_push,
                    d_packed, (void*)d_halo, (void*)d_xch})
      if (p) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
    if (done) cudaEventDestroy(done);
  }
};

struct Ccg {
  int S, nsys;
  std::vector<CcgClass*> classes;  // largest systems first
  cudaEvent_t begin = nullptr;
  CcgOut* d_out = nullptr;
  ~Ccg() {
    for (CcgClass* c : classes) delete c;
    if (begin) cudaEventDestroy(begin);
    if (d_out) cudaFree(d_out);
  }
};

namespace {

// The largest rows per thread whose five register vectors fit beside the product (about
// 60 of 128 registers), and a small form for systems of few rows.
template <typename VT, int NC, bool GRID>
struct Rpt {
  static constexpr int words = NC * (int)sizeof(VT) / 4;
  static constexpr int big = words == 1   ? 9
                             : words == 2 ? 6
                             : cc_planes<VT>(NC, 4, GRID) ? 4
                             : words <= 4 ? 3
                                          : 2;
  static constexpr int small = GRID ? (words <= 2 ? 4 : (words <= 4 ? 2 : 1)) : (words <= 2 ? 2 : 1);
};

template <typename VT, int LD, int NC, bool GRID>
void* pick(int rpt, int* big) {
  using R = Rpt<VT, NC, GRID>;
  *big = R::big;
  return rpt <= R::small ? (void*)k_ccg<VT, LD, NC, R::small, GRID>
                         : (void*)k_ccg<VT, LD, NC, R::big, GRID>;
}
template <typename VT, bool GRID>
void* pick_ld(int ld, int S, int rpt, int* big) {
  if (ld == 1) return pick<VT, 1, 1, GRID>(rpt, big);
  if (ld == 2) return pick<VT, 2, 2, GRID>(rpt, big);
  return S <= 3 ? pick<VT, 4, 3, GRID>(rpt, big) : pick<VT, 4, 4, GRID>(rpt, big);
}
void* pick_kernel(bool fp32, bool grid, int ld, int S, int rpt, int* big) {
  if (grid)
    return fp32 ? pick_ld<float, true>(ld, S, rpt, big) : pick_ld<double, true>(ld, S, rpt, big);
  return fp32 ? pick_ld<float, false>(ld, S, rpt, big) : pick_ld<double, false>(ld, S, rpt, big);
}
// 16-byte units of a published row
int row_units(bool fp32, int ld, int S) {
  const int nc = ld == 1 ? 1 : (ld == 2 ? 2 : (S <= 3 ? 3 : 4));
  return fp32 ? (nc + 2) / 3 : nc;
}

template <typename T>
cudaError_t dev_alloc(T** p, size_t n) {
  return cudaMalloc(reinterpret_cast<void**>(p), sizeof(T) * std::max<size_t>(n, 1));
}

struct CreateArgs {
  const tp_csr_op* op;
  const CcgSource* src;
  int max_it;
  double delta;
  const double* b;
  double* x;
  const double* rtol;
  CcgOut* out;
  cudaStream_t st;
};

template <typename VT>
void fill(CcgArgs<VT>& a, const CcgClass* h, const CreateArgs& ca, int win_cap) {
  const tp_csr_op* op = ca.op;
  a.parts = h->d_parts;
  a.order = h->d_order;
  a.S = op->S;
  a.max_it = ca.max_it;
  // FP32 recurrences drift: past a factor of some hundreds the true residual no longer
  // follows theirs.  Ten steps of 274,625 rows and three species at rtol 1e-8 from the
  // previous step: 3243 iterations with a refresh every factor 1000 (one step 480 instead of
  // 230), 2703 at 300, 2697 at 100; a refresh costs about four iterations.
  const double delta = sizeof(VT) == 4 ? std::max(ca.delta, 1.0 / 500.0) : ca.delta;
  a.delta2 = delta * delta;
  a.slices = h->d_slices;
  a.loc_col = h->d_cols;
  a.push = h->d_push;
  a.halo = h->d_halo;
  a.bar = reinterpret_cast<unsigned int*>(h->d_xch);
  a.sums = reinterpret_cast<ulonglong2*>(h->d_xch + 256);
  a.ubuf = a.sums + (size_t)2 * 16 * h->C;
  a.packed = static_cast<VT*>(h->d_packed);
  a.inK = sizeof(VT) == 4 ? (const VT*)op->K32 : (const VT*)op->K64;
  a.sK = static_cast<const VT*>(ca.src->sK);
  a.sell_slice = ca.src->slice_ptr;
  a.A64.indptr = op->indptr;
  a.A64.indices = op->indices;
  a.A64.K = op->K64;
  a.A64.M = nullptr;
  a.A64.diag = op->diag64;
  a.A64.bc = op->bc_mask;
  for (int s = 0; s < 4; s++) {
    a.A64.dscale[s] = s < op->S ? op->dscale[s] : 0.0;
    a.A64.cscale[s] = 0.0;
  }
  a.diag = sizeof(VT) == 4 ? (const VT*)op->diag32 : (const VT*)op->diag64;
  a.b = ca.b;
  a.x = ca.x;
  a.rtol = ca.rtol;
  a.out = ca.out;
  a.win_cap = win_cap;
  a.dyn_bytes = (int)h->dyn;
  a.wait_limit_ns = CC_WAIT_NS;
  a.wait_missing = 0;
}

// slices per warp of a system of n rows on C CTAs
int rows_per_thread(int64_t n, int C) {
  const int64_t per = ((n + 31) / 32 + C - 1) / C;
  return (int)((per + CC_W - 1) / CC_W);
}

cudaLaunchConfig_t launch_config(const CcgClass* c, cudaLaunchAttribute* attr, int clusters,
                                 cudaStream_t st) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = c->C;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(c->C * clusters);
  cfg.blockDim = dim3(CC_T);
  cfg.dynamicSmemBytes = c->dyn;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Tables of the systems `sys` (largest first) on clusters of C CTAs (grid: one system on C
// CTAs of the whole device); *ok = false when one does not fit.
int build_class(CcgClass* h, const CreateArgs& ca, int inner_fp32, const std::vector<int32_t>& sys,
                const std::vector<int32_t>& row0, const std::vector<int32_t>& rows, int C,
                bool grid, bool* ok) {
  *ok = false;
  const tp_csr_op* op = ca.op;
  cudaStream_t st = ca.st;
  const int nsys = (int)sys.size(), ld = op->ld;
  const size_t vt = inner_fp32 ? 4 : 8;
  const int64_t most = rows[sys[0]];
  int dev = 0, optin = 0, big = 0;
  TP_CUDA_TRY(cudaGetDevice(&dev));
  TP_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const int rpt = rows_per_thread(most, C);
  void* fn = pick_kernel(inner_fp32 != 0, grid, ld, op->S, rpt, &big);
  if (rpt > big || rpt * CC_T > (1 << CC_SRC_BITS)) return TP_OK;
  // columns of a window in planes, 0: rows of ld values
  const int nc = ld < 4 ? ld : (op->S <= 3 ? 3 : 4);
  const int planes = inner_fp32 && cc_planes<float>(nc, rpt, grid) ? nc : 0;
  const size_t rb = planes ? 4 * (size_t)planes : vt * ld;
  cudaFuncAttributes fa;
  TP_CUDA_TRY(cudaFuncGetAttributes(&fa, fn));
  const size_t dyn = ((size_t)optin - fa.sharedSizeBytes - 1024) & ~(size_t)15;
  h->fp32 = inner_fp32 ? 1 : 0;
  h->C = C;
  h->nsys = nsys;
  h->dyn = dyn;
  h->fn = fn;
  h->grid = grid;
  const int np = nsys * C;
  std::vector<CcgPart> parts(np);
  std::vector<int32_t> base(nsys), count(nsys);
  int64_t slice_off = 0;
  for (int q = 0; q < nsys; q++) {
    base[q] = row0[sys[q]];
    count[q] = rows[sys[q]];
    const int64_t per = (((int64_t)count[q] + 31) / 32 + C - 1) / C * 32;
    for (int k = 0; k < C; k++) {
      CcgPart& p = parts[(size_t)q * C + k];
      memset(&p, 0, sizeof(p));
      const int64_t a0 = std::min<int64_t>(k * per, count[q]);
      const int64_t a1 = std::min<int64_t>(a0 + per, count[q]);
      p.row0 = base[q] + (int32_t)a0;
      p.nrows = (int32_t)(a1 - a0);
      p.nslices = (p.nrows + 31) / 32;
      p.slice_off = (int32_t)slice_off;
      slice_off += p.nslices + 1;
    }
  }
  TP_CUDA_TRY(dev_alloc(&h->d_parts, np));
  TP_CUDA_TRY(dev_alloc(&h->d_slices, slice_off));
  TP_CUDA_TRY(cudaMemcpyAsync(h->d_parts, parts.data(), sizeof(CcgPart) * np,
                              cudaMemcpyHostToDevice, st));
  k_ccg_slices<<<np, 128, 0, st>>>(h->d_parts, op->indptr, h->d_slices,
                                   CC_W * (inner_fp32 ? 8 : 4));
  TP_LAUNCH_CHECK();
  TP_CUDA_TRY(cudaMemcpyAsync(parts.data(), h->d_parts, sizeof(CcgPart) * np,
                              cudaMemcpyDeviceToHost, st));
  std::vector<int32_t> sl_host(slice_off);
  TP_CUDA_TRY(cudaMemcpyAsync(sl_host.data(), h->d_slices, sizeof(int32_t) * slice_off,
                              cudaMemcpyDeviceToHost, st));
  TP_CUDA_TRY(cudaStreamSynchronize(st));
  int64_t entries = 0;
  for (CcgPart& p : parts) {
    p.entry_off = entries;
    entries += p.entries;
  }
  // scratch of the builder: per system first row and rows | bounds, push offsets, flag
  struct Tmp {
    int32_t* p = nullptr;
    ~Tmp() {
      if (p) cudaFree(p);
    }
  } tmp;
  const size_t n_bounds = grid ? 0 : (size_t)np * (C + 1), n_at = grid ? 0 : (size_t)np * C;
  TP_CUDA_TRY(dev_alloc(&tmp.p, 2 * (size_t)nsys + n_bounds + n_at + 1));
  int32_t *t_row0 = tmp.p, *t_rows = tmp.p + nsys, *t_bounds = tmp.p + 2 * (size_t)nsys,
          *t_at = t_bounds + n_bounds, *t_flag = t_at + n_at;
  TP_CUDA_TRY(dev_alloc(&h->d_cols, (size_t)entries));
  TP_CUDA_TRY(cudaMemcpyAsync(h->d_parts, parts.data(), sizeof(CcgPart) * np,
                              cudaMemcpyHostToDevice, st));
  TP_CUDA_TRY(cudaMemcpyAsync(t_row0, base.data(), sizeof(int32_t) * nsys,
                              cudaMemcpyHostToDevice, st));
  TP_CUDA_TRY(cudaMemcpyAsync(t_rows, count.data(), sizeof(int32_t) * nsys,
                              cudaMemcpyHostToDevice, st));
  TP_CUDA_TRY(cudaMemsetAsync(t_flag, 0, sizeof(int32_t), st));
  const size_t bits = 2 * sizeof(uint32_t) * (size_t)((most + 31) / 32);
  if (bits > 200 * 1024) return TP_OK;
  if (bits > 40 * 1024) {
    TP_CUDA_TRY(cudaFuncSetAttribute(k_ccg_halo<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     200 * 1024));
    TP_CUDA_TRY(cudaFuncSetAttribute(k_ccg_halo<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     200 * 1024));
  }
  const int unit = grid ? 1 : (int)rb;  // columns: window entries, or byte offsets
  k_ccg_halo<false><<<np, 512, bits, st>>>(h->d_parts, C, t_row0, t_rows, op->indptr,
                                           op->indices, h->d_slices, unit, planes, h->d_cols,
                                           grid ? nullptr : t_bounds, nullptr, nullptr, nullptr,
                                           t_flag);
  TP_LAUNCH_CHECK();
  std::vector<int32_t> bounds(n_bounds), at(n_at);
  int32_t flag = 0;
  TP_CUDA_TRY(cudaMemcpyAsync(parts.data(), h->d_parts, sizeof(CcgPart) * np,
                              cudaMemcpyDeviceToHost, st));
  if (!grid)
    TP_CUDA_TRY(cudaMemcpyAsync(bounds.data(), t_bounds, sizeof(int32_t) * n_bounds,
                              cudaMemcpyDeviceToHost, st));
  TP_CUDA_TRY(cudaMemcpyAsync(&flag, t_flag, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  TP_CUDA_TRY(cudaStreamSynchronize(st));
  if (flag) return TP_OK;
  // push lists: producer by producer, its consumers in rank order
  int64_t npush = 0;
  int win_cap = 0;
  for (int q = 0; q < nsys; q++)
    for (int k = 0; k < C; k++) {
      CcgPart& p = parts[(size_t)q * C + k];
      p.push_off = (int32_t)npush;
      if (grid) npush += p.nhalo;
      for (int j = 0; j < C && !grid; j++) {
        at[((size_t)q * C + k) * C + j] = (int32_t)npush;
        const int32_t* bj = &bounds[((size_t)q * C + j) * (C + 1)];
        // empty ranks past the last row share its bound: they own nothing
        if (p.nrows) npush += bj[k + 1] - bj[k];
      }
      p.npush = (int32_t)(npush - p.push_off);
      win_cap = std::max(win_cap, p.nrows + p.nhalo);
    }
  win_cap = (win_cap + 31) & ~31;
  // window columns are 16-bit
  if (npush > INT32_MAX || win_cap * (planes ? planes : unit) > 65536) return TP_OK;
  if (!grid && win_cap >= (1 << CC_SLOT_BITS)) return TP_OK;
  // what has to fit in shared memory (the kernel carves in the same order); columns and
  // values stream from L2 where they do not
  bool spill = false;
  for (const CcgPart& p : parts) {
    auto r16 = [](size_t v) { return (v + 15) & ~(size_t)15; };
    size_t need = 2 * 16 * 16 * sizeof(double) + rb * (size_t)win_cap;
    const size_t own = rb * (size_t)(planes ? 32 * p.nslices : p.nrows);
    need += r16(own) + r16(4 * ((size_t)p.nslices + 1)) + r16(4 * (size_t)p.npush);
    if (need > dyn) return TP_OK;
    if (op->diag64) need += r16(own);
    const size_t nval = (size_t)(p.entries - sl_host[p.slice_off + p.val_slice]);
    need += r16(2 * (size_t)p.entries) + r16(vt * nval);
    spill |= nval > 0 && need > dyn;
  }
  if ((int)dyn > fa.maxDynamicSharedSizeBytes)
    TP_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  if (grid) {
    int occ = 0;
    TP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, CC_T, dyn));
    if (occ < 1) return TP_OK;
    TP_CUDA_TRY(dev_alloc(&h->d_halo, (size_t)npush));
    h->xch_bytes = 256 + sizeof(ulonglong2) * ((size_t)2 * 16 * C +
                                               (size_t)most * row_units(inner_fp32 != 0, ld, op->S));
    TP_CUDA_TRY(dev_alloc(&h->d_xch, h->xch_bytes));
  } else {
    TP_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = launch_config(h, &attr, 1, st);
    int active = 0;
    if (cudaOccupancyMaxActiveClusters(&active, fn, &cfg) != cudaSuccess || active < 1) {
      cudaGetLastError();
      return TP_OK;
    }
  }
  if (!grid) TP_CUDA_TRY(dev_alloc(&h->d_push, (size_t)npush));
  TP_CUDA_TRY(dev_alloc(&h->d_order, (size_t)nsys));
  if (spill) TP_CUDA_TRY(cudaMalloc(&h->d_packed, vt * std::max<size_t>((size_t)entries, 1)));
  TP_CUDA_TRY(cudaMemcpyAsync(h->d_order, sys.data(), sizeof(int32_t) * nsys,
                              cudaMemcpyHostToDevice, st));
  TP_CUDA_TRY(cudaMemcpyAsync(h->d_parts, parts.data(), sizeof(CcgPart) * np,
                              cudaMemcpyHostToDevice, st));
  if (!grid)
    TP_CUDA_TRY(cudaMemcpyAsync(t_at, at.data(), sizeof(int32_t) * n_at, cudaMemcpyHostToDevice,
                                st));
  k_ccg_halo<true><<<np, 512, bits, st>>>(h->d_parts, C, t_row0, t_rows, op->indptr,
                                          op->indices, h->d_slices, unit, planes, h->d_cols, t_bounds,
                                          t_at, h->d_push, grid ? h->d_halo : nullptr, t_flag);
  TP_LAUNCH_CHECK();
  TP_CUDA_TRY(cudaStreamSynchronize(st));
  if (h->fp32)
    fill(h->af, h, ca, win_cap);
  else
    fill(h->ad, h, ca, win_cap);
  *ok = true;
  return TP_OK;
}

}  // namespace

int ccg_create(const tp_csr_op* op, int inner_fp32, const CcgSource& src, int max_it,
               double delta, const double* b, double* x, const double* rtol, bool allow_grid,
               cudaStream_t st, Ccg** out) {
  *out = nullptr;
  if (op->M64 || op->n_rows <= 0) return TP_OK;
  const int nsys = op->n_systems > 0 ? op->n_systems : 1;
  if (src.sK && nsys != 1) return TP_OK;
  if (inner_fp32 && !src.sK && !op->K32) return TP_OK;
  std::vector<int32_t> row0(nsys), rows(nsys), order(nsys);
  int64_t most = 0;
  for (int m = 0; m < nsys; m++) {
    const int64_t r0 = op->sys_row_ptr ? op->sys_row_ptr[m] : 0;
    const int64_t r1 = op->sys_row_ptr ? op->sys_row_ptr[m + 1] : op->n_rows;
    if (r0 < 0 || r1 < r0 || r1 > op->n_rows || r1 > INT32_MAX) return TP_OK;
    row0[m] = (int32_t)r0;
    rows[m] = (int32_t)(r1 - r0);
    order[m] = m;
    most = std::max(most, r1 - r0);
  }
  int big = 0;
  pick_kernel(inner_fp32 != 0, false, op->ld, op->S, 1, &big);
  // One system: a cluster up to where every SM is faster (us per iteration, cluster / all
  // SMs): one FP64 column 3.1 / 4.0 at 15.6k rows, 4.3 / 4.2 at 24k, 6.3 / 4.4 at 39k; two
  // 3.9 / 4.0 at 9.3k; three 5.0 / 4.3 and four 5.0 / 5.1 at 4.9k; one FP32 column 4.0 / 4.4
  // at 36k, 4.9 / 4.4 at 51k; two 3.5 / 4.1 and three 4.1 / 4.3 at 13.8k, 5.6 / 4.1 and
  // 5.5 / 4.4 at 24k; four 4.6 / 4.5 at 9.3k.
  bool grid = rows_per_thread(most, 16) > big;
  if (allow_grid && nsys == 1) {
    const int64_t limit = inner_fp32 ? (op->ld == 1 ? 40960 : (op->S <= 3 ? 16384 : 8192))
                                     : (op->ld == 1 ? 24576 : (op->ld == 2 ? 8192 : 4096));
    grid = grid || most > limit;
  }
  if (grid && !(allow_grid && nsys == 1)) return TP_OK;
  std::stable_sort(order.begin(), order.end(),
                   [&](int32_t p, int32_t q) { return rows[p] > rows[q]; });
  Ccg* h = new Ccg();
  struct Guard {
    Ccg* h;
    ~Guard() { delete h; }
  } guard{h};
  h->S = op->S;
  h->nsys = nsys;
  TP_CUDA_TRY(dev_alloc(&h->d_out, (size_t)nsys));
  TP_CUDA_TRY(cudaMemsetAsync(h->d_out, 0, sizeof(CcgOut) * (size_t)nsys, st));
  const CreateArgs ca{op, &src, max_it, delta, b, x, rtol, h->d_out, st};
  // Many systems: 8 CTAs where a system fits them (fewer SMs idle in its latencies: 64
  // meshes of 8..40 cells per side take 6.1 ms against 7.2 ms with 16 CTAs each; 4 CTAs for
  // the small ones change nothing), else 16; few systems: 16, the lower latency.
  const int least = nsys > 8 ? 8 : 16;
  auto fits8 = [&](int32_t m) { return least == 8 && rows_per_thread(rows[m], 8) <= big; };
  for (int at = 0; at < nsys;) {
    const int C = grid ? sm_count() : (fits8(order[at]) ? 8 : 16);
    int end = at + 1;
    while (end < nsys && (C == least || !fits8(order[end]))) end++;
    const std::vector<int32_t> sys(order.begin() + at, order.begin() + end);
    CcgClass* c = new CcgClass();
    h->classes.push_back(c);
    bool ok = false;
    const int rc = build_class(c, ca, inner_fp32, sys, row0, rows, C, grid, &ok);
    if (rc != TP_OK || !ok) return rc;
    at = end;
  }
  if (h->classes.size() > 1) {
    TP_CUDA_TRY(cudaEventCreateWithFlags(&h->begin, cudaEventDisableTiming));
    for (CcgClass* c : h->classes) {
      TP_CUDA_TRY(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
      TP_CUDA_TRY(cudaEventCreateWithFlags(&c->done, cudaEventDisableTiming));
    }
  }
  guard.h = nullptr;
  *out = h;
  return TP_OK;
}

int ccg_run(Ccg* h, cudaStream_t st) {
  // several cluster sizes: side by side on streams of their own, the largest systems first
  const bool fork = h->classes.size() > 1;
  if (fork) TP_CUDA_TRY(cudaEventRecord(h->begin, st));
  for (CcgClass* c : h->classes) {
    cudaStream_t s = fork ? c->stream : st;
    if (fork) TP_CUDA_TRY(cudaStreamWaitEvent(s, h->begin, 0));
    void* args[1] = {c->fp32 ? (void*)&c->af : (void*)&c->ad};
    if (c->grid) {
      TP_CUDA_TRY(cudaMemsetAsync(c->d_xch, 0, c->xch_bytes, s));
      TP_CUDA_TRY(cudaLaunchCooperativeKernel(c->fn, dim3(c->C), dim3(CC_T), args, c->dyn, s));
      continue;
    }
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = launch_config(c, &attr, c->nsys, s);
    TP_CUDA_TRY(cudaLaunchKernelExC(&cfg, c->fn, args));
    if (fork) {
      TP_CUDA_TRY(cudaEventRecord(c->done, s));
      TP_CUDA_TRY(cudaStreamWaitEvent(st, c->done, 0));
    }
  }
  return TP_OK;
}

int ccg_result(Ccg* h, tp_cg_result* res, int32_t* lane_iters, int32_t* lane_status,
               double* lane_rnorm, double* lane_bnorm, cudaStream_t st) {
  std::vector<CcgOut> o(h->nsys);
  TP_CUDA_TRY(cudaMemcpyAsync(o.data(), h->d_out, sizeof(CcgOut) * h->nsys,
                              cudaMemcpyDeviceToHost, st));
  TP_CUDA_TRY(cudaStreamSynchronize(st));
  int status = TP_OK, its = 0, rel = 0;
  for (int m = 0; m < h->nsys; m++) {
    its = std::max(its, o[m].iterations);
    rel = std::max(rel, o[m].n_reliable);
    if (status == TP_OK) status = o[m].status;
    for (int s = 0; s < h->S; s++) {
      const int64_t l = (int64_t)m * h->S + s;
      if (lane_iters) lane_iters[l] = o[m].lane_iters[s];
      if (lane_status) lane_status[l] = o[m].lane_status[s];
      if (lane_rnorm) lane_rnorm[l] = sqrt(std::max(o[m].lane_rtrue[s], 0.0));
      if (lane_bnorm) lane_bnorm[l] = sqrt(std::max(o[m].lane_bb[s], 0.0));
    }
  }
  if (res) {
    res->status = status;
    res->iterations = its;
    res->n_reliable = rel;
    res->n_lanes = h->nsys * h->S;
  }
  return TP_OK;
}

size_t ccg_smem(const Ccg* h) { return h->classes[0]->dyn; }
bool ccg_is_grid(const Ccg* h) { return h->classes[0]->grid; }

void ccg_set_wait(Ccg* h, unsigned long long limit_ns, unsigned int missing) {
  for (CcgClass* c : h->classes) {
    c->af.wait_limit_ns = c->ad.wait_limit_ns = limit_ns;
    c->af.wait_missing = c->ad.wait_missing = 8 * missing;
  }
}

void ccg_destroy(Ccg* h) { delete h; }

}  // namespace tp
