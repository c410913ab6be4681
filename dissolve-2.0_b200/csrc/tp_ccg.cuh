// tp_ccg.cuh -- cluster engine of the Krylov solves (tp_ccg.cu), used by the tp_cg_* and
// tp_pcg_* handles for systems that fit one thread-block cluster.
#pragma once
#include "tp_common.cuh"

namespace tp {

struct Ccg;

// Where the inner operator's values come from: the CSR values of the operator (sK == NULL:
// K64, or K32 for an FP32 inner solve) or a SELL-32 copy of one system (tp_sell order).
struct CcgSource {
  const void* sK = nullptr;
  const int32_t* slice_ptr = nullptr;
};

// allow_grid: one system past a cluster may take every SM (a cooperative launch per solve).
// *out stays NULL (and TP_OK is returned) when the systems do not fit the engine; the
// caller then keeps its own.  [sync]
int ccg_create(const tp_csr_op* op, int inner_fp32, const CcgSource& src, int max_it,
               double delta, const double* b, double* x, const double* rtol, bool allow_grid,
               cudaStream_t st, Ccg** out);
int ccg_run(Ccg* h, cudaStream_t st);
// summary over all systems, per-lane arrays (lane = system * S + column), any NULL  [sync]
int ccg_result(Ccg* h, tp_cg_result* res, int32_t* lane_iters, int32_t* lane_status,
               double* lane_rnorm, double* lane_bnorm, cudaStream_t st);
size_t ccg_smem(const Ccg* h);  // dynamic shared memory per CTA
bool ccg_is_grid(const Ccg* h);  // one system on every SM
// bound of the waits of the next runs; missing > 0 (tests) makes every wait run out
void ccg_set_wait(Ccg* h, unsigned long long limit_ns, unsigned int missing);
void ccg_destroy(Ccg* h);

}  // namespace tp
