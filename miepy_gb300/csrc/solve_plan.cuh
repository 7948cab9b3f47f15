// Plan records of the packed-operator solve, shared by the BiCGSTAB driver and its
// CUDA-core matrix pass (solve.cu) and the tensor-core matrix pass (gemv_tc.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gb_internal.h"

namespace gb {

struct Strip {          // GEMV work: blocks (i, j0 .. j0+nb-1) of cluster sys
    int sys, i, nb, pad;
    long long p0;       // first pair index (cluster-local)
};
struct Item {           // rows [r0, r0+nr) of cluster sys
    int sys, r0, nr, pad;
};
struct TcUnit {         // tensor-core pass: the pairs (i, j) of cluster sys with i < j, i0 <= i <
    int sys, i0, j0, nj;   // i0 + I (I of the plan), j0 <= j < j0 + nj; unit c of its rows
    int c, C;              // among C: row i's partials of its C units are contiguous
};
struct SysPlan {
    long long strip_row_base;   // index into row_strip (first block row of this cluster)
    long long strip_base;       // global index of the first strip of this cluster
    long long cw_off;           // element offset of this cluster's per-pair column partials
    long long cu_off;           // element offset of this cluster's per-strip row partials
    int vbeg, vend;             // vector items
    int rbeg, rend;             // reduce items
    // tensor-core pass: the cluster's N + 1 first terms of every row's partials in CU, then of
    // every column's in CW, in tc_rows; its first elements there
    long long tc_base, tc_cu, tc_cw;
};

struct KState {         // per (cluster, rhs) BiCGSTAB scalars
    double2 rho, alpha, omega, beta;   // FP64 solver
    double r0sq, bsq, rsq, tol2;       // (bsq, rsq also mirrored from the FP32 solver, for the host)
    float2 rho_f, alpha_f, omega_f, beta_f;   // FP32 solver
    float r0sq_f, bsq_f, rsq_f, tol2_f;
    int iters, restarts, done, status;
    int need_restart, maxiter, pad0, pad1;
};

// mask_mode: -1 all, 0 running clusters, 1 restarting clusters
template <int R>
__device__ __forceinline__ bool active_rhs(const KState* st, int sys, int rr, int mask_mode) {
    if (mask_mode < 0) return true;
    const KState& k = st[sys * R + rr];
    return (mask_mode == 0) ? (!k.done && !k.need_restart) : (k.need_restart != 0);
}
template <int R>
__device__ __forceinline__ bool any_active(const KState* st, int sys, int mask_mode) {
    bool a = false;
#pragma unroll
    for (int rr = 0; rr < R; rr++) a |= active_rhs<R>(st, sys, rr, mask_mode);
    return a;
}

// two bf16 in memory order; a float rounded to bf16
__device__ __forceinline__ unsigned bf2(float first, float second) {
    __nv_bfloat162 v = __floats2bfloat162_rn(first, second);
    return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ float bf_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// Tensor-core matrix pass (gemv_tc.cu) over units [ubeg, uend) of rows groups of I and one
// block size B: row partials per (row, unit) in CU and column partials per (row group,
// column) in CW, float2 terms of B R elements as +- column sums, from the bf16 hi/lo tiles
// of the matrix (mat_tc) and the operands Yu, Yw of the particles (tc_y_bytes(B, R) each,
// k_yprep_tc).  R is 4 or 8.
constexpr int kTcRows = 4;   // I at most
int launch_pgemv_tc(int R, const SysDev* sys, const TcUnit* units, long long ubeg, long long uend, int I,
                    const KState* st, int mask, const void* mat_tc, const void* Yu, const void* Yw, void* CU, void* CW,
                    const SysPlan* plan, const long long* tc_rows, int B, int* err, cudaStream_t stream);

// The R = 4 and 8 solves, applies and wait limit, compiled in their own unit
// (solve_multi.cu, which includes solve.cu with GB_SOLVE_MULTI_RHS defined) so that
// the two halves of the solver compile in parallel.
int solve_entry_multi(int nsys, const gb_system* sys, int R, int prec, double tol, int maxiter, double inner_tol,
                      int max_refine, const double* mat128, const float* mat64, const float* mat64lo,
                      const void* mat_tc, const double* pdiag, const double* tvec, const double* b, double* x,
                      void* workspace, size_t ws_bytes, int* status, int* iters, double* resid, cudaStream_t stream);
int apply_entry_multi(int nsys, const gb_system* sys, int R, int prec, const double* mat128, const float* mat64,
                      const float* mat64lo, const void* mat_tc, const double* tvec, const double* x, double* y,
                      void* workspace, size_t ws_bytes, int reps, int repeat, cudaStream_t stream);
int set_wait_limit_multi(long long cycles);

}   // namespace gb
