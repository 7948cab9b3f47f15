// Single-launch BiCGSTAB of small FP64 systems (solve_team.cu).
#pragma once

#include <cuda_runtime.h>

#include "gb_internal.h"
#include "solve_plan.cuh"

namespace gb {

struct TeamPlan {
    bool ok = false;         // the single-launch solver takes these systems
    bool cluster = false;    // a thread-block cluster per system (else a cooperative launch)
    bool resident = false;   // matrix rows in shared memory
    int G = 0;               // CTAs per system
    int tile = 4, cp = 1;    // rows per warp tile and column parts of a product
    long long cycles = 0;    // estimate of an iteration
    size_t smem = 0;
};

TeamPlan team_plan(int nsys, int Dmax, int R, bool packed);

// The wait limit of the current device's cooperative teams from that of the matrix pass's
// waits (gb_set_gemv_wait_limit): ten times as long, < 0 for the default.
int set_team_wait_limit(long long gemv_cycles);

// Solves nsys systems (sys: packed operator; null: one dense D x D matrix) from x = 0.
// err_cnt: nsys + 1 ints; vectors: at least 2 total_vec + 3 nsys R G complex values; the
// states of every (system, right-hand side) go to st; err_cnt[0] is set if a cooperative
// team's wait ran out.  Asynchronous.
int team_solve(const TeamPlan& t, int nsys, const SysDev* sys, int D, int R, const double2* mat, const double2* tvec,
               const double2* b, double2* x, KState* st, int* err_cnt, double2* vectors, long long total_vec, double tol,
               int maxiter, cudaStream_t stream);

}   // namespace gb
