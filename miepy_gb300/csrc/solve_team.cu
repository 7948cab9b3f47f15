// BiCGSTAB of small FP64 systems in one launch (solve_linear_system, cpp/src/
// interactions.cpp:347-368): the dense operator of the plugin, substrate and lattice
// routes, and the packed operator of small clusters.
//
// A system whose matrix the chip holds on its SMs is bound by launches and readbacks when
// every product, reduction and vector update is its own kernel: 7 to 9 launches per
// iteration, 50 to 70 us.  Here a team of G CTAs runs the whole iteration:
//   - each CTA owns D / G consecutive rows: their matrix rows (in shared memory, scaled
//     by the Mie factors on the packed route; streamed from memory where a dense matrix is
//     larger than the SMs hold) and their entries of every vector (in registers);
//   - a product gathers the operand vector from L2 (written by its owners) and needs only
//     the CTA's own rows; dot products go through one partial per CTA, summed by every
//     CTA in the same order, so each holds the same scalars and takes the same branches;
//   - five team barriers per iteration: operand p, <r0, v>, operand s, <t, t> and <t, s>,
//     <r, r> and <r0, r>.
// Teams of up to kClusterG CTAs are thread-block clusters with the hardware barrier
// (any number of systems per launch).  Larger systems take up to one CTA per SM in a
// cooperative launch with a barrier through L2, whose waits are bounded: where one runs out
// (other streams' kernels kept part of the team off the SMs) the launch-per-step solver
// takes the systems.
//
// FP64 issues one warp instruction per 64 cycles and SM sub-partition, whatever its lanes
// do, so the iteration's small steps count instructions too: a warp holds eight vector
// elements, real and imaginary parts in different lanes (a complex multiply-add is two
// instructions) and the parts of a dot product in different lane groups; quotients of the
// scalar step run in the lanes of one division; rows are tiled so that the lanes' partial
// sums reduce by halving exchanges (9 additions for four complex sums instead of 40), and
// the tile and the column split are those of the fewest instructions per sub-partition.
// Dense systems solved to 1e-10 with one right-hand side (14 iterations), a launch per step
// and in one: D = 80 705 -> 202 us, D = 224 803 -> 288, D = 600 897 -> 358, D = 1300 1312 ->
// 743, D = 2900 2842 -> 2247, D = 4000 4390 -> 3818.  Beyond that the products are all of
// it (4.85 ms either way at D = 4500): kTeamMaxD.  A step of five spheres, lmax 2 (D = 80,
// assembly and epilogue included): 440 -> 186 us.

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "gb_common.cuh"
#include "gb_internal.h"
#include "solve_plan.cuh"
#include "solve_team.h"

namespace {

using gb::KState;

constexpr int kTeamThreads = 256;
constexpr int kTeamWarps = kTeamThreads / 32;
constexpr int kClusterG = 16;        // CTAs of a cluster team
constexpr int kElems = 8;            // vector elements per warp
constexpr int kMaxElems = kElems * kTeamWarps;
constexpr int kMaxRestarts = 8;      // as the launch-per-step solver
// Cycles a cooperative team waits at a barrier (per device), ten times the matrix pass's
// limit, about 2 s: its CTAs may have to wait for other streams' kernels to leave their SMs.
constexpr int kDevices = 64;
std::atomic<long long> g_team_wait[kDevices];   // 0: the default
constexpr long long kTeamWaitCycles = 4000000000LL;
// A team's CTA takes at most half of an SM's shared memory and registers (two CTAs per SM),
// so that kernels of other streams run beside a solve, which lasts up to milliseconds: with
// 222 KB and 208 registers a mixed solve of N = 12, lmax 3 took 46.8 ms beside dense solves
// of D = 2880, and 0.71 ms with half (0.60 alone; 0.98 beside the launch-per-step solver).
// Fewer registers cost 1 to 2 %; dense rows beyond 110 KB are streamed (D = 1000, R = 1 620 ->
// 698 us); batches share the SMs (19 systems of D = 80 265 -> 186 us).  Packed rows are not in
// memory in that form: systems that half of every SM cannot hold (D above about 950) take
// whole SMs and leave the others free, a quarter where the rows fit the rest, else a
// sixteenth at least (D up to 1291, R = 2 1287).  D = 960 594 us with a launch per step, 402
// so, 347 with every SM; D = 1200 773, 526, 438; the mixed solve beside a stream of D = 1200
// solves 0.58 ms, 3.1 with every SM.
constexpr size_t kTeamSmem = 110 * 1024, kWholeSmem = 222 * 1024;
// a dense matrix up to this size (of 129 MB of L2) stays there between products
constexpr size_t kL2Matrix = 96 << 20;
// beyond this the products are all of the time and the launch-per-step solver streams the
// matrix with more warps
constexpr int kTeamMaxD = 4000;

struct TeamArgs {
    const gb::SysDev* sys;      // packed: [nsys]
    const double2* mat;         // packed blocks, or the dense matrix
    const double2* tvec;        // packed: Mie factors
    const double2* b;
    double2* x;
    KState* st;                 // [nsys][R]
    int* err;
    int* cnt;                   // [nsys] barrier arrivals
    double2 *g1, *g2;           // operand vectors, at the clusters' vec offsets
    double* part;               // [nsys][2 buffers][3 R][G]
    double tol;
    long long wait;             // limit of a cooperative team's barrier, in cycles
    int maxiter, D, G, resident, CP;   // D: the dense system; CP: column parts of a product
};

__device__ __forceinline__ double2 cquot(double2 a, double2 b) {
    const double den = b.x * b.x + b.y * b.y;
    return make_double2((a.x * b.x + a.y * b.y) / den, (a.y * b.x - a.x * b.y) / den);
}
__device__ __forceinline__ bool finite2(double2 a) { return isfinite(a.x) && isfinite(a.y); }

enum { STATE_RUNNING = -1 };

__device__ __forceinline__ bool finite1(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

// Eigen's BiCGSTAB scalars, the phases of the launch-per-step solver.  Phase 0 starts
// from |b|^2, phase 4 ends a restart (r0 = r = b - A x; the first one resets the count):
// one thread per right-hand side.
__device__ void team_scalars_rare(KState& k, int phase, double d0, double tol, int maxiter) {
    if (phase == 0) {
        k.bsq = k.r0sq = k.rsq = d0;
        k.tol2 = tol * tol * d0;
        k.rho = k.beta = make_double2(d0, 0.0);   // beta = (rho / 1) (1 / 1)
        k.alpha = k.omega = make_double2(1, 0);
        k.iters = k.restarts = k.need_restart = 0;
        k.maxiter = maxiter;
        k.done = 0;
        k.status = STATE_RUNNING;
        if (!isfinite(d0)) { k.done = 1; k.status = GB_NAN; }
        else if (d0 == 0.0 || !(k.rsq > k.tol2) || maxiter <= 0) { k.done = 1; k.status = GB_OK; }
        return;
    }
    if (!k.need_restart) return;
    k.need_restart = 0;
    k.rsq = k.r0sq = d0;
    const double2 old = k.rho;
    k.rho = make_double2(d0, 0.0);
    if (k.restarts++ == 0) k.iters = 0;
    if (!isfinite(k.rsq)) { k.done = 1; k.status = GB_NAN; return; }
    if (!(k.rsq > k.tol2)) { k.done = 1; k.status = GB_OK; return; }
    k.beta = cmul(cquot(k.rho, old), cquot(k.alpha, k.omega));
    if (!finite2(k.beta)) { k.done = 1; k.status = GB_BREAKDOWN; }
}

// Phases 1 (alpha), 2 (omega) and 3 (end of iteration), by the first warp: lane
// 4 rr + q holds part q of right-hand side rr, so the two (four in phase 3) quotients run
// in one division.  tot: per right-hand side the norm, and the dot's real and imaginary
// parts (<r0, v>; |t|^2, <s, t>; |r|^2, <r0, r>).
template <int R> __device__ __forceinline__ void team_scalars(KState* ks, int phase, const double* tot, int lane) {
    const int rr = min(lane >> 2, R - 1), q = lane & 3, c = q & 1;
    const bool mine = (lane >> 2) < R;
    KState& k = ks[rr];
    const double nrm = tot[3 * rr];
    const double2 d = make_double2(tot[3 * rr + 1], tot[3 * rr + 2]);
    const bool skip = k.done || k.need_restart;
    double2 a, b;   // the quotient a / b of this lane
    if (phase == 1) { a = k.rho; b = d; }
    else if (q < 2) { a = d; b = k.rho; }        // phase 3: rho / rho_old
    else { a = k.alpha; b = k.omega; }
    double num, den;
    if (phase == 2) {
        num = c ? -d.y : d.x;   // <t, s> / |t|^2 from the parts of <s, t>
        den = nrm;
    } else {
        num = fma(c ? a.y : a.x, b.x, (c ? -a.x : a.y) * b.y);
        den = fma(b.x, b.x, b.y * b.y);
    }
    double quo = num / den;
    if (phase == 2 && !(nrm > 0.0)) quo = 0.0;
    if (phase == 3) {   // beta = (rho / rho_old) (alpha / omega)
        const int base = lane & ~3;
        const double ax = __shfl_sync(0xffffffffu, quo, base), ay = __shfl_sync(0xffffffffu, quo, base | 1);
        const double bx = __shfl_sync(0xffffffffu, quo, base | 2), by = __shfl_sync(0xffffffffu, quo, base | 3);
        quo = fma(ax, c ? by : bx, (c ? ay : -ay) * (c ? bx : by));
    }
    const double oth = __shfl_xor_sync(0xffffffffu, quo, 1);
    __syncwarp();   // every lane has read the state
    if (!mine || q != 0 || skip) return;
    const double2 v = make_double2(quo, oth);
    const bool fin = finite1(quo) && finite1(oth);
    if (phase == 1) {
        k.alpha = v;
        if (!fin) { k.done = 1; k.status = (d.x == 0 && d.y == 0) ? GB_BREAKDOWN : GB_NAN; }
    } else if (phase == 2) {
        k.omega = v;
        if (!fin) { k.done = 1; k.status = GB_NAN; }
    } else {
        k.iters += 1;
        k.rsq = nrm;
        if (!finite1(nrm)) { k.done = 1; k.status = GB_NAN; return; }
        if (!(nrm > k.tol2)) { k.done = 1; k.status = GB_OK; return; }
        if (k.iters >= k.maxiter) { k.done = 1; k.status = GB_NOT_CONVERGED; return; }
        const double low = 2.220446049250313e-16 * 2.220446049250313e-16 * k.r0sq;
        // |rho| < low, with the root only where the larger part does not decide
        if (!(fabs(d.x) >= low || fabs(d.y) >= low) && sqrt(d.x * d.x + d.y * d.y) < low) {
            if (k.restarts >= kMaxRestarts) { k.done = 1; k.status = GB_BREAKDOWN; return; }
            k.need_restart = 1;
            return;
        }
        k.rho = d;   // <r0, r>
        k.beta = v;
        if (!fin) { k.done = 1; k.status = GB_NAN; }
    }
}

// TILE: rows per warp tile of a product.
template <int R, bool PACKED, bool CLUSTER, int TILE>
__global__ void __launch_bounds__(kTeamThreads, 2) k_team_bicgstab(const TeamArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ KState ks[R];
    __shared__ double ysum[kTeamWarps][TILE * 2 * R];
    __shared__ double dsum[kTeamWarps][3 * R];
    __shared__ double tot[3 * R];
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int G = a.G, sidx = blockIdx.x / G, member = blockIdx.x - sidx * G;
    gb::SysDev S{};
    if (PACKED) S = a.sys[sidx];
    const int D = PACKED ? S.D : a.D;
    const long long vo = PACKED ? S.vec_off : 0;
    const int rows_per = (D + G - 1) / G, r0 = min(member * rows_per, D), nr = min(rows_per, D - r0);
    double2* xs = reinterpret_cast<double2*>(smem);                 // [D][R]
    double2* rows = xs + (size_t)D * R;                             // [nr][D] (resident)
    const double2* grows = a.mat + (size_t)r0 * D;                  // dense rows in memory
    double* part = a.part + (size_t)sidx * 6 * R * G;
    // the thread's vector element (row er, right-hand side rr), its real (c = 0) or
    // imaginary part; lanes 16-31 repeat lanes 0-15 (the imaginary parts of the dots)
    const int elem = wid * kElems + (lane & 7), c = (lane >> 3) & 1, kind = lane >> 4;
    const bool own = elem < nr * R;
    const int er = own ? elem / R : 0, rr = own ? elem - er * R : 0;
    const long long ge = 2 * (vo + (long long)(r0 + er) * R + rr) + c;   // as doubles
    if (tid == 0) s_abort = 0;

    // ---- the CTA's matrix rows
    double2 tme = make_double2(1.0, 0.0);   // Mie factor of the own row's entry as an operand
    if (PACKED) {
        const int B = S.B, N = S.N;
        for (int e = tid; e < nr * D; e += kTeamThreads) {
            const int q = e / D, col = e - q * D, row = r0 + q;
            const int i = row / B, r = row - i * B, j = col / B, cc = col - j * B;
            double2 v = make_double2(0.0, 0.0);
            if (i != j) {   // T[i, j] = A_ij, T[j, i] = S A_ij S for i < j (times t_j, in the operand)
                const long long lo = min(i, j), hi = max(i, j), p = pair_start(lo, N) + (hi - lo - 1);
                v = __ldg(a.mat + S.mat_off + p * (long long)B * B + (long long)r * B + cc);
                if (i > j) {
                    const unsigned s = ((unsigned)(__ldg(S.rowinfo + r) ^ __ldg(S.rowinfo + cc)) >> 30) & 1u;
                    v = make_double2(flipd(v.x, s), flipd(v.y, s));
                }
            }
            rows[e] = v;
        }
        if (own) tme = a.tvec[S.t_off + r0 + er];
    } else if (a.resident) {
        for (int e = tid; e < nr * D; e += kTeamThreads) rows[e] = __ldg(grows + e);
    }

    int epoch = 0;
    // Every CTA of the team arrives before any passes.  False (for the whole CTA) once a
    // bounded wait has expired.
    auto team_barrier = [&]() -> bool {
        if (CLUSTER) {
            __syncwarp();   // the aligned barrier takes whole warps: callers come out of divergent stores
            asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
            return true;
        }
        __syncthreads();
        epoch++;
        if (tid == 0) {
            __threadfence();
            int* n = a.cnt + sidx;
            atomicAdd(n, 1);
            const int target = epoch * G;
            const long long t0 = clock64();
            for (;;) {
                int v;
                asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(n) : "memory");
                if (v >= target) break;
                if (clock64() - t0 > a.wait) {
                    s_abort = 1;
                    atomicExch(a.err, 1);
                    break;
                }
            }
        }
        __syncthreads();
        return s_abort == 0;
    };

    // (T g)[own rows] for the operand gathered from g; the own part returned
    const int tiles = (nr + TILE - 1) / TILE, CP = a.CP;
    auto product = [&](const double2* g) -> double {
        for (int e = tid; e < D * R; e += kTeamThreads) xs[e] = __ldcg(g + vo + e);
        __syncthreads();
        double y = 0.0;
        const double2* base = (PACKED || a.resident) ? rows : grows;
        for (int t0 = 0; t0 < tiles; t0 += kTeamWarps / CP) {
            const int t = t0 + wid / CP, cp = wid % CP;
            if (t < tiles) {
                const double2* m[TILE];
#pragma unroll
                for (int q = 0; q < TILE; q++) m[q] = base + (size_t)min(t * TILE + q, nr - 1) * D;
                double acc[TILE * 2 * R];
#pragma unroll
                for (int q = 0; q < TILE * 2 * R; q++) acc[q] = 0.0;
#pragma unroll 2
                for (int col = cp * 32 + lane; col < D; col += CP * 32) {
                    double2 xv[R];
#pragma unroll
                    for (int q = 0; q < R; q++) xv[q] = xs[col * R + q];
#pragma unroll
                    for (int q = 0; q < TILE; q++) {
                        const double2 v = m[q][col];
#pragma unroll
                        for (int w = 0; w < R; w++) {
                            double& re = acc[(q * R + w) * 2];
                            double& im = acc[(q * R + w) * 2 + 1];
                            re = fma(v.x, xv[w].x, re);
                            im = fma(v.x, xv[w].y, im);
                            re = fma(-v.y, xv[w].y, re);
                            im = fma(v.y, xv[w].x, im);
                        }
                    }
                }
                constexpr int V = TILE * 2 * R, SH = V == 4 ? 3 : V == 8 ? 2 : 1;   // 5 - log2 V
                const double s = halving_sum<V>(acc);
                if ((lane & ((1 << SH) - 1)) == 0) ysum[wid][lane >> SH] = s;
            }
            __syncthreads();
            // the own part of these tiles: its column parts in order
            const int tl = er / TILE - t0;
            if (own && tl >= 0 && tl < kTeamWarps / CP) {
                const int at = ((er % TILE) * R + rr) * 2 + c;
                for (int q = 0; q < CP; q++) y += ysum[tl * CP + q][at];
            }
            __syncthreads();
        }
        return y;
    };

    int buf = 0;
    // norm (u, the own part) and dot (w: conj(w) u) summed over the team's rows, then the
    // scalars of the phase, in every CTA alike
    auto dots = [&](bool with_norm, bool with_dot, double u, double w, int phase) -> bool {
        const int nw = max(1, (nr * R + kElems - 1) / kElems);
        if (wid < nw) {
            const double up = __shfl_xor_sync(0xffffffffu, u, 8);
            double nv = own && with_norm ? u * u : 0.0;
            double dv = own && with_dot ? (kind == 0 ? w * u : (c ? -w : w) * up) : 0.0;
#pragma unroll
            for (int o = 8; o >= R; o >>= 1) {
                if (with_norm) nv += __shfl_xor_sync(0xffffffffu, nv, o);
                if (with_dot) dv += __shfl_xor_sync(0xffffffffu, dv, o);
            }
            if ((lane & 15) < R) {
                dsum[wid][3 * (lane & 15) + 1 + kind] = dv;
                if (kind == 0) dsum[wid][3 * (lane & 15)] = nv;
            }
        }
        if (nw > 1) __syncthreads();
        else __syncwarp();
        double* p = part + (size_t)buf * 3 * R * G;
        if (tid < 3 * R) {
            double s = dsum[0][tid];
            for (int q = 1; q < nw; q++) s += dsum[q][tid];
            p[(size_t)tid * G + member] = s;
        }
        if (!team_barrier()) return false;
        buf ^= 1;
        if (wid < 3 * R && (wid % 3 ? with_dot : with_norm)) {   // a warp per value
            double s = 0.0;
            for (int q = lane; q < G; q += 32) s += __ldcg(p + (size_t)wid * G + q);
            for (int o = G > 16 ? 16 : 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) tot[wid] = s;
        }
        __syncthreads();
        if (phase == 0 || phase == 4) {
            if (tid < R) team_scalars_rare(ks[tid], phase, tot[3 * tid], a.tol, a.maxiter);
        } else if (wid == 0) {
            team_scalars<R>(ks, phase, tot, lane);
        }
        __syncthreads();
        return true;
    };
    // the own part of acc + s z for a complex s and the own part z of a vector
    auto cmadd = [&](double acc, double2 s, double z) {
        const double zp = __shfl_xor_sync(0xffffffffu, z, 8);
        return fma(s.x, z, fma(c ? s.y : -s.y, zp, acc));
    };
    auto cneg = [](double2 s) { return make_double2(-s.x, -s.y); };
    double* g1 = reinterpret_cast<double*>(a.g1);
    double* g2 = reinterpret_cast<double*>(a.g2);
    auto publish = [&](double* g, double z) {   // the operand, times the Mie factor
        const double o = PACKED ? cmadd(0.0, tme, z) : z;
        if (own && kind == 0) g[ge] = o;
    };

    const double bv = own ? reinterpret_cast<const double*>(a.b)[ge] : 0.0;
    double r = bv, rs = bv, p = 0.0, v = 0.0, s = 0.0, t = 0.0, x = 0.0;
    bool ok = dots(true, false, r, 0.0, 0);
    const long long most = ((long long)a.maxiter + 2) * (kMaxRestarts + 2) + 16;
    for (long long it = 0; ok; it++) {
        bool run = false, restart = false;
#pragma unroll
        for (int q = 0; q < R; q++) {
            run |= !ks[q].done;
            restart |= ks[q].need_restart != 0;
        }
        if (!run) break;
        if (it >= most) {
            if (tid == 0) atomicExch(a.err, 1);
            break;
        }
        if (restart) {   // r = b - (I + T) x, r0 = r for the right-hand sides that ask for it
            publish(g1, x);
            if (!(ok = team_barrier())) break;
            const double y = product(a.g1);
            if (ks[rr].need_restart) r = rs = bv - (x + y);
            if (!(ok = dots(true, false, r, 0.0, 4))) break;
        }
        const KState& k = ks[rr];
        auto active = [&]() { return !k.done && !k.need_restart; };   // (of the element's right-hand side)
        {
            const double q = cmadd(p, cneg(k.omega), v), np = cmadd(r, k.beta, q);
            if (active()) p = np;
        }
        publish(g1, p);
        if (!(ok = team_barrier())) break;
        double y = product(a.g1);
        if (active()) v = p + y;
        if (!(ok = dots(false, true, v, rs, 1))) break;
        {
            const double ns = cmadd(r, cneg(k.alpha), v);
            if (active()) s = ns;
        }
        publish(g2, s);
        if (!(ok = team_barrier())) break;
        y = product(a.g2);
        if (active()) t = s + y;
        // |t|^2 and <s, t>, the conjugate of <t, s>
        if (!(ok = dots(true, true, t, s, 2))) break;
        {
            const double nx = cmadd(cmadd(x, k.omega, s), k.alpha, p), q = cmadd(s, cneg(k.omega), t);
            if (active()) {
                x = nx;
                r = q;
            }
        }
        if (!(ok = dots(true, true, r, rs, 3))) break;
    }
    if (own && kind == 0) reinterpret_cast<double*>(a.x)[ge] = x;
    if (member == 0 && tid < R) a.st[sidx * R + tid] = ks[tid];
}

template <int R, bool PACKED, bool CLUSTER, int TILE>
int launch_team(const TeamArgs& a, int nsys, size_t smem, cudaStream_t stream) {
    auto kfn = k_team_bicgstab<R, PACKED, CLUSTER, TILE>;
    GB_CUDA_TRY(gb::ensure_dynamic_smem(reinterpret_cast<const void*>(kfn), smem));
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nsys * a.G));
    cfg.blockDim = dim3(kTeamThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (CLUSTER) {
        if (a.G > 8)
            GB_CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(kfn),
                                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)a.G;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kfn, a);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorInvalidClusterSize ||
        e == cudaErrorInvalidConfiguration) {   // no room for a team (part of a device): the caller's other path
        (void)cudaGetLastError();
        return gb_set_error(GB_UNSUPPORTED, "single-launch solve: %s", cudaGetErrorString(e));
    }
    GB_CUDA_TRY(e);
    gb::note_launch();
    return GB_OK;
}

template <int R, bool PACKED>
int launch_any(const TeamArgs& a, int nsys, const gb::TeamPlan& t, cudaStream_t s) {
    if (t.cluster) return t.tile == 2 ? launch_team<R, PACKED, true, 2>(a, nsys, t.smem, s)
                                      : launch_team<R, PACKED, true, 4>(a, nsys, t.smem, s);
    return t.tile == 2 ? launch_team<R, PACKED, false, 2>(a, nsys, t.smem, s)
                       : launch_team<R, PACKED, false, 4>(a, nsys, t.smem, s);
}

// FP64 instructions per sub-partition (its share of the warps' units) of one product with
// rows rows per CTA, for the best tile and column split.  Rows that come from HBM are bound
// by the loads in flight: there a round of tiles costs what all of its warps would take,
// idle ones included, and two or four warps share a tile (dense D = 3500, R = 1 3.73 -> 3.12
// ms, 3.53 with a launch per step; D = 2900 2.44 -> 2.24; where the matrix stays in L2, D =
// 2400, a warp per tile is as quick).
int product_cost(int rows, int D, int R, bool from_hbm, int* tile, int* cp) {
    int best = 1 << 30;
    for (int T = 4; T >= 2; T -= 2)
        for (int C = from_hbm ? 2 : 1; C <= (from_hbm ? 4 : kTeamWarps); C *= 2) {
            const int tiles = (rows + T - 1) / T, per = kTeamWarps / C;   // tiles per round of the warps
            const int step = (D + 32 * C - 1) / (32 * C) * 4 * T * R + (T == 4 ? 9 : 6) * R;
            int cost = 0;
            for (int t = 0; t < tiles; t += per) {
                const int warps = from_hbm ? kTeamWarps : std::min(per, tiles - t) * C;
                cost += (warps + 3) / 4 * step + C;
            }
            if (cost < best) {
                best = cost;
                *tile = T;
                *cp = C;
            }
        }
    return best;
}

}   // namespace

namespace gb {

// The team of a launch.  Cluster or cooperative by the iteration's estimated cycles: two
// products at 64 cycles an instruction, and five barriers with the exchange of operands
// and partial dots, measured at about 1500 cycles each in a cluster and 3300 through L2.
// A batch takes at most two CTAs per SM: beyond that the systems would queue, where the
// launch-per-step solver shares its launches between them (FP64 clusters of N = 5, lmax 2:
// 150 of them 622 -> 282 us, 300 of them 930 us in launches of their own).
TeamPlan team_plan(int nsys, int Dmax, int R, bool packed) {
    TeamPlan best;
    if (R > 2 || Dmax < 1 || Dmax > kTeamMaxD) return best;
    const int sms = sm_count();
    for (int form = 0; form < 2; form++) {
        TeamPlan t;
        t.cluster = form == 0;
        t.G = std::min(t.cluster ? kClusterG : sms / nsys, (Dmax + 3) / 4);
        if (t.cluster)   // a batch: fewer CTAs per system, down to what holds a system's elements
            while ((long long)nsys * t.G > sms && t.G > 1 && (Dmax + t.G / 2 - 1) / (t.G / 2) * R <= kMaxElems) t.G /= 2;
        if (t.G < 1 || (long long)nsys * t.G > 2LL * sms) continue;
        const int rows = (Dmax + t.G - 1) / t.G;
        if (rows * R > kMaxElems) continue;
        const size_t vec = sizeof(double2) * (size_t)Dmax * R, mat = sizeof(double2) * (size_t)rows * Dmax;
        t.resident = vec + mat <= kTeamSmem;
        t.smem = vec + (t.resident ? mat : 0);
        if (t.smem > kTeamSmem || (packed && !t.resident)) continue;
        const bool from_hbm = !t.resident && sizeof(double2) * (size_t)Dmax * Dmax > kL2Matrix;
        const long long waves = ((long long)nsys * t.G + sms - 1) / sms;
        t.cycles = waves * (2LL * 64 * product_cost(rows, Dmax, R, from_hbm, &t.tile, &t.cp) + 5 * (t.cluster ? 1500 : 3300));
        t.ok = true;
        if (!best.ok || t.cycles < best.cycles) best = t;
    }
    if (packed && !best.ok) {   // whole SMs: as few as hold the rows, or up to three quarters of all where that is quicker
        const size_t vec = sizeof(double2) * (size_t)Dmax * R, row = sizeof(double2) * (size_t)Dmax;
        const int most = vec < kWholeSmem ? (int)std::min<size_t>((kWholeSmem - vec) / row, kMaxElems / R) : 0;
        if (most < 1) return best;
        const int least = (Dmax + most - 1) / most;
        if ((long long)nsys * least > sms - sms / 16) return best;
        for (int G = least; G == least || (long long)nsys * G <= sms * 3 / 4; G++) {
            TeamPlan t;
            t.G = G;
            const int rows = (Dmax + G - 1) / G;
            t.resident = true;
            t.smem = vec + rows * row;
            t.cycles = 2LL * 64 * product_cost(rows, Dmax, R, false, &t.tile, &t.cp) + 5 * 3300;
            t.ok = true;
            if (!best.ok || t.cycles < best.cycles) best = t;
        }
    }
    return best;
}

int set_team_wait_limit(long long gemv_cycles) {
    int dev = 0;
    GB_CUDA_TRY(cudaGetDevice(&dev));
    const long long most = 0x7fffffffffffffffLL;
    const long long v = gemv_cycles < 0 ? 0 : gemv_cycles == 0 ? 1 : gemv_cycles > most / 10 ? most : 10 * gemv_cycles;
    g_team_wait[dev % kDevices].store(v, std::memory_order_relaxed);
    return GB_OK;
}

int team_solve(const TeamPlan& t, int nsys, const SysDev* sys, int D, int R, const double2* mat, const double2* tvec,
               const double2* b, double2* x, KState* st, int* err_cnt, double2* vectors, long long total_vec, double tol,
               int maxiter, cudaStream_t stream) {
    TeamArgs a{};
    a.sys = sys;
    a.mat = mat;
    a.tvec = tvec;
    a.b = b;
    a.x = x;
    a.st = st;
    a.err = err_cnt;
    a.cnt = err_cnt + 1;
    a.g1 = vectors;
    a.g2 = vectors + total_vec;
    a.part = reinterpret_cast<double*>(vectors + 2 * total_vec);
    a.tol = tol;
    a.maxiter = maxiter;
    a.D = D;
    a.G = t.G;
    a.resident = t.resident;
    a.CP = t.cp;
    int dev = 0;
    GB_CUDA_TRY(cudaGetDevice(&dev));
    const long long limit = g_team_wait[dev % kDevices].load(std::memory_order_relaxed);
    a.wait = limit ? limit : kTeamWaitCycles;
    GB_CUDA_TRY(cudaMemsetAsync(err_cnt, 0, sizeof(int) * (size_t)(nsys + 1), stream));
    if (R == 1) return sys ? launch_any<1, true>(a, nsys, t, stream) : launch_any<1, false>(a, nsys, t, stream);
    return sys ? launch_any<2, true>(a, nsys, t, stream) : launch_any<2, false>(a, nsys, t, stream);
}

}   // namespace gb
