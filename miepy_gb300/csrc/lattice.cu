// Lattice sums of a periodic cluster (sphere_aggregate_tmatrix_periodic,
// interactions.py:153-186): for every ordered pair (i, j) the sums over the cells c, and
// the origin where i != j, of
//   G[p][mu] = e^{-i k khat.c} P_p^mu(cos theta) h_p(k r) e^{i mu phi}
// of the separation pos_i - pos_j - c.  The translation blocks are linear in G, so the
// assembler forms each block once from the summed table (assemble.cu, mode 2); the origin's
// term is the aggregate's own block.
//
// Bound by the FP64 pipe (one warp instruction per 64 cycles and SM sub-partition), so the
// work per (pair, cell, p, |mu|) is kept to 8 instructions and every lane has a cell:
//   - a CTA takes one pair and a chunk of cells.  Phase A, a thread per cell: cos theta,
//     u = sin theta e^{i phi} and w h_p (w the Bloch factor), whose recurrence
//     h_{p+1} = (2p+1)/x h_p - h_{p-1} starts from one sincos of k r - k khat.c;
//   - phase B, a warp per |mu| (spread so that the sub-partitions carry equal sums), lanes
//     over the cells: u^|mu| and the monic Legendre column q_p, then the four real sums
//     q (Re, Im w h_p)(Re, Im u^|mu|), from which both signs of mu follow;
//   - the lanes reduce by halving exchanges, the Legendre scale kappa_p^mu and the
//     (-1)^mu (p-mu)!/(p+mu)! of negative orders multiply the sums once.
// A pair's chunks put their tables into the pair's own block of the output, which the
// assembler reads back (in order: the result does not depend on scheduling) and then
// overwrites.  Small blocks have room for few tables (two at lmax 1), so where the pairs
// are few as well a chunk's cells are shared by a cluster of up to eight CTAs, whose sums
// the first one adds in order (whole aggregates of 5040 cells: N = 1, lmax 1 126 -> 29 us,
// lmax 3 63 -> 35; N = 2, lmax 1 126 -> 29; N = 6, lmax 1 127 -> 75).  All pairs i = j share
// one sum.  5040 cells, the whole aggregate, against a
// thread per cell for the special functions, the table entries in passes over shared memory
// and atomic adds of the blocks: N = 5, lmax 2 465 -> 84 us, N = 30, lmax 3 21.5 -> 2.9 ms
// (74 % of the FP64 pipe's time for 300 instructions per cell), N = 30, lmax 4 39.3 -> 4.5 ms.

#include <algorithm>

#include "gb_common.cuh"
#include "gb_internal.h"
#include "lattice.h"

namespace {

constexpr int kLatThreads = 256;
constexpr int kPortableCluster = 8;
constexpr int kPM = 2 * GB_LMAX_MAX + 2;

struct LatArgs {
    int N, ncell, nch, per;      // chunks per pair, cells per chunk (the origin is cell 0)
    int split, sub;              // CTAs per chunk (a cluster, if several), cells of each
    const double* pos;
    const double* cells;
    double k, kx, ky, kz;
    const double* neg_ratio;     // [PM][PM]
    double2* out;
    long long ld;
    double kappa[kPM * (kPM + 1) / 2];   // (2p-1)!! / (p-mu)!
};

template <int L> __host__ __device__ constexpr int stage_cells() { return L <= 4 ? 512 : L <= 7 ? 256 : 128; }

// Column MU over the staged cells, added to sums[4 (p - MU) ..] (re re, im im, re im, im re).
template <int L, int MU>
__device__ __forceinline__ void column(const double* __restrict__ st, int n, double* __restrict__ sums) {
    constexpr int PM = 2 * L + 2, SC = stage_cells<L>(), NP = PM - MU, NV = 4 * NP;
    const int lane = threadIdx.x & 31;
    double acc[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) acc[q] = 0.0;
#pragma unroll 1
    for (int c = lane; c < n; c += 32) {
        const double ct = st[2 * PM * SC + c], ux = st[(2 * PM + 1) * SC + c], uy = st[(2 * PM + 2) * SC + c];
        double cr = 1.0, ci = 0.0, br = ux, bi = uy;   // u^MU by binary powering
#pragma unroll
        for (int e = MU; e; e >>= 1) {
            if (e & 1) {
                const double t = cr * br - ci * bi;
                ci = cr * bi + ci * br;
                cr = t;
            }
            if (e > 1) {
                const double t = br * br - bi * bi;
                bi = 2.0 * br * bi;
                br = t;
            }
        }
        double qa = 0.0, qb = 1.0;
#pragma unroll
        for (int q = 0; q < NP; q++) {
            const int p = MU + q;
            if (q > 0) {
                const double g = -(double)((p - 1 - MU) * (p - 1 + MU)) / (double)((2 * p - 3) * (2 * p - 1));
                const double qn = q == 1 ? ct * qb : fma(g, qa, ct * qb);
                qa = qb;
                qb = qn;
            }
            const double hr = st[2 * p * SC + c], hi = st[(2 * p + 1) * SC + c];
            if (MU == 0) {
                acc[4 * q] = fma(qb, hr, acc[4 * q]);
                acc[4 * q + 3] = fma(qb, hi, acc[4 * q + 3]);
            } else {
                const double a = qb * hr, b = qb * hi;
                acc[4 * q] = fma(a, cr, acc[4 * q]);
                acc[4 * q + 1] = fma(b, ci, acc[4 * q + 1]);
                acc[4 * q + 2] = fma(a, ci, acc[4 * q + 2]);
                acc[4 * q + 3] = fma(b, cr, acc[4 * q + 3]);
            }
        }
    }
#pragma unroll
    for (int q0 = 0; q0 < NV; q0 += 32) {
        constexpr int LAST = NV % 32;
        if (q0 + 32 <= NV) {
            double v[32];
#pragma unroll
            for (int q = 0; q < 32; q++) v[q] = acc[q0 + q < NV ? q0 + q : 0];
            const double s = halving_sum<32>(v);
            sums[q0 + lane] += s;
        } else {
            constexpr int V = LAST <= 8 ? 8 : LAST <= 16 ? 16 : 32, SH = V == 8 ? 2 : V == 16 ? 1 : 0;
            double v[V];
#pragma unroll
            for (int q = 0; q < V; q++) v[q] = (q < LAST && q0 + q < NV) ? acc[q0 + q < NV ? q0 + q : 0] : 0.0;
            const double s = halving_sum<V>(v);
            const int at = lane >> SH;
            if ((lane & ((1 << SH) - 1)) == 0 && at < LAST) sums[q0 + at] += s;
        }
    }
}

// The tasks |mu| = 1, 2, .., 2L, 0 in snake order over the four sub-partitions, warps s and
// s + 4 of sub-partition s in turn.
template <int L, int T>
__device__ __forceinline__ void columns(int warp, const double* st, int n, double (*sums)[4 * (2 * L + 2)]) {
    if constexpr (T <= 2 * L) {
        constexpr int MU = T < 2 * L ? T + 1 : 0, row = T / 4, pos = T % 4;
        constexpr int owner = (row & 1 ? 3 - pos : pos) + 4 * (row & 1);
        if (warp == owner) column<L, MU>(st, n, sums[MU]);
        columns<L, T + 1>(warp, st, n, sums);
    }
}

// Every thread of the cluster arrives before any passes.
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}
// *p of the cluster's CTA rank
__device__ __forceinline__ double cluster_read(const double* p, unsigned rank) {
    unsigned at;
    double v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
    return v;
}

// SPLIT: a.split CTAs per chunk (a kernel of its own, so that the other keeps its registers)
template <int L, bool SPLIT>
__global__ void __launch_bounds__(kLatThreads) k_lattice_sums(const __grid_constant__ LatArgs a) {
    constexpr int PM = 2 * L + 2, MM = 2 * L, SC = stage_cells<L>();
    extern __shared__ __align__(16) double st[];                // [2 PM + 3][SC]
    __shared__ double sums[MM + 1][4 * PM];
    const int tid = threadIdx.x, warp = tid >> 5;
    // pairs: (0, 0) for every i = j, then the ordered pairs i != j
    const unsigned unit = SPLIT ? blockIdx.x / a.split : blockIdx.x;
    const int pair = unit / a.nch, chunk = unit - pair * a.nch;
    const int rank = SPLIT ? blockIdx.x - unit * a.split : 0;
    int i = 0, j = 0;
    if (pair > 0) {
        i = (pair - 1) / (a.N - 1);
        j = (pair - 1) - i * (a.N - 1);
        j += j >= i;
    }
    const double px = a.pos[3 * i] - a.pos[3 * j], py = a.pos[3 * i + 1] - a.pos[3 * j + 1],
                 pz = a.pos[3 * i + 2] - a.pos[3 * j + 2];
    for (int e = tid; e < (MM + 1) * 4 * PM; e += kLatThreads) (&sums[0][0])[e] = 0.0;
    int cb = chunk * a.per, c1 = min((chunk + 1) * a.per, a.ncell + 1);
    if constexpr (SPLIT) {
        cb += rank * a.sub;
        c1 = min(c1, cb + a.sub);
    }
    for (int c0 = cb; c0 < c1; c0 += SC) {
        const int n = min(SC, c1 - c0);
        __syncthreads();
        // ---- A: one thread per cell
        for (int e = tid; e < n; e += kLatThreads) {
            const int cell = c0 + e - 1;   // -1: the origin
            double lx = 0.0, ly = 0.0, lz = 0.0;
            if (cell >= 0) {
                lx = a.cells[3LL * cell];
                ly = a.cells[3LL * cell + 1];
                lz = a.cells[3LL * cell + 2];
            }
            const bool none = cell < 0 && pair == 0;   // a particle has no block with itself
            const double dx = none ? 1.0 : px - lx, dy = py - ly, dz = pz - lz;
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double r = sqrt(r2), inv = 1.0 / r;
            const double ix = 1.0 / (a.k * r);
            double s, c;
            sincos(a.k * (r - (a.kx * lx + a.ky * ly + a.kz * lz)), &s, &c);
            // w h_0 = -i e^{i (k r - k khat.c)} / (k r), w h_1 = (1/x - i) w h_0
            double ar = none ? 0.0 : s * ix, ai = none ? 0.0 : -c * ix;
            double br = fma(ar, ix, ai), bi = fma(ai, ix, -ar);
            st[e] = ar;
            st[SC + e] = ai;
            st[2 * SC + e] = br;
            st[3 * SC + e] = bi;
#pragma unroll
            for (int p = 2; p < PM; p++) {
                const double f = (2 * p - 1) * ix;
                const double nr = fma(f, br, -ar), ni = fma(f, bi, -ai);
                ar = br;
                ai = bi;
                br = nr;
                bi = ni;
                st[2 * p * SC + e] = nr;
                st[(2 * p + 1) * SC + e] = ni;
            }
            st[2 * PM * SC + e] = dz * inv;
            st[(2 * PM + 1) * SC + e] = dx * inv;
            st[(2 * PM + 2) * SC + e] = dy * inv;
        }
        __syncthreads();
        // ---- B: a warp per |mu|
        columns<L, 0>(warp, st, n, sums);
    }
    __syncthreads();
    if constexpr (SPLIT) {   // the other CTAs' sums, in order
        cluster_barrier();
        if (rank == 0)
            for (int e = tid; e < (MM + 1) * 4 * PM; e += kLatThreads) {
                double* at = &sums[0][0] + e;
                double v = *at;
                for (int q = 1; q < a.split; q++) v += cluster_read(at, q);
                *at = v;
            }
        cluster_barrier();   // (their shared memory lives until it is read)
        if (rank) return;
    }
    // the chunk's table, entries p^2 + p + mu, into the pair's block (all of i = j: the
    // one sum into every diagonal block)
    const int B = 2 * L * (L + 2), copies = pair == 0 ? a.N : 1;
    for (int e = tid; e < PM * (2 * MM + 1); e += kLatThreads) {
        const int p = e / (2 * MM + 1), mu = e - p * (2 * MM + 1) - MM, am = mu < 0 ? -mu : mu;
        if (am > p) continue;
        const double* x = sums[am] + 4 * (p - am);
        double f = a.kappa[p * (p + 1) / 2 + am];
        double2 g;
        if (mu >= 0) {
            g = make_double2(f * (x[0] - x[1]), f * (x[2] + x[3]));
        } else {
            f *= a.neg_ratio[p * PM + am];
            g = make_double2(f * (x[0] + x[1]), f * (x[3] - x[2]));
        }
        const int at = chunk * (PM * PM) + p * p + p + mu;
        for (int q = 0; q < copies; q++) {
            const long long bi = pair == 0 ? q : i, bj = pair == 0 ? q : j;
            a.out[(bi * B + at / B) * a.ld + bj * B + at % B] = g;
        }
    }
}

template <int L>
int launch(LatArgs a, cudaStream_t stream) {
    const size_t smem = sizeof(double) * (2 * (2 * L + 2) + 3) * stage_cells<L>();
    auto kfn = a.split > 1 ? k_lattice_sums<L, true> : k_lattice_sums<L, false>;
    GB_CUDA_TRY(gb::ensure_dynamic_smem(reinterpret_cast<const void*>(kfn), smem));
    const long long pairs = 1 + (long long)a.N * (a.N - 1);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.blockDim = dim3(kLatThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    for (;; a.split = kPortableCluster) {
        a.sub = (a.per + a.split - 1) / a.split;
        cfg.gridDim = dim3((unsigned)(pairs * a.nch * a.split));
        at[0].val.clusterDim.x = (unsigned)a.split;
        cfg.numAttrs = a.split > 1 ? 1 : 0;
        if (a.split > kPortableCluster)
            GB_CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(kfn),
                                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kfn, a);
        if (a.split > kPortableCluster && (e == cudaErrorInvalidClusterSize || e == cudaErrorLaunchOutOfResources ||
                                           e == cudaErrorInvalidConfiguration)) {   // (part of a device)
            (void)cudaGetLastError();
            continue;
        }
        GB_CUDA_TRY(e);
        break;
    }
    gb::note_launch();
    return GB_OK;
}

}   // namespace

namespace gb {

// Chunks per pair: enough CTAs for three per SM, in equal chunks of at least 128 cells, as
// many as the pair's block has room for tables ((2L+2)^2 of its B^2 entries each).
int lattice_chunks(int N, int lmax, int ncell) {
    const long long B = 2LL * lmax * (lmax + 2), room = B * B / ((2 * lmax + 2) * (2 * lmax + 2));
    const long long pairs = 1 + (long long)N * (N - 1), want = (3LL * sm_count() + pairs - 1) / pairs;
    return (int)std::max<long long>(1, std::min({room, want, (ncell + 128LL) / 128}));
}

// CTAs per chunk: where the chunks are fewer than the SMs, as many more as still have an SM
// each and 16 cells, up to sixteen.  (Beyond one per SM the clusters queue: N = 2, lmax 5, 5040
// cells 79 us with 102 CTAs, 112 with 408.)
static int lattice_split(int N, int ncell, int nch) {
    const long long units = (1 + (long long)N * (N - 1)) * nch;
    int k = 1;
    while (k < 16 && 2 * k * units <= sm_count() && 2LL * k * nch * 16 <= ncell + 1) k *= 2;
    return k;
}

int launch_lattice_sums(int N, int lmax, const double* pos, double k, const double* cells, int ncell, double kx, double ky,
                        double kz, const double* neg_ratio, double2* out, long long ld, cudaStream_t stream) {
    LatArgs a{};
    a.N = N;
    a.ncell = ncell;
    a.nch = lattice_chunks(N, lmax, ncell);
    a.per = (ncell + 1 + a.nch - 1) / a.nch;
    a.split = lattice_split(N, ncell, a.nch);
    a.pos = pos;
    a.cells = cells;
    a.k = k;
    a.kx = kx;
    a.ky = ky;
    a.kz = kz;
    a.neg_ratio = neg_ratio;
    a.out = out;
    a.ld = ld;
    for (int p = 0; p < 2 * lmax + 2; p++)
        for (int m = 0; m <= p; m++) {
            double v = 1.0;
            for (int q = 1; q <= p; q++) v *= 2 * q - 1;
            for (int q = 2; q <= p - m; q++) v /= q;
            a.kappa[p * (p + 1) / 2 + m] = v;
        }
    switch (lmax) {
        case 1: return launch<1>(a, stream);
        case 2: return launch<2>(a, stream);
        case 3: return launch<3>(a, stream);
        case 4: return launch<4>(a, stream);
        case 5: return launch<5>(a, stream);
        case 6: return launch<6>(a, stream);
        case 7: return launch<7>(a, stream);
        case 8: return launch<8>(a, stream);
        default: return launch<9>(a, stream);
    }
}

}   // namespace gb
