// Cluster expansion coefficients and far fields.
//
// p_cluster: the scattered field of every particle re-expanded about one origin
// (cluster_coefficients, vsh/cluster_coefficients.py:14-53): for particle i at
// x_i != origin, with (r, theta, phi) of origin - x_i,
//   p_cluster[0][n,m] += sum_{v,u} a_i(v,u) A + b_i(v,u) B
//   p_cluster[1][n,m] += sum_{v,u} a_i(v,u) B + b_i(v,u) A,
// A, B = vsh_translation(m, n, u, v, r, theta, phi, k, incident)
// (cpp/src/vsh_translation.cpp:428-470): the folded Gaunt coefficients of the cross
// tables times G[p][mu] = P_p^mu(cos theta) j_p(k r) e^{i mu phi}.  j_p follows the
// reference's upward recurrence (cpp/src/special.cpp:20-45), which loses digits for
// p > k r, as the reference's own values do.  A particle at the origin adds its own
// coefficients.  One CTA per particle writes its contribution; a second kernel sums
// the particles in index order (deterministic).

#include <algorithm>
#include <cstring>
#include <vector>

#include "gb_common.cuh"
#include "gb_internal.h"

namespace {

constexpr int kCCThreads = 256;
constexpr int kPMax = 2 * GB_LMAX_MAX + 2;      // orders p <= Lc + Lin + 1
constexpr int kMUMax = 4 * GB_LMAX_MAX + 1;     // |mu| <= Lc + Lin

__device__ __forceinline__ double2 mul_ipow_cc(double2 z, int k) {
    switch (k & 3) {
        case 0: return z;
        case 1: return make_double2(-z.y, z.x);
        case 2: return make_double2(-z.x, -z.y);
        default: return make_double2(z.y, -z.x);
    }
}

__global__ void __launch_bounds__(kCCThreads)
k_cluster_contrib(int N, int Lin, int Lc, const double* __restrict__ pos, const double2* __restrict__ p_scat,
                  double k, double ox, double oy, double oz, const int4* __restrict__ nmvu,
                  const int2* __restrict__ qab, const double* __restrict__ cA, const double* __restrict__ cB,
                  int Q, const double* __restrict__ neg_ratio, double2* __restrict__ contrib) {
    __shared__ double jp[kPMax];
    __shared__ double Pl[kPMax][kPMax];
    __shared__ double2 eph[kMUMax];
    __shared__ double2 G[kPMax][kMUMax];
    __shared__ double geo[6];
    const int ri = Lin * (Lin + 2), rc = Lc * (Lc + 2);
    const int PM = Lc + Lin + 1;            // orders p = 0 .. Lc + Lin
    const int MO = Lc + Lin;                // |mu| <= MO
    const int MU = 2 * MO + 1;
    const int PMn = Lc + Lin + 2;           // stride of neg_ratio
    const int tid = threadIdx.x;
    for (int i = blockIdx.x; i < N; i += gridDim.x) {
        const double2* ps = p_scat + (long long)i * 2 * ri;
        double2* out = contrib + (long long)i * 2 * rc;
        const double dx = ox - pos[3 * i], dy = oy - pos[3 * i + 1], dz = oz - pos[3 * i + 2];
        if (dx == 0.0 && dy == 0.0 && dz == 0.0) {   // particle at the origin: its own coefficients
            for (int e = tid; e < 2 * rc; e += kCCThreads) {
                const int a = e / rc, r = e % rc;
                out[e] = (r < ri) ? ps[a * ri + r] : make_double2(0.0, 0.0);
            }
            __syncthreads();
            continue;
        }
        if (tid == 0) {
            const double rho2 = dx * dx + dy * dy;
            const double rad = sqrt(rho2 + dz * dz);
            const double rho = sqrt(rho2);
            geo[0] = dz / rad;                           // cos(theta)
            geo[1] = rho / rad;                          // sin(theta)
            geo[2] = rho2 > 0.0 ? dx / rho : 1.0;        // cos(phi); phi = 0 on the z axis
            geo[3] = rho2 > 0.0 ? dy / rho : 0.0;        // sin(phi)
            // j_p(k r) by the reference's upward recurrence
            const double z = k * rad;
            double sz, cz;
            sincos(z, &sz, &cz);
            double j2p = sz / z;
            jp[0] = j2p;
            if (PM > 1) {
                double j1 = j2p / z - cz / z;
                jp[1] = j1;
                for (int p = 2; p < PM; p++) {
                    const double jn = (2.0 * p - 1.0) / z * j1 - j2p;
                    j2p = j1;
                    j1 = jn;
                    jp[p] = jn;
                }
            }
        }
        __syncthreads();
        // Legendre P_p^mu (no Condon-Shortley phase), one thread per mu; e^{i mu phi}
        if (tid < PM) {
            const int mu = tid;
            const double x = geo[0], u = geo[1];
            double pmm = 1.0;
            for (int kk = 1; kk <= mu; kk++) pmm *= (2 * kk - 1) * u;
            Pl[mu][mu] = pmm;
            if (mu + 1 < PM) {
                double pa = pmm, pb = x * (2 * mu + 1) * pmm;
                Pl[mu + 1][mu] = pb;
                for (int q = mu + 2; q < PM; q++) {
                    const double pc = ((2 * q - 1) * x * pb - (q + mu - 1) * pa) / (double)(q - mu);
                    Pl[q][mu] = pc;
                    pa = pb;
                    pb = pc;
                }
            }
        } else if (tid >= 64 && tid < 64 + MO + 1) {
            const int mu = tid - 64;
            int e = mu;
            double2 acc = make_double2(1.0, 0.0), base = make_double2(geo[2], geo[3]);
            while (e) {
                if (e & 1) acc = cmul(acc, base);
                base = cmul(base, base);
                e >>= 1;
            }
            eph[MO + mu] = acc;
            eph[MO - mu] = make_double2(acc.x, -acc.y);
        }
        __syncthreads();
        for (int e = tid; e < PM * MU; e += kCCThreads) {
            const int q = e / MU, mi = e % MU, mu = mi - MO, am = mu < 0 ? -mu : mu;
            double2 g = make_double2(0.0, 0.0);
            if (am <= q) {
                double P = Pl[q][am];
                if (mu < 0) P *= neg_ratio[q * PMn + am];
                const double f = P * jp[q];
                g = make_double2(f * eph[mi].x, f * eph[mi].y);
            }
            G[q][mi] = g;
        }
        __syncthreads();
        // one thread per outgoing mode (n, m): sum over the particle's modes (v, u)
        for (int r = tid; r < rc; r += kCCThreads) {
            double2 acc0 = make_double2(0.0, 0.0), acc1 = make_double2(0.0, 0.0);
            for (int s = 0; s < ri; s++) {
                const int t = r * ri + s;
                const int4 e4 = nmvu[t];
                const int2 qq = qab[t];
                const int mi = (e4.w - e4.y) + MO;
                const int nv = e4.x + e4.z;
                double2 sa = make_double2(0.0, 0.0), sb = make_double2(0.0, 0.0);
                for (int q = 0; q <= qq.x; q++) {
                    const double c = cA[(size_t)t * Q + q];
                    const double2 gv = G[nv - 2 * q][mi];
                    sa.x = fma(c, gv.x, sa.x);
                    sa.y = fma(c, gv.y, sa.y);
                }
                for (int q = 1; q <= qq.y; q++) {
                    const double c = cB[(size_t)t * Q + q];
                    const double2 gv = G[nv - 2 * q + 1][mi];
                    sb.x = fma(c, gv.x, sb.x);
                    sb.y = fma(c, gv.y, sb.y);
                }
                const double2 A = mul_ipow_cc(sa, nv), Bt = mul_ipow_cc(sb, nv + 1);
                const double2 a = ps[s], b = ps[ri + s];
                cfma(acc0, a, A);
                cfma(acc0, b, Bt);
                cfma(acc1, a, Bt);
                cfma(acc1, b, A);
            }
            out[r] = acc0;
            out[rc + r] = acc1;
        }
        __syncthreads();
    }
}

__global__ void k_cluster_sum(int N, int n2rc, const double2* __restrict__ contrib, double2* __restrict__ out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n2rc) return;
    double2 s = make_double2(0.0, 0.0);
    for (int i = 0; i < N; i++) {
        const double2 v = contrib[(long long)i * n2rc + e];
        s.x += v.x;
        s.y += v.y;
    }
    out[e] = s;
}

}   // namespace

extern "C" {

size_t gb_cluster_coefficients_workspace_size(int N, int lmax_cluster) {
    if (N < 1 || lmax_cluster < 1) return 0;
    return sizeof(double2) * 2 * (size_t)lmax_to_rmax(lmax_cluster) * N;
}

int gb_cluster_coefficients(int N, int lmax, const double* pos, const double* p_scat, double k, const double* origin,
                            int lmax_cluster, double* p_cluster, void* workspace, size_t ws_bytes, void* stream) {
    if (N < 1 || !pos || !p_scat || !origin || !p_cluster || !workspace)
        return gb_set_error(GB_BAD_ARG, "bad cluster-coefficient arguments");
    if (lmax < 1 || lmax > GB_LMAX_MAX || lmax_cluster < 1 || lmax_cluster > GB_LMAX_MAX)
        return gb_set_error(GB_UNSUPPORTED, "orders must be in 1..%d (got %d, %d)", GB_LMAX_MAX, lmax, lmax_cluster);
    if (ws_bytes < gb_cluster_coefficients_workspace_size(N, lmax_cluster))
        return gb_set_error(GB_OVER_BUDGET, "workspace too small for %d particles", N);
    if (lmax_to_rmax(lmax_cluster) > kCCThreads * 64) return gb_set_error(GB_UNSUPPORTED, "lmax_cluster too large");
    cudaStream_t s = (cudaStream_t)stream;
    const gb::CrossTables* T = nullptr;
    int e = gb::get_cross_tables(lmax_cluster, lmax, s, &T);
    if (e) return e;
    double o[3];
    memcpy(o, origin, sizeof(o));   // host array
    const int grid = std::min(N, gb::sm_count() * 8);
    double2* contrib = static_cast<double2*>(workspace);
    gb::note_launch();
    k_cluster_contrib<<<grid, kCCThreads, 0, s>>>(N, lmax, lmax_cluster, pos, reinterpret_cast<const double2*>(p_scat),
                                                  k, o[0], o[1], o[2], T->nmvu, T->qab, T->cA, T->cB, T->Q,
                                                  T->neg_ratio, contrib);
    GB_CUDA_TRY(cudaGetLastError());
    const int n2rc = 2 * lmax_to_rmax(lmax_cluster);
    gb::note_launch();
    k_cluster_sum<<<(n2rc + 127) / 128, 128, 0, s>>>(N, n2rc, contrib, reinterpret_cast<double2*>(p_cluster));
    GB_CUDA_TRY(cudaGetLastError());
    return GB_OK;
}

}   // extern "C"
