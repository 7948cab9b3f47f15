// K8: fields of a cluster on a set of points.
//
// Near field: sphere_cluster.E_field / H_field (sphere_cluster.py:244-391): outside the
// spheres the outgoing expansions of p_scat about every particle are summed (expand_E,
// vsh/expansion.py:13-42); a point inside sphere i instead takes the interior expansion
// of p_int[i] with j_n(k_int r) (complex argument).  H fields use expand_H: the
// polarisation-swapped coefficients times -i sqrt(eps/mu).  Far field: the far-field form
// of the expansions (expand_E_far, vsh/expansion.py:45-77) at Cartesian points, or at
// (R, theta, phi) about the origin in theta and phi components (E_angular / H_angular,
// sphere_cluster.py:393-426).  The sums per (point, particle) are in expansion.cuh.
//
// k_field64 (FP64).  Bound by the FP64 pipe (a warp instruction per 64 cycles and SM
// sub-partition), so a lane takes one point and the particles of a group of 32 points are
// split over 1 to 8 warps, enough warps to fill every sub-partition evenly; the warps'
// sums are added in order (deterministic).  The folded coefficients of a tile of
// particles are formed by the CTA in shared memory.  Against a thread per point with FP64
// trigonometry and complex divisions per mode: far fields at 7200 directions of 50
// spheres, lmax 4, 3237 -> 355 us; a whole E_field call on 97 x 100 points around 25
// spheres, lmax 4, 5.28 -> 1.40 ms (the kernel was 4.17 ms of it).
//
// k_field32 (FP32 exterior sums for large maps: a 512 x 512 plane around thousands of
// spheres is ~5e8 point-particle terms).  Bound by the FP32 pipe; a thread takes two
// points in packed f32x2 arithmetic and reads every folded coefficient once for both
// (16-byte broadcast loads of duplicated pairs).  Coordinates, from the first particle's
// position, are split into two floats so that separations keep FP32 accuracy without FP64
// arithmetic (their error is 2^-48 of the extent of points and particles, wherever the
// origin lies); k r is reduced with a
// two-float k / pi, which the phase of distant spheres needs.  Points inside a sphere are
// found by the FP32 distance, decided in FP64 and collected, so that their FP64 interior
// expansions run on full warps.  512 x 512 points, 2000 spheres, lmax 3: 30.7 -> 7.6 ms
// (535 warp instructions per particle and 64 points; with fewer than three warps per sub-partition, the
// last of its 1.7 waves, the packed FMA pipe is 54 % busy).

#include <algorithm>

#include "expansion.cuh"
#include "gb_common.cuh"
#include "gb_internal.h"

namespace {

using namespace gbx;

constexpr int kLF = 8;              // largest expansion order of the near-field kernels
constexpr int kLFF = GB_LMAX_MAX;   // largest order of the angular far field
constexpr int kTileBytes = 32 * 1024;

struct FieldArgs {
    int N, Npts, interior, swap;
    const double* pos;
    const double* radius;
    const double2* p_scat;
    const double2* p_int;
    double k;
    const double2* k_int;
    const double* pts;                        // [Npts][3], or R, theta, phi
    const double *th, *ph;
    double ox, oy, oz;
    double2 pref;                             // 1, or the magnetic prefactor
    const double2* hfac_int;
    double2* out;
    FoldW fold;
};

__device__ __forceinline__ double2 cdivd(double2 a, double2 b) {
    const double den = 1.0 / (b.x * b.x + b.y * b.y);
    return make_double2((a.x * b.x + a.y * b.y) * den, (a.y * b.x - a.x * b.y) * den);
}

// j_n of complex x, n = 0..L + 1.  The upward recurrence (the reference's,
// cpp/src/special.cpp:20-45) multiplies its rounding errors by about
// |y_n / j_n| ~ ((2n-1)!!)^2 / |x|^(2n+1) once n > |x|, so it serves only |x| >= L + 2;
// below that the values come from Miller's downward recurrence
// j_{n-1} = (2n+1)/x j_n - j_{n+1}, started at n = L + 26 from (j, j+1) = (1, 0) and
// normalised by j_0 = sin(x)/x or j_1 = j_0/x - cos(x)/x, whichever is larger in modulus
// (they have no common zero).
template <int L>
__device__ __forceinline__ void bessel_j(double2 x, double2 ix, double2 (&z)[L + 2]) {
    constexpr int NP = L + 2;
    double s, c, sh = 0.0, ch = 1.0;
    sincos(x.x, &s, &c);
    if (x.y != 0.0) {
        sh = sinh(x.y);
        ch = cosh(x.y);
    }
    const double2 e0 = cmul(make_double2(s * ch, c * sh), ix);
    const double2 t1 = cmul(e0, ix), u1 = cmul(make_double2(c * ch, -s * sh), ix);
    const double2 e1 = make_double2(t1.x - u1.x, t1.y - u1.y);
    if (x.x * x.x + x.y * x.y >= (double)(NP * NP)) {
        z[0] = e0;
        z[1] = e1;
#pragma unroll
        for (int n = 2; n < NP; n++) {
            const double2 f = make_double2((2 * n - 1) * ix.x, (2 * n - 1) * ix.y);
            const double2 a = cmul(f, z[n - 1]);
            z[n] = make_double2(a.x - z[n - 2].x, a.y - z[n - 2].y);
        }
        return;
    }
    double2 hi = make_double2(0.0, 0.0), cur = make_double2(1.0, 0.0);   // j_{n+1}, j_n (unscaled)
    auto down = [&](int n) {   // j_{n-1}
        const double2 a = cmul(make_double2((2 * n + 1) * ix.x, (2 * n + 1) * ix.y), cur);
        const double2 lo = make_double2(a.x - hi.x, a.y - hi.y);
        hi = cur;
        cur = lo;
    };
#pragma unroll 1
    for (int n = NP + 24; n > NP; n--) {
        down(n);
        if (fabs(cur.x) + fabs(cur.y) > 1e150) {   // keep the unnormalised values finite
            hi = make_double2(hi.x * 1e-150, hi.y * 1e-150);
            cur = make_double2(cur.x * 1e-150, cur.y * 1e-150);
        }
    }
#pragma unroll
    for (int n = NP; n >= 1; n--) {
        down(n);
        z[n - 1] = cur;
        if (fabs(cur.x) + fabs(cur.y) > 1e150) {
            hi = make_double2(hi.x * 1e-150, hi.y * 1e-150);
            cur = make_double2(cur.x * 1e-150, cur.y * 1e-150);
#pragma unroll
            for (int q = 0; q < NP; q++)
                if (q >= n - 1) z[q] = make_double2(z[q].x * 1e-150, z[q].y * 1e-150);
        }
    }
    const bool use0 = e0.x * e0.x + e0.y * e0.y >= e1.x * e1.x + e1.y * e1.y;
    const double2 sc = use0 ? cdivd(e0, z[0]) : cdivd(e1, z[1]);
#pragma unroll
    for (int n = 0; n < NP; n++) z[n] = cmul(sc, z[n]);
}

// The interior field of sphere i at (X, Y, Z), written to out.
template <int L>
__device__ __noinline__ void interior_field(const FieldArgs& a, int i, double X, double Y, double Z, double2* out) {
    constexpr int rmax = L * (L + 2);
    const double dx = X - a.pos[3 * i], dy = Y - a.pos[3 * i + 1], dz = Z - a.pos[3 * i + 2];
    const double rho2 = dx * dx + dy * dy;
    double inv_r, r;
    root(rho2 + dz * dz, inv_r, r);
    Dir<double> d;
    direction(dx, dy, dz, rho2, inv_r, d);
    const double2 ki = a.k_int[i];
    const double2 x = make_double2(ki.x * r, ki.y * r);
    const double2 ix = cdivd(make_double2(1.0, 0.0), x);
    double2 z[L + 2];
    bessel_j<L>(x, ix, z);
    const double2* ca = a.p_int + (long long)i * 2 * rmax + (a.swap ? rmax : 0);
    const double2* cb = a.p_int + (long long)i * 2 * rmax + (a.swap ? 0 : rmax);
    auto radial = [&](int n) {
        const double2 q = cmul(make_double2(n * ix.x, n * ix.y), z[n]);
        Rad<double> f;
        f.zr = z[n].x; f.nzr = -z[n].x; f.zi = z[n].y; f.nzi = -z[n].y;
        f.dr = z[n - 1].x - q.x; f.di = z[n - 1].y - q.y; f.ndi = -f.di;
        f.hr = (n + 1) * q.x; f.hi = (n + 1) * q.y; f.nhi = -f.hi;
        return f;
    };
    auto coef = [&](int n, int m, CV<double>(&v)[4]) {
        double2 w[4];
        fold_nm(a.fold, REGULAR, n, m, ca, cb, w);
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = CV<double>{w[q].x, w[q].y};
    };
    CV<double> Er{0, 0}, Et{0, 0}, Ep{0, 0}, E[3] = {{0, 0}, {0, 0}, {0, 0}};
    expansion<L, REGULAR, double>(d, radial, coef, Er, Et, Ep);
    add_cartesian<true, double>(d, Er, Et, Ep, E);
    const double2 pref = a.hfac_int && a.swap ? a.hfac_int[i] : make_double2(1.0, 0.0);
    for (int c = 0; c < 3; c++) out[c] = cmul(pref, make_double2(E[c].x, E[c].y));
}

// Item it of a tile's folding work: particle it / (entries), entry (n, m) in order.
template <int L>
__device__ __forceinline__ void fold_item(int e, int& n, int& m) {
    n = 1;
    while ((n + 1) * (n + 2) / 2 - 1 <= e) n++;
    m = e - (n * (n + 1) / 2 - 1);
}
__host__ __device__ constexpr int fold_entries(int L) { return L * (L + 3) / 2; }   // (n, m), 1 <= n <= L, 0 <= m <= n
template <int L>
__host__ __device__ constexpr int fold_slot(int n, int m) { return m == 0 ? fold_n(n) : fold_n(n) + 3 + 4 * (m - 1); }

// blockDim = 32 PG PS: warp w takes the points of group w / PS and the particles q with
// q % PS == w % PS of every tile.  ANGULAR: points (R, theta, phi) about the origin, out
// [Npts][2]; otherwise Cartesian points, out [Npts][3].
template <int L, int FORM, bool ANGULAR>
__global__ void __launch_bounds__(256) k_field64(const __grid_constant__ FieldArgs a, int PS) {
    constexpr int rmax = L * (L + 2), NC = fold_count(L), NE = fold_entries(L);
    constexpr int kTile = kTileBytes / (NC * 16) < 32 ? kTileBytes / (NC * 16) : 32;
    static_assert(kTile >= 1, "a particle's coefficients fit in a tile");
    __shared__ __align__(16) double2 tile[kTileBytes / 16];
    __shared__ double spos[32][3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, PG = (blockDim.x >> 5) / PS;
    const int split = w % PS;
    const int pt = (blockIdx.x * PG + w / PS) * 32 + lane;
    const bool valid = pt < a.Npts;
    double X = 0, Y = 0, Z = 0, st0 = 0, ct0 = 1, sp0 = 0, cp0 = 1;
    if (valid) {
        if (ANGULAR) {
            sincos(a.th[pt], &st0, &ct0);
            sincos(a.ph[pt], &sp0, &cp0);
            const double R = a.pts[pt];
            X = a.ox + R * st0 * cp0;
            Y = a.oy + R * st0 * sp0;
            Z = a.oz + R * ct0;
        } else {
            X = a.pts[3LL * pt];
            Y = a.pts[3LL * pt + 1];
            Z = a.pts[3LL * pt + 2];
        }
    }
    const double ik = 1.0 / a.k;
    int inside = -1;
    CV<double> E[3] = {{0, 0}, {0, 0}, {0, 0}};
    const int step = PS * (kTile / PS > 0 ? kTile / PS : 1);
    for (int t0 = 0; t0 < a.N; t0 += step) {
        const int cnt = min(step, a.N - t0);
        __syncthreads();
        for (int e = threadIdx.x; e < cnt * 3; e += blockDim.x) spos[e / 3][e % 3] = a.pos[3LL * t0 + e];
        for (int e = threadIdx.x; e < cnt * NE; e += blockDim.x) {
            const int q = e / NE;
            int n, m;
            fold_item<L>(e - q * NE, n, m);
            const double2* c = a.p_scat + (long long)(t0 + q) * 2 * rmax;
            double2 v[4];
            fold_nm(a.fold, FORM, n, m, c + (a.swap ? rmax : 0), c + (a.swap ? 0 : rmax), v);
            double2* dst = tile + q * NC + fold_slot<L>(n, m);
            for (int i = 0; i < (m ? 4 : 3); i++) dst[i] = v[i];
        }
        __syncthreads();
        if (!valid) continue;
#pragma unroll 1
        for (int q = split; q < cnt; q += PS) {
            const double dx = X - spos[q][0], dy = Y - spos[q][1], dz = Z - spos[q][2];
            const double rho2 = dx * dx + dy * dy, r2 = rho2 + dz * dz;
            if (FORM == OUTGOING && a.interior) {
                const double rs = a.radius[t0 + q];
                if (r2 < rs * rs) inside = t0 + q;   // the last match wins, as in the reference's loop
            }
            double inv_r, r;
            root(r2, inv_r, r);
            Dir<double> d;
            direction(dx, dy, dz, rho2, inv_r, d);
            double s, c;
            sincos(a.k * r, &s, &c);
            const double ix = ik * inv_r;
            const double2* cf = tile + q * NC;
            auto coef = [&](int n, int m, CV<double>(&v)[4]) {
#pragma unroll
                for (int i = 0; i < (m ? 4 : 3); i++) {
                    const double2 u = cf[fold_slot<L>(n, m) + i];
                    v[i] = CV<double>{u.x, u.y};
                }
            };
            Outgoing<double> h;
            if (FORM == OUTGOING) h.start(s, c, ix);
            CV<double> Er{0, 0}, Et{0, 0}, Ep{0, 0};
            expansion<L, FORM, double>(d, h, coef, Er, Et, Ep);
            if (FORM == FAR) {   // e^{ikr} / (kr)
                const double fr = c * ix, fi = s * ix;
                CV<double> t{0, 0}, p{0, 0};
                caxpy(t, fr, fi, -fi, Et);
                caxpy(p, fr, fi, -fi, Ep);
                Et = t;
                Ep = p;
            }
            add_cartesian<FORM == OUTGOING, double>(d, Er, Et, Ep, E);
        }
    }
    // the splits' sums, added in order by the group's first warp
    if (PS > 1) {
        __syncthreads();
        double* red = reinterpret_cast<double*>(tile);           // [warps][6][32]
        int* rin = reinterpret_cast<int*>(red + 8 * 6 * 32);     // [warps][32]
        if (split) {
            for (int c = 0; c < 3; c++) {
                red[(w * 6 + 2 * c) * 32 + lane] = E[c].x;
                red[(w * 6 + 2 * c + 1) * 32 + lane] = E[c].y;
            }
            rin[w * 32 + lane] = inside;
        }
        __syncthreads();
        if (split) return;
        for (int q = 1; q < PS; q++) {
            for (int c = 0; c < 3; c++) {
                E[c].x += red[((w + q) * 6 + 2 * c) * 32 + lane];
                E[c].y += red[((w + q) * 6 + 2 * c + 1) * 32 + lane];
            }
            inside = max(inside, rin[(w + q) * 32 + lane]);
        }
    }
    if (!valid) return;
    if (ANGULAR) {   // Cartesian -> (theta, phi) components at the point
        const double tt[3] = {ct0 * cp0, ct0 * sp0, -st0}, pp[3] = {-sp0, cp0, 0.0};
        double2 Eth = make_double2(0, 0), Eph = make_double2(0, 0);
        for (int c = 0; c < 3; c++) {
            Eth.x += E[c].x * tt[c]; Eth.y += E[c].y * tt[c];
            Eph.x += E[c].x * pp[c]; Eph.y += E[c].y * pp[c];
        }
        a.out[2LL * pt] = cmul(a.pref, Eth);
        a.out[2LL * pt + 1] = cmul(a.pref, Eph);
        return;
    }
    if (FORM == OUTGOING && inside >= 0) {
        if constexpr (FORM == OUTGOING) interior_field<L>(a, inside, X, Y, Z, a.out + 3LL * pt);
        return;
    }
    for (int c = 0; c < 3; c++) a.out[3LL * pt + c] = cmul(a.pref, make_double2(E[c].x, E[c].y));
}

// ------------------------------------------------------------ FP32 field --
constexpr int kThreads32 = 128;
constexpr int kPoints32 = 2 * kThreads32;

__device__ __forceinline__ float rsqrt_approx(float v) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ float2 bc(float v) { return make_float2(v, v); }

template <int L>
__global__ void __launch_bounds__(kThreads32, L <= 4 ? 4 : 2)
k_field32(const __grid_constant__ FieldArgs a, float kpi_h, float kpi_l, float ik) {
    constexpr int rmax = L * (L + 2), NC = fold_count(L), NE = fold_entries(L);
    constexpr int kTile = kTileBytes / (NC * 16) < 32 ? kTileBytes / (NC * 16) : 32;
    __shared__ __align__(16) float4 tile[kTile * NC];   // (re, re, im, im)
    __shared__ float4 spos[kTile][2];                   // x.h, y.h, z.h, test radius^2; x.l, y.l, z.l
    __shared__ int n_in, list[kPoints32];
    const int tid = threadIdx.x;
    const long long p0 = (long long)blockIdx.x * kPoints32 + tid, p1 = p0 + kThreads32;
    const double o[3] = {a.pos[0], a.pos[1], a.pos[2]};
    float2 Xh[3], Xl[3];
    for (int c = 0; c < 3; c++) {
        const double u = p0 < a.Npts ? a.pts[3 * p0 + c] - o[c] : 0.0, v = p1 < a.Npts ? a.pts[3 * p1 + c] - o[c] : 0.0;
        Xh[c] = make_float2((float)u, (float)v);
        Xl[c] = make_float2((float)(u - (double)Xh[c].x), (float)(v - (double)Xh[c].y));
    }
    if (tid == 0) n_in = 0;
    int in0 = -1, in1 = -1;
    const float2 zero = make_float2(0.f, 0.f);
    CV<float2> E[3] = {{zero, zero}, {zero, zero}, {zero, zero}};
    for (int t0 = 0; t0 < a.N; t0 += kTile) {
        const int cnt = min(kTile, a.N - t0);
        __syncthreads();
        for (int q = tid; q < cnt; q += kThreads32) {
            float h[3], l[3];
            for (int c = 0; c < 3; c++) {
                const double v = a.pos[3LL * (t0 + q) + c] - o[c];
                h[c] = (float)v;
                l[c] = (float)(v - (double)h[c]);
            }
            // points nearer than this are decided in FP64
            const double rs = a.interior ? a.radius[t0 + q] : 0.0;
            spos[q][0] = make_float4(h[0], h[1], h[2], a.interior ? (float)(rs * rs * 1.0001) : -1.f);
            spos[q][1] = make_float4(l[0], l[1], l[2], 0.f);
        }
        for (int e = tid; e < cnt * NE; e += kThreads32) {
            const int q = e / NE;
            int n, m;
            fold_item<L>(e - q * NE, n, m);
            const double2* c = a.p_scat + (long long)(t0 + q) * 2 * rmax;
            double2 v[4];
            fold_nm(a.fold, OUTGOING, n, m, c + (a.swap ? rmax : 0), c + (a.swap ? 0 : rmax), v);
            float4* dst = tile + q * NC + fold_slot<L>(n, m);
            for (int i = 0; i < (m ? 4 : 3); i++) {
                const float x = (float)v[i].x, y = (float)v[i].y;
                dst[i] = make_float4(x, x, y, y);
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int q = 0; q < cnt; q++) {
            const float4 ph = spos[q][0], pl = spos[q][1];
            // (Xh - ph) exactly by TwoSum, its error added to the low parts: the separation
            // rounded once, as an FP64 difference rounded to FP32 would be
            auto diff = [](float2 xh, float2 xl, float p_h, float p_l) {
                const float2 p = bc(p_h), t = vsub(xh, p), bb = vsub(t, xh);
                const float2 e = vsub(vsub(xh, vsub(t, bb)), vadd(p, bb));
                return vadd(t, vadd(e, vsub(xl, bc(p_l))));
            };
            const float2 dx = diff(Xh[0], Xl[0], ph.x, pl.x), dy = diff(Xh[1], Xl[1], ph.y, pl.y),
                         dz = diff(Xh[2], Xl[2], ph.z, pl.z);
            const float2 rho2 = vfma(dx, dx, vmul(dy, dy));
            const float2 r2 = vfma(dz, dz, rho2);
            if (fminf(r2.x, r2.y) < ph.w) {   // perhaps inside: the last match wins
                const double* pp = a.pos + 3LL * (t0 + q);
                const double rs = a.radius[t0 + q];
                auto test = [&](long long pt, int& in) {
                    if (pt >= a.Npts) return;
                    const double x = a.pts[3 * pt] - pp[0], y = a.pts[3 * pt + 1] - pp[1], z = a.pts[3 * pt + 2] - pp[2];
                    if (x * x + y * y + z * z < rs * rs) in = t0 + q;
                };
                test(p0, in0);
                test(p1, in1);
            }
            // r and 1/r, each corrected by a Newton step; likewise 1/rho
            float2 ir = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
            float2 r = vmul(r2, ir);
            r = vfma(vfma(vneg(r), r, r2), vmul(bc(0.5f), ir), r);
            ir = vfma(vfma(vneg(r), ir, bc(1.f)), ir, ir);
            const bool ax0 = !(rho2.x > 1e-36f), ax1 = !(rho2.y > 1e-36f);   // phi = 0 on the z axis
            float2 ih = make_float2(rsqrt_approx(rho2.x), rsqrt_approx(rho2.y));
            float2 rho = vmul(rho2, ih);
            rho = vfma(vfma(vneg(rho), rho, rho2), vmul(bc(0.5f), ih), rho);
            ih = vfma(vfma(vneg(rho), ih, bc(1.f)), ih, ih);
            Dir<float2> d;
            d.ct = vmul(dz, ir);
            d.st = vmul(rho, ir);
            d.cp = vmul(dx, ih);
            d.sp = vmul(dy, ih);
            if (ax0) { d.st.x = 0.f; d.cp.x = 1.f; d.sp.x = 0.f; }
            if (ax1) { d.st.y = 0.f; d.cp.y = 1.f; d.sp.y = 0.f; }
            // k r = pi (2 j + f): f from the two-float k / pi
            const float2 u = vmul(r, bc(kpi_h));
            const float2 j = make_float2(2.f * rintf(0.5f * u.x), 2.f * rintf(0.5f * u.y));
            const float2 f = vfma(r, bc(kpi_l), vfma(r, bc(kpi_h), vneg(j)));
            float2 s, c;
            sincospif(f.x, &s.x, &c.x);
            sincospif(f.y, &s.y, &c.y);
            Outgoing<float2> h;
            h.start(s, c, vmul(ir, bc(ik)));
            const float4* cf = tile + q * NC;
            auto coef = [&](int n, int m, CV<float2>(&v)[4]) {
#pragma unroll
                for (int i = 0; i < (m ? 4 : 3); i++) {
                    const float4 w = cf[fold_slot<L>(n, m) + i];
                    v[i] = CV<float2>{make_float2(w.x, w.y), make_float2(w.z, w.w)};
                }
            };
            CV<float2> Er{zero, zero}, Et{zero, zero}, Ep{zero, zero};
            expansion<L, OUTGOING, float2>(d, h, coef, Er, Et, Ep);
            add_cartesian<true, float2>(d, Er, Et, Ep, E);
        }
    }
    auto store = [&](long long pt, int in, bool second) {
        if (pt >= a.Npts) return;
        if (in >= 0) {
            list[atomicAdd(&n_in, 1)] = tid + (second ? kThreads32 : 0);
            // the sphere's index waits in the point's own output (read back below)
            a.out[3 * pt] = make_double2((double)in, 0.0);
            return;
        }
        for (int c = 0; c < 3; c++)
            a.out[3 * pt + c] = cmul(a.pref, second ? make_double2(E[c].x.y, E[c].y.y) : make_double2(E[c].x.x, E[c].y.x));
    };
    store(p0, in0, false);
    store(p1, in1, true);
    __syncthreads();
    for (int e = tid; e < n_in; e += kThreads32) {
        const long long pt = (long long)blockIdx.x * kPoints32 + list[e];
        const int i = (int)a.out[3 * pt].x;
        interior_field<L>(a, i, a.pts[3 * pt], a.pts[3 * pt + 1], a.pts[3 * pt + 2], a.out + 3 * pt);
    }
}

template <int L, int FORM, bool ANGULAR>
int launch64(const FieldArgs& a, cudaStream_t s) {
    // splits of the particles: enough warps for three per SM sub-partition
    const long long groups = ((long long)a.Npts + 31) / 32, want = 12LL * gb::sm_count();
    int PS = 1;
    while (PS < 8 && 2 * PS <= a.N && groups * PS < want) PS *= 2;
    const int PG = groups * PS >= want && PS < 4 ? 4 / PS : 1;
    const unsigned grid = (unsigned)((groups + PG - 1) / PG);
    gb::note_launch();
    k_field64<L, FORM, ANGULAR><<<grid, 32 * PG * PS, 0, s>>>(a, PS);
    GB_CUDA_TRY(cudaGetLastError());
    return GB_OK;
}

template <int L>
int launch32(const FieldArgs& a, cudaStream_t s) {
    const double kpi = a.k / 3.14159265358979323846;
    const float h = (float)kpi, l = (float)(kpi - (double)h);
    gb::note_launch();
    k_field32<L><<<(unsigned)((a.Npts + (long long)kPoints32 - 1) / kPoints32), kThreads32, 0, s>>>(a, h, l,
                                                                                                    (float)(1.0 / a.k));
    GB_CUDA_TRY(cudaGetLastError());
    return GB_OK;
}

FieldArgs field_args(int N, const double* pos, const double* p_scat, double k, int Npts, const double* pts, int magnetic,
                     double hfac_re, double hfac_im, double* out) {
    FieldArgs a{};
    a.N = N;
    a.Npts = Npts;
    a.swap = magnetic != 0;
    a.pos = pos;
    a.p_scat = reinterpret_cast<const double2*>(p_scat);
    a.k = k;
    a.pts = pts;
    a.pref = magnetic ? make_double2(hfac_re, hfac_im) : make_double2(1.0, 0.0);
    a.out = reinterpret_cast<double2*>(out);
    static const FoldW w = fold_weights();
    a.fold = w;
    return a;
}

// one instance per order
#define GB_BY_LMAX8(CALL)                                            \
    switch (lmax) {                                                  \
        case 1: return CALL(1);                                      \
        case 2: return CALL(2);                                      \
        case 3: return CALL(3);                                      \
        case 4: return CALL(4);                                      \
        case 5: return CALL(5);                                      \
        case 6: return CALL(6);                                      \
        case 7: return CALL(7);                                      \
        default: return CALL(8);                                     \
    }

int near_field(bool fp32, int N, int lmax, const double* pos, const double* radius, const double* p_scat,
               const double* p_int, double k, const double* k_int, int Npts, const double* pts, int interior,
               int magnetic, double hfac_re, double hfac_im, const double* hfac_int, double* out, void* stream) {
    if (N < 1 || Npts < 0 || !pos || !p_scat || !pts || !out) return gb_set_error(GB_BAD_ARG, "bad field arguments");
    if (interior && (!radius || !p_int || !k_int)) return gb_set_error(GB_BAD_ARG, "interior fields need radius, p_int, k_int");
    if (magnetic && interior && !hfac_int) return gb_set_error(GB_BAD_ARG, "interior H fields need hfac_int");
    if (Npts == 0) return GB_OK;
    if (lmax < 1 || lmax > kLF) return gb_set_error(GB_UNSUPPORTED, "near field supports lmax 1..%d (got %d)", kLF, lmax);
    FieldArgs a = field_args(N, pos, p_scat, k, Npts, pts, magnetic, hfac_re, hfac_im, out);
    a.interior = interior != 0;
    a.radius = radius;
    a.p_int = reinterpret_cast<const double2*>(p_int);
    a.k_int = reinterpret_cast<const double2*>(k_int);
    a.hfac_int = reinterpret_cast<const double2*>(hfac_int);
    const cudaStream_t s = (cudaStream_t)stream;
#define GB_F32(Lv) launch32<Lv>(a, s)
#define GB_F64(Lv) launch64<Lv, OUTGOING, false>(a, s)
    if (fp32) GB_BY_LMAX8(GB_F32)
    GB_BY_LMAX8(GB_F64)
#undef GB_F32
#undef GB_F64
}

}   // namespace

extern "C" int gb_near_field(int N, int lmax, const double* pos, const double* radius, const double* p_scat,
                             const double* p_int, double k, const double* k_int, int Npts, const double* pts,
                             int interior, int magnetic, double hfac_re, double hfac_im, const double* hfac_int,
                             double* out, void* stream) {
    return near_field(false, N, lmax, pos, radius, p_scat, p_int, k, k_int, Npts, pts, interior, magnetic, hfac_re,
                      hfac_im, hfac_int, out, stream);
}

// Same arguments and result as gb_near_field, with the exterior sums in FP32.
extern "C" int gb_near_field32(int N, int lmax, const double* pos, const double* radius, const double* p_scat,
                               const double* p_int, double k, const double* k_int, int Npts, const double* pts,
                               int interior, int magnetic, double hfac_re, double hfac_im, const double* hfac_int,
                               double* out, void* stream) {
    return near_field(true, N, lmax, pos, radius, p_scat, p_int, k, k_int, Npts, pts, interior, magnetic, hfac_re,
                      hfac_im, hfac_int, out, stream);
}

// The far-field form of every particle's outgoing expansion, summed at the points
// (sphere_cluster.E_field / H_field with far=True, sphere_cluster.py:244-391, with
// expand_E_far / expand_H_far, vsh/expansion.py:45-77,96-108): no interior
// expansions; H fields swap the coefficients and take the prefactor hfac.
extern "C" int gb_far_field_expansions(int N, int lmax, const double* pos, const double* p_scat, double k, int Npts,
                                       const double* pts, int magnetic, double hfac_re, double hfac_im, double* out,
                                       void* stream) {
    if (N < 1 || Npts < 0 || !pos || !p_scat || !pts || !out) return gb_set_error(GB_BAD_ARG, "bad field arguments");
    if (lmax < 1 || lmax > kLF) return gb_set_error(GB_UNSUPPORTED, "far field supports lmax 1..%d (got %d)", kLF, lmax);
    if (Npts == 0) return GB_OK;
    const FieldArgs a = field_args(N, pos, p_scat, k, Npts, pts, magnetic, hfac_re, hfac_im, out);
    const cudaStream_t s = (cudaStream_t)stream;
#define GB_FAR(Lv) launch64<Lv, FAR, false>(a, s)
    GB_BY_LMAX8(GB_FAR)
#undef GB_FAR
}

extern "C" int gb_far_field(int N, int lmax, const double* pos, const double* p_scat, double k, const double* origin,
                            int Npts, const double* radius, const double* theta, const double* phi, int magnetic,
                            double hfac_re, double hfac_im, double* out, void* stream) {
    if (N < 1 || Npts < 0 || !pos || !p_scat || !origin || !out) return gb_set_error(GB_BAD_ARG, "bad far-field arguments");
    if (lmax < 1 || lmax > kLFF) return gb_set_error(GB_UNSUPPORTED, "far field supports lmax 1..%d", kLFF);
    if (Npts == 0) return GB_OK;
    if (!radius || !theta || !phi) return gb_set_error(GB_BAD_ARG, "null point arrays");
    FieldArgs a = field_args(N, pos, p_scat, k, Npts, radius, magnetic, hfac_re, hfac_im, out);
    a.th = theta;
    a.ph = phi;
    a.ox = origin[0];   // host array
    a.oy = origin[1];
    a.oz = origin[2];
    const cudaStream_t s = (cudaStream_t)stream;
#define GB_ANG(Lv) launch64<Lv, FAR, true>(a, s)
    if (lmax == 9) return GB_ANG(9);
    if (lmax == 10) return GB_ANG(10);
    GB_BY_LMAX8(GB_ANG)
#undef GB_ANG
}
