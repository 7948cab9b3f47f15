// One particle's VSH expansion at one separation vector, shared by the near-field and
// far-field kernels (expand_E / expand_E_far, vsh/expansion.py:13-77; N and M of
// vsh/vsh_functions.py:40-109).
//
// The sums are arranged for the fewest operations per (point, particle), because the
// FP64 pipe (one warp instruction per 64 cycles and SM sub-partition) or the FP32 pipe
// bounds every kernel that uses them:
//   - the angles enter through cos/sin of theta and phi straight from the separation
//     (no acos, atan2 or per-mode sincos), e^{i m phi} by m - 1 complex products;
//   - P_n^m(cos theta) = kappa_nm sin(theta) q_nm with q monic in cos(theta)
//     (q_nm = cos q_{n-1,m} - gamma q_{n-2,m}: two operations), so pi = m kappa q and
//     tau = kappa (n cos q_nm - (n+m)(n-m)/(2n-1) q_{n-1,m}) need no division by
//     sin(theta) and stay finite on the axis;
//   - E_mn, kappa and the negative-order Legendre factor fold into the coefficients:
//     E_mn P_n^m of order -m is (-1)^m the one of order m, so with w = |E_mn| kappa,
//     A = w (c_m + (-1)^m c_-m) and D = i w (c_m - (-1)^m c_-m) (times the powers of i),
//       c_m e + (+-) c_-m e*  =  cos(m phi) A + sin(m phi) D            (even: s)
//       i (c_m e - (+-) c_-m e*) = cos(m phi) D - sin(m phi) A          (odd: id)
//     which serve P, tau (s) and pi (id) of both orders: 26 multiply-adds per +-m pair;
//   - the radial functions multiply the sums over m once per n.
// In the far form the radial factors (-i)^n fold into the coefficients too.
#pragma once

#include "gb_common.cuh"

namespace gbx {

// ----------------------------------------------------------- value types --
// double: one point; float2: two points in packed f32x2 arithmetic.
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ double vneg(double a) { return -a; }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return fsub2(a, b); }
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }
template <class V> __device__ __forceinline__ V vset(double v);
template <> __device__ __forceinline__ double vset<double>(double v) { return v; }
template <> __device__ __forceinline__ float2 vset<float2>(double v) { return make_float2((float)v, (float)v); }

template <class V> struct CV { V x, y; };
// acc += s z for real s
template <class V> __device__ __forceinline__ void axpy(CV<V>& acc, V s, const CV<V>& z) {
    acc.x = vfma(s, z.x, acc.x);
    acc.y = vfma(s, z.y, acc.y);
}
// acc += (a + i b) z with nb = -b
template <class V> __device__ __forceinline__ void caxpy(CV<V>& acc, V a, V b, V nb, const CV<V>& z) {
    acc.x = vfma(a, z.x, acc.x);
    acc.x = vfma(nb, z.y, acc.x);
    acc.y = vfma(a, z.y, acc.y);
    acc.y = vfma(b, z.x, acc.y);
}

// ---------------------------------------------------------- coefficients --
// w_nm = |E_mn| kappa_nm = sqrt((2n+1)(n-m)! / (n(n+1)(n+m)!)) (2n-1)!! / (n-m)!, m >= 0.
struct FoldW {
    double w[(GB_LMAX_MAX + 1) * (GB_LMAX_MAX + 2) / 2];
};
__host__ __device__ constexpr int fold_at(int n, int m) { return n * (n + 1) / 2 + m; }
inline FoldW fold_weights() {
    FoldW f{};
    for (int n = 1; n <= GB_LMAX_MAX; n++)
        for (int m = 0; m <= n; m++) {
            double ratio = 1.0, odd = 1.0, low = 1.0;   // (n-m)!/(n+m)!, (2n-1)!!, (n-m)!
            for (int q = n - m + 1; q <= n + m; q++) ratio /= q;
            for (int q = 1; q <= n; q++) odd *= 2 * q - 1;
            for (int q = 2; q <= n - m; q++) low *= q;
            f.w[fold_at(n, m)] = sqrt((2.0 * n + 1) / ((double)n * (n + 1)) * ratio) * odd / low;
        }
    return f;
}

// Folded coefficients of one particle: for every n, the m = 0 entry (a for P, a and b for
// tau: 3 complex values), then A_a, D_a, A_b, D_b of m = 1..n (4 complex values each).
__host__ __device__ constexpr int fold_count(int L) { return 3 * L + 2 * L * (L + 1); }
__host__ __device__ constexpr int fold_n(int n) { return 3 * (n - 1) + 2 * (n - 1) * n; }   // start of order n

__device__ __forceinline__ double2 mul_i(double2 z, int k) {
    switch (k & 3) {
        case 0: return z;
        case 1: return make_double2(-z.y, z.x);
        case 2: return make_double2(-z.x, -z.y);
        default: return make_double2(z.y, -z.x);
    }
}

enum Form { OUTGOING = 0, REGULAR = 1, FAR = 2 };
// powers of i of the N (a) and M (b) coefficients: i i^n outgoing, -i i^n regular; far:
// the radial (-i)^n and (-i)^(n+1) folded in
__device__ __forceinline__ int phase_a(int form, int n) { return form == FAR ? 1 : n + (form == REGULAR ? 3 : 1); }
__device__ __forceinline__ int phase_b(int form, int n) { return form == FAR ? 0 : n + (form == REGULAR ? 3 : 1); }

// The 3 (m = 0) or 4 folded values of (n, m) from the particle's coefficients ca (N) and
// cb (M), each [rmax].
__device__ __forceinline__ void fold_nm(const FoldW& f, int form, int n, int m, const double2* __restrict__ ca,
                                        const double2* __restrict__ cb, double2 (&v)[4]) {
    const int r = n * n + n - 1;   // of (n, 0)
    const double w = f.w[fold_at(n, m)];
    const int pa = phase_a(form, n), pb = phase_b(form, n);
    if (m == 0) {
        const double2 a = ca[r], b = cb[r];
        v[0] = mul_i(make_double2(w * a.x, w * a.y), pa);
        v[1] = mul_i(make_double2(-n * w * a.x, -n * w * a.y), pa);   // tau_n0 = -P_n1
        v[2] = mul_i(make_double2(-n * w * b.x, -n * w * b.y), pb);
        return;
    }
    const double sg = (m & 1) ? -w : w;
    const double2 ap = ca[r + m], am = ca[r - m], bp = cb[r + m], bm = cb[r - m];
    v[0] = mul_i(make_double2(fma(sg, am.x, w * ap.x), fma(sg, am.y, w * ap.y)), pa);
    v[1] = mul_i(make_double2(fma(-sg, am.x, w * ap.x), fma(-sg, am.y, w * ap.y)), pa + 1);
    v[2] = mul_i(make_double2(fma(sg, bm.x, w * bp.x), fma(sg, bm.y, w * bp.y)), pb);
    v[3] = mul_i(make_double2(fma(-sg, bm.x, w * bp.x), fma(-sg, bm.y, w * bp.y)), pb + 1);
}

// ------------------------------------------------------------- the sums --
template <class V> struct Dir { V ct, st, cp, sp; };   // cos/sin of theta and phi

// Radial factors of one n: z_n, (z x)'/x = z_{n-1} - n z_n / x, n (n+1) z_n / x, with the
// negated parts that their products take (packed arithmetic negates no operand).
template <class V> struct Rad { V zr, nzr, zi, nzi, dr, di, ndi, hr, hi, nhi; };

// Adds the expansion's spherical components (E_r, E_theta, E_phi).  radial(n) gives Rad
// for n = 1..L in order (unused in the far form); coef(n, m, v) the folded values.
template <int L, int FORM, class V, class RadialFn, class CoefFn>
__device__ __forceinline__ void expansion(const Dir<V>& d, RadialFn radial, CoefFn coef, CV<V>& Er, CV<V>& Et, CV<V>& Ep) {
    const V zero = vset<V>(0.0);
    V er[L + 1], ei[L + 1], nei[L + 1];   // e^{i m phi}
    V qc[L + 1], qp[L + 1];               // q_nm and q_{n-1,m}, m >= 1
    V p0 = vset<V>(1.0), p0p = zero, diag = vset<V>(1.0);
    CV<V> Ft{zero, zero}, Fp{zero, zero}, Fq{zero, zero};   // far: sums over n
#pragma unroll
    for (int n = 1; n <= L; n++) {
        {   // m = 0: monic P_n
            const V t = vmul(d.ct, p0);
            const double g = n < 2 ? 0.0 : -(double)((n - 1) * (n - 1)) / (double)((2 * n - 3) * (2 * n - 1));
            const V pn = n < 2 ? t : vfma(vset<V>(g), p0p, t);
            p0p = p0;
            p0 = pn;
        }
#pragma unroll
        for (int m = 1; m < n; m++) {
            const double g = -(double)((n - 1 - m) * (n - 1 + m)) / (double)((2 * n - 3) * (2 * n - 1));
            const V t = vmul(d.ct, qc[m]);
            const V q = (n - 1 == m) ? t : vfma(vset<V>(g), qp[m], t);
            qp[m] = qc[m];
            qc[m] = q;
        }
        if (n == 1) {
            er[1] = d.cp;
            ei[1] = d.sp;
        } else {
            diag = vmul(diag, d.st);
            er[n] = vfma(nei[n - 1], d.sp, vmul(er[n - 1], d.cp));
            ei[n] = vfma(ei[n - 1], d.cp, vmul(er[n - 1], d.sp));
        }
        nei[n] = vneg(ei[n]);
        qc[n] = diag;
        qp[n] = zero;
        const V nct = vmul(vset<V>((double)n), d.ct);
        CV<V> R{zero, zero}, T{zero, zero}, T2{zero, zero}, F{zero, zero}, F2{zero, zero};
        {
            CV<V> v[4];
            coef(n, 0, v);
            const V t0 = vmul(d.st, qc[1]);
            if (FORM != FAR) R = CV<V>{vmul(p0, v[0].x), vmul(p0, v[0].y)};
            if (FORM != FAR) {
                T = CV<V>{vmul(t0, v[1].x), vmul(t0, v[1].y)};
                F2 = CV<V>{vmul(t0, v[2].x), vmul(t0, v[2].y)};
            } else {
                axpy(Ft, t0, v[1]);
                axpy(Fq, t0, v[2]);
            }
        }
#pragma unroll
        for (int m = 1; m <= n; m++) {
            CV<V> v[4];   // A_a, D_a, A_b, D_b
            coef(n, m, v);
            const CV<V> sa{vfma(ei[m], v[1].x, vmul(er[m], v[0].x)), vfma(ei[m], v[1].y, vmul(er[m], v[0].y))};
            const CV<V> ia{vfma(nei[m], v[0].x, vmul(er[m], v[1].x)), vfma(nei[m], v[0].y, vmul(er[m], v[1].y))};
            const CV<V> sb{vfma(ei[m], v[3].x, vmul(er[m], v[2].x)), vfma(ei[m], v[3].y, vmul(er[m], v[2].y))};
            const CV<V> ib{vfma(nei[m], v[2].x, vmul(er[m], v[3].x)), vfma(nei[m], v[2].y, vmul(er[m], v[3].y))};
            const double g = -(double)((n + m) * (n - m)) / (double)(2 * n - 1);
            V tau = vmul(nct, qc[m]);
            if (m < n) tau = vfma(vset<V>(g), qp[m], tau);
            const V mp = (m == 1) ? qc[m] : vmul(vset<V>((double)m), qc[m]);
            if (FORM != FAR) {
                axpy(R, vmul(d.st, qc[m]), sa);
                axpy(T, tau, sa);
                axpy(T2, mp, ib);
                axpy(F, mp, ia);
                axpy(F2, tau, sb);
            } else {
                axpy(Ft, tau, sa);
                axpy(Ft, mp, ib);
                axpy(Fp, mp, ia);
                axpy(Fq, tau, sb);
            }
        }
        if (FORM != FAR) {
            const Rad<V> z = radial(n);
            caxpy(Er, z.hr, z.hi, z.nhi, R);
            caxpy(Et, z.dr, z.di, z.ndi, T);
            caxpy(Et, z.zr, z.zi, z.nzi, T2);
            caxpy(Ep, z.dr, z.di, z.ndi, F);
            caxpy(Ep, z.nzr, z.nzi, z.zi, F2);   // - z F2
        }
    }
    if (FORM == FAR) {
        Et.x = vadd(Et.x, Ft.x);
        Et.y = vadd(Et.y, Ft.y);
        Ep.x = vadd(Ep.x, vsub(Fp.x, Fq.x));
        Ep.y = vadd(Ep.y, vsub(Fp.y, Fq.y));
    }
}

// E (Cartesian) += (E_r, E_theta, E_phi) along the direction's unit vectors.
template <bool RADIAL, class V>
__device__ __forceinline__ void add_cartesian(const Dir<V>& d, const CV<V>& Er, const CV<V>& Et, const CV<V>& Ep,
                                              CV<V> (&E)[3]) {
    const V nsp = vneg(d.sp), nst = vneg(d.st);
    CV<V> h{vmul(Et.x, d.ct), vmul(Et.y, d.ct)};
    if (RADIAL) axpy(h, d.st, Er);
    axpy(E[0], d.cp, h);
    axpy(E[0], nsp, Ep);
    axpy(E[1], d.sp, h);
    axpy(E[1], d.cp, Ep);
    if (RADIAL) axpy(E[2], d.ct, Er);
    axpy(E[2], nst, Et);
}

// ------------------------------------------------------------- geometry --
// 1/sqrt(v) and sqrt(v), the root corrected by one Newton step.
__device__ __forceinline__ void root(double v, double& inv, double& s) {
    inv = rsqrt(v);
    s = v * inv;
    s = fma(fma(-s, s, v), 0.5 * inv, s);
}
__device__ __forceinline__ void direction(double dx, double dy, double dz, double rho2, double inv_r, Dir<double>& d) {
    double cp = 1.0, sp = 0.0, rho = 0.0;   // phi = 0 on the z axis
    if (rho2 > 0.0) {
        double inv;
        root(rho2, inv, rho);
        cp = dx * inv;
        sp = dy * inv;
    }
    d.ct = dz * inv_r;
    d.st = rho * inv_r;
    d.cp = cp;
    d.sp = sp;
}

// h_n(x) = j_n + i y_n of real x by the upward recurrences, one n per call (n = 1, 2, ...).
template <class V> struct Outgoing {
    V ix, ja, ya, jb, yb;   // n - 1 and n
    __device__ __forceinline__ Rad<V> operator()(int n) {
        if (n > 1) {
            const V f = vmul(vset<V>((double)(2 * n - 1)), ix);
            const V jn = vfma(f, jb, vneg(ja)), yn = vfma(f, yb, vneg(ya));
            ja = jb;
            ya = yb;
            jb = jn;
            yb = yn;
        }
        Rad<V> r;
        const V nix = vmul(vset<V>((double)n), ix);
        const V qr = vmul(nix, jb), qi = vmul(nix, yb);
        r.zr = jb;
        r.nzr = vneg(jb);
        r.zi = yb;
        r.nzi = vneg(yb);
        r.dr = vsub(ja, qr);
        r.di = vsub(ya, qi);
        r.ndi = vsub(qi, ya);
        r.hr = vmul(vset<V>((double)(n + 1)), qr);
        r.hi = vmul(vset<V>((double)(n + 1)), qi);
        r.nhi = vmul(vset<V>(-(double)(n + 1)), qi);
        return r;
    }
    // from sin(x), cos(x) and 1/x
    __device__ __forceinline__ void start(V s, V c, V inv_x) {
        ix = inv_x;
        ja = vmul(s, inv_x);
        ya = vneg(vmul(c, inv_x));
        jb = vfma(ja, inv_x, ya);
        yb = vfma(ya, inv_x, vneg(ja));
    }
};

}   // namespace gbx
