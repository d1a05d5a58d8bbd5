/*
 * gexs_device.cuh — device arithmetic of the cross-section kernels.
 *
 * FP64 helpers round every operation as written (no fused multiply-add), so
 * that grid frequencies, window limits and Humlicek region limits are the
 * same doubles the reference computes: BaseProfile.cpp:17-21 builds the
 * grid as start + i*dfreq and Managers/CPU/OpenMPManager.cpp:399-408 and
 * compute/CPU/profiles.cpp:17-28 compare such values against thresholds.
 */
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "../../include/gexs_b200.h"
#include "gh_nodes.h"

namespace gexs {

/* ------------------------------------------------ exactly-rounded FP64 ops */
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

/* grid frequency f_j = nu_start + j*dnu, two roundings */
__device__ __forceinline__ double grid_f(double nu_start, double dnu, int64_t j)
{
    return dadd(nu_start, dmul((double)j, dnu));
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

/* ---------------------------------------------------- Humlicek W4 pieces
 * K(x, y) = Re w(x + iy) by Humlicek's four regions (compute/CPU/profiles.cpp
 * :11-44, constants as there).  T = y - i x.  The caller selects the region.
 * Region I has the closed form Re[T c/(1/2 + T^2)] = c y (p + x^2) /
 * ((p + x^2)^2 - 2 x^2), p = 1/2 + y^2; regions II-IV use complex Horner
 * evaluation in real arithmetic and Re(N/D) = (Nr Dr + Ni Di)/|D|^2. */
template <typename R> struct HC;
template <> struct HC<float> {
    static __device__ __forceinline__ float k(double v) { return (float)v; }
};
template <> struct HC<double> {
    static __device__ __forceinline__ double k(double v) { return v; }
};

template <typename R>
__device__ __forceinline__ R hum_region1(R x, R y)
{
    R x2 = x * x;
    R num = x2 + (R(0.5) + y * y);
    R den = num * num - R(2) * x2;
    return HC<R>::k(0.5641896) * y * num / den;
}

/* 1/d in FP64: the hardware's approximate reciprocal refined by one step of
 * Householder's third-order iteration, r (1 + e + e^2) with e = 1 - d r
 * (e ~ 2^-20, so the truncation is ~2^-60): three FMAs against the longer
 * instruction sequence of the IEEE division.  For finite d with 1/d normal
 * (no special cases); within 1 ulp of the correctly rounded value: against
 * __drcp_rn on 6e8 random d of 2^-1021 to 2^1022, 0.03% differ by one ulp
 * and none by more. */
__device__ __forceinline__ double rcp_f64(double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

/* Regions II-IV with every rounding written out: a bin's value depends on
 * which products the compiler contracts, and the core kernel has two copies
 * of each region (its dense and its sparse walk), chosen by the 32 lines of
 * a group.  Left to the compiler, 1183 of 80,001 bins of a 2000-line FP64
 * list differed between tile shapes, by up to 47 ulp (region IV cancels). */
__device__ __forceinline__ double re_div(double nr, double ni, double dr, double di)
{
    /* |d|^2 is between ~1e-1 and ~1e30 in regions II-IV */
    return dmul(fma(nr, dr, dmul(ni, di)), rcp_f64(fma(dr, dr, dmul(di, di))));
}

template <typename R> __device__ __forceinline__ R hum_region2(R x, R y);
template <>
__device__ __forceinline__ double hum_region2<double>(double x, double y)
{
    /* T (1.410474 + .5641896 U) / (.75 + U (3 + U)), U = T^2 */
    const double ur = fma(-x, x, dmul(y, y)), ui = dmul(dmul(-2.0, x), y);
    const double ar = fma(.5641896, ur, 1.410474), ai = dmul(.5641896, ui);
    /* N = T * a, T = (y, -x) */
    const double nr = fma(x, ai, dmul(y, ar)), ni = fma(y, ai, -dmul(x, ar));
    /* D = .75 + U*(3+U) */
    const double br = dadd(3.0, ur);
    const double dr = dadd(.75, fma(ur, br, -dmul(ui, ui)));
    const double di = fma(ur, ui, dmul(ui, br));
    return re_div(nr, ni, dr, di);
}

/* FP32: one approximate reciprocal (1 ulp) instead of an IEEE division */
template <>
__device__ __forceinline__ float hum_region2<float>(float x, float y)
{
    const float c0 = (float)1.410474, c1 = (float).5641896;
    const float ur = __fmaf_rn(-x, x, __fmul_rn(y, y)), ui = __fmul_rn(__fmul_rn(-2.f, x), y);
    const float ar = __fmaf_rn(c1, ur, c0), ai = __fmul_rn(c1, ui);
    const float nr = __fmaf_rn(x, ai, __fmul_rn(y, ar)), ni = __fmaf_rn(y, ai, -__fmul_rn(x, ar));
    const float br = __fadd_rn(3.f, ur);
    const float dr = __fadd_rn(.75f, __fmaf_rn(ur, br, -__fmul_rn(ui, ui)));
    const float di = __fmaf_rn(ur, ui, __fmul_rn(ui, br));
    return __fmul_rn(__fmaf_rn(nr, dr, __fmul_rn(ni, di)),
                     rcp_approx(__fmaf_rn(dr, dr, __fmul_rn(di, di))));
}

/* p = c + t*p */
__device__ __forceinline__ void cmul_add(double& pr, double& pi, double tr, double ti, double c)
{
    const double r = fma(tr, pr, -dmul(ti, pi));
    pi = fma(tr, pi, dmul(ti, pr));
    pr = dadd(c, r);
}

__device__ __forceinline__ double hum_region3(double x, double y)
{
    const double tr = y, ti = -x;
    double nr = .5642236, ni = 0.0;
    cmul_add(nr, ni, tr, ti, 3.778987);
    cmul_add(nr, ni, tr, ti, 11.96482);
    cmul_add(nr, ni, tr, ti, 20.20933);
    cmul_add(nr, ni, tr, ti, 16.4955);
    double dr = 1.0, di = 0.0;
    cmul_add(dr, di, tr, ti, 6.699398);
    cmul_add(dr, di, tr, ti, 21.69274);
    cmul_add(dr, di, tr, ti, 39.27121);
    cmul_add(dr, di, tr, ti, 38.82363);
    cmul_add(dr, di, tr, ti, 16.4955);
    return re_div(nr, ni, dr, di);
}

__device__ __forceinline__ float expcos(float a, float b) { return expf(a) * cosf(b); }

__device__ __forceinline__ double hum_region4(double x, double y)
{
    /* exp(U) - T P(U)/Q(U); P, Q written as polynomials in V = -U */
    const double ur = fma(-x, x, dmul(y, y)), ui = dmul(dmul(-2.0, x), y);
    const double vr = -ur, vi = -ui;
    double pr = .56419, pi = 0.0;
    cmul_add(pr, pi, vr, vi, 1.320522);
    cmul_add(pr, pi, vr, vi, 35.76683);
    cmul_add(pr, pi, vr, vi, 219.0313);
    cmul_add(pr, pi, vr, vi, 1540.787);
    cmul_add(pr, pi, vr, vi, 3321.9905);
    cmul_add(pr, pi, vr, vi, 36183.31);
    double qr = 1.0, qi = 0.0;
    cmul_add(qr, qi, vr, vi, 1.841439);
    cmul_add(qr, qi, vr, vi, 61.57037);
    cmul_add(qr, qi, vr, vi, 364.2191);
    cmul_add(qr, qi, vr, vi, 2186.181);
    cmul_add(qr, qi, vr, vi, 9022.228);
    cmul_add(qr, qi, vr, vi, 24322.84);
    cmul_add(qr, qi, vr, vi, 32066.6);
    /* T * P, T = (y, -x) */
    const double nr = fma(x, pi, dmul(y, pr)), ni = fma(y, pi, -dmul(x, pr));
    return dsub(dmul(exp(ur), cos(ui)), re_div(nr, ni, qr, qi));
}

/* p(z) of a polynomial with real coefficients c[0..N] (ascending) at the
 * complex z with s = 2 Re z and q = |z|^2, by division by z's quadratic
 * factor (Knuth, TAOCP 2, 4.6.4): two FMAs per coefficient against four of
 * the complex Horner form.  p = u + z v. */
template <int N>
__device__ __forceinline__ void quad_horner(const double (&c)[N + 1], double s, double q,
                                            double& u, double& v)
{
    double b1 = c[N], b2 = 0.0;
#pragma unroll
    for (int k = N - 1; k >= 1; --k) {
        const double b = k == N - 1 ? fma(s, b1, c[k]) : fma(s, b1, fma(-q, b2, c[k]));
        b2 = b1; b1 = b;
    }
    v = b1;
    u = fma(-q, b2, c[0]);
}

/* Regions III and IV for the FP32 form's core: the rational parts in FP64
 * (their real part comes out of a mostly imaginary quotient, so FP32
 * rounding would be amplified), exp(U) cos(Im U) in FP32.  The division by
 * the quadratic factor loses a few bits more than complex Horner (~2e-13 of
 * the result), far below the FP32 form's rounding.  In region IV |x| < 5.5
 * and y < 0.195|x| - 0.176, so Re U >= -30.25 (no underflow), |Im U| < 10,
 * and Re w = exp-term + a non-negative part: the FP32 error of the exp term
 * (a few 1e-7 of that term) is at most a few 1e-7 of the result. */
__device__ __forceinline__ double hum_region3_core(double x, double y)
{
    /* T = (y, -x) */
    const double s = 2.0 * y, q = fma(x, x, y * y);
    const double cn[5] = {16.4955, 20.20933, 11.96482, 3.778987, .5642236};
    const double cd[6] = {16.4955, 38.82363, 39.27121, 21.69274, 6.699398, 1.0};
    double nu, nv, du, dv;
    quad_horner<4>(cn, s, q, nu, nv);
    quad_horner<5>(cd, s, q, du, dv);
    const double nr = fma(y, nv, nu), ni = -x * nv, dr = fma(y, dv, du), di = -x * dv;
    return fma(nr, dr, ni * di) * rcp_f64(fma(dr, dr, di * di));
}

__device__ __forceinline__ double hum_region4_core(double x, double y)
{
    /* V = -U = (x^2 - y^2, 2 x y); P, Q polynomials in V */
    const double vr = fma(x, x, -(y * y)), vi = 2.0 * x * y;
    const double h = fma(x, x, y * y), s = 2.0 * vr, q = h * h;
    const double cp[7] = {36183.31, 3321.9905, 1540.787, 219.0313, 35.76683, 1.320522, .56419};
    const double cq[8] = {32066.6, 24322.84, 9022.228, 2186.181, 364.2191, 61.57037, 1.841439, 1.0};
    double pu, pv, qu, qv;
    quad_horner<6>(cp, s, q, pu, pv);
    quad_horner<7>(cq, s, q, qu, qv);
    const double pr = fma(vr, pv, pu), pi = vi * pv, qr = fma(vr, qv, qu), qi = vi * qv;
    const double nr = fma(y, pr, x * pi), ni = fma(y, pi, -(x * pr));
    return (double)expcos((float)-vr, (float)-vi) -
           fma(nr, qr, ni * qi) * rcp_f64(fma(qr, qr, qi * qi));
}

/* regions II-IV by the tests of compute/CPU/profiles.cpp:24,31 */
static __device__ __noinline__ double hum_core_f64(double x, double y)
{
    if (dadd(x, y) >= 5.5) return hum_region2<double>(x, y);
    if (y >= dsub(dmul(0.195, x), 0.176)) return hum_region3(x, y);
    return hum_region4(x, y);
}

/* --------------------------------------------------- Gauss-Hermite Voigt
 * sum_k w_k (A + B)/(A B), A = y2 + (x - t_k)^2, B = y2 + (x + t_k)^2,
 * ascending t_k; the caller multiplies by y/pi. */
template <int NODES> struct GH;
template <> struct GH<16> { static constexpr int NP = 8; };
template <> struct GH<32> { static constexpr int NP = 16; };

template <int NODES>
__host__ __device__ __forceinline__ constexpr double gh_t(int k)
{
    constexpr double t16[8] = {GEXS_GH16_T_LIST};
    constexpr double t32[16] = {GEXS_GH32_T_LIST};
    return NODES == 16 ? t16[k] : t32[k];
}
template <int NODES>
__host__ __device__ __forceinline__ constexpr double gh_w(int k)
{
    constexpr double w16[8] = {GEXS_GH16_W_LIST};
    constexpr double w32[16] = {GEXS_GH32_W_LIST};
    return NODES == 16 ? w16[k] : w32[k];
}

/* FP32, NP pairs of bins on packed f32x2 instructions, nodes outermost so
 * that a node's constants serve every pair: eight packed instructions and
 * two MUFU reciprocals per pair and node pair.  Both pipes then need 16
 * cycles of a scheduler per warp; one bin at a time took 16 + 2 issues.
 * Every rounding is that of the scalar sum w (A + B) * rcp(A B). */
template <int NODES, int NP>
__device__ __forceinline__ void gh_sum2_f32(const float2 (&x)[NP], float y2, float2 (&acc)[NP])
{
    const float2 yy = make_float2(y2, y2);
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < GH<NODES>::NP; ++k) {
        const float t = (float)gh_t<NODES>(k), w = (float)gh_w<NODES>(k);
        const float2 tp = make_float2(t, t), tm = make_float2(-t, -t), ww = make_float2(w, w);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const float2 d1 = __fadd2_rn(x[j], tm), d2 = __fadd2_rn(x[j], tp);
            const float2 A = __ffma2_rn(d1, d1, yy), B = __ffma2_rn(d2, d2, yy);
            const float2 D = __fmul2_rn(A, B);
            float2 r;
            r.x = rcp_approx(D.x); r.y = rcp_approx(D.y);
            acc[j] = __ffma2_rn(__fmul2_rn(ww, __fadd2_rn(A, B)), r, acc[j]);
        }
    }
}

/* Lines much narrower than a node spacing (y < 1/8): near a node t_k the
 * term w_k / (y^2 + (x - t_k)^2) is a spike of width y, and an x carried
 * in one float (absolute error ~1e-7 x) would put a relative error of
 * about 1e-7 x / |x - t_k| on it.  Here x is the unevaluated pair xs + xl
 * (x_pair below, error ~1e-13) and x - t_k is taken against the node split
 * the same way, so every difference keeps its relative accuracy. */
template <int NODES, int NP>
__device__ __forceinline__ void gh_sum2_f32_pair(const float2 (&xs)[NP], const float2 (&xl)[NP],
                                                 float y2, float2 (&acc)[NP])
{
    const float2 yy = make_float2(y2, y2);
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < GH<NODES>::NP; ++k) {
        const double tk = gh_t<NODES>(k);
        const float th = (float)tk, tl = (float)(tk - (double)th), w = (float)gh_w<NODES>(k);
        const float2 tp = make_float2(th, th), tm = make_float2(-th, -th);
        const float2 lm = make_float2(-tl, -tl), ww = make_float2(w, w);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            /* xs - th is exact when xs is within a factor 2 of th (Sterbenz) */
            const float2 d1 = __fadd2_rn(__fadd2_rn(xs[j], tm), __fadd2_rn(xl[j], lm));
            const float2 d2 = __fadd2_rn(xs[j], tp);
            const float2 A = __ffma2_rn(d1, d1, yy), B = __ffma2_rn(d2, d2, yy);
            const float2 D = __fmul2_rn(A, B);
            float2 r;
            r.x = rcp_approx(D.x); r.y = rcp_approx(D.y);
            acc[j] = __ffma2_rn(__fmul2_rn(ww, __fadd2_rn(A, B)), r, acc[j]);
        }
    }
}

/* x = (n - fc) dx as the pair xs + xl from n (an exact integer in float),
 * dx = dxh + dxl and mf = -fc dx = mfh + mfl (each split from FP64 on the
 * host of the record): TwoProduct of n dxh and TwoSum with mfh, written
 * with _rn intrinsics so that no step is contracted into an FMA. */
__device__ __forceinline__ void x_pair(float n, float dxh, float dxl, float mfh, float mfl,
                                       float& xs, float& xl)
{
    const float p = __fmul_rn(n, dxh);
    const float e1 = __fmaf_rn(n, dxh, -p);
    const float s = __fadd_rn(p, mfh);
    const float bb = __fsub_rn(s, p);
    const float e2 = __fadd_rn(__fsub_rn(p, __fsub_rn(s, bb)), __fsub_rn(mfh, bb));
    const float lo = __fadd_rn(__fadd_rn(e1, e2), __fmaf_rn(n, dxl, mfl));
    /* |x|: the profile is even in x */
    if (s < 0.f) { xs = -s; xl = -lo; } else { xs = s; xl = lo; }
}

/* same sum as 1/A + 1/B per pair: no A*B product, safe for |x| > 1e9 */
template <int NODES>
__device__ __forceinline__ float gh_sum_f32_wide(float x, float y2)
{
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < GH<NODES>::NP; ++k) {
        float t = (float)gh_t<NODES>(k), w = (float)gh_w<NODES>(k);
        float d1 = x - t, d2 = x + t;
        float A = fmaf(d1, d1, y2), B = fmaf(d2, d2, y2);
        acc = fmaf(w, 1.f / A + 1.f / B, acc);
    }
    return acc;
}

/* the sum as the reference writes it, any x and y */
template <int NODES>
__device__ __noinline__ double gh_sum_f64(double x, double y2)
{
    double acc = 0.0;
#pragma unroll 1
    for (int k = 0; k < GH<NODES>::NP; ++k) {
        double d1 = dsub(x, gh_t<NODES>(k)), d2 = dadd(x, gh_t<NODES>(k));
        double A = dadd(y2, dmul(d1, d1)), B = dadd(y2, dmul(d2, d2));
        acc = dadd(acc, dmul(gh_w<NODES>(k), ddiv(dadd(A, B), dmul(A, B))));
    }
    return acc;
}

/* the same with refined reciprocals, for 1e-100 <= y and |x|, y <= 1e60: 11
 * FP64 instructions per node pair */
template <int NODES>
__device__ __forceinline__ double gh_sum_f64_near(double x, double y2)
{
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < GH<NODES>::NP; ++k) {
        const double d1 = dsub(x, gh_t<NODES>(k)), d2 = dadd(x, gh_t<NODES>(k));
        const double A = fma(d1, d1, y2), B = fma(d2, d2, y2);
        acc = fma(dmul(gh_w<NODES>(k), dadd(A, B)), rcp_f64(dmul(A, B)), acc);
    }
    return acc;
}

/* sum_k w_k t_k^(2 m) over all nodes */
template <int NODES>
__host__ __device__ constexpr double gh_moment(int m)
{
    double s = 0.0;
    for (int k = 0; k < GH<NODES>::NP; ++k) {
        double v = 2.0 * gh_w<NODES>(k);
        for (int i = 0; i < 2 * m; ++i) v *= gh_t<NODES>(k);
        s += v;
    }
    return s;
}

/* Far from the nodes (|x| >= GH_FAR) the quadrature's own asymptotic
 * series: sum_k w_k / (z - t_k) = (1/z) p(1/z^2) with p's coefficients the
 * moments above, whose real part over y is (A + B (3 x^2 - y^2) / |z|^4) /
 * |z|^2 for p(zeta) = A + B zeta (quad_horner).  Seven terms: the first one
 * left out is below 2e-17 of the sum.  27 FP64 instructions whatever the
 * number of nodes, against 90 (16 nodes) or 180 (32). */
constexpr double GH_FAR = 32.0;
template <int NODES>
__device__ __forceinline__ double gh_sum_f64_far(double x, double y2)
{
    constexpr double c[7] = {gh_moment<NODES>(0), gh_moment<NODES>(1), gh_moment<NODES>(2),
                             gh_moment<NODES>(3), gh_moment<NODES>(4), gh_moment<NODES>(5),
                             gh_moment<NODES>(6)};
    /* every rounding written out: two copies give the same bits */
    const double x2 = dmul(x, x), inv = rcp_f64(fma(x, x, y2)), i2 = dmul(inv, inv);
    double a, b;
    quad_horner<6>(c, dmul(dmul(2.0, fma(x, x, -y2)), i2), i2, a, b);
    return dmul(fma(b, dmul(fma(3.0, x2, -y2), i2), a), inv);
}

/* ------------------------------------------------ bin-averaged erf difference */
__device__ __forceinline__ float erf_bin_f32(float xm, float xp, int form)
{
    if (form == GEXS_ERF_LITERAL || xm < 0.f) return erff(xp) - erff(xm);
    return erfcf(xm) - erfcf(xp);
}
/* a call: four inlined functions at two places would not fit the
 * instruction cache */
static __device__ __noinline__ double erf_bin_f64(double xm, double xp, int form)
{
    if (form == GEXS_ERF_LITERAL || xm < 0.0) return dsub(erf(xp), erf(xm));
    return dsub(erfc(xm), erfc(xp));
}

/* ---------------------------------------------------- interval search
 * first t in [lo, hi] with pred(t) true, pred monotone false -> true and
 * pred(hi) assumed true (hi may be one past the range).  Gallops from the
 * guess g, then bisects. */
template <typename P>
__device__ __forceinline__ int first_true(int lo, int hi, int g, const P& pred)
{
    if (lo >= hi) return hi;
    g = max(lo, min(g, hi - 1));
    int l, r;                        /* pred(l) false (or l = lo-1), pred(r) true */
    if (pred(g)) {
        r = g; int step = 1;
        for (;;) {
            int c = r - step;
            if (c < lo) { l = lo - 1; break; }
            if (!pred(c)) { l = c; break; }
            r = c; step <<= 1;
        }
    } else {
        l = g; int step = 1;
        for (;;) {
            int c = l + step;
            if (c >= hi) { r = hi; break; }
            if (pred(c)) { r = c; break; }
            l = c; step <<= 1;
        }
    }
    while (r - l > 1) {
        int m = l + ((r - l) >> 1);
        if (pred(m)) r = m; else l = m;
    }
    return r;
}

}  // namespace gexs
