// e^{iQ} for a Hermitian traceless 3x3 Q by the Cayley-Hamilton theorem
// (Morningstar & Peardon, Phys. Rev. D 69 (2004) 054501, eqs. 23-34) — the
// method of the reference's exp(const SU3&) (src/Math/su3.cpp:96-183):
//
//   c0 = det Q = tr(Q^3)/3,  c1 = tr(Q^2)/2,  c0max = 2 (c1/3)^{3/2}
//   theta = acos(c0/c0max),  u = sqrt(c1/3) cos(theta/3),  w = sqrt(c1) sin(theta/3)
//   h0 = (u^2 - w^2) e^{2iu} + e^{-iu} [8u^2 cos w + 2iu (3u^2 + w^2) xi(w)]
//   h1 = 2u e^{2iu} - e^{-iu} [2u cos w - i (3u^2 - w^2) xi(w)]
//   h2 = e^{2iu} - e^{-iu} [cos w + 3iu xi(w)]
//   f_j = h_j / (9u^2 - w^2),   e^{iQ} = f0 + f1 Q + f2 Q^2
//
// with c0 < 0 handled by f_j(-c0) = (-1)^j conj(f_j(c0)) and xi(w) = sin(w)/w
// replaced by its series for |w| < 0.05, both as the reference does.
//
// Deliberate differences from the reference, all where it returns NaN:
//   * c0/c0max is clamped to 1 (rounding can push it above 1 for a doubly
//     degenerate spectrum, where the reference's acos gives NaN);
//   * c1 below a tiny threshold (Q = 0, e.g. a cold field) uses the series
//     1 + iQ - Q^2/2, where the reference computes 0/0.
// tr(Q^3)/3 is evaluated as det Q (equal for traceless Q) and Q^2 from its six
// independent entries; both agree with the reference to rounding.
//
// For small Q (c1 <= YM_SERIES_C1, which holds for every link of a flow at
// eps <= 0.02) the coefficients f_j come instead from the truncated power
// series of e^{iQ} reduced by the same Cayley-Hamilton identity (ch_series):
// exact to the working precision, with no acos / sincos / sqrt / division.
// The result equals the closed form to rounding; the closed form remains for
// larger Q.
#pragma once
#include "su3.cuh"

namespace ym {

// e^{iQ} = (1 + f0m1) + f1 Q + f2 Q^2.  The constant coefficient is kept as
// f0 - 1, so that e^{iQ} - 1 (small for small Q) is formed without rounding a
// 1 into it: an FP32 link update U + (e^{iQ} - 1) U then carries only the
// rounding of the stored link, not that of e^{iQ}'s entries near 1, which
// otherwise drifts the FP32 flow systematically (t^2 E about 1e-6 off at t = 2
// with reunitarisation every 10 steps).
template <class S>
struct ChCoef {
    Cx<S> f0m1, f1, f2;
};

template <class S>
__device__ __forceinline__ S ch_small_c1();
template <>
__device__ __forceinline__ double ch_small_c1<double>() { return 1e-60; }
template <>
__device__ __forceinline__ float ch_small_c1<float>() { return 1e-20f; }

// The same coefficients from the power series of e^{iQ}, for small Q.  By the
// Cayley-Hamilton theorem Q^3 = c1 Q + c0, so every power reduces to
// Q^n = A_n + B_n Q + C_n Q^2 with A_n = c0 C_{n-1}, B_n = C_{n+1} and
//   C_2 = 1, C_3 = 0, C_4 = c1, C_5 = c0, C_6 = c1^2, C_7 = 2 c0 c1,
//   C_8 = c1^3 + c0^2, C_9 = 3 c0 c1^2, C_10 = c1^4 + 3 c0^2 c1,
//   C_11 = 4 c0 c1^3 + c0^3, C_12 = c1^5 + 6 c0^2 c1^2,
// and f_j = sum_n i^n {A,B,C}_n / n!.  Truncating after Q^N is truncating
// the series of e^{iQ} itself: the error is below rho^{N+1}/(N+1)! e^rho with
// rho the largest |eigenvalue| of Q, rho^2 <= 4 c1 / 3.  No transcendental
// function, no division and no cancellation: every term is a small correction
// to (1, i, -1/2), and f0 - 1 is the sum of the terms alone.  Collected by
// coefficient: 11 operations in FP32 and 34 in FP64, against 32 and 72 for the
// recursion term by term.
//
// Where the series replaces the closed form: c1 <= YM_SERIES_C1, i.e. every
// eigenvalue of Q within rho <= sqrt(4 YM_SERIES_C1 / 3) = 0.163 of zero.  The
// flow stays far inside it (eps Z at eps = 0.02 has c1 <= 0.011 on the
// benchmark fields, Haar-mixed included).  Terms: FP64 up to Q^11 (truncation
// below 0.163^12/12! = 7e-19), FP32 up to Q^6 (below 0.163^7/7! = 2e-9).
#define YM_SERIES_C1 0.02

__device__ __forceinline__ ChCoef<float> ch_series(float c0, float c1) {
    ChCoef<float> f;
    f.f0m1 = cx(mul_rn(mul_rn(c0, c0), -1.f / 720.f), mul_rn(c0, fmaf(c1, 1.f / 120.f, -1.f / 6.f)));
    f.f1 = cx(mul_rn(c0, fmaf(c1, -1.f / 360.f, 1.f / 24.f)), fmaf(c1, fmaf(c1, 1.f / 120.f, -1.f / 6.f), 1.f));
    f.f2 = cx(fmaf(c1, fmaf(c1, -1.f / 720.f, 1.f / 24.f), -0.5f), mul_rn(c0, 1.f / 120.f));
    return f;
}

__device__ __forceinline__ ChCoef<double> ch_series(double c0, double c1) {
    constexpr double k4 = 1.0 / 24, k5 = 1.0 / 120, k6 = 1.0 / 720, k7 = 1.0 / 5040, k8 = 1.0 / 40320,
                     k9 = 1.0 / 362880, k10 = 1.0 / 3628800, k11 = 1.0 / 39916800;
    const double q = mul_rn(c0, c0), p = mul_rn(c1, c1), c3 = mul_rn(c1, p);
    const double s8 = c3 + q, s10 = mul_rn(c1, fma(3.0, q, c3)), s11 = fma(4.0, c3, q), s12 = mul_rn(p, fma(6.0, q, c3));
    ChCoef<double> f;
    f.f0m1 = cx(mul_rn(q, fma(-3.0 * k10, p, fma(2.0 * k8, c1, -k6))),
                mul_rn(c0, fma(-k11, s10, fma(k9, s8, fma(-k7, p, fma(k5, c1, -1.0 / 6))))));
    f.f1 = cx(mul_rn(c0, fma(-k10, s11, fma(3.0 * k8, p, fma(-2.0 * k6, c1, k4)))),
              fma(-k11, s12, fma(k9, s10, fma(-k7, s8, fma(k5, p, fma(-1.0 / 6, c1, 1.0))))));
    f.f2 = cx(fma(-k10, s10, fma(k8, s8, fma(-k6, p, fma(k4, c1, -0.5)))),
              mul_rn(c0, fma(-k11, s11, fma(3.0 * k9, p, fma(-2.0 * k7, c1, k5)))));
    return f;
}

// Cayley-Hamilton coefficients from c0 = det Q and c1 = tr(Q^2)/2, in type S.
template <class S>
__device__ __forceinline__ ChCoef<S> ch_coefficients(S c0, S c1) {
    ChCoef<S> f;
    if (!(c1 > ch_small_c1<S>())) {  // also catches NaN c1: falls to the series
        f.f0m1 = cx(S(0), S(0));
        f.f1 = cx(S(0), S(1));
        f.f2 = cx(S(-0.5), S(0));
        return f;
    }
    const bool neg = c0 < S(0);
    if (neg) c0 = -c0;
    const S inv_sqrt3 = S(0.57735026918962576451);
    const S c1sqrt = sqrt(c1);
    const S c0max = c1 * c1sqrt * inv_sqrt3 * S(2.0 / 3.0);
    S x = c0 / c0max;
    x = x > S(1) ? S(1) : x;
    const S theta = acos(x);
    S st, ct;
    sincos(theta * S(1.0 / 3.0), &st, &ct);
    const S w = c1sqrt * st;
    const S u = c1sqrt * inv_sqrt3 * ct;
    const S u2 = u * u, w2 = w * w;
    S sw, cw;
    sincos(w, &sw, &cw);
    const S xi = fabs(w) < S(0.05) ? S(1) - w2 / S(6) * (S(1) - w2 / S(20) * (S(1) - w2 / S(42))) : sw / w;
    S su, cu;
    sincos(u, &su, &cu);
    const S cmu = cu, smu = -su;  // e^{-iu}
    const S c2u = cmu * cmu - smu * smu, s2u = S(-2) * cmu * smu;  // e^{2iu}
    const S cwcmu = cw * cmu, cwsmu = cw * smu, xicmu = xi * cmu, xismu = xi * smu;
    S h0r = (u2 - w2) * c2u + S(8) * u2 * cwcmu - S(2) * u * (S(3) * u2 + w2) * xismu;
    S h0i = (u2 - w2) * s2u + S(8) * u2 * cwsmu + S(2) * u * (S(3) * u2 + w2) * xicmu;
    S h1r = S(2) * u * c2u - S(2) * u * cwcmu - (S(3) * u2 - w2) * xismu;
    S h1i = S(2) * u * s2u - S(2) * u * cwsmu + (S(3) * u2 - w2) * xicmu;
    S h2r = c2u - cwcmu + S(3) * u * xismu;
    S h2i = s2u - cwsmu - S(3) * u * xicmu;
    if (neg) {
        h0i = -h0i;
        h1r = -h1r;
        h2i = -h2i;
    }
    const S norm = S(1) / (S(9) * u2 - w2);
    f.f0m1 = cx(h0r * norm - S(1), h0i * norm);
    f.f1 = cx(h1r * norm, h1i * norm);
    f.f2 = cx(h2r * norm, h2i * norm);
    return f;
}

template <class R>
struct QSquared {  // Q^2, Hermitian: real diagonal and the upper triangle
    R a00, a11, a22;
    Cx<R> a01, a02, a12;
};

// (every multiply-add below is written out, so that kernels sharing this code
// round alike)
//
// |q01|^2, |q02|^2, |q12|^2: shared by Q^2, c0 and c1.
template <class R>
struct OffNorms {
    R n01, n02, n12;
};
template <class R>
__device__ __forceinline__ OffNorms<R> off_norms(const Herm8<R>& q) {
    OffNorms<R> n;
    n.n01 = fma(q.z01.re, q.z01.re, mul_rn(q.z01.im, q.z01.im));
    n.n02 = fma(q.z02.re, q.z02.re, mul_rn(q.z02.im, q.z02.im));
    n.n12 = fma(q.z12.re, q.z12.re, mul_rn(q.z12.im, q.z12.im));
    return n;
}

template <class R>
__device__ __forceinline__ QSquared<R> q_squared(const Herm8<R>& q, R q22, const OffNorms<R>& n) {
    QSquared<R> s;
    s.a00 = fma(q.d0, q.d0, n.n01 + n.n02);
    s.a11 = fma(q.d1, q.d1, n.n01 + n.n12);
    s.a22 = fma(q22, q22, n.n02 + n.n12);
    // (Q^2)_01 = q00 q01 + q01 q11 + q02 conj(q12);  q00 + q11 = -q22
    s.a01 = cx(fma(-q22, q.z01.re, fma(q.z02.re, q.z12.re, mul_rn(q.z02.im, q.z12.im))),
               fma(-q22, q.z01.im, fma(q.z02.im, q.z12.re, -mul_rn(q.z02.re, q.z12.im))));
    // (Q^2)_02 = q00 q02 + q01 q12 + q02 q22;  q00 + q22 = -q11
    s.a02 = cx(fma(-q.d1, q.z02.re, fma(q.z01.re, q.z12.re, -mul_rn(q.z01.im, q.z12.im))),
               fma(-q.d1, q.z02.im, fma(q.z01.re, q.z12.im, mul_rn(q.z01.im, q.z12.re))));
    // (Q^2)_12 = conj(q01) q02 + q11 q12 + q12 q22;  q11 + q22 = -q00
    s.a12 = cx(fma(-q.d0, q.z12.re, fma(q.z01.re, q.z02.re, mul_rn(q.z01.im, q.z02.im))),
               fma(-q.d0, q.z12.im, fma(q.z01.re, q.z02.im, -mul_rn(q.z01.im, q.z02.re))));
    return s;
}

// c1 = tr(Q^2)/2 = q00^2 + q00 q11 + q11^2 + |q01|^2 + |q02|^2 + |q12|^2 and c0 =
// det Q, in Q's own type.
template <class R>
__device__ __forceinline__ R c1_of(const Herm8<R>& q, R q22, const OffNorms<R>& n) {
    return fma(-q.d0, q22, fma(q.d1, q.d1, (n.n01 + n.n02) + n.n12));
}
template <class R>
__device__ __forceinline__ R c0_of(const Herm8<R>& q, R q22, const OffNorms<R>& n) {
    const R pr = fma(q.z01.re, q.z12.re, -mul_rn(q.z01.im, q.z12.im));  // q01 q12
    const R pi = fma(q.z01.re, q.z12.im, mul_rn(q.z01.im, q.z12.re));
    const R re3 = fma(pr, q.z02.re, mul_rn(pi, q.z02.im));  // Re(q01 q12 conj(q02))
    return fma(R(2), re3, fma(q.d0, fma(q.d1, q22, -n.n12), fma(-q.d1, n.n02, -mul_rn(q22, n.n01))));
}

// det Q for Hermitian Q: q00 q11 q22 + 2 Re(q01 q12 conj(q02)) - q00|q12|^2 - q11|q02|^2 - q22|q01|^2
template <class S, class R>
__device__ __forceinline__ S herm_det(const Herm8<R>& q, R q22r) {
    const S a = S(q.d0), b = S(q.d1), c = S(q22r);
    const S xr = S(q.z01.re), xi = S(q.z01.im), yr = S(q.z02.re), yi = S(q.z02.im);
    const S zr = S(q.z12.re), zi = S(q.z12.im);
    const S pr = fma(xr, zr, -mul_rn(xi, zi)), pi = fma(xr, zi, mul_rn(xi, zr));  // q01 q12
    const S re3 = fma(pr, yr, mul_rn(pi, yi));                                     // Re(q01 q12 conj(q02))
    const S nz = fma(zr, zr, mul_rn(zi, zi)), ny = fma(yr, yr, mul_rn(yi, yi)), nx = fma(xr, xr, mul_rn(xi, xi));
    return fma(S(2), re3, fma(a, fma(b, c, -nz), fma(-b, ny, -mul_rn(c, nx))));
}

template <class S, class R>
__device__ __forceinline__ S herm_c1(const Herm8<R>& q, R q22r) {
    const S a = S(q.d0), b = S(q.d1), c = S(q22r);
    const S n = fma(S(q.z01.re), S(q.z01.re), fma(S(q.z01.im), S(q.z01.im), fma(S(q.z02.re), S(q.z02.re),
                fma(S(q.z02.im), S(q.z02.im), fma(S(q.z12.re), S(q.z12.re), mul_rn(S(q.z12.im), S(q.z12.im)))))));
    return fma(S(0.5), fma(a, a, fma(b, b, mul_rn(c, c))), n);
}

// Threshold on c0/c0max above which the mixed path evaluates the coefficients in
// FP64: near a doubly degenerate spectrum acos loses about half the significand.
#define YM_DEGENERATE_X 0.98

__device__ __forceinline__ ChCoef<double> exp_coefficients(const Herm8<double>& q, double q22,
                                                           const OffNorms<double>& n) {
    const double c0 = c0_of(q, q22, n), c1 = c1_of(q, q22, n);
    if (c1 <= YM_SERIES_C1) return ch_series(c0, c1);
    return ch_coefficients<double>(c0, c1);
}

// Mixed path: the FP32 series for small Q; otherwise the FP32 closed form
// unless the spectrum is nearly degenerate (or tiny), then the closed form in
// FP64 from the FP32 entries.
__device__ __forceinline__ ChCoef<float> exp_coefficients(const Herm8<float>& q, float q22, const OffNorms<float>& n) {
    const float c0 = c0_of(q, q22, n);
    const float c1 = c1_of(q, q22, n);
    if (c1 <= float(YM_SERIES_C1)) return ch_series(c0, c1);
    const float c1s = sqrtf(c1);
    const float c0max = c1 * c1s * 0.38490017945975050f;  // 2/(3 sqrt 3)
    const float x = fabsf(c0) / c0max;
    if (x < float(YM_DEGENERATE_X) && c1 > 1e-12f) return ch_coefficients<float>(c0, c1);
    ChCoef<double> d = ch_coefficients<double>(herm_det<double>(q, q22), herm_c1<double>(q, q22));
    ChCoef<float> f;
    f.f0m1 = cx(float(d.f0m1.re), float(d.f0m1.im));
    f.f1 = cx(float(d.f1.re), float(d.f1.im));
    f.f2 = cx(float(d.f2.re), float(d.f2.im));
    return f;
}

// E = e^{iQ} = f0 + f1 Q + f2 Q^2 as a full matrix.
template <class R>
__device__ __forceinline__ void exp_iq(const Herm8<R>& q, M3<R>& e) {
    const R q22 = -(q.d0 + q.d1);
    const OffNorms<R> n = off_norms(q);
    const ChCoef<R> f = exp_coefficients(q, q22, n);
    const QSquared<R> s = q_squared(q, q22, n);
    // diagonal: 1 + f0m1 + f1 q_ii + f2 (Q^2)_ii  (q_ii and (Q^2)_ii real)
    e.e[0][0] = cx(R(1) + (f.f0m1.re + f.f1.re * q.d0 + f.f2.re * s.a00), f.f0m1.im + f.f1.im * q.d0 + f.f2.im * s.a00);
    e.e[1][1] = cx(R(1) + (f.f0m1.re + f.f1.re * q.d1 + f.f2.re * s.a11), f.f0m1.im + f.f1.im * q.d1 + f.f2.im * s.a11);
    e.e[2][2] = cx(R(1) + (f.f0m1.re + f.f1.re * q22 + f.f2.re * s.a22), f.f0m1.im + f.f1.im * q22 + f.f2.im * s.a22);
    // off-diagonal: f1 q_ij + f2 (Q^2)_ij; lower entries use the conjugates of q and Q^2
#define YM_OFFD(I, J, QV, SV)                                                                     \
    e.e[I][J] = cx(f.f1.re * QV.re - f.f1.im * QV.im + f.f2.re * SV.re - f.f2.im * SV.im,         \
                   f.f1.re * QV.im + f.f1.im * QV.re + f.f2.re * SV.im + f.f2.im * SV.re);        \
    e.e[J][I] = cx(f.f1.re * QV.re + f.f1.im * QV.im + f.f2.re * SV.re + f.f2.im * SV.im,         \
                   -f.f1.re * QV.im + f.f1.im * QV.re - f.f2.re * SV.im + f.f2.im * SV.re);
    YM_OFFD(0, 1, q.z01, s.a01)
    YM_OFFD(0, 2, q.z02, s.a02)
    YM_OFFD(1, 2, q.z12, s.a12)
#undef YM_OFFD
}

// Rows 0 and 1 of e^{iQ} - 1 (enough to update an SU(3) link through its
// first two rows as U + (e^{iQ} - 1) U).
template <class R>
__device__ __forceinline__ void expm1_iq_rows2(const Herm8<R>& q, Rows2<R>& e) {
    const R q22 = -(q.d0 + q.d1);
    const OffNorms<R> n = off_norms(q);
    const ChCoef<R> f = exp_coefficients(q, q22, n);
    const QSquared<R> s = q_squared(q, q22, n);
    e.e[0][0] = cx(fma(f.f2.re, s.a00, fma(f.f1.re, q.d0, f.f0m1.re)), fma(f.f2.im, s.a00, fma(f.f1.im, q.d0, f.f0m1.im)));
    e.e[1][1] = cx(fma(f.f2.re, s.a11, fma(f.f1.re, q.d1, f.f0m1.re)), fma(f.f2.im, s.a11, fma(f.f1.im, q.d1, f.f0m1.im)));
    // upper entries f1 q_ij + f2 (Q^2)_ij; e10 from the conjugates of q01 and (Q^2)_01
    auto upper = [&](const Cx<R>& z, const Cx<R>& w) {
        return cx(fma(f.f1.re, z.re, fma(-f.f1.im, z.im, fma(f.f2.re, w.re, -mul_rn(f.f2.im, w.im)))),
                  fma(f.f1.re, z.im, fma(f.f1.im, z.re, fma(f.f2.re, w.im, mul_rn(f.f2.im, w.re)))));
    };
    e.e[0][1] = upper(q.z01, s.a01);
    e.e[0][2] = upper(q.z02, s.a02);
    e.e[1][2] = upper(q.z12, s.a12);
    e.e[1][0] = upper(cx(q.z01.re, -q.z01.im), cx(s.a01.re, -s.a01.im));
}

}  // namespace ym
