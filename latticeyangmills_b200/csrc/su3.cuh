// SU(3) algebra on the device, templated on the arithmetic type (double for the
// FP64 path, float for the mixed path).
//
// A link is a 3x3 complex matrix, row-major, the same element order as the
// reference's SU3 (include/Math/su3.h:63: 18 doubles, (re, im) interleaved).
// Products are written out with fused multiply-adds; the reference evaluates
// the same sums without FMA (su3.h:143-183), so the two agree to rounding.
#pragma once
#include <cuda_runtime.h>

namespace ym {

template <class R>
struct Cx {
    R re, im;
};

template <class R>
struct M3 {
    Cx<R> e[3][3];
};

// Hermitian traceless generator stored as 8 reals:
//   d0 = Z00, d1 = Z11 (Z22 = -d0 - d1, real diagonal),
//   z01, z02, z12 the upper off-diagonal entries (lower = conjugate).
template <class R>
struct Herm8 {
    R d0, d1;
    Cx<R> z01, z02, z12;
};

template <class R>
__device__ __forceinline__ Cx<R> cx(R re, R im) {
    Cx<R> c;
    c.re = re;
    c.im = im;
    return c;
}

// A product that the compiler leaves rounded as it stands: contracted into the
// sums that use it or not, it would make kernels that share this code differ
// by rounding.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// c = op(a) * op(b) with op = identity or dagger (DA / DB).
template <bool DA, bool DB, class R>
__device__ __forceinline__ void mmul(const M3<R>& a, const M3<R>& b, M3<R>& c) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            R re = R(0), im = R(0);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const R xr = DA ? a.e[k][i].re : a.e[i][k].re;
                const R xi = DA ? -a.e[k][i].im : a.e[i][k].im;
                const R yr = DB ? b.e[j][k].re : b.e[k][j].re;
                const R yi = DB ? -b.e[j][k].im : b.e[k][j].im;
                re = fma(xr, yr, re);
                re = fma(-xi, yi, re);
                im = fma(xr, yi, im);
                im = fma(xi, yr, im);
            }
            c.e[i][j] = cx(re, im);
        }
    }
}

// c += op(a) * op(b)
template <bool DA, bool DB, class R>
__device__ __forceinline__ void mmul_acc(const M3<R>& a, const M3<R>& b, M3<R>& c) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            R re = c.e[i][j].re, im = c.e[i][j].im;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const R xr = DA ? a.e[k][i].re : a.e[i][k].re;
                const R xi = DA ? -a.e[k][i].im : a.e[i][k].im;
                const R yr = DB ? b.e[j][k].re : b.e[k][j].re;
                const R yi = DB ? -b.e[j][k].im : b.e[k][j].im;
                re = fma(xr, yr, re);
                re = fma(-xi, yi, re);
                im = fma(xr, yi, im);
                im = fma(xi, yr, im);
            }
            c.e[i][j] = cx(re, im);
        }
    }
}

template <class R>
__device__ __forceinline__ void mzero(M3<R>& a) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) a.e[i][j] = cx(R(0), R(0));
}

template <class R>
__device__ __forceinline__ R re_trace(const M3<R>& a) {
    return a.e[0][0].re + a.e[1][1].re + a.e[2][2].re;
}

// Entry k of row 2 of the SU(3) matrix whose rows 0 and 1 are those of a
// (M3 or Rows2): conj(r0 x r1).  Every multiply-add is written out, so every
// kernel rebuilds the same row 2 bit for bit.
template <class R, class M>
__device__ __forceinline__ Cx<R> row2_entry_of(const M& a, int k) {
    const int i = (k + 1) % 3, j = (k + 2) % 3;
    const Cx<R> p = a.e[0][i], q = a.e[1][j], r = a.e[0][j], s = a.e[1][i];
    const R re = fma(p.re, q.re, fma(-p.im, q.im, -fma(r.re, s.re, -r.im * s.im)));
    const R im = fma(p.re, q.im, fma(p.im, q.re, -fma(r.re, s.im, r.im * s.re)));
    return cx(re, -im);
}

// Row 2 of an SU(3) matrix from rows 0 and 1.
template <class R>
__device__ __forceinline__ void reconstruct_row2(M3<R>& a) {
#pragma unroll
    for (int k = 0; k < 3; k++) a.e[2][k] = row2_entry_of<R>(a, k);
}

// ---------------------------------------------------------------------------
// Products of SU(3) matrices through their first two rows.  For A, B in SU(3)
// the product is in SU(3), so rows 0 and 1 of op(A) op(B) (18 complex
// multiply-adds) determine row 2 = conj(row0 x row1) (6 complex products):
// 24 instead of 27 complex multiply-adds, and a chain of products needs only
// the first two rows of its running left factor.
// ---------------------------------------------------------------------------
template <class R>
struct Rows2 {
    Cx<R> e[2][3];
};

// c(rows 0,1) = op(a) * op(b).  DA: a is read through its columns (dagger), so all
// of a's rows are needed; otherwise only a's rows 0 and 1 are read.
template <bool DA, bool DB, class R, class MA>
__device__ __forceinline__ void mmul_rows2(const MA& a, const M3<R>& b, Rows2<R>& c) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            R re = R(0), im = R(0);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const R xr = DA ? a.e[k][i].re : a.e[i][k].re;
                const R xi = DA ? -a.e[k][i].im : a.e[i][k].im;
                const R yr = DB ? b.e[j][k].re : b.e[k][j].re;
                const R yi = DB ? -b.e[j][k].im : b.e[k][j].im;
                re = fma(xr, yr, re);
                re = fma(-xi, yi, re);
                im = fma(xr, yi, im);
                im = fma(xi, yr, im);
            }
            c.e[i][j] = cx(re, im);
        }
    }
}

// row 2 of an SU(3) matrix given by its first two rows, entry k
template <class R>
__device__ __forceinline__ Cx<R> row2_entry(const Rows2<R>& a, int k) {
    return row2_entry_of<R>(a, k);
}

// acc += the SU(3) matrix whose first two rows are a
template <class R>
__device__ __forceinline__ void madd_su3_rows2(M3<R>& acc, const Rows2<R>& a) {
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            acc.e[i][j].re += a.e[i][j].re;
            acc.e[i][j].im += a.e[i][j].im;
        }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const Cx<R> r = row2_entry(a, k);
        acc.e[2][k].re += r.re;
        acc.e[2][k].im += r.im;
    }
}

template <class R>
__device__ __forceinline__ void full_from_rows2(const Rows2<R>& a, M3<R>& m) {
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) m.e[i][j] = a.e[i][j];
#pragma unroll
    for (int k = 0; k < 3; k++) m.e[2][k] = row2_entry(a, k);
}

// Products of SU(3) links through their first two rows (third row rebuilt as conj(r0 x r1))
// save 22% of the staple multiply-adds but rebuild a row from rounded rows.
// In FP64 that costs nothing measurable; in FP32 the rebuilt rows of the fused
// kernel's staples carried a systematic bias that grew linearly with flow time
// (t^2<E> at t = 4 on 32^4 drifted 4e-6 from FP64 against 5e-7 with full
// products, measured before the link update took its e^{iQ} - 1 form), so the
// fused kernel's FP32 staples form all three rows.  The plaquette field and
// the observables form their products through two rows in every precision
// (t = 4 error against FP64 1.0e-7 either way).
template <class R>
struct kTwoRowStaples {
    static constexpr bool value = sizeof(R) == 8;
};

// Entry (i,j) of u * w (full matrices).
template <class R>
__device__ __forceinline__ Cx<R> mul_entry(const M3<R>& u, const M3<R>& w, int i, int j) {
    R re = R(0), im = R(0);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        re = fma(u.e[i][k].re, w.e[k][j].re, re);
        re = fma(-u.e[i][k].im, w.e[k][j].im, re);
        im = fma(u.e[i][k].re, w.e[k][j].im, im);
        im = fma(u.e[i][k].im, w.e[k][j].re, im);
    }
    return cx(re, im);
}

// Im of entry (i,i) of u * w.
template <class R>
__device__ __forceinline__ R mul_diag_im(const M3<R>& u, const M3<R>& w, int i) {
    R im = R(0);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        im = fma(u.e[i][k].re, w.e[k][i].im, im);
        im = fma(u.e[i][k].im, w.e[k][i].re, im);
    }
    return im;
}

// Flow generator of X = U Omega (Omega the staple sum):
//   Z = (i/2) [X - X^+]_traceless   (Hermitian, traceless),
// the quantity the reference returns from PureGauge::computeDerivative
// (src/Actions/puregauge.cpp:62-79, where X is formed as (Omega^+ U^+)^+).  Only
// the six off-diagonal entries and the imaginary diagonal of X are computed:
// (i/2)(a + ib) = (-b/2, a/2) with a + ib = X_ij - conj(X_ji).
template <class R>
__device__ __forceinline__ Herm8<R> force_from_u_omega(const M3<R>& u, const M3<R>& w) {
    Herm8<R> z;
    const R i0 = mul_diag_im(u, w, 0), i1 = mul_diag_im(u, w, 1), i2 = mul_diag_im(u, w, 2);
    const R mean = (i0 + i1 + i2) * R(1.0 / 3.0);
    z.d0 = mean - i0;
    z.d1 = mean - i1;
    const Cx<R> x01 = mul_entry(u, w, 0, 1), x10 = mul_entry(u, w, 1, 0);
    const Cx<R> x02 = mul_entry(u, w, 0, 2), x20 = mul_entry(u, w, 2, 0);
    const Cx<R> x12 = mul_entry(u, w, 1, 2), x21 = mul_entry(u, w, 2, 1);
    z.z01 = cx(R(-0.5) * (x01.im + x10.im), R(0.5) * (x01.re - x10.re));
    z.z02 = cx(R(-0.5) * (x02.im + x20.im), R(0.5) * (x02.re - x20.re));
    z.z12 = cx(R(-0.5) * (x12.im + x21.im), R(0.5) * (x12.re - x21.re));
    return z;
}

// The generator (i/2)[X - X^+]_traceless of X = B C^+ for X in SU(3), from B's
// first two rows: rows 0 and 1 of X (six entries), then of row 2 = conj(row0 x row1) only
// X_20, X_21 and Im X_22.  92 multiply-adds, against 90 plus the 27 that
// rebuild B's row 2 for the full form.  trace (optional): Re tr X, for four
// more.
template <class R>
__device__ __forceinline__ Herm8<R> force_from_b2_cdag(const Rows2<R>& b, const M3<R>& c, R* trace = nullptr) {
    Cx<R> x[2][3];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {  // (B C^+)_ij = sum_k b_ik conj(c_jk)
            R re = R(0), im = R(0);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                re = fma(b.e[i][k].re, c.e[j][k].re, re);
                re = fma(b.e[i][k].im, c.e[j][k].im, re);
                im = fma(b.e[i][k].im, c.e[j][k].re, im);
                im = fma(-b.e[i][k].re, c.e[j][k].im, im);
            }
            x[i][j] = cx(re, im);
        }
    // row 2 = conj(row0 x row1): X_2k = conj(X_0i X_1j - X_0j X_1i), (i, j) = (k+1, k+2) mod 3
    auto cross = [&](int i, int j) {
        const Cx<R> p = x[0][i], q = x[1][j], r = x[0][j], s = x[1][i];
        const R re = fma(p.re, q.re, fma(-p.im, q.im, -fma(r.re, s.re, -r.im * s.im)));
        const R im = fma(p.re, q.im, fma(p.im, q.re, -fma(r.re, s.im, r.im * s.re)));
        return cx(re, -im);
    };
    const Cx<R> x20 = cross(1, 2), x21 = cross(2, 0);
    const R i2 = -fma(x[0][0].re, x[1][1].im, fma(x[0][0].im, x[1][1].re, -fma(x[0][1].re, x[1][0].im, x[0][1].im * x[1][0].re)));
    if (trace) *trace = x[0][0].re + x[1][1].re + cross(0, 1).re;
    Herm8<R> z;
    const R i0 = x[0][0].im, i1 = x[1][1].im;
    const R mean = mul_rn(i0 + i1 + i2, R(1.0 / 3.0));
    z.d0 = mean - i0;
    z.d1 = mean - i1;
    z.z01 = cx(R(-0.5) * (x[0][1].im + x[1][0].im), R(0.5) * (x[0][1].re - x[1][0].re));
    z.z02 = cx(R(-0.5) * (x[0][2].im + x20.im), R(0.5) * (x[0][2].re - x20.re));
    z.z12 = cx(R(-0.5) * (x[1][2].im + x21.im), R(0.5) * (x[1][2].re - x21.re));
    return z;
}

// The same generator with every row of X multiplied out, 108 multiply-adds, for
// products whose unitarity is not to be relied on: with h the product's
// deviation from it, the completed row 2 puts h's entries 02 and 12 into the
// generator (which vanish for one link, but not for a product), the full
// product only h times the field strength.
template <class R>
__device__ __forceinline__ Herm8<R> force_from_b_cdag(const M3<R>& b, const M3<R>& c) {
    auto entry = [&](int i, int j) {  // (B C^+)_ij = sum_k b_ik conj(c_jk)
        R re = R(0), im = R(0);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            re = fma(b.e[i][k].re, c.e[j][k].re, re);
            re = fma(b.e[i][k].im, c.e[j][k].im, re);
            im = fma(b.e[i][k].im, c.e[j][k].re, im);
            im = fma(-b.e[i][k].re, c.e[j][k].im, im);
        }
        return cx(re, im);
    };
    Herm8<R> z;
    const R i0 = entry(0, 0).im, i1 = entry(1, 1).im, i2 = entry(2, 2).im;
    const R mean = mul_rn(i0 + i1 + i2, R(1.0 / 3.0));
    z.d0 = mean - i0;
    z.d1 = mean - i1;
    const Cx<R> x01 = entry(0, 1), x10 = entry(1, 0);
    const Cx<R> x02 = entry(0, 2), x20 = entry(2, 0);
    const Cx<R> x12 = entry(1, 2), x21 = entry(2, 1);
    z.z01 = cx(R(-0.5) * (x01.im + x10.im), R(0.5) * (x01.re - x10.re));
    z.z02 = cx(R(-0.5) * (x02.im + x20.im), R(0.5) * (x02.re - x20.re));
    z.z12 = cx(R(-0.5) * (x12.im + x21.im), R(0.5) * (x12.re - x21.re));
    return z;
}

// acc += v^+ h v for a Hermitian traceless h and v in SU(3) (Hermitian and
// traceless again: its diagonal d0, d1 and upper triangle are formed).  With
// d2 = h22, v^+ h v = v^+ (h - d2) v + d2, and h - d2 = A + A^+ for the upper
// triangular A with half its diagonal, whose third row is zero: w = A v has
// two rows, and v^+ (h - d2) v = v^+ w + (v^+ w)^+ sums over two rows of v.
// 113 multiply-adds, against 139 for h v and the needed entries of v^+ (h v).
// The stage kernel that makes three of these per link is bound by its issue
// slots: at 32^4 on B200 0.165 -> 0.148 ms per launch (FP32-12, with the row 2
// of the links in four multiply-adds per component instead of five), 0.167 ->
// 0.160 (FP32-18), 0.350 -> 0.337 (FP64).
template <class R>
__device__ __forceinline__ void herm_conj_add(const M3<R>& v, const Herm8<R>& h, Herm8<R>& acc) {
    const R d2 = -(h.d0 + h.d1);
    const R a0 = R(0.5) * (h.d0 - d2), a1 = R(0.5) * (h.d1 - d2);
    Rows2<R> w;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const Cx<R> a = v.e[0][j], b = v.e[1][j], c = v.e[2][j];
        // row 0: a0 a + z01 b + z02 c
        w.e[0][j].re = fma(a0, a.re, fma(h.z01.re, b.re, fma(-h.z01.im, b.im, fma(h.z02.re, c.re, -h.z02.im * c.im))));
        w.e[0][j].im = fma(a0, a.im, fma(h.z01.re, b.im, fma(h.z01.im, b.re, fma(h.z02.re, c.im, h.z02.im * c.re))));
        // row 1: a1 b + z12 c
        w.e[1][j].re = fma(a1, b.re, fma(h.z12.re, c.re, -h.z12.im * c.im));
        w.e[1][j].im = fma(a1, b.im, fma(h.z12.re, c.im, h.z12.im * c.re));
    }
    auto diag = [&](int i, R& out) {  // out += d2 + 2 Re (v^+ w)_ii
        R re = v.e[0][i].re * w.e[0][i].re;
        re = fma(v.e[0][i].im, w.e[0][i].im, re);
        re = fma(v.e[1][i].re, w.e[1][i].re, re);
        re = fma(v.e[1][i].im, w.e[1][i].im, re);
        out = fma(R(2), re, out + d2);
    };
    auto entry = [&](int i, int j, Cx<R>& out) {  // out += (v^+ w)_ij + conj((v^+ w)_ji)
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const Cx<R> vi = v.e[k][i], vj = v.e[k][j], wi = w.e[k][i], wj = w.e[k][j];
            out.re = fma(vi.re, wj.re, out.re);
            out.re = fma(vi.im, wj.im, out.re);
            out.re = fma(vj.re, wi.re, out.re);
            out.re = fma(vj.im, wi.im, out.re);
            out.im = fma(vi.re, wj.im, out.im);
            out.im = fma(-vi.im, wj.re, out.im);
            out.im = fma(vj.im, wi.re, out.im);
            out.im = fma(-vj.re, wi.im, out.im);
        }
    };
    diag(0, acc.d0);
    diag(1, acc.d1);
    entry(0, 1, acc.z01);
    entry(0, 2, acc.z02);
    entry(1, 2, acc.z12);
}

template <class R>
__device__ __forceinline__ Herm8<R> h8_axpby(R a, const Herm8<R>& x, R b, const Herm8<R>& y) {
    Herm8<R> r;
    r.d0 = fma(a, x.d0, -mul_rn(b, y.d0));
    r.d1 = fma(a, x.d1, -mul_rn(b, y.d1));
    r.z01 = cx(fma(a, x.z01.re, -mul_rn(b, y.z01.re)), fma(a, x.z01.im, -mul_rn(b, y.z01.im)));
    r.z02 = cx(fma(a, x.z02.re, -mul_rn(b, y.z02.re)), fma(a, x.z02.im, -mul_rn(b, y.z02.im)));
    r.z12 = cx(fma(a, x.z12.re, -mul_rn(b, y.z12.re)), fma(a, x.z12.im, -mul_rn(b, y.z12.im)));
    return r;
}

template <class R>
__device__ __forceinline__ Herm8<R> h8_scale(R a, const Herm8<R>& x) {
    Herm8<R> r;
    r.d0 = mul_rn(a, x.d0);
    r.d1 = mul_rn(a, x.d1);
    r.z01 = cx(mul_rn(a, x.z01.re), mul_rn(a, x.z01.im));
    r.z02 = cx(mul_rn(a, x.z02.re), mul_rn(a, x.z02.im));
    r.z12 = cx(mul_rn(a, x.z12.re), mul_rn(a, x.z12.im));
    return r;
}

// a x + y
template <class R>
__device__ __forceinline__ Herm8<R> h8_axpy(R a, const Herm8<R>& x, const Herm8<R>& y) {
    Herm8<R> r;
    r.d0 = fma(a, x.d0, y.d0);
    r.d1 = fma(a, x.d1, y.d1);
    r.z01 = cx(fma(a, x.z01.re, y.z01.re), fma(a, x.z01.im, y.z01.im));
    r.z02 = cx(fma(a, x.z02.re, y.z02.re), fma(a, x.z02.im, y.z02.im));
    r.z12 = cx(fma(a, x.z12.re, y.z12.re), fma(a, x.z12.im, y.z12.im));
    return r;
}

template <class R>
__device__ __forceinline__ Herm8<R> h8_neg(const Herm8<R>& x) {
    Herm8<R> r;
    r.d0 = -x.d0;
    r.d1 = -x.d1;
    r.z01 = cx(-x.z01.re, -x.z01.im);
    r.z02 = cx(-x.z02.re, -x.z02.im);
    r.z12 = cx(-x.z12.re, -x.z12.im);
    return r;
}

}  // namespace ym
