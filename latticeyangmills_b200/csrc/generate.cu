// Gauge-field generation on the device: Metropolis updates of the Wilson
// action, the step before the flow.  The reference's generator app
// (src/Apps/gaugefieldfactory.cpp:192-220) does not compile and draws from an
// unseedable generator; this restates its intended update with a seeded,
// counter-based random stream:
//
//   per link, `hits` proposals U' = X U with X a product R S T of three SU(2)
//   elements embedded in the (0,1), (0,2), (1,2) blocks, each with
//   x0 = +-sqrt(1 - eps^2) (sign of a uniform draw) and an eps-long vector of
//   uniform direction (src/Math/random.cpp:71-156), or X^+ U with equal
//   probability: R S T is not distributed like its inverse T^+ S^+ R^+, and
//   without the X^+ choice the proposal is not symmetric and the chain misses
//   detailed balance;
//   accept when exp(-dS) > r,  dS = -(beta/3) Re tr[(U' - U) A],
//   A the staple sum of the link (the action written at
//   src/Actions/puregauge.cpp:28, staples as puregauge.cpp:36-54).
//
// The sweep is a checkerboard: for each direction mu and site parity, every
// link U_mu(x) of that parity is updated in parallel (its staples involve no
// link of the same direction and parity), in place.  The random numbers of a
// (link, sweep, hit) come from Philox4x32-10 keyed by the seed with counter
// (link index, sweep, hit, call), so the chain does not depend on the launch
// shape; oracle/ymoracle.c runs the same chain on the CPU.
#include <cmath>

#include "field.cuh"
#include "kernels.h"

namespace ym {

namespace {

__device__ __forceinline__ uint4 philox_g(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint64_t p0 = uint64_t(0xD2511F53u) * c.x, p1 = uint64_t(0xCD9E8D57u) * c.z;
        c = make_uint4(uint32_t(p1 >> 32) ^ c.y ^ k.x, uint32_t(p1), uint32_t(p0 >> 32) ^ c.w ^ k.y, uint32_t(p0));
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

// Uniform (w + 1/2) / 2^32 of a random word.
__device__ __forceinline__ double unit(uint32_t w) { return (double(w) + 0.5) * 2.3283064365386963e-10; }

// 2 w + 1 - 2^32, exactly: 2^33 (unit(w) - 1/2), from the word set into a
// double's low bits (one addition instead of a conversion).
__device__ __forceinline__ double centred(uint32_t w) {
    return __hiloint2double(int(0x43300000u | (w >> 31)), int((w << 1) | 1u)) - (4503599627370496.0 + 4294967296.0);
}

// An embedded SU(2) element [[a, b], [-conj b, conj a]] from four random words:
// Re a = +-x0 with the first word's sign, the other three components eps long
// in a uniform direction.
template <class R>
struct Su2 {
    Cx<R> a, b;
};

// 1 / sqrt(n) by Newton's iteration from the FP32 value (relative error below
// 2^-22, then 2^-43, then FP64 rounding); n within FP32's range.  No branch, so
// several proposals' chains can be interleaved.
__device__ __forceinline__ double rsqrt_newton(double n) {
    double y = double(rsqrtf(float(n)));
    const double hn = 0.5 * n;
#pragma unroll
    for (int i = 0; i < 2; i++) y = fma(y, fma(-hn * y, y, 0.5), y);
    return y;
}

template <class R>
__device__ __forceinline__ Su2<R> su2_from(const uint4& o, double eps, double x0) {
    const double v1 = centred(o.y), v2 = centred(o.z), v3 = centred(o.w);
    const double len = eps * rsqrt_newton(fma(v1, v1, fma(v2, v2, v3 * v3)));
    Su2<R> m;
    m.a = cx(R(o.x < 0x80000000u ? -x0 : x0), R(v3 * len));
    m.b = cx(R(v2 * len), R(v1 * len));
    return m;
}

template <class R>
__device__ __forceinline__ Cx<R> cmul(const Cx<R>& x, const Cx<R>& y) {
    return cx(fma(x.re, y.re, -x.im * y.im), fma(x.re, y.im, x.im * y.re));
}
// x y + z w
template <class R>
__device__ __forceinline__ Cx<R> cmul2(const Cx<R>& x, const Cx<R>& y, const Cx<R>& z, const Cx<R>& w) {
    return cx(fma(x.re, y.re, fma(-x.im, y.im, fma(z.re, w.re, -z.im * w.im))),
              fma(x.re, y.im, fma(x.im, y.re, fma(z.re, w.im, z.im * w.re))));
}
template <class R>
__device__ __forceinline__ Cx<R> neg_conj(const Cx<R>& x) {
    return cx(-x.re, x.im);
}
template <class R>
__device__ __forceinline__ Cx<R> conj_of(const Cx<R>& x) {
    return cx(x.re, -x.im);
}

// R S T of SU(2) elements in the (0,1), (0,2) and (1,2) blocks: twelve complex
// products, the zeros of the factors left out.
template <class R>
__device__ __forceinline__ void rst_product(const Su2<R>& r, const Su2<R>& s, const Su2<R>& t, M3<R>& x) {
    const Cx<R> rc = neg_conj(r.b), rd = conj_of(r.a);  // row 1 of R
    const Cx<R> sc = neg_conj(s.b), sd = conj_of(s.a);  // row 2 of S
    const Cx<R> tc = neg_conj(t.b), td = conj_of(t.a);  // row 2 of T
    const Cx<R> p02 = cmul(r.a, s.b), p12 = cmul(rc, s.b);
    x.e[0][0] = cmul(r.a, s.a);
    x.e[0][1] = cmul2(r.b, t.a, p02, tc);
    x.e[0][2] = cmul2(r.b, t.b, p02, td);
    x.e[1][0] = cmul(rc, s.a);
    x.e[1][1] = cmul2(rd, t.a, p12, tc);
    x.e[1][2] = cmul2(rd, t.b, p12, td);
    x.e[2][0] = sc;
    x.e[2][1] = cmul(sd, tc);
    x.e[2][2] = cmul(sd, td);
}

// exp(x) > r for r = unit(w), in FP32: 1, 0, or -1 where the two are closer
// than the FP32 evaluation can be off (about one call in 10^5, and NaN).
__device__ __forceinline__ int exp_exceeds_fp32(double x, uint32_t w) {
    const float xf = float(x);
    const float e = expf(xf), r = fmaf(float(w), 2.3283064e-10f, 1.1641532e-10f);
    // x rounded to FP32: |x| 2^-24; expf: 2 ulp; r: 2 roundings; doubled
    const float off = fmaf(e, fmaf(fabsf(xf), 1.2e-7f, 5e-7f), r * 3e-7f);
    return fabsf(e - r) > off ? int(e > r) : -1;
}

// This lane's part of the staple sum: every `group`-th of the three directions
// nu != mu, from the `j`-th.
template <class F>
__device__ __forceinline__ M3<typename F::Real> staple_part(const F& u, const Geo& g, int s, const int c[4], int mu,
                                                            int j, int group) {
    using R = typename F::Real;
    M3<R> omega;
    mzero(omega);
    const int cmu = g.coord(c, mu);
    const int s_pm = g.hop_rt(s, cmu, mu, +1);
#pragma unroll 1
    for (int k = j; k < 3; k += group) {
        const int nu = k + (k >= mu ? 1 : 0);
        const int cnu = g.coord(c, nu);
        const int s_pn = g.hop_rt(s, cnu, nu, +1);
        const int s_mn = g.hop_rt(s, cnu, nu, -1);
        const int s_pm_mn = g.hop_rt(s_mn, cmu, mu, +1);
        M3<R> t;
        mmul<false, true>(u.template load<false>(nu, s_pm), u.template load<false>(mu, s_pn), t);
        mmul_acc<false, true>(t, u.template load<false>(nu, s), omega);
        mmul<true, true>(u.template load<false>(nu, s_pm_mn), u.template load<false>(mu, s_mn), t);
        mmul_acc<false, false>(t, u.template load<false>(nu, s_mn), omega);
    }
    return omega;
}

constexpr int kMetroThreads = 64;

// Proposal `hit` of link l: X, the acceptance draw's word, and beta/3 Re tr[(U' -
// U) A] = beta/3 Re tr[(X - 1) W], W = U A.
template <class R>
__device__ __forceinline__ double propose(uint32_t l0, uint32_t l1, uint32_t sweep, uint32_t hit, uint2 key,
                                          double eps, double x0, double beta_3, const M3<R>& W, M3<R>& X,
                                          uint32_t& draw) {
    const uint4 oa = philox_g(make_uint4(l0, l1, sweep, hit), key);
    const uint4 ob = philox_g(make_uint4(l0, l1 ^ (1u << 24), sweep, hit), key);
    const uint4 oc = philox_g(make_uint4(l0, l1 ^ (2u << 24), sweep, hit), key);
    const uint4 od = philox_g(make_uint4(l0, l1 ^ (3u << 24), sweep, hit), key);
    M3<R> m;
    rst_product(su2_from<R>(oa, eps, x0), su2_from<R>(ob, eps, x0), su2_from<R>(oc, eps, x0), m);
    const bool inverse = od.y < 0x80000000u;  // X^+ with probability 1/2
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            X.e[i][j] = cx(inverse ? m.e[j][i].re : m.e[i][j].re, inverse ? -m.e[j][i].im : m.e[i][j].im);
    R dtr = R(0);
#pragma unroll
    for (int i = 0; i < 3; i++) {  // one sum per row of X
        R d = R(0);
#pragma unroll
        for (int j = 0; j < 3; j++) {
            d = fma(i == j ? X.e[i][j].re - R(1) : X.e[i][j].re, W.e[j][i].re, d);
            d = fma(-X.e[i][j].im, W.e[j][i].im, d);
        }
        dtr += d;
    }
    draw = od.x;
    return beta_3 * double(dtr);
}

// G lanes per link of the (mu, parity) class (1, 2, 4 or 8); link h's site is the
// one of that parity in the x pair (2h, 2h + 1) (extents are even).  The lanes
// of a link share its staples, then draw the next G proposals against the same
// link, one each; the first accepted one is taken and the later ones are drawn
// again from the new link, so the chain is that of one proposal after another.
// The trace change of a proposal needs W = U A only, so U and W are multiplied
// by X only when it is accepted.
//
// One proposal in nine is accepted (eps = 0.24), so nearly every hit some links
// of a warp have two 3x3 products to do and most have none.  U, W and the
// accepted X stand in shared memory and the warp does the products together:
// six lanes per accepted link, each a column of X U or X W, five links at a
// time.
//
// Bound by the chain of a hit and the few warps that 168 registers (FP64) and
// a small lattice's links leave.  FP64, 30 hits, per launch on B200, before
// (each thread multiplying its own link) and now: 12^4 (4 lanes) 27.0 -> 24.1
// us, 16^4 53.0 -> 47.6, 24^4 206 -> 184, 32^4 600 -> 525; FP32-12 16^4 37.9 ->
// 37.1, 32^4 458 -> 386.  (One thread per site, half of them idle, and dense
// products for every proposal: 16^4 153 us, 32^4 2.4 ms.)  Two or three
// proposals per thread at a time gained nothing, nor did drawing the next hit's
// X during this one's test (16^4 47.9 us, 24^4 225), reading W's triangle
// instead of forming X^+ (48.1, 184) or 7 blocks per SM (53, 210).
template <class F, int G>
__global__ void __launch_bounds__(kMetroThreads, G == 1 ? 5 : 6)
    metropolis_kernel(F u, Geo g, int mu, int parity, double beta_3, double eps, double x0, int hits, uint64_t seed,
                      uint32_t sweep, unsigned long long* accepted) {
    using R = typename F::Real;
    constexpr int kLinks = kMetroThreads / G, kWarpLinks = 32 / G;
    __shared__ Cx<R> uw[18][kLinks];  // U, then W
    __shared__ Cx<R> xs[9][kLinks];
    __shared__ int takers[kLinks];  // the links of a warp that accepted, in order
    const int lane = int(threadIdx.x & 31), j = lane & (G - 1), slot = int(threadIdx.x) / G;
    int* const warp_takers = takers + slot / kWarpLinks * kWarpLinks;
    const int col = (lane % 6) % 3 + ((lane % 6) / 3) * 9;  // this lane's column in uw: entries col, col + 3, col + 6
    const int h2 = 2 * (int(blockIdx.x) * kLinks + slot);
    const bool link = h2 < g.V;
    grid_wait();
    int s = 0;
    {
        M3<R> U, A, W;
        mzero(U);
        mzero(A);
        if (link) {
            int c[4];
            g.coords(h2, c);
            const int odd = (c[1] + c[2] + c[3] + parity) & 1;
            s = h2 + odd;
            c[0] += odd;
            A = staple_part(u, g, s, c, mu, j, G);
            U = u.template load<false>(mu, s);
        }
#pragma unroll
        for (int o = 1; o < G; o <<= 1)
#pragma unroll
            for (int e = 0; e < 9; e++) {
                A.e[e / 3][e % 3].re += __shfl_xor_sync(0xffffffffu, A.e[e / 3][e % 3].re, o);
                A.e[e / 3][e % 3].im += __shfl_xor_sync(0xffffffffu, A.e[e / 3][e % 3].im, o);
            }
        mmul<false, false>(U, A, W);
        if (j == 0) {
#pragma unroll
            for (int e = 0; e < 9; e++) {
                uw[e][slot] = U.e[e / 3][e % 3];
                uw[9 + e][slot] = W.e[e / 3][e % 3];
            }
        }
        __syncwarp();
    }
    const uint64_t l = uint64_t(s) * 4 + uint64_t(mu);
    const uint32_t l0 = uint32_t(l), l1 = uint32_t(l >> 32);
    const uint2 key = make_uint2(uint32_t(seed), uint32_t(seed >> 32) ^ 0x4D455452u);
    unsigned acc = 0;  // of this lane's proposals
    int h = link ? 0 : hits;
    while (__any_sync(0xffffffffu, h < hits)) {
        M3<R> X, W;
#pragma unroll
        for (int e = 0; e < 9; e++) W.e[e / 3][e % 3] = uw[9 + e][slot];
        uint32_t draw;
        const double x = propose(l0, l1, sweep, uint32_t(h + j), key, eps, x0, beta_3, W, X, draw);
        int ok = exp_exceeds_fp32(x, draw);
        if (ok < 0) ok = exp(x) > unit(draw);
        unsigned taken = __ballot_sync(0xffffffffu, ok && h + j < hits);  // one lane per link that accepts, its first
        int first = 0;
        if (G > 1) {
            const unsigned mine = (taken >> (lane & ~(G - 1))) & ((1u << G) - 1u);
            first = mine ? __ffs(int(mine)) - 1 : G - 1;
            taken = __ballot_sync(0xffffffffu, mine && j == first);
        }
        if (taken >> lane & 1u) {
#pragma unroll
            for (int e = 0; e < 9; e++) xs[e][slot] = X.e[e / 3][e % 3];
            warp_takers[__popc(taken & ((1u << lane) - 1u))] = slot;
            acc++;
        }
        __syncwarp();
        for (int r = lane < 30 ? lane / 6 : kWarpLinks; r < __popc(taken); r += 5) {
            const int o = warp_takers[r];
            const Cx<R> y[3] = {uw[col][o], uw[col + 3][o], uw[col + 6][o]};
#pragma unroll
            for (int i = 0; i < 3; i++) {  // the sums of mmul
                R re = R(0), im = R(0);
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const Cx<R> a = xs[3 * i + k][o];
                    re = fma(a.re, y[k].re, re);
                    re = fma(-a.im, y[k].im, re);
                    im = fma(a.re, y[k].im, im);
                    im = fma(a.im, y[k].re, im);
                }
                uw[col + 3 * i][o] = cx(re, im);
            }
        }
        __syncwarp();
        h += first + 1;
    }
    const unsigned changed = __ballot_sync(0xffffffffu, acc != 0) >> (lane & ~(G - 1)) & ((1u << G) - 1u);
    grid_release();
    if (changed && j == 0) {
        M3<R> U;
#pragma unroll
        for (int e = 0; e < 9; e++) U.e[e / 3][e % 3] = uw[e][slot];
        u.store(mu, s, U);
    }
    // warp sum, one atomic per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0 && acc) atomicAdd(accepted, (unsigned long long)acc);
}

template <class F>
cudaError_t launch_metro_typed(void* u, const Geo& g, int mu, int parity, double beta, double eps, int hits,
                               uint64_t seed, uint32_t sweep, unsigned long long* accepted, cudaStream_t st) {
    const unsigned links = unsigned(g.V / 2);
    const double x0 = std::sqrt(std::fma(-eps, eps, 1.0));
    auto launch = [&](auto kernel, unsigned lanes) {
        const unsigned per_block = kMetroThreads / lanes;
        return launch_chained(true, kernel, (links + per_block - 1) / per_block, kMetroThreads, st, F{u, g.V}, g, mu,
                              parity, beta / 3.0, eps, x0, hits, seed, sweep, accepted);
    };
    // Few links leave the SMs short of warps, and a launch lasts as long as one
    // link's chain of hits: more lanes per link draw more of the chain at once.
    // Every count is the fastest until its blocks no longer fit the GPU at once
    // (6 a SM at 168 registers, 148 SMs; 8 lanes until 2 a SM, where a hit of the
    // narrower form is as short).  us per launch on B200 (30 hits) at 1 / 2 / 4
    // / 8 lanes, FP64: 2048 links 33.1 / 22.1 / 15.1 / 13.7, 4096 33.1 / 22.1 /
    // 16.1 / 16.8, 13824 34.9 / 28.4 / 25.4 / 36.3, 15552 35.1 / 28.9 / 35.5 /
    // 42.9, 27648 45.4 / 37.8 / 45.5 / 65.0, 29376 46.8 / 53.2 / 52.7 / 68.8;
    // FP32-12: 2048 27.3 / 18.5 / 13.4 / 11.5, 13824 28.0 / 24.0 / 21.5 / 30.3,
    // 15552 28.0 / 24.3 / 25.5 / 32.5, 27648 36.4 / 31.0 / 39.4 / 49.3, 29376
    // 36.6 / 37.9 / 40.2 / 51.7.
    constexpr unsigned kSms = 148, kResident = 6 * kSms;
    if (links <= 2 * kSms * (kMetroThreads / 8)) return launch(metropolis_kernel<F, 8>, 8);
    if (links <= kResident * (kMetroThreads / 4)) return launch(metropolis_kernel<F, 4>, 4);
    if (links <= kResident * (kMetroThreads / 2)) return launch(metropolis_kernel<F, 2>, 2);
    // Past one wave of one-lane FP64 blocks the few blocks of the second take a
    // chain's time alone; half as many links per block even that out until the
    // second wave is a third full: 57344 links 88.3 / 81.7 us, 65536 99.5 / 89.1,
    // 73728 102.0 / 92.9, but 90112 108.4 / 117.8.  (FP32 blocks fit 8 a SM and
    // gain nothing: 77824 links 77.8 / 79.8.)
    constexpr unsigned kWave = kResident * kMetroThreads;
    if (sizeof(typename F::Real) == 8 && links > kWave && links <= kWave / 3 * 4) return launch(metropolis_kernel<F, 2>, 2);
    return launch(metropolis_kernel<F, 1>, 1);
}

}  // namespace

cudaError_t launch_metropolis(int prec, void* u, const Geo& g, int mu, int parity, double beta, double eps, int hits,
                              uint64_t seed, uint32_t sweep, unsigned long long* accepted, cudaStream_t st) {
    switch (prec) {
        case kFP64: return launch_metro_typed<FieldD18>(u, g, mu, parity, beta, eps, hits, seed, sweep, accepted, st);
        case kFP32_18: return launch_metro_typed<FieldF18>(u, g, mu, parity, beta, eps, hits, seed, sweep, accepted, st);
        case kFP32_12: return launch_metro_typed<FieldF12>(u, g, mu, parity, beta, eps, hits, seed, sweep, accepted, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ym
