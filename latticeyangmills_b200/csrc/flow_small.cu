// The RK3 stage and the observables of small lattices, one launch each.
//
// A lattice of a few thousand sites fills the GPU with less than one wave of
// blocks, so a launch lasts as long as one thread's chain of loads and products.
// Here the chain is cut into its independent plaquette loops, one per thread,
// 18 (stage) or 24 (observables) per site, which meet in shared memory:
//
//   stage        D_mu(x) = sum_{nu != mu} [ s_{mu nu} H_p(x) - L_{mu nu}(x) ], where H_p(x)
//                is the generator (i/2)[.]_TL of the plaquette of plane p = {mu, nu}
//                and L_{mu nu}(x) that of the loop x -> x-nu -> x-nu+mu -> x+mu -> x
//                (the lower staple's, src/Actions/puregauge.cpp:36-54); then one
//                thread per link finishes as the other stage kernels do.
//   observables  each clover leaf's generator (observables.cu), summed per plane.
//
// Bound by launch latency and by one wave's chain: loads, one loop's products
// (4.5 warps per scheduler), a barrier, one link's exponential.  8^4 on B200,
// us per step / per measured step: FP64 20.5 / 35.7 -> 15.1 / 23.8, FP32-12 (as
// fused staple kernels) 17.4 / 27.5 -> 11.3 / 18.3.
//
// The stage's loops are multiplied out in all three rows.  Links drift from
// SU(3) by their rounding (until a reunitarisation, FP64 ones for good), and a
// loop whose row 2 is completed from the others carries that drift into its
// generator (force_from_b_cdag).  The two-kernel stage completes its
// plaquettes too, but takes a link's upper and lower loops from the same ones,
// so that the error cancels along the lattice; loops completed one by one do
// not: after 400 steps of eps = 0.01 from a = 0.35 without reunitarisation, at
// 8^4, rms error of the links against the flow in higher precision 1.11e-15
// (FP64) and 6.1e-7 (FP32) in two rows, 7.5e-16 and 4.3e-7 in three, 7.6e-16 and
// 4.4e-7 in the two-kernel stage.  Two rows run 14.5 (FP64) and 10.7 us (FP32-12)
// per step; the lower loops as transported plaquettes, as exact, 17.3 and 11.4.
//
// Stage forms 0 and 1 of a configuration of at most kSmallSites sites run this
// kernel, whole lattices, slabs and blocks alike (the rule goes by the whole
// configuration's volume), so decomposed flows stay bit-identical to whole ones.
#include "flow_device.cuh"
#include "kernels.h"
#include "observables.cuh"

namespace ym {

namespace {

// Generator of the loop x -> x-nu -> x-nu+mu -> x+mu -> x, begun with
// U_nu(x-nu)^+ and closed with U_mu(x)^+ (clover leaf Q4), through two rows.
template <class F>
__device__ __forceinline__ Herm8<typename F::Real> lower_loop(const F& u, const Geo& g, int s, const int c[4], int mu,
                                                              int nu) {
    using R = typename F::Real;
    const int w = g.hop_rt(s, g.coord(c, nu), nu, -1);
    const int w_pm = g.hop_rt(w, g.coord(c, mu), mu, +1);
    Rows2<R> b, t;
    mmul_rows2<true, false>(u.template load<false>(nu, w), u.template load<false>(mu, w), t);
    mmul_rows2<false, false>(t, u.template load<false>(nu, w_pm), b);
    return force_from_b2_cdag(b, u.template load<false>(mu, s));
}

// The stage's loops, every row multiplied out: the plaquette of plane (a, b) and
// lower_loop's loop.
template <class F>
__device__ __forceinline__ Herm8<typename F::Real> stage_plaquette(const F& u, const Geo& g, int s, const int c[4],
                                                                   int a, int b) {
    using R = typename F::Real;
    M3<R> t, x;
    mmul<false, false>(u.template load<false>(a, s), u.template load<false>(b, g.hop_rt(s, g.coord(c, a), a, +1)), t);
    mmul<false, true>(t, u.template load<false>(a, g.hop_rt(s, g.coord(c, b), b, +1)), x);
    return force_from_b_cdag(x, u.template load<false>(b, s));
}
template <class F>
__device__ __forceinline__ Herm8<typename F::Real> stage_lower_loop(const F& u, const Geo& g, int s, const int c[4],
                                                                    int mu, int nu) {
    using R = typename F::Real;
    const int w = g.hop_rt(s, g.coord(c, nu), nu, -1);
    const int w_pm = g.hop_rt(w, g.coord(c, mu), mu, +1);
    M3<R> t, x;
    mmul<true, false>(u.template load<false>(nu, w), u.template load<false>(mu, w), t);
    mmul<false, false>(t, u.template load<false>(nu, w_pm), x);
    return force_from_b_cdag(x, u.template load<false>(mu, s));
}

// Generators of the clover leaves Q2 and Q3 of plane (mu, nu) (observables.cu).
template <class F>
__device__ __forceinline__ Herm8<typename F::Real> leaf_q2(const F& u, const Geo& g, int s, const int c[4], int mu,
                                                           int nu) {
    using R = typename F::Real;
    const int y = g.hop_rt(s, g.coord(c, mu), mu, -1);
    const int y_pn = g.hop_rt(y, g.coord(c, nu), nu, +1);
    Rows2<R> b, t;
    M3<R> close;
    mmul_rows2<true, false>(u.template load<false>(mu, y), u.template load<false>(nu, y), t);
    full_from_rows2(t, close);
    mmul_rows2<false, true>(u.template load_rows2<false>(nu, s), u.template load<false>(mu, y_pn), b);
    return force_from_b2_cdag(b, close);
}

template <class F>
__device__ __forceinline__ Herm8<typename F::Real> leaf_q3(const F& u, const Geo& g, int s, const int c[4], int mu,
                                                           int nu) {
    using R = typename F::Real;
    const int y = g.hop_rt(s, g.coord(c, mu), mu, -1);
    const int w = g.hop_rt(s, g.coord(c, nu), nu, -1);
    const int z = g.hop_rt(y, g.coord(c, nu), nu, -1);
    Rows2<R> b, t;
    M3<R> close;
    mmul_rows2<true, true>(u.template load<false>(nu, w), u.template load<false>(mu, z), t);
    full_from_rows2(t, close);
    mmul_rows2<true, true>(u.template load<false>(mu, y), u.template load<false>(nu, z), b);
    return force_from_b2_cdag(b, close);
}

// Generators of one block's loops, [loop][component][lane].
template <class R, int N>
struct LoopStore {
    R v[N][8][32];
    __device__ __forceinline__ void put(int loop, int lane, const Herm8<R>& h) {
        R(*d)[32] = v[loop];
        d[0][lane] = h.d0;
        d[1][lane] = h.d1;
        d[2][lane] = h.z01.re;
        d[3][lane] = h.z01.im;
        d[4][lane] = h.z02.re;
        d[5][lane] = h.z02.im;
        d[6][lane] = h.z12.re;
        d[7][lane] = h.z12.im;
    }
    __device__ __forceinline__ Herm8<R> get(int loop, int lane) const {
        const R(*d)[32] = v[loop];
        Herm8<R> h;
        h.d0 = d[0][lane];
        h.d1 = d[1][lane];
        h.z01 = cx(d[2][lane], d[3][lane]);
        h.z02 = cx(d[4][lane], d[5][lane]);
        h.z12 = cx(d[6][lane], d[7][lane]);
        return h;
    }
};

template <class R>
__device__ __forceinline__ Herm8<R> h8_add(const Herm8<R>& a, const Herm8<R>& b) {
    return h8_axpy(R(1), a, b);
}

constexpr int kStageThreads = 18 * 32;

// One block per 32 sites: warps 3 mu + k the lower loops of link mu and its
// k-th other direction, warps 12 + p the plaquettes of plane p; then warps
// 0..3 the links.  HALO: a slab's boundary links also go into its neighbours'
// halos, as in rk_link_update_to.
template <class F, int STAGE, bool HALO>
__global__ void __launch_bounds__(kStageThreads, 1)
    rk_small_stage_kernel(F in, F out, ForceField<typename F::Real> zf, Geo g, typename F::Real eps,
                          HaloTargets<F> h) {
    using R = typename F::Real;
    __shared__ LoopStore<R, 18> loops;
    const int w = int(threadIdx.x >> 5), lane = int(threadIdx.x & 31);
    const int s = g.site0 + int(blockIdx.x) * 32 + lane;
    const bool active = s < g.site1;
    int c[4];
    g.coords(active ? s : g.site0, c);
    grid_wait();
    if (active) {
        if (w < 12) {
            const int mu = w / 3, k = w - 3 * mu;
            loops.put(w, lane, stage_lower_loop(in, g, s, c, mu, k + (k >= mu ? 1 : 0)));
        } else {
            const int p = w - 12;
            loops.put(w, lane, stage_plaquette(in, g, s, c, plane_a(p), plane_b(p)));
        }
    }
    const int mu = w;
    Herm8<R> prev = {};
    if (STAGE != 0 && w < 4 && active) prev = zf.load(mu, s);  // arrives while the block's loops finish
    __syncthreads();
    if (w >= 4 || !active) return;
    Herm8<R> d;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int nu = k + (k >= mu ? 1 : 0);
        const int p = mu < nu ? plane_index(mu, nu) : plane_index(nu, mu);
        const R sg = mu < nu ? R(1) : R(-1);
        const Herm8<R> part = h8_axpy(sg, loops.get(12 + p, lane), h8_neg(loops.get(3 * mu + k, lane)));
        d = k == 0 ? part : h8_add(part, d);
    }
    const M3<R> u = in.template load<false>(mu, s);
    const Rows2<R> un = rk_finish_from<F, STAGE>(out, zf, eps, s, mu, d, u, prev);
    if constexpr (HALO) {
        if (c[3] == 1) h.lower.store_rows2(mu, h.lower_t * h.slice_sites + (s - h.slice_sites), un);
        if (c[3] == h.nt) h.upper.store_rows2(mu, s - h.nt * h.slice_sites, un);
    }
}

constexpr int kSmallObsThreads = 12 * 32;

// One block per 32 sites: warp 2 p the leaves Q1 and Q3 of plane p, warp 2 p + 1
// Q2 and Q4; their sums give S = (i/2)[C]_TL (G = -2i S), warps 0..5 take the
// energy of one plane each, warps 0..2 then the charge of one pair each.  The
// block that finishes last folds the partials, in block order (a second launch
// would take as long as this one).
template <class F>
__global__ void __launch_bounds__(kSmallObsThreads, 1)
    small_observables_kernel(F u, Geo g, double* partials, unsigned* done, double inv_18v, double* out) {
    using R = typename F::Real;
    __shared__ LoopStore<R, 6> half, full;
    __shared__ bool last;
    const int w = int(threadIdx.x >> 5), lane = int(threadIdx.x & 31);
    const int s = g.site0 + int(blockIdx.x) * 32 + lane;
    bool active = s < g.site1;
    int c[4];
    g.coords(active ? s : g.site0, c);
    active = active && g.interior(c);  // a block's halo sites are its neighbours'
    grid_wait();
    double plaq = 0.0, energy = 0.0, topc = 0.0;
    Herm8<R> sum;
    if (active) {
        const int p = w >> 1, mu = plane_a(p), nu = plane_b(p);
        if (w & 1) {
            sum = h8_add(leaf_q2(u, g, s, c, mu, nu), lower_loop(u, g, s, c, mu, nu));
            half.put(p, lane, sum);
        } else {
            R t;
            sum = plane_generator<false>(u, g, s, c, mu, nu, &t);
            sum = h8_add(leaf_q3(u, g, s, c, mu, nu), sum);
            plaq = double(t);
        }
    }
    __syncthreads();
    if (active && !(w & 1)) {
        sum = h8_add(half.get(w >> 1, lane), sum);
        energy = -4.0 * double(herm_trace_mul(sum, sum));
        full.put(w >> 1, lane, sum);
    }
    __syncthreads();
    if (active && w < 3) {  // pairs (01,23), (02,13), (03,12): planes k and 5 - k
        const double t = 4.0 * double(herm_trace_mul(full.get(w, lane), full.get(5 - w, lane)));
        topc = w == 1 ? -t : t;
    }
    block_sum3(plaq, energy, topc);
    if (threadIdx.x == 0) {
        partials[3 * blockIdx.x + 0] = plaq;
        partials[3 * blockIdx.x + 1] = energy;
        partials[3 * blockIdx.x + 2] = topc;
        __threadfence();
        last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;  // wraps to 0 for the next launch
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    plaq = energy = topc = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
        plaq += __ldcg(partials + 3 * i + 0);
        energy += __ldcg(partials + 3 * i + 1);
        topc += __ldcg(partials + 3 * i + 2);
    }
    block_sum3(plaq, energy, topc);
    if (threadIdx.x == 0) write_row(plaq, energy, topc, inv_18v, out);
}

unsigned site_groups(const Geo& g) { return unsigned((g.site1 - g.site0 + 31) / 32); }

template <class F, bool HALO>
cudaError_t launch_small_typed(int stage, const void* uin, void* uout, void* z, const Geo& g, double eps,
                               const HaloTargets<F>& h, bool chained, cudaStream_t st) {
    using R = typename F::Real;
    const F in{const_cast<void*>(uin), g.V}, out{uout, g.V};
    const ForceField<R> zf{z, g.V};
    const R e = R(stage == 0 ? eps * 0.25 : eps);
    auto launch = [&](auto kernel) {
        return launch_chained(chained, kernel, site_groups(g), kStageThreads, st, in, out, zf, g, e, h);
    };
    switch (stage) {
        case 0: return launch(rk_small_stage_kernel<F, 0, HALO>);
        case 1: return launch(rk_small_stage_kernel<F, 1, HALO>);
        default: return launch(rk_small_stage_kernel<F, 2, HALO>);
    }
}

template <class F>
cudaError_t launch_small_halo_typed(int stage, const void* uin, void* uout, void* z, const Geo& g, double eps,
                                    void* lower_out, int lower_v, int lower_t, void* upper_out, int upper_v,
                                    cudaStream_t st) {
    const HaloTargets<F> h{F{lower_out, lower_v}, F{upper_out, upper_v}, g.site0, (g.site1 - g.site0) / g.site0,
                           lower_t};
    return launch_small_typed<F, true>(stage, uin, uout, z, g, eps, h, false, st);
}

template <class F>
cudaError_t launch_small_obs_typed(const void* u, const Geo& g, double* partials, double* out, bool chained,
                                   cudaStream_t st) {
    unsigned* done = reinterpret_cast<unsigned*>(partials + small_partials(g) - 1);
    return launch_chained(chained, small_observables_kernel<F>, site_groups(g), kSmallObsThreads, st,
                          F{const_cast<void*>(u), g.V}, g, partials, done, 1.0 / (18.0 * double(g.vglobal)), out);
}

}  // namespace

cudaError_t launch_small_stage(int prec, int stage, const void* uin, void* uout, void* z, const Geo& g, double eps,
                               bool chained, cudaStream_t st) {
    switch (prec) {
        case kFP64: return launch_small_typed<FieldD18, false>(stage, uin, uout, z, g, eps, {}, chained, st);
        case kFP32_18: return launch_small_typed<FieldF18, false>(stage, uin, uout, z, g, eps, {}, chained, st);
        case kFP32_12: return launch_small_typed<FieldF12, false>(stage, uin, uout, z, g, eps, {}, chained, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_small_stage_halo(int prec, int stage, const void* uin, void* uout, void* z, const Geo& g, double eps,
                                    void* lower_out, int lower_v, int lower_t, void* upper_out, int upper_v,
                                    cudaStream_t st) {
    switch (prec) {
        case kFP64:
            return launch_small_halo_typed<FieldD18>(stage, uin, uout, z, g, eps, lower_out, lower_v, lower_t,
                                                     upper_out, upper_v, st);
        case kFP32_18:
            return launch_small_halo_typed<FieldF18>(stage, uin, uout, z, g, eps, lower_out, lower_v, lower_t,
                                                     upper_out, upper_v, st);
        case kFP32_12:
            return launch_small_halo_typed<FieldF12>(stage, uin, uout, z, g, eps, lower_out, lower_v, lower_t,
                                                     upper_out, upper_v, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_small_observables(int prec, const void* u, const Geo& g, double* partials, double* out,
                                     bool chained, cudaStream_t st) {
    switch (prec) {
        case kFP64: return launch_small_obs_typed<FieldD18>(u, g, partials, out, chained, st);
        case kFP32_18: return launch_small_obs_typed<FieldF18>(u, g, partials, out, chained, st);
        case kFP32_12: return launch_small_obs_typed<FieldF12>(u, g, partials, out, chained, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ym
