// K1 as two kernels: the RK3 stage of one configuration with its force built
// from a stored plaquette field.
//
// Each link's generator D_mu(x) = (i/2)[U Omega - (U Omega)^+]_TL
// (src/Actions/puregauge.cpp:36-79) is a sum over the six plaquettes through
// the link, each read from the link's own corner.  With
//   P_ab(x) = U_a(x) U_b(x+a) U_a(x+b)^+ U_b(x)^+,   a < b, six planes per site,
//   H_ab(x) = (i/2)[P_ab(x) - P_ab(x)^+]_TL          (Hermitian traceless, 8 reals),
// the upper loop of link (mu, x) in plane (mu, nu) is P_{mu nu}(x) and the lower
// loop is U_nu(y)^+ P_{mu nu}(y)^+ U_nu(y) with y = x - nu; P_{nu mu} = P_{mu nu}^+,
// and (i/2)[.]_TL commutes with the conjugation by a unitary matrix, so
//   D_mu(x) = sum_{nu != mu} s_{mu nu} [ H_p(x) - U_nu(y)^+ H_p(y) U_nu(y) ],
// with p the plane {mu, nu} and s_{mu nu} = +1 for mu < nu, -1 otherwise.
//
// plaq_field_kernel forms the six H_p(x) of every site (three SU(3) products
// each, 8 reals stored); rk_split_stage_kernel then builds D from three
// conjugations v^+ H v per link and finishes the stage as the fused kernel does
// (device code in flow_device.cuh, shared with the ensemble kernels).
// Per link that is 6 x 3 / 4 + 3 x (1 + 1/2) products' worth of multiply-adds
// in place of 13, for 2 x 6 x 8 reals of plaquette field per site written and
// read.
#include "flow_device.cuh"
#include "kernels.h"
#include "observables.cuh"

namespace ym {

// Planes per thread of the plaquette-field kernel (below): two for the FP32
// forms; one in FP64, where a pair needs 132 registers (2 blocks of 6 warps
// per SM) and a single plane 80: at 32^4 on B200 the FP64 field kernel runs
// 0.294 -> 0.270 ms per launch, the two-kernel FP64 step 1.80 -> 1.73 ms.
template <class F>
struct PlaqPlanesPerThread {
    static constexpr int value = sizeof(typename F::Real) == 8 ? 1 : 2;
};

// One thread per (site, pair of planes): six warps cover 64 sites, warps
// 3k .. 3k + 2 the planes {(0,1), (0,2)}, {(0,3), (1,3)}, {(1,2), (2,3)} of
// site group k (the two planes of a pair share one of the site's links,
// loaded once).  The second plane's loads issue during the first plane's
// products: against one plane per thread, the FP32-18 kernel ran 16 % faster
// at 32^4 on B200 (0.180 -> 0.151 ms), the 12-real one 1.6 % (0.148 -> 0.146).
// With one plane per thread (PlaqPlanesPerThread 1) six warps cover 32 sites,
// warp w plane w.

template <class F>
__global__ void __launch_bounds__(192, PlaqMinBlocks<F>::value) plaq_field_kernel(F u, ForceField<typename F::Real> hf, Geo g) {
    const int w = int(threadIdx.x >> 5);
    // FP32: blocks walk the lattice from its end, so the stage kernel that
    // follows starts at site 0, whose links and plane generators this launch
    // touched last and are still in L2: 1 % off the FP32-12 step at 32^4 on
    // B200, in bursts (0.7535 -> 0.747 ms) and in the power-capped steady
    // state (0.886 -> 0.878); in FP64 the field kernel itself runs 9 % slower
    // that way (0.274 -> 0.298 ms), so FP64 keeps the ascending order
    const int blk = sizeof(typename F::Real) == 4 ? int(gridDim.x - 1 - blockIdx.x) : int(blockIdx.x);
    int c[4];
    if (PlaqPlanesPerThread<F>::value == 1) {
        const int s = g.site0 + blk * 32 + int(threadIdx.x & 31);
        if (s >= g.site1) return;
        g.coords(s, c);
        grid_wait();
        const auto h = plane_generator<false>(u, g, s, c, plane_a(w), plane_b(w));
        grid_release();
        hf.store(w, s, h);
        return;
    }
    const int s = g.site0 + (blk * 2 + w / 3) * 32 + int(threadIdx.x & 31);
    if (s >= g.site1) return;
    const int pr = w % 3;
    const int p0 = pr == 0 ? 0 : (pr == 1 ? 2 : 3);
    const int p1 = pr == 0 ? 1 : (pr == 1 ? 4 : 5);
    g.coords(s, c);
    grid_wait();
    // both planes before either store: the link the two share is loaded once
    const auto h0 = plane_generator<false>(u, g, s, c, plane_a(p0), plane_b(p0));
    const auto h1 = plane_generator<false>(u, g, s, c, plane_a(p1), plane_b(p1));
    grid_release();
    hf.store(p0, s, h0);
    hf.store(p1, s, h1);
}

// One thread per link: four warps (directions) per 32 sites.
template <class F, int STAGE, class FO>
__global__ void __launch_bounds__(128, SplitMinBlocks<F>::value)
    rk_split_stage_kernel(F in, FO out, ForceField<typename F::Real> zf, ForceField<typename F::Real> hf, Geo g,
                          typename F::Real eps) {
    const int mu = int(threadIdx.x >> 5) & 3;
    const int s = g.site0 + int(blockIdx.x) * 32 + int(threadIdx.x & 31);
    grid_wait();
    if (s >= g.site1) return;
    split_link_update<F, STAGE, FO, false>(in, out, zf, hf, g, eps, s, mu);
}

// The same for a time slab, storing its boundary links into its neighbours'
// halos (the two-kernel form of rk_stage_halo_kernel).
template <class F, int STAGE>
__global__ void __launch_bounds__(128, SplitMinBlocks<F>::value)
    rk_split_stage_halo_kernel(F in, F out, ForceField<typename F::Real> zf, ForceField<typename F::Real> hf, Geo g,
                               typename F::Real eps, HaloTargets<F> h) {
    const int mu = int(threadIdx.x >> 5) & 3;
    const int s = g.site0 + int(blockIdx.x) * 32 + int(threadIdx.x & 31);
    if (s >= g.site1) return;
    split_link_update_to<F, STAGE, true>(in, out, zf, hf, g, eps, s, mu, h);
}

template <class F>
static cudaError_t launch_split_halo_typed(int stage, const void* uin, void* uout, void* z, const void* hp,
                                           const Geo& g, double eps, void* lower_out, int lower_v, int lower_t,
                                           void* upper_out, int upper_v, cudaStream_t st) {
    using R = typename F::Real;
    F in{const_cast<void*>(uin), g.V}, out{uout, g.V};
    ForceField<R> zf{z, g.V}, hf{const_cast<void*>(hp), g.V};
    HaloTargets<F> h{F{lower_out, lower_v}, F{upper_out, upper_v}, g.site0, (g.site1 - g.site0) / g.site0, lower_t};
    const dim3 grid(unsigned((g.site1 - g.site0 + 31) / 32));
    const R e = R(stage == 0 ? eps * 0.25 : eps);
    switch (stage) {
        case 0: rk_split_stage_halo_kernel<F, 0><<<grid, 128, 0, st>>>(in, out, zf, hf, g, e, h); break;
        case 1: rk_split_stage_halo_kernel<F, 1><<<grid, 128, 0, st>>>(in, out, zf, hf, g, e, h); break;
        default: rk_split_stage_halo_kernel<F, 2><<<grid, 128, 0, st>>>(in, out, zf, hf, g, e, h); break;
    }
    return cudaGetLastError();
}

template <class F>
static cudaError_t launch_plaq_typed(const void* u, void* h, const Geo& g, bool chained, cudaStream_t st) {
    F in{const_cast<void*>(u), g.V};
    ForceField<typename F::Real> hf{h, g.V};
    const unsigned groups = unsigned((g.site1 - g.site0 + 31) / 32);
    return launch_chained(chained, plaq_field_kernel<F>, PlaqPlanesPerThread<F>::value == 1 ? groups : (groups + 1) / 2,
                          192, st, in, hf, g);
}

template <class F, class FO = F>
static cudaError_t launch_split_typed(int stage, const void* uin, void* uout, void* z, const void* h, const Geo& g,
                                      double eps, bool chained, cudaStream_t st) {
    using R = typename F::Real;
    const F in{const_cast<void*>(uin), g.V};
    const FO out{uout, g.V};
    ForceField<R> zf{z, g.V}, hf{const_cast<void*>(h), g.V};
    const unsigned grid = unsigned((g.site1 - g.site0 + 31) / 32);
    const R e = R(stage == 0 ? eps * 0.25 : eps);
    auto launch = [&](auto kernel) { return launch_chained(chained, kernel, grid, 128, st, in, out, zf, hf, g, e); };
    switch (stage) {
        case 0: return launch(rk_split_stage_kernel<F, 0, FO>);
        case 1: return launch(rk_split_stage_kernel<F, 1, FO>);
        default: return launch(rk_split_stage_kernel<F, 2, FO>);
    }
}

// The plaquette-field kernel of a measurement: the same field, and the sum of
// Re tr P over the sites [count0, count1) that are the context's own, one
// FP64 partial per warp (no barrier: a block's warps retire apart, as in
// plaq_field_kernel; one partial per block after a barrier ran 0.123 / 0.154 ms
// in FP32-12 / -18 at 32^4 on B200 against 0.112 / 0.123).  FP64 takes 96
// registers at three resident blocks: 0.255 ms, against 0.291 at
// plaq_field_kernel's 80.
template <class F>
__global__ void __launch_bounds__(192, sizeof(typename F::Real) == 8 ? 3 : PlaqMinBlocks<F>::value)
    plaq_field_sum_kernel(F u, ForceField<typename F::Real> hf, Geo g, int count0, int count1, double* partials) {
    using R = typename F::Real;
    constexpr int kPlanes = PlaqPlanesPerThread<F>::value;
    const int w = int(threadIdx.x >> 5);
    const int s = g.site0 + (int(blockIdx.x) * kPlanes + (kPlanes == 1 ? 0 : w / 3)) * 32 + int(threadIdx.x & 31);
    R t0 = R(0), t1 = R(0);
    bool counts = false;
    grid_wait();
    if (s < g.site1) {
        int c[4];
        g.coords(s, c);
        counts = s >= count0 && s < count1 && g.interior(c);
        if (kPlanes == 1) {
            hf.store(w, s, plane_generator<false>(u, g, s, c, plane_a(w), plane_b(w), &t0));
        } else {
            const int pr = w % 3;
            const int p0 = pr == 0 ? 0 : (pr == 1 ? 2 : 3);
            const int p1 = pr == 0 ? 1 : (pr == 1 ? 4 : 5);
            const auto h0 = plane_generator<false>(u, g, s, c, plane_a(p0), plane_b(p0), &t0);
            const auto h1 = plane_generator<false>(u, g, s, c, plane_a(p1), plane_b(p1), &t1);
            hf.store(p0, s, h0);
            hf.store(p1, s, h1);
        }
    }
    const double sum = warp_sum(counts ? double(t0) + double(t1) : 0.0);
    if ((threadIdx.x & 31) == 0) partials[int64_t(blockIdx.x) * 6 + w] = sum;
}

static int plaq_blocks(int prec, const Geo& g) {
    const int groups = (g.site1 - g.site0 + 31) / 32;
    return prec == kFP64 ? groups : (groups + 1) / 2;
}

int plaq_sum_partials(int prec, const Geo& g) { return 6 * plaq_blocks(prec, g); }

template <class F>
static cudaError_t launch_plaq_sum_typed(const void* u, void* h, const Geo& g, int count0, int count1,
                                         double* partials, bool chained, cudaStream_t st) {
    F in{const_cast<void*>(u), g.V};
    ForceField<typename F::Real> hf{h, g.V};
    return launch_chained(chained, plaq_field_sum_kernel<F>, unsigned(plaq_blocks(sizeof(typename F::Real) == 8 ? kFP64 : kFP32_18, g)), 192, st, in, hf, g, count0, count1, partials);
}

cudaError_t launch_plaq_field_sum(int prec, const void* u, void* h, const Geo& g, int count0, int count1,
                                  double* partials, cudaStream_t st, bool rows_in, bool chained) {
    if (g.site1 <= g.site0) return cudaErrorInvalidValue;
    switch (prec) {
        case kFP64:
            if (rows_in) return launch_plaq_sum_typed<FieldD18Rows>(u, h, g, count0, count1, partials, chained, st);
            return launch_plaq_sum_typed<FieldD18>(u, h, g, count0, count1, partials, chained, st);
        case kFP32_18: return launch_plaq_sum_typed<FieldF18>(u, h, g, count0, count1, partials, chained, st);
        case kFP32_12: return launch_plaq_sum_typed<FieldF12>(u, h, g, count0, count1, partials, chained, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_plaq_field(int prec, const void* u, void* h, const Geo& g, cudaStream_t st, bool rows_in,
                              bool chained) {
    if (small_lattice(g)) return cudaSuccess;  // its stage kernel forms its own plaquettes
    switch (prec) {
        case kFP64:
            if (rows_in) return launch_plaq_typed<FieldD18Rows>(u, h, g, chained, st);
            return launch_plaq_typed<FieldD18>(u, h, g, chained, st);
        case kFP32_18: return launch_plaq_typed<FieldF18>(u, h, g, chained, st);
        case kFP32_12: return launch_plaq_typed<FieldF12>(u, h, g, chained, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_rk_split_stage_halo(int prec, int stage, const void* uin, void* uout, void* z, const void* h,
                                       const Geo& g, double eps, void* lower_out, int lower_v, int lower_t,
                                       void* upper_out, int upper_v, cudaStream_t st) {
    if (g.site0 <= 0 || g.site0 % 32 || (g.site1 - g.site0) % g.site0) return cudaErrorInvalidValue;
    if (small_lattice(g))
        return launch_small_stage_halo(prec, stage, uin, uout, z, g, eps, lower_out, lower_v, lower_t, upper_out,
                                       upper_v, st);
    switch (prec) {
        case kFP64:
            return launch_split_halo_typed<FieldD18>(stage, uin, uout, z, h, g, eps, lower_out, lower_v, lower_t,
                                                     upper_out, upper_v, st);
        case kFP32_18:
            return launch_split_halo_typed<FieldF18>(stage, uin, uout, z, h, g, eps, lower_out, lower_v, lower_t,
                                                     upper_out, upper_v, st);
        case kFP32_12:
            return launch_split_halo_typed<FieldF12>(stage, uin, uout, z, h, g, eps, lower_out, lower_v, lower_t,
                                                     upper_out, upper_v, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_rk_split_stage(int prec, int stage, const void* uin, void* uout, void* z, const void* h,
                                  const Geo& g, double eps, cudaStream_t st, bool rows_in, bool rows_out, bool chained) {
    if (small_lattice(g)) return launch_small_stage(prec, stage, uin, uout, z, g, eps, chained, st);
    switch (prec) {
        case kFP64:
            if (rows_in && rows_out) return launch_split_typed<FieldD18Rows>(stage, uin, uout, z, h, g, eps, chained, st);
            if (rows_in) return launch_split_typed<FieldD18Rows, FieldD18>(stage, uin, uout, z, h, g, eps, chained, st);
            if (rows_out) return launch_split_typed<FieldD18, FieldD18Rows>(stage, uin, uout, z, h, g, eps, chained, st);
            return launch_split_typed<FieldD18>(stage, uin, uout, z, h, g, eps, chained, st);
        case kFP32_18: return launch_split_typed<FieldF18>(stage, uin, uout, z, h, g, eps, chained, st);
        case kFP32_12: return launch_split_typed<FieldF12>(stage, uin, uout, z, h, g, eps, chained, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ym
