// K2: plaquette, clover energy and clover topological charge
// (src/Observables/superobs.cpp:31-128), one thread per (site, plane), or from
// the two-kernel stage's plaquette field (launch_measure_from_field).
//
// Per plane (mu < nu) the four clover leaves, all oriented the same way,
//   Q1 = U_mu(x) U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+
//   Q2 = U_nu(x) U_mu(x-mu+nu)^+ U_nu(x-mu)^+ U_mu(x-mu)
//   Q3 = U_mu(x-mu)^+ U_nu(x-mu-nu)^+ U_mu(x-mu-nu) U_nu(x-nu)
//   Q4 = U_nu(x-nu)^+ U_mu(x-nu) U_nu(x+mu-nu) U_mu(x)^+
// give C = sum Q and G = [C - C^+]_traceless.  The reference adds Q1 and Q3 and
// subtracts Q4^+ and Q2^+ (superobs.cpp:47-74); after C - C^+ both sums give the
// same G.  Per site:
//   plaq   += Re tr Q1                        (:71, normalised by 18 V at :125)
//   energy += Re tr(G_{mu nu} G_{mu nu})      (:109, raw, no 1/8 factor)
//   topc   -= Re tr(G01 G23) + Re tr(G02 G13^+) + Re tr(G03 G12)   (:114-124, / 256 pi^2)
// Planes are visited in the pairs (01,23), (02,13), (03,12) so only two G are
// live at a time.  Site values are accumulated in FP64 whatever the link
// precision: warp shuffles, a shared-memory tree, one partial per block, and a
// single-block fold in a fixed order (deterministic, no atomics), in place of
// the reference's MPI_Allreduce (:24-28).
#include <algorithm>

#include "kernels.h"
#include "observables.cuh"

namespace ym {

// One block of 1024 threads per row: thread i folds partials i, i+1024, ... in
// order, then the block tree.  Output (plaq, topc, energy, nonfinite flag).
__global__ void __launch_bounds__(1024) obs_finalize_kernel(const double* partials, int nblocks, double inv_18v,
                                                            double* out) {
    grid_wait();
    partials += int64_t(blockIdx.x) * 3 * nblocks;
    out += 4 * blockIdx.x;
    double a = 0.0, b = 0.0, c = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < nblocks; i += blockDim.x) {
        a += partials[3 * i + 0];
        b += partials[3 * i + 1];
        c += partials[3 * i + 2];
    }
    block_sum3(a, b, c);
    if (threadIdx.x == 0) write_row(a, b, c, inv_18v, out);
}

int obs_blocks(const Geo& g) {
    const int groups = (g.site1 - g.site0 + kObsSites - 1) / kObsSites;
    return groups < kObsMaxBlocks ? groups : kObsMaxBlocks;
}

cudaError_t launch_observables(int prec, const void* u, const Geo& g, double* partials, cudaStream_t st) {
    const unsigned nb = unsigned(obs_blocks(g));
    if (nb == 0) return cudaErrorInvalidValue;
    auto launch = [&](auto f) {
        return launch_chained(false, observables_kernel<decltype(f)>, nb, kObsThreads, st, f, g, partials);
    };
    void* const links = const_cast<void*>(u);
    switch (prec) {
        case kFP64: return launch(FieldD18{links, g.V});
        case kFP32_18: return launch(FieldF18{links, g.V});
        case kFP32_12: return launch(FieldF12{links, g.V});
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_obs_finalize(const double* partials, int nblocks, const Geo& g, double* out, cudaStream_t st,
                                bool chained, int rows) {
    return launch_chained(chained, obs_finalize_kernel, unsigned(rows), 1024, st, partials, nblocks,
                          1.0 / (18.0 * double(g.vglobal)), out);
}

template <class F>
static cudaError_t launch_clover_typed(const void* u, const void* h, const Geo& g, int blocks, const double* plaq,
                                       int nplaq, double* partials, bool chained, cudaStream_t st) {
    const F in{const_cast<void*>(u), g.V};
    const ForceField<typename F::Real> hf{const_cast<void*>(h), g.V};
    return launch_chained(chained, clover_field_kernel<F>, unsigned(blocks), 96, st, in, hf, g, plaq, nplaq, partials);
}

static int clover_blocks(const Geo& g) { return std::min((g.site1 - g.site0 + 31) / 32, kCloverMaxBlocks); }

int measure_partials(int prec, const Geo& field, const Geo& own) {
    return plaq_sum_partials(prec, field) + kFoldRows * 3 * clover_blocks(own);
}

// Contexts on the two-kernel stage measure this way: the field is needed by
// the next stage 0 in any case, and even alone (one evaluation, field
// included) it is the faster form at every size from 16^3 x 32 up: FP64 24^3 x
// 48 0.55 -> 0.39 ms; below, both are a few launches long (8^4 FP64: 9.3 + 2.9
// us against 4.9 + 6.7 + 2.9, of which the next step saves the first).
cudaError_t launch_measure_from_field(int prec, const void* u, void* h, const Geo& field, const Geo& own,
                                      double* partials, int slot, cudaStream_t st, bool rows_in, bool chained) {
    const int np = plaq_sum_partials(prec, field), nc = clover_blocks(own);
    if (np < 1 || nc < 1 || slot < 0 || slot >= kFoldRows) return cudaErrorInvalidValue;
    const cudaError_t e =
        launch_plaq_field_sum(prec, u, h, field, own.site0, own.site1, partials, st, rows_in, chained);
    if (e != cudaSuccess) return e;
    double* const cp = partials + np + int64_t(slot) * 3 * nc;
    switch (prec) {
        case kFP64:
            if (rows_in) return launch_clover_typed<FieldD18Rows>(u, h, own, nc, partials, np, cp, chained, st);
            return launch_clover_typed<FieldD18>(u, h, own, nc, partials, np, cp, chained, st);
        case kFP32_18: return launch_clover_typed<FieldF18>(u, h, own, nc, partials, np, cp, chained, st);
        case kFP32_12: return launch_clover_typed<FieldF12>(u, h, own, nc, partials, np, cp, chained, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_fold_rows(int prec, const Geo& field, const Geo& own, const double* partials, int rows, double* out,
                             cudaStream_t st, bool chained) {
    if (rows < 1 || rows > kFoldRows) return cudaErrorInvalidValue;
    return launch_obs_finalize(partials + plaq_sum_partials(prec, field), clover_blocks(own), own, out, st, chained,
                               rows);
}

}  // namespace ym
