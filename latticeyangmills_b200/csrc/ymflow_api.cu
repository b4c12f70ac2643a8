// C ABI of libymflow (declared in include/ymflow.h): the flow context, its
// device buffers, the RK3 step sequence (optionally replayed as a CUDA graph)
// and the measurement schedule of the reference's WilsonFlow::applyWilsonFlow
// (src/Apps/wilsonflow.cpp:115-136).
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <map>
#include <mutex>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "context.h"

using namespace ym;


namespace ym {

int fail(ymflow_ctx* c, int code, const std::string& msg) {
    if (c) c->err = msg;
    return code;
}

int cuda_fail(ymflow_ctx* c, cudaError_t e, const char* what) {
    cudaGetLastError();  // reported here: the next call's launches do not find it again
    return fail(c, status_of(e), cuda_message(e, what));
}

}  // namespace ym

namespace {

thread_local std::string g_create_error;


int64_t link_count(const ymflow_ctx* c) { return 4 * c->geo.V; }

int dev_alloc(ymflow_ctx* c, void** p, size_t bytes, const char* what) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return cuda_fail(c, e, what);
    }
    c->bytes += int64_t(bytes);
    return YMFLOW_OK;
}

// .bin-layout device buffer of at least `bytes` (the whole field by default)
int ensure_staging(ymflow_ctx* c, size_t bytes = 0) {
    if (bytes == 0) bytes = size_t(link_count(c)) * 18 * sizeof(double);
    if (c->staging && c->staging_bytes >= bytes) return YMFLOW_OK;
    if (c->staging) {
        cudaFree(c->staging);
        c->bytes -= int64_t(c->staging_bytes);
        c->staging = nullptr;
        c->staging_bytes = 0;
    }
    const int r = dev_alloc(c, (void**)&c->staging, bytes, "staging buffer");
    if (r == YMFLOW_OK) c->staging_bytes = bytes;
    return r;
}

// Whether a measurement goes through the plaquette field: where the stages do.
bool measures_from_field(const ymflow_ctx* c) {
    return c->stage_form == 1 && c->hfield && !small_lattice(c->geo);
}

int ensure_partials(ymflow_ctx* c) {
    int n = small_lattice(c->geo) ? small_partials(c->geo) : 3 * obs_blocks(c->geo);
    if (measures_from_field(c)) n = std::max(n, measure_partials(c->prec, plaq_range(c->geo, c->slab), c->geo));
    if (n <= c->partial_cap) return YMFLOW_OK;
    if (c->partials) {
        cudaFree(c->partials);
        c->bytes -= int64_t(c->partial_cap) * sizeof(double);
        c->partials = nullptr;
        c->partial_cap = 0;
    }
    int r = dev_alloc(c, (void**)&c->partials, size_t(n) * sizeof(double), "observable partials");
    if (r != YMFLOW_OK) return r;
    YM_CK(c, cudaMemsetAsync(c->partials, 0, size_t(n) * sizeof(double), c->stream), "clear partials");
    c->partial_cap = n;
    return r;
}

}  // namespace

namespace ym {
void set_create_error(const std::string& msg) { g_create_error = msg; }
}  // namespace ym

namespace ym {

int ensure_meas(ymflow_ctx* c, int rows) {
    if (rows <= c->meas_cap) return YMFLOW_OK;
    if (c->meas) {
        cudaFree(c->meas);
        c->bytes -= int64_t(c->meas_cap) * 4 * sizeof(double);
        c->meas = nullptr;
    }
    if (c->meas_host) {
        cudaFreeHost(c->meas_host);
        c->meas_host = nullptr;
    }
    c->meas_cap = 0;
    int r = dev_alloc(c, (void**)&c->meas, size_t(rows) * 4 * sizeof(double), "measurement rows");
    if (r != YMFLOW_OK) return r;
    cudaError_t e = cudaMallocHost((void**)&c->meas_host, size_t(rows) * 4 * sizeof(double));
    if (e != cudaSuccess) return cuda_fail(c, e, "pinned measurement rows");
    c->meas_cap = rows;
    return YMFLOW_OK;
}

}  // namespace ym

namespace {

// The tiling of the shared-memory stage kernel used by default: among the
// (ty, tz) that tile the lattice into at least one unit per SM, the one with
// the least recomputed face work per site (ties: the smaller tile), two links
// per thread on the 64-register kernel.  false if
// none qualifies (small lattices, x extents whose lines do not fill whole
// warps, slabs).
bool default_tile(const ymflow_ctx* c, TileShape* out) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    bool found = false;
    double best = 0.0;
    for (int ty = 1; ty <= c->geo.n[1]; ty++) {
        for (int tz = 1; tz <= c->geo.n[2]; tz++) {
            TileShape tp;
            if (!make_tile_shape(c->prec, c->geo, ty, tz, &tp, true, 2, 1) || tp.units < sms) continue;
            const double cost = double(tp.nfy + tp.nfz) / tp.ns + 1e-6 * tp.ns;
            if (!found || cost < best) {
                if (tile_grid(c->prec, c->device, &tp) != cudaSuccess) {
                    cudaGetLastError();
                    continue;
                }
                *out = tp;
                best = cost;
                found = true;
            }
        }
    }
    return found;
}

// YMFLOW_OPT_TILE's value of a tiling
int64_t tile_option(const TileShape& tp) {
    return (int64_t(tp.lean) << 36) | (int64_t(tp.lpt) << 32) | (int64_t(tp.ty) << 16) | int64_t(tp.tz);
}

void drop_graphs(ymflow_ctx* c) {
    for (cudaGraphExec_t& g : c->graph) {
        if (g) cudaGraphExecDestroy(g);
        g = nullptr;
    }
}

// Whether the steps of a call pass links on as their rows 0 and 1: whole
// lattices on the two-kernel FP64 stage.
bool steps_by_rows(const ymflow_ctx* c) {
    return c->prec == YMFLOW_FP64 && c->stage_form == 1 && !c->slab && !c->is_block && !small_lattice(c->geo);
}

constexpr int kRowsIn = 1, kRowsOut = 2;

// The link buffers that the three stages of a step read and write.
struct StageBuffers {
    const void* in[3];
    void* out[3];
};

// A step from u[from] into the other buffer.
StageBuffers step_buffers(const ymflow_ctx* c, int from) {
    void* const a = c->u[from];
    void* const b = c->u[1 - from];
    return {{a, b, a}, {b, a, b}};
}

// The launches of one RK3 step over `io`: per stage the fused
// stage kernel, or the plaquette-field kernel and the stage kernel built on it
// (stage_form 1).  field_ready: the plaquette field already holds io.in[0]'s
// (stage 0 needs no field kernel).  rows (FP64, stage_form 1): bit 0, io.in[0]
// was written by a stage of the same call; bit 1, another step of the call
// follows: the links between a call's steps, and between its stages, are
// stored and read as their rows 0 and 1 (FieldD18Rows).  ev (optional): three events per stage, before the stage,
// after its plaquette-field kernel (at once for the fused form) and after it.
cudaError_t enqueue_step(ymflow_ctx* c, const StageBuffers& io, double eps, cudaEvent_t* ev, bool field_ready,
                         int rows) {
    const void* const* in = io.in;
    void* const* out = io.out;
    for (int s = 0; s < 3; s++) {
        if (ev) cudaEventRecord(ev[3 * s], c->stream);
        cudaError_t e = cudaSuccess;
        if (c->stage_form == 1) {
            const bool rows_in = s > 0 || (rows & kRowsIn), rows_out = s < 2 || (rows & kRowsOut);
            if (s > 0 || !field_ready)
                e = launch_plaq_field(c->prec, in[s], c->hfield, c->geo, c->stream, rows_in, true);
            if (e != cudaSuccess) return e;
            if (ev) cudaEventRecord(ev[3 * s + 1], c->stream);
            e = launch_rk_split_stage(c->prec, s, in[s], out[s], c->z, c->hfield, c->geo, eps, c->stream, rows_in,
                                      rows_out, true);
        } else if (c->stage_form == 2) {
            if (ev) cudaEventRecord(ev[3 * s + 1], c->stream);
            e = launch_rk_tile_stage(c->prec, s, in[s], out[s], c->z, c->geo, c->tile, eps, c->stream);
        } else {
            if (ev) cudaEventRecord(ev[3 * s + 1], c->stream);
            e = launch_rk_stage(c->prec, s, in[s], out[s], c->z, c->geo, eps, c->block, c->stream, true);
        }
        if (e != cudaSuccess) return e;
        if (ev) cudaEventRecord(ev[3 * s + 2], c->stream);
    }
    return cudaSuccess;
}

// One RK3 step of a slab: each stage's new links are followed by the halo
// exchange of that buffer, which the next stage reads.
int run_step_slab(ymflow_ctx* c, double eps, cudaEvent_t* ev, bool field_ready) {
    const int from = c->cur;
    const int in[3] = {from, 1 - from, from};
    for (int s = 0; s < 3; s++) {
        if (ev) cudaEventRecord(ev[3 * s], c->stream);
        if (c->stage_form == 1) {
            if (s > 0 || !field_ready)
                YM_CK(c, launch_plaq_field(c->prec, c->u[in[s]], c->hfield, plaq_range(c->geo, true), c->stream),
                      "plaquette-field launch");
            if (ev) cudaEventRecord(ev[3 * s + 1], c->stream);
            YM_CK(c, launch_rk_split_stage(c->prec, s, c->u[in[s]], c->u[1 - in[s]], c->z, c->hfield, c->geo, eps,
                                           c->stream),
                  "stage launch");
        } else {
            if (ev) cudaEventRecord(ev[3 * s + 1], c->stream);
            YM_CK(c, launch_rk_stage(c->prec, s, c->u[in[s]], c->u[1 - in[s]], c->z, c->geo, eps, c->block,
                                     c->stream),
                  "stage launch");
        }
        if (ev) cudaEventRecord(ev[3 * s + 2], c->stream);
        const int r = slab_exchange(c, 1 - in[s]);
        if (r != YMFLOW_OK) return r;
    }
    c->cur = 1 - from;
    return YMFLOW_OK;
}

// The step over `io` as an executable graph (stage form 2).
int capture_step(ymflow_ctx* c, const StageBuffers& io, double eps, cudaGraphExec_t* exec) {
    cudaGraph_t g = nullptr;
    YM_CK(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal), "begin step capture");
    cudaError_t le = enqueue_step(c, io, eps, nullptr, false, 0);
    cudaError_t ee = cudaStreamEndCapture(c->stream, &g);
    if (le != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        return cuda_fail(c, le, "stage launch during capture");
    }
    YM_CK(c, ee, "end step capture");
    cudaError_t ie = cudaGraphInstantiate(exec, g, 0);
    cudaGraphDestroy(g);
    YM_CK(c, ie, "instantiate step graph");
    return YMFLOW_OK;
}

// One RK3 step of the current field, step `s` of the `nsteps` (from 1) of a
// call.  field_ready: the plaquette field holds the current links' (a
// measurement has just been enqueued, and nothing has changed the links
// since).  Forms 0 and 1 launch their kernels chained (launch_chained), which
// is faster than a replayed graph at every size, most of all between a step and
// a measurement: us per step / per measured step on B200, graphs of unchained
// launches against chained launches of the same kernels, 12^4 FP64 41.9 / 60
// against 38.1 / 52, 16^4 FP32-12 57.5 / 78 against 53.9 / 71, 16^3 x 32
// FP32-12 102.9 / 133 against 97.5 / 124 (graphs of chained launches lie
// between); and a context's first steps build no graph.  The tile form's one
// kernel per stage is replayed.
int run_step(ymflow_ctx* c, double eps, int s, int nsteps, cudaEvent_t* ev, bool field_ready = false) {
    if (c->slab) return run_step_slab(c, eps, ev, field_ready);
    const int from = c->cur;
    if (c->use_graph && c->stage_form == 2 && !ev) {
        if (!c->graph[from] || c->graph_eps[from] != eps || c->graph_block[from] != c->block) {
            if (c->graph[from]) cudaGraphExecDestroy(c->graph[from]);
            c->graph[from] = nullptr;
            const int r = capture_step(c, step_buffers(c, from), eps, &c->graph[from]);
            if (r != YMFLOW_OK) return r;
            c->graph_eps[from] = eps;
            c->graph_block[from] = c->block;
        }
        YM_CK(c, cudaGraphLaunch(c->graph[from], c->stream), "launch step graph");
    } else {
        const int rows = steps_by_rows(c) ? (s > 1 ? kRowsIn : 0) | (s < nsteps ? kRowsOut : 0) : 0;
        YM_CK(c, enqueue_step(c, step_buffers(c, from), eps, ev, field_ready, rows), "stage launch");
    }
    c->cur = 1 - from;
    return YMFLOW_OK;
}

}  // namespace

namespace ym {

cudaError_t enqueue_stage(ymflow_ctx* c, int stage, const void* in, void* out, double eps) {
    if (c->stage_form == 1) {
        const cudaError_t e = launch_plaq_field(c->prec, in, c->hfield, c->geo, c->stream);
        if (e != cudaSuccess) return e;
        return launch_rk_split_stage(c->prec, stage, in, out, c->z, c->hfield, c->geo, eps, c->stream);
    }
    if (c->stage_form == 2) return launch_rk_tile_stage(c->prec, stage, in, out, c->z, c->geo, c->tile, eps, c->stream);
    return launch_rk_stage(c->prec, stage, in, out, c->z, c->geo, eps, c->block, c->stream);
}

// Folds the `n` rows up to `last` whose partials enqueue_measure has left.
static int fold_rows(ymflow_ctx* c, int last, int n) {
    if (n == 0) return YMFLOW_OK;
    const bool chained = !c->slab && !c->is_block;
    YM_CK(c, launch_fold_rows(c->prec, plaq_range(c->geo, c->slab), c->geo, c->partials, n,
                              c->meas + 4 * (last - n + 1), c->stream, chained),
          "observables fold");
    return YMFLOW_OK;
}

// Observables of the current field into meas row `row` (device).
int enqueue_measure(ymflow_ctx* c, int row, bool rows_in, int* pending) {
    int r = ensure_partials(c);
    if (r != YMFLOW_OK) return r;
    // Kernels of a whole lattice follow one another on its stream alone, so they
    // may be launched on each other's heels; slabs and blocks also wait for
    // their neighbours' streams.
    const bool chained = !c->slab && !c->is_block;
    if (small_lattice(c->geo)) {
        YM_CK(c, launch_small_observables(c->prec, c->u[c->cur], c->geo, c->partials, c->meas + 4 * row, chained,
                                          c->stream),
              "observables launch");
    } else if (measures_from_field(c)) {
        YM_CK(c, launch_measure_from_field(c->prec, c->u[c->cur], c->hfield, plaq_range(c->geo, c->slab), c->geo,
                                           c->partials, pending ? *pending : 0, c->stream, rows_in, chained),
              "observables launch");
        if (pending && ++*pending < kFoldRows) return YMFLOW_OK;
        if ((r = fold_rows(c, row, pending ? *pending : 1)) != YMFLOW_OK) return r;
        if (pending) *pending = 0;
    } else {
        YM_CK(c, launch_observables(c->prec, c->u[c->cur], c->geo, c->partials, c->stream), "observables launch");
        YM_CK(c, launch_obs_finalize(c->partials, obs_blocks(c->geo), c->geo, c->meas + 4 * row, c->stream),
              "observables fold");
    }
    if (c->slab && c->comm) return slab_reduce_row(c, c->meas + 4 * row);
    return YMFLOW_OK;
}


// Loads the kernels of a call's steps and measurements (LoadOnly): whole lattices
// in forms 0 and 1.  (Form 2's were loaded when the context was created.)
int load_flow_kernels(ymflow_ctx* c) {
    if (c->slab || c->is_block || c->stage_form == 2 || c->kernels_form == c->stage_form) return YMFLOW_OK;
    const bool by_rows = steps_by_rows(c);
    LoadOnly load;
    for (int rows : {kRowsOut, kRowsIn | kRowsOut, kRowsIn}) {  // a call's first step, those inside it, its last
        YM_CK(c, enqueue_step(c, step_buffers(c, c->cur), 0.0, nullptr, false, by_rows ? rows : 0), "stage kernels");
        if (!by_rows) break;
    }
    for (bool rows_in : {false, true}) {
        const int r = enqueue_measure(c, 0, rows_in && by_rows);
        if (r != YMFLOW_OK) return r;
    }
    c->kernels_form = c->stage_form;
    return YMFLOW_OK;
}

void fill_obs(const ymflow_ctx* c, const double* m, int64_t step, double t, ymflow_obs* o) {
    o->step = int32_t(step);
    o->pad = 0;
    o->t = t;
    o->plaq = m[0];
    o->topc = m[1];
    o->energy = m[2];
    o->t2E = -t * t * m[2] / (64.0 * double(c->geo.vglobal));
}

// A slab measures and flows only once connected; its halos are refreshed from
// the neighbours first (the field may have been uploaded or initialised since).
int slab_prepare(ymflow_ctx* c) {
    if (c->is_block)
        return fail(c, YMFLOW_ERR_STATE, "block context: flow and measure its group with ymflow_block_group_flow");
    if (!c->slab) return YMFLOW_OK;
    if (!c->comm)
        return fail(c, YMFLOW_ERR_STATE,
                    "slab context not connected: call ymflow_slab_connect, or flow its group with "
                    "ymflow_slab_group_flow");
    return slab_exchange(c, c->cur);
}

}  // namespace ym

extern "C" {

const char* ymflow_version(void) { return "ymflow 0.1 (sm_100a)"; }

int ymflow_device_count(int* count) {
    if (!count) return YMFLOW_ERR_ARG;
    *count = 0;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return YMFLOW_OK;
    }
    int k = 0;
    for (int d = 0; d < n; d++) {
        int major = 0;
        if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, d) == cudaSuccess && major == 10) k++;
    }
    *count = k;
    return YMFLOW_OK;
}

}  // extern "C"

namespace ym {

ymflow_ctx* create_context(const int dims[4], int64_t config_sites, int precision, int device, int* status) {
    auto set = [&](int s, const std::string& m) {
        if (status) *status = s;
        g_create_error = m;
    };
    if (!dims) {
        set(YMFLOW_ERR_ARG, "dims is NULL");
        return nullptr;
    }
    int64_t V = 1;
    for (int i = 0; i < 4; i++) {
        if (dims[i] < 1 || dims[i] > 4096) {
            set(YMFLOW_ERR_ARG, "lattice extents must be in 1..4096");
            return nullptr;
        }
        V *= dims[i];
    }
    if (precision < YMFLOW_FP64 || precision > YMFLOW_FP32_12) {
        set(YMFLOW_ERR_ARG, "unknown precision");
        return nullptr;
    }
    if (V >= (int64_t(1) << 31) || !volume_addressable(precision, V)) {
        set(YMFLOW_ERR_ARG, "lattice volume too large (4 V link bytes must stay below 64 GiB)");
        return nullptr;
    }
    std::string why;
    if (!device_usable(device, &why)) {
        set(YMFLOW_ERR_NODEVICE, why);
        return nullptr;
    }
    ymflow_ctx* c = new (std::nothrow) ymflow_ctx();
    if (!c) {
        set(YMFLOW_ERR_OOM, "host allocation failed");
        return nullptr;
    }
    DeviceGuard guard(device);
    c->device = device;
    c->prec = precision;
    for (int i = 0; i < 4; i++) c->dims[i] = dims[i];
    c->geo = make_geo(dims);
    // FP64 re-reads time-neighbour links from DRAM (traffic 1.3x the compulsory
    // bytes); a tiled block order keeps them in L2: 3 % faster at 32^4.  Only
    // the FP64 stage kernels use it: the FP32 forms' working set already fits
    // L2, and they lose 3 % with it.
    set_tiled_order(c->geo, 512);
    int r = YMFLOW_OK;
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) r = YMFLOW_ERR_CUDA;
    const size_t ub = link_field_bytes(c->prec, V);
    const size_t zb = force_field_bytes(c->prec, V);
    if (r == YMFLOW_OK) r = dev_alloc(c, &c->u[0], ub, "link buffer 0");
    if (r == YMFLOW_OK) r = dev_alloc(c, &c->u[1], ub, "link buffer 1");
    if (r == YMFLOW_OK) r = dev_alloc(c, &c->z, zb, "force buffer");
    if (r == YMFLOW_OK) r = dev_alloc(c, (void**)&c->deviation, sizeof(unsigned long long), "drift flag");
    // Every precision flows with the plaquette-field form of the force (fewer
    // multiply-adds per link than the staple form) as two kernels through a
    // stored plaquette field: at 32^4 on B200 0.77 against 1.16 ms per step
    // (FP32-12) and 1.73 against 2.05 (FP64).  Where the FP64 plaquette field
    // (384 bytes per site) does not fit beside the links, FP64 keeps the fused
    // staple kernel.  FP32 configurations of at most 8192 sites, whose steps are
    // bound by their launches, keep the one-launch fused kernel; by the whole
    // configuration's volume, so that its slabs and blocks, however cut, take
    // the same form as one another and as the whole lattice.  (us per step with
    // one launch per stage / two, FP32-12: 8^3 x 12 16.7 / 17.5, 7 x 9 x 8 x 13 17.3 /
    // 18.3, 10^4 21.0 / 19.9; FP32-18: 18.6 / 18.6, 19.2 / 19.7, 22.9 / 20.9.  The
    // line is drawn for steps without a measurement: measured every step the
    // two kernels, whose field the measurement shares, are ahead below it too,
    // 29.3 / 22.9 and 30.7 / 24.1 at 8^3 x 12.  Up to kSmallSites forms 0 and 1 are
    // flow_small.cu's.)  The one-kernel form with a tile's plane generators in
    // shared memory is prepared (its default tiling) for
    // YMFLOW_OPT_STAGE_FORM 2 and the autotuner, which times every form.
    if (r == YMFLOW_OK && prepare_tile_kernels(c->prec) != cudaSuccess) {
        const cudaError_t e = cudaGetLastError();
        r = cuda_fail(c, e == cudaSuccess ? cudaErrorInvalidValue : e, "tile kernel set-up");
    }
    if (r == YMFLOW_OK) c->tile_ok = default_tile(c, &c->tile);
    const bool launch_bound = c->prec != YMFLOW_FP64 && (config_sites > 0 ? config_sites : V) <= 8192;
    if (r == YMFLOW_OK && !launch_bound) {
        r = dev_alloc(c, &c->hfield, plane_field_bytes(c->prec, V), "plaquette field");
        if (r == YMFLOW_OK) {
            c->stage_form = 1;
        } else if (c->prec == YMFLOW_FP64 && r == YMFLOW_ERR_OOM) {
            r = YMFLOW_OK;
            c->err.clear();
        }
    }
    if (r == YMFLOW_OK) r = ensure_partials(c);
    if (r == YMFLOW_OK) r = ensure_meas(c, 16);
    if (r == YMFLOW_OK && (cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess))
        r = YMFLOW_ERR_CUDA;
    if (r != YMFLOW_OK) {
        set(r, c->err.empty() ? "context setup failed" : c->err);
        ymflow_destroy(c);
        return nullptr;
    }
    if (status) *status = YMFLOW_OK;
    return c;
}

}  // namespace ym

extern "C" {

ymflow_ctx* ymflow_create(const int dims[4], int precision, int device, int* status) {
    return create_context(dims, 0, precision, device, status);
}

ymflow_ctx* ymflow_create_slab(const int global_dims[4], int t0, int nt, int precision, int device, int* status) {
    auto set = [&](int s, const std::string& m) {
        if (status) *status = s;
        g_create_error = m;
    };
    if (!global_dims) {
        set(YMFLOW_ERR_ARG, "global_dims is NULL");
        return nullptr;
    }
    for (int i = 0; i < 4; i++)
        if (global_dims[i] < 1 || global_dims[i] > 4096) {
            set(YMFLOW_ERR_ARG, "lattice extents must be in 1..4096");
            return nullptr;
        }
    if (nt < 1 || t0 < 0 || int64_t(t0) + nt > global_dims[3] || nt + 2 > 4096) {
        set(YMFLOW_ERR_ARG, "slab slices [t0, t0 + nt) outside the lattice's time extent");
        return nullptr;
    }
    const int64_t vs = int64_t(global_dims[0]) * global_dims[1] * global_dims[2];
    if (vs % 32 != 0) {
        set(YMFLOW_ERR_ARG, "a slab needs a spatial volume (x y z) divisible by 32");
        return nullptr;
    }
    if (vs * global_dims[3] >= (int64_t(1) << 31)) {
        set(YMFLOW_ERR_ARG, "lattice volume must be below 2^31 sites");
        return nullptr;
    }
    const int local[4] = {global_dims[0], global_dims[1], global_dims[2], nt + 2};
    ymflow_ctx* c = create_context(local, vs * global_dims[3], precision, device, status);
    if (!c) return nullptr;
    c->slab = true;
    c->geo.tile_groups = 0;  // the interior range starts at a halo slice: plain order
    c->t0 = t0;
    c->nt = nt;
    for (int i = 0; i < 4; i++) c->gdims[i] = global_dims[i];
    c->geo.site0 = int(vs);
    c->geo.site1 = int(vs * (nt + 1));
    c->geo.global0 = int64_t(t0) * vs;
    c->geo.vglobal = vs * global_dims[3];
    c->use_graph = false;
    // slabs flow with the two-kernel stage (or the fused kernel where its
    // plaquette field did not fit): the tile kernel covers whole-lattice
    // contexts only
    c->tile_ok = false;
    if (c->stage_form == 2) {
        DeviceGuard guard(device);
        const int r = dev_alloc(c, &c->hfield, plane_field_bytes(c->prec, c->geo.V), "plaquette field");
        if (r != YMFLOW_OK) {
            if (status) *status = r;
            g_create_error = c->err;
            ymflow_destroy(c);
            return nullptr;
        }
        c->stage_form = 1;
    }
    return c;
}

void ymflow_destroy(ymflow_ctx* c) {
    if (!c) return;
    DeviceGuard guard(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    slab_release(c);
    drop_graphs(c);
    for (void* p : {c->u[0], c->u[1], c->z, c->hfield, (void*)c->staging, (void*)c->partials, (void*)c->meas,
                    (void*)c->deviation})
        if (p) cudaFree(p);
    if (c->meas_host) cudaFreeHost(c->meas_host);
    for (cudaEvent_t e : c->events) cudaEventDestroy(e);
    if (c->ev0) cudaEventDestroy(c->ev0);
    if (c->ev1) cudaEventDestroy(c->ev1);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
}

const char* ymflow_last_error(const ymflow_ctx* c) {
    if (!c) return g_create_error.c_str();
    return c->err.c_str();
}

int ymflow_upload(ymflow_ctx* c, const double* links) {
    if (!c || !links) return fail(c, YMFLOW_ERR_ARG, "null argument to ymflow_upload");
    if (c->is_block)
        return ymflow_upload_sites(c, links, 0,
                                   int64_t(c->geo.bext[0]) * c->geo.bext[1] * c->geo.bext[2] * c->geo.bext[3], 0);
    return ymflow_upload_sites(c, links, 0, int64_t(c->geo.site1 - c->geo.site0), 0);
}

int ymflow_download(ymflow_ctx* c, double* links) {
    if (!c || !links) return fail(c, YMFLOW_ERR_ARG, "null argument to ymflow_download");
    if (c->is_block)
        return ymflow_download_sites(c, links, 0,
                                     int64_t(c->geo.bext[0]) * c->geo.bext[1] * c->geo.bext[2] * c->geo.bext[3], 0);
    return ymflow_download_sites(c, links, 0, int64_t(c->geo.site1 - c->geo.site0), 0);
}

namespace {

int check_site_range(ymflow_ctx* c, const void* p, int64_t first, int64_t n, int flags) {
    if (!c) return YMFLOW_ERR_ARG;
    if (!p && n > 0) return fail(c, YMFLOW_ERR_ARG, "null links pointer");
    const int64_t own = c->is_block ? int64_t(c->geo.bext[0]) * c->geo.bext[1] * c->geo.bext[2] * c->geo.bext[3]
                                 : int64_t(c->geo.site1 - c->geo.site0);
    if (first < 0 || n < 0 || first + n > own)
        return fail(c, YMFLOW_ERR_ARG, "site range outside the lattice (or the slab / block)");
    if (flags & ~YMFLOW_IO_BIG_ENDIAN) return fail(c, YMFLOW_ERR_ARG, "unknown flags");
    return YMFLOW_OK;
}

}  // namespace

int ymflow_load_file(ymflow_ctx* c, const char* path, int flags, int64_t chunk_sites) {
    NvtxRange range("ymflow_load_file");
    if (!c || !path) return YMFLOW_ERR_ARG;
    if (flags & ~YMFLOW_IO_BIG_ENDIAN) return fail(c, YMFLOW_ERR_ARG, "unknown flags");
    if (c->is_block)
        return fail(c, YMFLOW_ERR_STATE, "a block's sites are not one run of the file: upload them (ymflow_upload)");
    const int64_t n = c->geo.site1 - c->geo.site0;  // this context's sites
    const int64_t site_bytes = 4 * 18 * int64_t(sizeof(double));
    const int64_t chunk = std::min<int64_t>(chunk_sites > 0 ? chunk_sites : 65536, n);
    FILE* f = std::fopen(path, "rb");
    if (!f) return fail(c, YMFLOW_ERR_ARG, std::string("cannot open ") + path);
    std::fseek(f, 0, SEEK_END);
    const int64_t file_bytes = std::ftell(f);
    if (file_bytes != c->geo.vglobal * site_bytes) {
        std::fclose(f);
        return fail(c, YMFLOW_ERR_ARG, std::string(path) + ": " + std::to_string(file_bytes) + " bytes, expected " +
                                           std::to_string(c->geo.vglobal * site_bytes));
    }
    std::fseek(f, long(c->geo.global0 * site_bytes), SEEK_SET);  // a slab's part starts at its first site
    DeviceGuard guard(c->device);
    int r = ensure_staging(c, size_t(2 * chunk * site_bytes));
    double* pinned[2] = {nullptr, nullptr};
    cudaEvent_t done[2] = {nullptr, nullptr};
    auto cleanup = [&]() {
        for (int i = 0; i < 2; i++) {
            if (done[i]) cudaEventDestroy(done[i]);
            if (pinned[i]) cudaFreeHost(pinned[i]);
        }
        std::fclose(f);
    };
    for (int i = 0; i < 2 && r == YMFLOW_OK; i++) {
        cudaError_t e = cudaMallocHost((void**)&pinned[i], size_t(chunk * site_bytes));
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming);
        if (e != cudaSuccess) r = cuda_fail(c, e, "pinned read buffers");
    }
    // Double buffering: the host reads chunk k+1 from the file while the device
    // copies and packs chunk k; a buffer is refilled once its copy has completed.
    for (int64_t first = 0, k = 0; first < n && r == YMFLOW_OK; first += chunk, k++) {
        const int b = int(k & 1);
        const int64_t m = std::min(chunk, n - first);
        cudaError_t e = cudaEventSynchronize(done[b]);
        if (e != cudaSuccess) {
            r = cuda_fail(c, e, "read buffer wait");
            break;
        }
        if (std::fread(pinned[b], size_t(site_bytes), size_t(m), f) != size_t(m)) {
            r = fail(c, YMFLOW_ERR_ARG, std::string(path) + ": short read");
            break;
        }
        double* dst = c->staging + size_t(b) * size_t(chunk) * 72;
        e = cudaMemcpyAsync(dst, pinned[b], size_t(m * site_bytes), cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess) e = cudaEventRecord(done[b], c->stream);
        if (e == cudaSuccess)
            e = launch_pack_range(c->prec, dst, c->u[c->cur], c->geo, c->geo.site0 + int(first), int(m),
                                  (flags & YMFLOW_IO_BIG_ENDIAN) != 0, c->stream);
        if (e != cudaSuccess) r = cuda_fail(c, e, "load copy");
    }
    if (r == YMFLOW_OK) {
        const cudaError_t e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) r = cuda_fail(c, e, "load");
    }
    cleanup();
    if (r != YMFLOW_OK) return r;
    c->loaded = true;
    c->step = 0;
    c->t = 0.0;
    return YMFLOW_OK;
}

int ymflow_upload_sites(ymflow_ctx* c, const double* links, int64_t first_site, int64_t nsites, int flags) {
    NvtxRange range("ymflow_upload_sites");
    int r = check_site_range(c, links, first_site, nsites, flags);
    if (r != YMFLOW_OK || nsites == 0) return r;
    DeviceGuard guard(c->device);
    const size_t bytes = size_t(nsites) * 4 * 18 * sizeof(double);
    r = ensure_staging(c, bytes);
    if (r != YMFLOW_OK) return r;
    YM_CK(c, transfer_upload(c->device, c->staging, links, bytes, c->stream), "upload copy");
    YM_CK(c, launch_pack_range(c->prec, c->staging, c->u[c->cur], c->geo, c->geo.site0 + int(first_site), int(nsites),
                               (flags & YMFLOW_IO_BIG_ENDIAN) != 0, c->stream),
          "pack launch");
    YM_CK(c, cudaStreamSynchronize(c->stream), "upload");
    c->loaded = true;
    c->step = 0;
    c->t = 0.0;
    return YMFLOW_OK;
}

int ymflow_download_sites(ymflow_ctx* c, double* links, int64_t first_site, int64_t nsites, int flags) {
    NvtxRange range("ymflow_download_sites");
    int r = check_site_range(c, links, first_site, nsites, flags);
    if (r != YMFLOW_OK) return r;
    if (!c->loaded) return fail(c, YMFLOW_ERR_STATE, "no links loaded");
    if (nsites == 0) return YMFLOW_OK;
    DeviceGuard guard(c->device);
    const size_t bytes = size_t(nsites) * 4 * 18 * sizeof(double);
    r = ensure_staging(c, bytes);
    if (r != YMFLOW_OK) return r;
    YM_CK(c, launch_unpack_range(c->prec, c->u[c->cur], c->staging, c->geo, c->geo.site0 + int(first_site),
                                 int(nsites),
                                 (flags & YMFLOW_IO_BIG_ENDIAN) != 0, c->stream),
          "unpack launch");
    YM_CK(c, transfer_download(c->device, links, c->staging, bytes, c->stream), "download copy");
    YM_CK(c, cudaStreamSynchronize(c->stream), "download");
    return YMFLOW_OK;
}

int ymflow_init_links(ymflow_ctx* c, int kind, double a, uint64_t seed, uint32_t config, double haar_frac) {
    if (!c) return YMFLOW_ERR_ARG;
    if (kind != YMFLOW_FIELD_COLD && kind != YMFLOW_FIELD_EXPIAH) return fail(c, YMFLOW_ERR_ARG, "unknown field kind");
    if (!(haar_frac >= 0.0 && haar_frac <= 1.0)) return fail(c, YMFLOW_ERR_ARG, "haar_frac outside [0, 1]");
    if (c->is_block) return fail(c, YMFLOW_ERR_STATE, "seeded fields fill whole lattices and slabs; upload a block's part");
    DeviceGuard guard(c->device);
    YM_CK(c, launch_init_links(c->prec, c->u[c->cur], c->geo, kind == YMFLOW_FIELD_COLD ? kCold : kExpIAH, a, seed,
                               config, c->stream),
          "init launch");
    if (haar_frac > 0.0)
        YM_CK(c, launch_haar_mix(c->prec, c->u[c->cur], c->geo, haar_frac, seed, config, c->stream), "haar launch");
    YM_CK(c, cudaStreamSynchronize(c->stream), "init links");
    c->loaded = true;
    c->step = 0;
    c->t = 0.0;
    return YMFLOW_OK;
}

int ymflow_generate_metropolis(ymflow_ctx* c, int start, double beta, double su3eps, int sweeps, int hits,
                               uint64_t seed, double* acceptance) {
    NvtxRange range("ymflow_generate_metropolis");
    if (!c) return YMFLOW_ERR_ARG;
    if (c->slab || c->is_block)
        return fail(c, YMFLOW_ERR_STATE, "generation runs on a whole-lattice context, not a slab or block");
    if (sweeps < 0 || hits < 1 || !(su3eps > 0.0 && su3eps < 1.0) || !std::isfinite(beta))
        return fail(c, YMFLOW_ERR_ARG, "need sweeps >= 0, hits >= 1, 0 < su3eps < 1, finite beta");
    if (start != YMFLOW_FIELD_COLD && start != YMFLOW_FIELD_HOT && start != YMFLOW_FIELD_CURRENT)
        return fail(c, YMFLOW_ERR_ARG, "start must be COLD, HOT or CURRENT");
    for (int i = 0; i < 4; i++)  // with an odd extent the periodic wrap joins two sites of one parity
        if (c->dims[i] % 2) return fail(c, YMFLOW_ERR_ARG, "the checkerboard update needs even extents");
    if (start == YMFLOW_FIELD_CURRENT && !c->loaded) return fail(c, YMFLOW_ERR_STATE, "no links loaded");
    DeviceGuard guard(c->device);
    if (start != YMFLOW_FIELD_CURRENT) {
        YM_CK(c, launch_init_links(c->prec, c->u[c->cur], c->geo, kCold, 0.0, seed, 0, c->stream), "cold start");
        if (start == YMFLOW_FIELD_HOT)
            YM_CK(c, launch_haar_mix(c->prec, c->u[c->cur], c->geo, 1.0, seed, 0, c->stream), "hot start");
        c->gen_sweep = 0;
    }
    YM_CK(c, cudaMemsetAsync(c->deviation, 0, sizeof(unsigned long long), c->stream), "reset counter");
    for (int sw = 0; sw < sweeps; sw++) {
        for (int mu = 0; mu < 4; mu++)
            for (int parity = 0; parity < 2; parity++)
                YM_CK(c, launch_metropolis(c->prec, c->u[c->cur], c->geo, mu, parity, beta, su3eps, hits, seed,
                                           c->gen_sweep + uint32_t(sw), c->deviation, c->stream),
                      "metropolis sweep");
        if (c->prec != YMFLOW_FP64)
            YM_CK(c, launch_reunitarize(c->prec, c->u[c->cur], c->geo, nullptr, c->stream), "reunitarise");
    }
    c->gen_sweep += uint32_t(sweeps);
    unsigned long long acc = 0;
    YM_CK(c, cudaMemcpyAsync(&acc, c->deviation, sizeof(acc), cudaMemcpyDeviceToHost, c->stream), "counter copy");
    YM_CK(c, cudaStreamSynchronize(c->stream), "generate");
    if (acceptance) {
        const double tries = double(sweeps) * double(hits) * 4.0 * double(c->geo.V);
        *acceptance = tries > 0 ? double(acc) / tries : 0.0;
    }
    c->loaded = true;
    c->step = 0;
    c->t = 0.0;
    return YMFLOW_OK;
}

int ymflow_observables(ymflow_ctx* c, ymflow_obs* out) {
    NvtxRange range("ymflow_observables");
    if (!c || !out) return fail(c, YMFLOW_ERR_ARG, "null argument to ymflow_observables");
    if (!c->loaded) return fail(c, YMFLOW_ERR_STATE, "no links loaded");
    DeviceGuard guard(c->device);
    int r = slab_prepare(c);
    if (r != YMFLOW_OK) return r;
    r = enqueue_measure(c, 0);
    if (r != YMFLOW_OK) return r;
    YM_CK(c, cudaMemcpyAsync(c->meas_host, c->meas, 4 * sizeof(double), cudaMemcpyDeviceToHost, c->stream),
          "observables copy");
    YM_CK(c, cudaStreamSynchronize(c->stream), "observables");
    fill_obs(c, c->meas_host, c->step, c->t, out);
    if (c->meas_host[3] != 0.0) return fail(c, YMFLOW_ERR_NONFINITE, "non-finite observable");
    return YMFLOW_OK;
}

int ymflow_flow(ymflow_ctx* c, double eps, int nsteps, int measure_every, int reunit_every, ymflow_obs* out,
                int out_cap, int* n_out) {
    NvtxRange range("ymflow_flow");
    if (!c) return YMFLOW_ERR_ARG;
    if (n_out) *n_out = 0;
    if (nsteps < 0 || !std::isfinite(eps)) return fail(c, YMFLOW_ERR_ARG, "nsteps < 0 or eps not finite");
    if (!c->loaded) return fail(c, YMFLOW_ERR_STATE, "no links loaded");
    int rows = 1;
    for (int s = 1; s <= nsteps; s++)
        if ((measure_every > 0 && s % measure_every == 0) || s == nsteps) rows++;
    if (out && out_cap < rows) return fail(c, YMFLOW_ERR_CAPACITY, "output holds " + std::to_string(out_cap) +
                                                                       " rows, flow needs " + std::to_string(rows));
    DeviceGuard guard(c->device);
    int r = ensure_meas(c, rows);
    if (r != YMFLOW_OK) return r;
    std::vector<int64_t> row_step(rows);
    std::vector<double> row_t(rows);
    if ((r = load_flow_kernels(c)) != YMFLOW_OK) return r;
    const bool reunit = c->prec != YMFLOW_FP64 && reunit_every > 0;
    if (reunit) YM_CK(c, cudaMemsetAsync(c->deviation, 0, sizeof(unsigned long long), c->stream), "reset drift");
    if ((r = slab_prepare(c)) != YMFLOW_OK) return r;
    int row = 0;
    int unfolded = 0;
    int* const pending = c->slab || c->is_block ? nullptr : &unfolded;  // a slab's or block's row is summed over its group
    if ((r = enqueue_measure(c, row, false, pending)) != YMFLOW_OK) return r;
    row_step[row] = c->step;
    row_t[row] = c->t;
    row++;
    const bool from_field = measures_from_field(c);
    const bool by_rows = steps_by_rows(c);
    bool field_ready = from_field;  // a measured row leaves its plaquette field for the next step's stage 0
    for (int s = 1; s <= nsteps; s++) {
        if ((r = run_step(c, eps, s, nsteps, nullptr, field_ready)) != YMFLOW_OK) return r;
        field_ready = false;
        c->step++;
        c->t += eps;
        if (reunit && s % reunit_every == 0)
            YM_CK(c, launch_reunitarize(c->prec, c->u[c->cur], c->geo, c->deviation, c->stream), "reunitarise");
        if ((measure_every > 0 && s % measure_every == 0) || s == nsteps) {
            if ((r = enqueue_measure(c, row, by_rows, pending)) != YMFLOW_OK) return r;
            row_step[row] = c->step;
            row_t[row] = c->t;
            row++;
            field_ready = from_field;
        }
    }
    if ((r = fold_rows(c, row - 1, unfolded)) != YMFLOW_OK) return r;
    YM_CK(c, cudaMemcpyAsync(c->meas_host, c->meas, size_t(rows) * 4 * sizeof(double), cudaMemcpyDeviceToHost,
                             c->stream),
          "measurement copy");
    unsigned long long dev_bits = 0;
    if (reunit)
        YM_CK(c, cudaMemcpyAsync(&dev_bits, c->deviation, sizeof(dev_bits), cudaMemcpyDeviceToHost, c->stream),
              "drift copy");
    YM_CK(c, cudaStreamSynchronize(c->stream), "flow");
    bool nonfinite = false;
    for (int i = 0; i < rows; i++) {
        if (out) fill_obs(c, c->meas_host + 4 * i, row_step[i], row_t[i], out + i);
        if (c->meas_host[4 * i + 3] != 0.0) nonfinite = true;
    }
    if (n_out) *n_out = rows;
    if (nonfinite) return fail(c, YMFLOW_ERR_NONFINITE, "non-finite observable during the flow");
    if (reunit) {
        double d;
        std::memcpy(&d, &dev_bits, sizeof(d));
        if (d > 1e-3) return fail(c, YMFLOW_ERR_UNITARITY, "links drifted from SU(3): |row norm - 1| = " +
                                                                std::to_string(d));
    }
    return YMFLOW_OK;
}

int ymflow_derivative(ymflow_ctx* c, int mu, double* z_host) {
    if (!c || !z_host || mu < 0 || mu > 3) return fail(c, YMFLOW_ERR_ARG, "bad argument to ymflow_derivative");
    if (!c->loaded) return fail(c, YMFLOW_ERR_STATE, "no links loaded");
    if (c->slab || c->is_block)
        return fail(c, YMFLOW_ERR_STATE, "ymflow_derivative runs on a whole-lattice context, not a slab or block");
    DeviceGuard guard(c->device);
    int r = ensure_staging(c);
    if (r != YMFLOW_OK) return r;
    YM_CK(c, launch_force(c->prec, mu, c->u[c->cur], c->geo, c->staging, c->stream), "force launch");
    YM_CK(c, transfer_download(c->device, z_host, c->staging, size_t(c->geo.V) * 18 * sizeof(double), c->stream),
          "force copy");
    YM_CK(c, cudaStreamSynchronize(c->stream), "derivative");
    return YMFLOW_OK;
}

int ymflow_su3_exp(const double* q_host, double* r_host, int64_t n, int device) {
    if (!q_host || !r_host || n < 0) return YMFLOW_ERR_ARG;
    if (n == 0) return YMFLOW_OK;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return YMFLOW_ERR_NODEVICE;
    }
    DeviceGuard guard(device);
    double* d = nullptr;
    const size_t bytes = size_t(n) * 18 * sizeof(double);
    if (cudaMalloc(&d, 2 * bytes) != cudaSuccess) {
        cudaGetLastError();
        return YMFLOW_ERR_OOM;
    }
    cudaError_t e = cudaMemcpy(d, q_host, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = launch_exp(d, d + size_t(n) * 18, n, nullptr);
    if (e == cudaSuccess) e = cudaMemcpy(r_host, d + size_t(n) * 18, bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? YMFLOW_OK : YMFLOW_ERR_CUDA;
}

int ymflow_reset_time(ymflow_ctx* c) {
    if (!c) return YMFLOW_ERR_ARG;
    c->step = 0;
    c->t = 0.0;
    return YMFLOW_OK;
}

int ymflow_set_time(ymflow_ctx* c, int64_t step, double t) {
    if (!c) return YMFLOW_ERR_ARG;
    if (step < 0 || !std::isfinite(t)) return fail(c, YMFLOW_ERR_ARG, "step < 0 or t not finite");
    c->step = step;
    c->t = t;
    return YMFLOW_OK;
}

int ymflow_time_kernels(ymflow_ctx* c, double eps, int nsteps, float* elapsed_ms, float* field_ms, float* stage_ms) {
    NvtxRange range("ymflow_time_kernels");
    if (!c || !elapsed_ms || nsteps < 1) return fail(c, YMFLOW_ERR_ARG, "bad argument to ymflow_time_kernels");
    if (!c->loaded) return fail(c, YMFLOW_ERR_STATE, "no links loaded");
    DeviceGuard guard(c->device);
    if (int r = slab_prepare(c)) return r;
    if (int r = load_flow_kernels(c)) return r;
    const bool per_kernel = field_ms || stage_ms;
    const size_t nev = per_kernel ? size_t(9) * nsteps : 0;
    while (c->events.size() < nev) {
        cudaEvent_t e;
        YM_CK(c, cudaEventCreate(&e), "event create");
        c->events.push_back(e);
    }
    const bool reunit = c->prec != YMFLOW_FP64 && c->timed_reunit > 0;
    YM_CK(c, cudaEventRecord(c->ev0, c->stream), "event record");
    for (int s = 0; s < nsteps; s++) {
        int r = run_step(c, eps, s + 1, nsteps, per_kernel ? c->events.data() + 9 * s : nullptr);
        if (r != YMFLOW_OK) return r;
        c->step++;
        c->t += eps;
        if (reunit && (s + 1) % c->timed_reunit == 0)
            YM_CK(c, launch_reunitarize(c->prec, c->u[c->cur], c->geo, c->deviation, c->stream), "reunitarise");
    }
    YM_CK(c, cudaEventRecord(c->ev1, c->stream), "event record");
    YM_CK(c, cudaEventSynchronize(c->ev1), "timed steps");
    YM_CK(c, cudaEventElapsedTime(elapsed_ms, c->ev0, c->ev1), "elapsed time");
    if (per_kernel) {
        double field = 0.0, stage = 0.0;
        for (int i = 0; i < 3 * nsteps; i++) {
            float a = 0.f, b = 0.f;
            YM_CK(c, cudaEventElapsedTime(&a, c->events[3 * i], c->events[3 * i + 1]), "kernel time");
            YM_CK(c, cudaEventElapsedTime(&b, c->events[3 * i + 1], c->events[3 * i + 2]), "kernel time");
            field += a;
            stage += b;
        }
        if (field_ms) *field_ms = float(field);
        if (stage_ms) *stage_ms = float(stage);
    }
    return YMFLOW_OK;
}

int ymflow_time_steps(ymflow_ctx* c, double eps, int nsteps, float* elapsed_ms, float* kernel_ms) {
    float field = 0.f, stage = 0.f;
    const int r = ymflow_time_kernels(c, eps, nsteps, elapsed_ms, kernel_ms ? &field : nullptr,
                                      kernel_ms ? &stage : nullptr);
    if (r == YMFLOW_OK && kernel_ms) *kernel_ms = field + stage;
    return r;
}

}  // extern "C"

namespace {

// Milliseconds per unmeasured step in the context's current form, launched as
// run_step launches the steps inside a call (chained; FP64 links as two rows;
// form 2 replayed), but every stage running from the current links into the
// other buffer: the current field is untouched and the generator buffer, which
// every step's stage 0 writes, is scratch.
int time_step(ymflow_ctx* c, double eps, float* ms) {
    void* const a = c->u[c->cur];
    void* const b = c->u[1 - c->cur];
    const StageBuffers io = {{a, a, a}, {b, b, b}};
    const int rows = steps_by_rows(c) ? kRowsIn | kRowsOut : 0;
    cudaGraphExec_t exec = nullptr;
    int r = YMFLOW_OK;
    if (c->use_graph && c->stage_form == 2) r = capture_step(c, io, eps, &exec);
    if (r == YMFLOW_ERR_OOM) r = YMFLOW_OK;  // launched directly
    auto timed = [&](int reps) -> int {
        YM_CK(c, cudaEventRecord(c->ev0, c->stream), "event record");
        for (int i = 0; i < reps; i++)
            YM_CK(c, exec ? cudaGraphLaunch(exec, c->stream) : enqueue_step(c, io, eps, nullptr, false, rows),
                  "autotune launch");
        YM_CK(c, cudaEventRecord(c->ev1, c->stream), "event record");
        YM_CK(c, cudaEventSynchronize(c->ev1), "autotune timing");
        YM_CK(c, cudaEventElapsedTime(ms, c->ev0, c->ev1), "elapsed time");
        *ms /= float(reps);
        return YMFLOW_OK;
    };
    if (r == YMFLOW_OK) r = timed(1);  // warm-up
    if (r == YMFLOW_OK) r = timed(2);
    // short steps again, enough of them to outlast the first launches' latency
    if (r == YMFLOW_OK && *ms < 1.f) r = timed(20);
    if (exec) cudaGraphExecDestroy(exec);
    return r;
}

struct TuneChoice {
    int form;
    int64_t tile;  // YMFLOW_OPT_TILE value (form 2)
};
std::mutex g_tune_mu;
std::map<std::array<int, 6>, TuneChoice> g_tune_cache;  // (dims, precision, device) -> choice

}  // namespace

extern "C" {

int ymflow_autotune(ymflow_ctx* c, double eps, int* stage_form, int* tile_y, int* tile_z) {
    NvtxRange range("ymflow_autotune");
    if (!c || !std::isfinite(eps)) return fail(c, YMFLOW_ERR_ARG, "bad argument to ymflow_autotune");
    if (c->slab || c->is_block) return fail(c, YMFLOW_ERR_ARG, "slab and block contexts keep the stage form of their group");
    if (!c->loaded) return fail(c, YMFLOW_ERR_STATE, "no links loaded");
    DeviceGuard guard(c->device);
    YM_CK(c, cudaStreamSynchronize(c->stream), "autotune");
    const std::array<int, 6> key = {c->dims[0], c->dims[1], c->dims[2], c->dims[3], c->prec, c->device};
    auto apply = [&](const TuneChoice& ch) -> int {
        if (ch.form == 2) {
            const int r = ymflow_set_option(c, YMFLOW_OPT_TILE, ch.tile);
            if (r != YMFLOW_OK) return r;
        }
        return ymflow_set_option(c, YMFLOW_OPT_STAGE_FORM, ch.form);
    };
    auto report = [&]() {
        if (stage_form) *stage_form = c->stage_form;
        if (tile_y) *tile_y = c->stage_form == 2 ? c->tile.ty : 0;
        if (tile_z) *tile_z = c->stage_form == 2 ? c->tile.tz : 0;
    };
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune_cache.find(key);
        if (it != g_tune_cache.end()) {
            const int r = apply(it->second);
            if (r == YMFLOW_OK) report();
            return r;
        }
    }
    const bool had_hfield = c->hfield != nullptr;
    std::vector<TuneChoice> cands = {{0, 0}, {1, 0}};
    if (small_lattice(c->geo)) cands = {{c->stage_form == 1 ? 1 : 0, 0}};  // forms 0 and 1 run the same kernel
    for (int ty = 1; ty <= c->geo.n[1]; ty++)
        for (int tz = 1; tz <= c->geo.n[2]; tz++)
            for (int lpt : {1, 2, 4})
                for (int lean : {0, 1}) {
                    TileShape tp;
                    if (make_tile_shape(c->prec, c->geo, ty, tz, &tp, true, lpt, lean))
                        cands.push_back({2, tile_option(tp)});
                }
    // Two passes: every candidate, then again those within 20 % of the first
    // pass's best, each keeping its faster time.  The clock drifts under the
    // power cap while the candidates run; the second pass times the close
    // ones at the same clock.
    TuneChoice best = {c->stage_form, c->tile_ok ? tile_option(c->tile) : 0};
    std::vector<float> tmin(cands.size(), -1.f);
    float best_ms = 0.f;
    bool any = false;
    for (int pass = 0; pass < 2; pass++) {
        const float bound = best_ms * 1.2f;
        for (size_t i = 0; i < cands.size(); i++) {
            if (pass == 1 && (tmin[i] < 0.f || tmin[i] > bound)) continue;
            int r = apply(cands[i]);
            if (r != YMFLOW_OK) continue;  // e.g. no device memory for the plaquette field
            float ms = 0.f;
            r = time_step(c, eps, &ms);
            if (r != YMFLOW_OK) return r;
            if (tmin[i] < 0.f || ms < tmin[i]) tmin[i] = ms;
            if (!any || tmin[i] < best_ms) {
                best = cands[i];
                best_ms = tmin[i];
                any = true;
            }
        }
        if (!any) return fail(c, YMFLOW_ERR_STATE, "autotune: no stage form could run");
    }
    int r = apply(best);
    if (r != YMFLOW_OK) return r;
    if (c->stage_form != 1 && !had_hfield && c->hfield) {  // drop the plaquette field tuning allocated
        cudaFree(c->hfield);
        c->bytes -= int64_t(plane_field_bytes(c->prec, c->geo.V));
        c->hfield = nullptr;
    }
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune_cache[key] = best;
    }
    report();
    return YMFLOW_OK;
}

int ymflow_set_option(ymflow_ctx* c, int key, int64_t value) {
    if (!c) return YMFLOW_ERR_ARG;
    switch (key) {
        case YMFLOW_OPT_BLOCK:  // four warps (one per direction) per 32 sites
            if (value != 128) return fail(c, YMFLOW_ERR_ARG, "stage block must be 128 (compiled launch bounds)");
            c->block = int(value);
            return YMFLOW_OK;
        case YMFLOW_OPT_OBS_BLOCK:  // fixed: six warps (one per plane) per 32 sites
            if (value != 192) return fail(c, YMFLOW_ERR_ARG, "observables block is 192 (six warps per 32 sites)");
            return YMFLOW_OK;
        case YMFLOW_OPT_GRAPH:
            c->use_graph = value != 0;
            return YMFLOW_OK;
        case YMFLOW_OPT_STAGE_FORM: {
            if (value < 0 || value > 2)
                return fail(c, YMFLOW_ERR_ARG, "stage form is 0 (fused), 1 (two kernels) or 2 (shared-memory tile)");
            if (value == 2 && !c->tile_ok)
                return fail(c, YMFLOW_ERR_ARG, "no tiling of this lattice for the shared-memory stage kernel "
                                               "(set one with YMFLOW_OPT_TILE)");
            DeviceGuard guard(c->device);
            if (value == 1 && !c->hfield) {
                const int r = dev_alloc(c, &c->hfield, plane_field_bytes(c->prec, c->geo.V), "plaquette field");
                if (r != YMFLOW_OK) return r;
            }
            if (c->stage_form != int(value)) {
                YM_CK(c, cudaStreamSynchronize(c->stream), "stage form switch");
                drop_graphs(c);
            }
            c->stage_form = int(value);
            return YMFLOW_OK;
        }
        case YMFLOW_OPT_TILE: {
            const int ty = int((value >> 16) & 0xffff), tz = int(value & 0xffff);
            const int lpt = int((value >> 32) & 0xf) ? int((value >> 32) & 0xf) : 4;
            const int lean = int((value >> 36) & 1);
            TileShape tp;
            if (value < 0 || (value >> 37) != 0 || !make_tile_shape(c->prec, c->geo, ty, tz, &tp, true, lpt, lean))
                return fail(c, YMFLOW_ERR_ARG, "tile (" + std::to_string(ty) + ", " + std::to_string(tz) +
                                                   ") does not tile this lattice's (y, z) in whole warps of x lines "
                                                   "within 64..512 threads and 227 KB of shared memory");
            DeviceGuard guard(c->device);
            YM_CK(c, tile_grid(c->prec, c->device, &tp), "tile occupancy");
            YM_CK(c, cudaStreamSynchronize(c->stream), "tile switch");
            drop_graphs(c);
            c->tile = tp;
            c->tile_ok = true;
            return YMFLOW_OK;
        }
        case YMFLOW_OPT_TIMED_REUNIT:
            if (value < 0 || value > (1 << 30)) return fail(c, YMFLOW_ERR_ARG, "timed reunitarisation period < 0");
            c->timed_reunit = int(value);
            return YMFLOW_OK;
        default: return fail(c, YMFLOW_ERR_ARG, "unknown option");
    }
}

int ymflow_get_option(const ymflow_ctx* c, int key, int64_t* value) {
    if (!c || !value) return YMFLOW_ERR_ARG;
    switch (key) {
        case YMFLOW_OPT_BLOCK: *value = c->block; return YMFLOW_OK;
        case YMFLOW_OPT_OBS_BLOCK: *value = 192; return YMFLOW_OK;
        case YMFLOW_OPT_GRAPH: *value = c->use_graph ? 1 : 0; return YMFLOW_OK;
        case YMFLOW_OPT_STAGE_FORM: *value = c->stage_form; return YMFLOW_OK;
        case YMFLOW_OPT_TILE: *value = c->tile_ok ? tile_option(c->tile) : 0; return YMFLOW_OK;
        case YMFLOW_OPT_TIMED_REUNIT: *value = c->timed_reunit; return YMFLOW_OK;
        default: return YMFLOW_ERR_ARG;
    }
}

int ymflow_host_alloc(int64_t bytes, void** ptr) {
    if (!ptr || bytes <= 0) return YMFLOW_ERR_ARG;
    *ptr = nullptr;
    cudaError_t e = cudaMallocHost(ptr, size_t(bytes));
    if (e != cudaSuccess) {
        cudaGetLastError();
        *ptr = nullptr;
        return e == cudaErrorMemoryAllocation ? YMFLOW_ERR_OOM : YMFLOW_ERR_CUDA;
    }
    return YMFLOW_OK;
}

int ymflow_host_free(void* ptr) {
    if (!ptr) return YMFLOW_OK;
    return cudaFreeHost(ptr) == cudaSuccess ? YMFLOW_OK : YMFLOW_ERR_CUDA;
}

int ymflow_device_bytes(const ymflow_ctx* c, int64_t* bytes) {
    if (!c || !bytes) return YMFLOW_ERR_ARG;
    *bytes = c->bytes;
    return YMFLOW_OK;
}

}  // extern "C"
