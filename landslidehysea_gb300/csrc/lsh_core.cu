// lsh_core.cu -- sm_103a kernels and the C ABI (include/lsh.h) of the
// two-layer finite-volume time step.
//
// Layout in HBM: FP64 structure-of-arrays, one array of nx*ny doubles per
// variable (h1 q1x q1y h2 q2x q2y H), row-major (cell j*nx + i).  The step:
//   order 1 (the reference scheme, ShallowWater.cu:391-442):
//     a flux pass over all edges (one thread each) writes every edge's terms
//     to planes; the cell update (one thread per cell) adds its four edges'
//     terms in the reference's colour order, with the positivity limiter,
//     updates the state IN PLACE, folds the cells' rates into one 64-bit
//     atomicMax on the bit pattern of the (non-negative) double; a clock
//     kernel advances t and dt on the device and lists the tiles that the
//     next step has to visit.  No host sync per step, no texture copy-back
//     (ShallowWater.cu:447-454), so a run of steps is one CUDA graph launch.
//   order 2: minmod reconstruction kernel + the same two passes on face
//     values, twice (Heun / TVD-RK2), the second update averaging with the
//     step's initial state.
//   Parameters that flux_fits refuses, and a device without room for the edge
//   planes, take the reference's 4 colour passes (hor-even, hor-odd, ver-even,
//   ver-odd) into 7 accumulators and a volume kernel, with the same bits.
// The FP64 math lives in lsh_scheme.cuh.

#include <cuda_runtime.h>

#include <algorithm>
#include <utility>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/lsh.h"
#include "lsh_passes.cuh"
#include "lsh_scheme.cuh"
#include "lsh_run_until.h"
#include "lsh_setup.h"
#include "lsh_kernels.cuh"

using lsh::Consts;
using lsh::EdgeIn;
using lsh::Geo;
using lsh::TimeRec;

namespace {

using lsh::kCellBlock;
using lsh::kEdgeBlock;
using lsh::kRateInitBits;
using lsh::KArgs;
using lsh::dt_of;
using lsh::do_edge;
using lsh::face_rest;
constexpr int kGraphChunk = 16;

thread_local std::string g_last_error;

// FP64 throughput probe: 8 independent DFMA chains per thread.
__global__ void k_fp64_probe(double* out, int iters, double a, double b) {
    double x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = threadIdx.x * 1e-3 + k;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = fma(x[k], a, b);
    }
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += x[k];
    if (s == 12345.678) out[0] = s;  // keeps the chains live; never true in practice
}

// h1 - H at the listed cells (lsh_get_gauge_eta); NaN for a cell off the grid.
__global__ void k_gauge_eta(const double* __restrict__ h1, const double* __restrict__ H, const int* cells, int n,
                            long long N, double* out) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const int c = cells[g];
    out[g] = (c >= 0 && c < N) ? h1[c] - H[c] : __longlong_as_double(0x7ff8000000000000LL);
}

}  // namespace

// ------------------------------------------------------------------ context

struct lsh_ctx {
    lsh_params p;
    Consts c;
    int device = 0;
    cudaStream_t own = nullptr;     // created by the library; used for graph capture
    cudaStream_t stream = nullptr;  // where work runs (own, or the caller's)
    size_t N = 0;
    void* slab = nullptr;           // one device allocation for every array
    double* X[7] = {};              // state (X[6] = H)
    double* Y[6] = {};              // order-2 stage buffer
    double* acc[7] = {};
    double* sx[7] = {};
    double* sy[7] = {};
    double* eta_max = nullptr;
    double* eta_time = nullptr;
    unsigned char* szero = nullptr;  // order 2: per-cell "stored slopes are zero" flags
    void* edge_mem = nullptr;        // the flux pass's edge buffers (null: the colour passes run)
    FluxMem flux{};
    unsigned* dep_ctr = nullptr;     // pass-overlap counters: kernels_per_step segments of dep_stride
    int dep_stride = 0;              // 0: the step's passes run as plain, fully ordered launches
    double* geo_buf = nullptr;
    Geo geo{};
    TimeRec* tm = nullptr;
    TimeRec* tm_host = nullptr;     // pinned mirror for reads
    int* gauge_cells = nullptr;     // lsh_get_gauge_eta: device copy of the last cell list
    double* gauge_out = nullptr;    // and its gathered values
    int gauge_cap = 0;
    std::vector<int> gauge_host;    // the cell list gauge_cells holds
    cudaGraphExec_t g_chunk = nullptr, g_one = nullptr;
    long long launches = 0;
    int kernels_per_step = 0;
    bool has_state = false;
};

namespace {

int fail_cuda(cudaError_t e, const char* what) {
    g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
    (void)cudaGetLastError();
    return (e == cudaErrorMemoryAllocation) ? LSH_ERR_GPU_OOM : LSH_ERR_CUDA;
}

#define LSH_CUDA(call)                                          \
    do {                                                        \
        cudaError_t e_ = (call);                                \
        if (e_ != cudaSuccess) return fail_cuda(e_, #call);     \
    } while (0)

int check_params(const lsh_params* p) {
    if (const char* why = lsh::params_problem(p)) {
        g_last_error = why;
        return LSH_ERR_INVALID;
    }
    return LSH_OK;
}

KArgs base_args(const lsh_ctx* ctx) {
    KArgs a;
    std::memset(&a, 0, sizeof(a));
    a.c = ctx->c;
    a.geo = ctx->geo;
    for (int k = 0; k < 7; ++k) {
        a.acc[k] = ctx->acc[k];
        a.sx[k] = ctx->sx[k]; a.sy[k] = ctx->sy[k];
        a.sxw[k] = ctx->sx[k]; a.syw[k] = ctx->sy[k];
    }
    a.eta_max = ctx->eta_max;
    a.eta_time = ctx->eta_time;
    a.szero = ctx->szero;
    a.tm = ctx->tm;
    return a;
}

dim3 grid_h(const lsh_ctx* ctx, int par) { return edge_grid_h(ctx->p.nx, ctx->p.ny, par); }
dim3 grid_v(const lsh_ctx* ctx, int par) { return edge_grid_v(ctx->p.nx, ctx->p.ny, par); }


// The arguments of a step's stages: order 1 in place; order 2 X -> Y, then
// Y -> X with the average.
void stage_args(const lsh_ctx* ctx, KArgs& a1, KArgs& a2) {
    a1 = a2 = base_args(ctx);
    for (int k = 0; k < 7; ++k) a1.W[k] = a2.W[k] = ctx->X[k];
    for (int k = 0; k < 6; ++k) {
        a1.Wout[k] = (ctx->p.order == 1) ? ctx->X[k] : ctx->Y[k];
        a2.W[k] = ctx->Y[k];
        a2.Wout[k] = ctx->X[k];
        a2.Xavg[k] = ctx->X[k];
    }
    if (!ctx->edge_mem) return;
    a1.eb = a2.eb = ctx->flux.eb;
    a2.eb.stage = 1;
    for (int l = 0; l < 2; ++l) {
        if (ctx->p.order == 1) a1.eb.depth[l] = a1.eb.depth_out[l] = ctx->Y[3 * l];
        else { a1.eb.depth[l] = a1.W[3 * l]; a2.eb.depth[l] = a2.W[3 * l]; }
    }
}

// Enqueue one time step; returns the number of kernels launched.  `mark` is
// called after each launch where they run one after the other.
template <class Mark>
int enqueue_step(const lsh_ctx* ctx, cudaStream_t s, bool ordered, Mark&& mark) {
    KArgs a1, a2;
    stage_args(ctx, a1, a2);
    const int nx = ctx->p.nx, ny = ctx->p.ny, order = ctx->p.order;
    const double two_cfl = 2.0 * ctx->p.cfl;
    if (ctx->edge_mem)
        return enqueue_flux_step(a1, a2, ctx->flux.map, ordered ? nullptr : ctx->dep_ctr, two_cfl, s, mark);
    if (ctx->dep_ctr && !ordered)
        return enqueue_step_overlap(nx, ny, order, a1, a2, ctx->dep_ctr, ctx->dep_stride, ctx->tm, two_cfl, s);
    const dim3 nbc = cell_grid(nx, ny);
    auto edges = [&](auto ord, const KArgs& a) {
        constexpr int O = decltype(ord)::value;
        k_edges_h<true, O><<<grid_h(ctx, 0), edge_block_h(), 0, s>>>(a, 0); mark();
        k_edges_h<false, O><<<grid_h(ctx, 1), edge_block_h(), 0, s>>>(a, 1); mark();
        k_edges_v<O><<<grid_v(ctx, 0), edge_block_v(), 0, s>>>(a, 0); mark();
        k_edges_v<O><<<grid_v(ctx, 1), edge_block_v(), 0, s>>>(a, 1); mark();
    };
    if (order == 1) {
        edges(std::integral_constant<int, 1>(), a1);
        k_volume<0><<<nbc, cell_block(), 0, s>>>(a1); mark();
    } else {
        k_recon<<<nbc, cell_block(), 0, s>>>(a1); mark();
        edges(std::integral_constant<int, 2>(), a1);
        k_volume<1><<<nbc, cell_block(), 0, s>>>(a1); mark();
        k_recon<<<nbc, cell_block(), 0, s>>>(a2); mark();
        edges(std::integral_constant<int, 2>(), a2);
        k_volume<2><<<nbc, cell_block(), 0, s>>>(a2); mark();
    }
    k_advance<<<1, 1, 0, s>>>(ctx->tm, two_cfl); mark();
    return ctx->kernels_per_step;
}

int build_graph(lsh_ctx* ctx, int nsteps, cudaGraphExec_t* out) {
    cudaGraph_t graph = nullptr;
    LSH_CUDA(cudaStreamBeginCapture(ctx->own, cudaStreamCaptureModeThreadLocal));
    for (int i = 0; i < nsteps; ++i) enqueue_step(ctx, ctx->own, false, [] {});
    cudaError_t e = cudaStreamEndCapture(ctx->own, &graph);
    if (e != cudaSuccess) return fail_cuda(e, "cudaStreamEndCapture");
    e = cudaGraphInstantiate(out, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return fail_cuda(e, "cudaGraphInstantiate");
    return LSH_OK;
}

int err_bits_to_status(int bits) {
    for (int s = 1; s < 31; ++s)
        if (bits & (1 << s)) return s;
    return LSH_OK;
}

int upload_state(lsh_ctx* ctx, const double* const src[LSH_NVARS], cudaMemcpyKind kind, double* dt0_out) {
    const size_t bytes = ctx->N * sizeof(double);
    for (int k = 0; k < 7; ++k) {
        if (!src[k]) { g_last_error = "null state pointer"; return LSH_ERR_INVALID; }
        LSH_CUDA(cudaMemcpyAsync(ctx->X[k], src[k], bytes, kind, ctx->stream));
    }
    KArgs a = base_args(ctx);
    for (int k = 0; k < 7; ++k) a.W[k] = ctx->X[k];
    const dim3 nbc = cell_grid(ctx->p.nx, ctx->p.ny);
    cudaStream_t s = ctx->stream;
    k_init_eta<<<nbc, cell_block(), 0, s>>>(a);
    TimeRec init{};
    init.rmax_bits = kRateInitBits;
    init.t_end = INFINITY;
    init.dt_min = ctx->p.dt_min;
    LSH_CUDA(cudaMemcpyAsync(ctx->tm, &init, sizeof(TimeRec), cudaMemcpyHostToDevice, s));
    launch_init_wave(a, ctx->p.nx, ctx->p.ny, s);
    k_cell_dt<<<nbc, cell_block(), 0, s>>>(a);
    k_init_finish<<<1, 1, 0, s>>>(ctx->tm, 2.0 * ctx->p.cfl);
    ctx->launches += 7;
    if (ctx->edge_mem) {
        launch_all_busy(ctx->flux.map, s);
        ctx->launches += 1;
    }
    LSH_CUDA(cudaGetLastError());
    LSH_CUDA(cudaMemcpyAsync(ctx->tm_host, ctx->tm, sizeof(TimeRec), cudaMemcpyDeviceToHost, s));
    LSH_CUDA(cudaStreamSynchronize(s));
    ctx->has_state = true;
    if (dt0_out) *dt0_out = ctx->tm_host->dt;
    return LSH_OK;
}

int read_time(lsh_ctx* ctx) {
    LSH_CUDA(cudaMemcpyAsync(ctx->tm_host, ctx->tm, sizeof(TimeRec), cudaMemcpyDeviceToHost, ctx->stream));
    LSH_CUDA(cudaStreamSynchronize(ctx->stream));
    return LSH_OK;
}

// t_end and `done` into the device record, from the host copy that read_time
// has just filled (a small H2D copy on the stream).
int put_t_end(lsh_ctx* ctx, double t_end) {
    ctx->tm_host->t_end = t_end;
    ctx->tm_host->done = (ctx->tm_host->t >= t_end || ctx->tm_host->err) ? 1 : 0;
    LSH_CUDA(cudaMemcpyAsync(ctx->tm, ctx->tm_host, sizeof(TimeRec), cudaMemcpyHostToDevice, ctx->stream));
    return LSH_OK;
}

// lsh_run_until's view of a context (lsh_run_until.h)
struct CtxClock {
    lsh_ctx* ctx;
    TimeRec& rec() { return *ctx->tm_host; }
    int read() { return read_time(ctx); }
    int put(double t_end) { return put_t_end(ctx, t_end); }
    int step(int n) { return lsh_step(ctx, n); }
    int failed() { return err_bits_to_status(ctx->tm_host->err); }
};

}  // namespace

extern "C" {

int lsh_params_default(lsh_params* p) {
    if (!p) return LSH_ERR_INVALID;
    std::memset(p, 0, sizeof(*p));
    p->nx = p->ny = 1;
    p->order = 1;
    p->coords = LSH_COORDS_CARTESIAN;
    p->friction_law = LSH_FRICTION_COULOMB;
    p->dx = p->dy = 1.0;
    p->radius = 6378136.6;
    p->borde_sup = p->borde_inf = p->borde_izq = p->borde_der = -1.0;
    p->cfl = 0.9;
    p->r = 0.5;
    p->gravity = 9.81;
    p->eps_h = 5e-3;
    p->L = p->H = 1.0;
    p->peso = p->beta = 1.0;
    return LSH_OK;
}

int lsh_check_device(void) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) { (void)cudaGetLastError(); return 1; }
    if (n == 0) return 1;
    for (int d = 0; d < n; ++d) {
        cudaDeviceProp prop;
        if (cudaGetDeviceProperties(&prop, d) == cudaSuccess && prop.major >= 1) return 0;
    }
    return 2;
}

const char* lsh_status_string(int s) {
    switch (s) {
        case LSH_OK: return "ok";
        case LSH_ERR_GPU_OOM: return "not enough GPU memory";
        case LSH_ERR_HOST_OOM: return "not enough CPU memory";
        case LSH_ERR_INVALID: return "invalid argument";
        case LSH_ERR_CUDA: return "CUDA error";
        case LSH_ERR_NUMERIC: return "NaN or Inf in the state";
        case LSH_ERR_IO: return "file missing or malformed";
        case LSH_ERR_NO_DEVICE: return "no CUDA device";
        case LSH_ERR_TIMEOUT: return "bounded device wait timed out";
        case LSH_ERR_STALL: return "time step below dt_min";
        default: return "unknown status";
    }
}

const char* lsh_last_error(void) { return g_last_error.c_str(); }

int lsh_create(const lsh_params* p, int device, lsh_ctx** out) {
    if (!out) return LSH_ERR_INVALID;
    *out = nullptr;
    if (int s = check_params(p)) return s;
    if (lsh_check_device() != 0) { g_last_error = "no CUDA device"; return LSH_ERR_NO_DEVICE; }
    lsh_ctx* ctx = new (std::nothrow) lsh_ctx();
    if (!ctx) return LSH_ERR_HOST_OOM;
    ctx->p = *p;
    ctx->c = lsh::make_consts(*p);
    ctx->N = size_t(p->nx) * p->ny;
    auto bail = [&](int s) { lsh_destroy(ctx); return s; };
    if (device >= 0) {
        cudaError_t e = cudaSetDevice(device);
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaSetDevice"));
    }
    {
        cudaError_t e = cudaGetDevice(&ctx->device);
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaGetDevice"));
        e = cudaStreamCreateWithFlags(&ctx->own, cudaStreamNonBlocking);
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaStreamCreate"));
        ctx->stream = ctx->own;
    }
    // one slab: X(7) + Y(6) + acc + eta(2) [+ sx, sy (14)] arrays of N, geometry, time record
    const size_t n_pad = (ctx->N + 31) & ~size_t(31);  // 256-byte aligned arrays
    const size_t geo_n = size_t(7) * (p->ny + 1);
    size_t dep_bytes = 0;
    // The slab of the flux pass and cell update (`flux`: only the wave
    // accumulator, which the initial-dt pass uses) or of the colour passes,
    // with the pass-overlap counters: one per tile row (block row) of each
    // pass of a step, when a launch of rows up to 65535 covers the grid.
    auto slab_bytes = [&](bool flux) {
        const int n_arrays = 7 + 6 + (flux ? 1 : 7) + 2 + ((p->order == 2) ? 14 : 0);
        ctx->kernels_per_step = (p->order == 1) ? 6 : 13;
        if (flux) ctx->dep_stride = (tiles_y(p->ny) <= 65535) ? flux_dep_stride(p->ny) : 0;
        else ctx->dep_stride = dep_stride_for(p->nx, p->ny);
        dep_bytes = size_t(ctx->dep_stride) * ctx->kernels_per_step * sizeof(unsigned);
        return (size_t(n_arrays) * n_pad + ((geo_n + 31) & ~size_t(31))) * sizeof(double) + 256 +
               ((p->order == 2) ? n_pad : 0) +  // + one byte per cell: slopes-are-zero flags
               ((dep_bytes + 255) & ~size_t(255));
    };
    // The flux pass and cell update where the parameters allow it and its edge
    // buffers fit the device beside the rest; the colour passes, which need 0.6
    // of the memory, where they do not (256 MB stay free for the caller and for
    // what the context allocates later).
    if (lsh::flux_fits(*p)) {
        cudaError_t e = cudaMalloc(&ctx->edge_mem, FluxMem{}.layout(nullptr, p->nx, p->ny, p->order));
        if (e == cudaSuccess) e = cudaMalloc(&ctx->slab, slab_bytes(true));
        size_t room = 0, total = 0;
        if (e == cudaSuccess && cudaMemGetInfo(&room, &total) == cudaSuccess && room < (size_t(256) << 20)) {
            cudaFree(ctx->slab);
            e = cudaErrorMemoryAllocation;
        }
        if (e != cudaSuccess) {
            if (ctx->edge_mem) cudaFree(ctx->edge_mem);
            ctx->edge_mem = ctx->slab = nullptr;
            if (e != cudaErrorMemoryAllocation) return bail(fail_cuda(e, "cudaMalloc edge buffers"));
            (void)cudaGetLastError();
        }
    }
    {
        cudaError_t e = ctx->slab ? cudaSuccess : cudaMalloc(&ctx->slab, slab_bytes(false));
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaMalloc"));
        e = cudaMallocHost((void**)&ctx->tm_host, sizeof(TimeRec));
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaMallocHost"));
    }
    if (ctx->edge_mem) {
        ctx->flux.layout(static_cast<unsigned char*>(ctx->edge_mem), p->nx, p->ny, p->order);
        cudaError_t e = cudaMemsetAsync(ctx->flux.clear, 0, ctx->flux.clear_bytes, ctx->own);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->own);
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaMemset cell marks"));
    }
    double* cur = static_cast<double*>(ctx->slab);
    for (int k = 0; k < 7; ++k) { ctx->X[k] = cur; cur += n_pad; }
    for (int k = 0; k < 6; ++k) { ctx->Y[k] = cur; cur += n_pad; }
    for (int k = ctx->edge_mem ? 6 : 0; k < 7; ++k) { ctx->acc[k] = cur; cur += n_pad; }
    ctx->eta_max = cur; cur += n_pad;
    ctx->eta_time = cur; cur += n_pad;
    if (p->order == 2) {
        for (int k = 0; k < 7; ++k) { ctx->sx[k] = cur; cur += n_pad; }
        for (int k = 0; k < 7; ++k) { ctx->sy[k] = cur; cur += n_pad; }
    }
    ctx->geo_buf = cur;
    cur += (geo_n + 31) & ~size_t(31);
    ctx->tm = reinterpret_cast<TimeRec*>(cur);
    unsigned char* tail = reinterpret_cast<unsigned char*>(cur) + 256;
    if (p->order == 2) {
        ctx->szero = tail;
        tail += n_pad;
        // no slope is known to be zero yet; wait before the legacy-stream copies below
        cudaError_t e = cudaMemsetAsync(ctx->szero, 0, n_pad, ctx->own);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->own);
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaMemset slope flags"));
    }
    if (ctx->dep_stride) {
        ctx->dep_ctr = reinterpret_cast<unsigned*>(tail);
        cudaError_t e = cudaMemsetAsync(ctx->dep_ctr, 0, dep_bytes, ctx->own);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->own);
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaMemset pass counters"));
    }

    const size_t st = size_t(p->ny + 1);
    std::vector<double> g(geo_n, 0.0);
    lsh::fill_geo(*p, g.data(), st);
    {
        cudaError_t e = cudaMemcpy(ctx->geo_buf, g.data(), geo_n * sizeof(double), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) return bail(fail_cuda(e, "cudaMemcpy geometry"));
    }
    ctx->geo.area = ctx->geo_buf;
    ctx->geo.len_v = ctx->geo_buf + st;
    ctx->geo.len_h = ctx->geo_buf + 2 * st;
    ctx->geo.tanR = ctx->geo_buf + 3 * st;
    ctx->geo.wx = ctx->geo_buf + 4 * st;
    ctx->geo.wy = ctx->geo_buf + 5 * st;
    ctx->geo.inv_area = ctx->geo_buf + 6 * st;
    *out = ctx;
    return LSH_OK;
}

int lsh_destroy(lsh_ctx* ctx) {
    if (!ctx) return LSH_OK;
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    if (ctx->g_chunk) cudaGraphExecDestroy(ctx->g_chunk);
    if (ctx->g_one) cudaGraphExecDestroy(ctx->g_one);
    if (ctx->slab) cudaFree(ctx->slab);
    if (ctx->edge_mem) cudaFree(ctx->edge_mem);
    if (ctx->gauge_cells) cudaFree(ctx->gauge_cells);
    if (ctx->tm_host) cudaFreeHost(ctx->tm_host);
    if (ctx->own) cudaStreamDestroy(ctx->own);
    (void)cudaGetLastError();
    delete ctx;
    return LSH_OK;
}

int lsh_set_stream(lsh_ctx* ctx, void* s) {
    if (!ctx) return LSH_ERR_INVALID;
    ctx->stream = s ? static_cast<cudaStream_t>(s) : ctx->own;
    return LSH_OK;
}

int lsh_set_state(lsh_ctx* ctx, const double* const host_state[LSH_NVARS], double* dt0_out) {
    if (!ctx || !host_state) return LSH_ERR_INVALID;
    return upload_state(ctx, host_state, cudaMemcpyHostToDevice, dt0_out);
}

int lsh_set_state_device(lsh_ctx* ctx, const double* const dev_state[LSH_NVARS], double* dt0_out) {
    if (!ctx || !dev_state) return LSH_ERR_INVALID;
    return upload_state(ctx, dev_state, cudaMemcpyDeviceToDevice, dt0_out);
}

int lsh_step(lsh_ctx* ctx, int nsteps) {
    if (!ctx || nsteps < 0) return LSH_ERR_INVALID;
    if (!ctx->has_state) { g_last_error = "lsh_set_state has not been called"; return LSH_ERR_INVALID; }
    if (nsteps == 0) return LSH_OK;
    if (!ctx->g_chunk) { if (int s = build_graph(ctx, kGraphChunk, &ctx->g_chunk)) return s; }
    if (!ctx->g_one) { if (int s = build_graph(ctx, 1, &ctx->g_one)) return s; }
    const int full = nsteps / kGraphChunk, rest = nsteps % kGraphChunk;
    for (int i = 0; i < full; ++i) LSH_CUDA(cudaGraphLaunch(ctx->g_chunk, ctx->stream));
    for (int i = 0; i < rest; ++i) LSH_CUDA(cudaGraphLaunch(ctx->g_one, ctx->stream));
    ctx->launches += (long long)nsteps * ctx->kernels_per_step;
    return LSH_OK;
}

int lsh_synchronize(lsh_ctx* ctx) {
    if (!ctx) return LSH_ERR_INVALID;
    if (int s = read_time(ctx)) return s;
    return err_bits_to_status(ctx->tm_host->err);
}

int lsh_run_until(lsh_ctx* ctx, double t_end, long long max_steps, long long* steps_done) {
    if (!ctx) return LSH_ERR_INVALID;
    if (!ctx->has_state) { g_last_error = "lsh_set_state has not been called"; return LSH_ERR_INVALID; }
    CtxClock c{ctx};
    return lsh::run_until(c, t_end, max_steps, 8 * kGraphChunk, steps_done);
}

int lsh_get_state(lsh_ctx* ctx, double* const host_state[LSH_NVARS]) {
    if (!ctx || !host_state) return LSH_ERR_INVALID;
    const size_t bytes = ctx->N * sizeof(double);
    for (int k = 0; k < 7; ++k)
        if (host_state[k]) LSH_CUDA(cudaMemcpyAsync(host_state[k], ctx->X[k], bytes, cudaMemcpyDeviceToHost, ctx->stream));
    LSH_CUDA(cudaStreamSynchronize(ctx->stream));
    return LSH_OK;
}

int lsh_get_state_device(lsh_ctx* ctx, double* const dev_state[LSH_NVARS]) {
    if (!ctx || !dev_state) return LSH_ERR_INVALID;
    const size_t bytes = ctx->N * sizeof(double);
    for (int k = 0; k < 7; ++k)
        if (dev_state[k]) LSH_CUDA(cudaMemcpyAsync(dev_state[k], ctx->X[k], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    return LSH_OK;
}

int lsh_get_time(lsh_ctx* ctx, double* t, double* dt_next, long long* steps) {
    if (!ctx) return LSH_ERR_INVALID;
    if (int s = read_time(ctx)) return s;
    if (t) *t = ctx->tm_host->t;
    if (dt_next) *dt_next = ctx->tm_host->dt;
    if (steps) *steps = ctx->tm_host->steps;
    return LSH_OK;
}

int lsh_get_eta_max(lsh_ctx* ctx, double* eta_max, double* eta_time) {
    if (!ctx) return LSH_ERR_INVALID;
    const size_t bytes = ctx->N * sizeof(double);
    if (eta_max) LSH_CUDA(cudaMemcpyAsync(eta_max, ctx->eta_max, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    if (eta_time) LSH_CUDA(cudaMemcpyAsync(eta_time, ctx->eta_time, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    LSH_CUDA(cudaStreamSynchronize(ctx->stream));
    return LSH_OK;
}

int lsh_get_gauge_eta(lsh_ctx* ctx, int n, const int* cells, double* out) {
    if (!ctx || n < 0 || (n > 0 && (!cells || !out))) return LSH_ERR_INVALID;
    if (n == 0) return LSH_OK;
    if (n > ctx->gauge_cap) {
        // one buffer: n cell indices, then n values (256-byte aligned)
        if (ctx->gauge_cells) { cudaFree(ctx->gauge_cells); ctx->gauge_cells = nullptr; ctx->gauge_cap = 0; }
        const size_t idx_bytes = (size_t(n) * sizeof(int) + 255) & ~size_t(255);
        void* buf = nullptr;
        LSH_CUDA(cudaMalloc(&buf, idx_bytes + size_t(n) * sizeof(double)));
        ctx->gauge_cells = static_cast<int*>(buf);
        ctx->gauge_out = reinterpret_cast<double*>(static_cast<char*>(buf) + idx_bytes);
        ctx->gauge_cap = n;
        ctx->gauge_host.clear();
    }
    cudaStream_t s = ctx->stream;
    if (ctx->gauge_host.size() != size_t(n) || !std::equal(cells, cells + n, ctx->gauge_host.begin())) {
        ctx->gauge_host.assign(cells, cells + n);
        LSH_CUDA(cudaMemcpyAsync(ctx->gauge_cells, ctx->gauge_host.data(), size_t(n) * sizeof(int),
                                 cudaMemcpyHostToDevice, s));
    }
    k_gauge_eta<<<(n + 127) / 128, 128, 0, s>>>(ctx->X[0], ctx->X[6], ctx->gauge_cells, n, (long long)ctx->N,
                                                ctx->gauge_out);
    ctx->launches += 1;
    LSH_CUDA(cudaGetLastError());
    LSH_CUDA(cudaMemcpyAsync(out, ctx->gauge_out, size_t(n) * sizeof(double), cudaMemcpyDeviceToHost, s));
    LSH_CUDA(cudaStreamSynchronize(s));
    return LSH_OK;
}

int lsh_get_masks(lsh_ctx* ctx, uint8_t* mask) {
    if (!ctx || !mask) return LSH_ERR_INVALID;
    std::vector<double> h1(ctx->N), h2(ctx->N), qx(ctx->N), qy(ctx->N);
    double* dst[LSH_NVARS] = {h1.data(), nullptr, nullptr, h2.data(), qx.data(), qy.data(), nullptr};
    if (int s = lsh_get_state(ctx, dst)) return s;
    const double eps = ctx->p.eps_h;
    for (size_t i = 0; i < ctx->N; ++i) {
        uint8_t m = 0;
        if (h1[i] >= eps) m |= 1;
        if (h2[i] >= eps) { m |= 2; if (qx[i] == 0.0 && qy[i] == 0.0) m |= 4; }
        mask[i] = m;
    }
    return LSH_OK;
}

int lsh_profile_step(lsh_ctx* ctx, float* ms_out, int cap, int* n_kernels) {
    if (!ctx || !ms_out || cap < 1) return LSH_ERR_INVALID;
    if (!ctx->has_state) { g_last_error = "lsh_set_state has not been called"; return LSH_ERR_INVALID; }
    cudaStream_t s = ctx->stream;
    const int nk = ctx->kernels_per_step;
    std::vector<cudaEvent_t> ev(nk + 1);
    for (auto& e : ev) LSH_CUDA(cudaEventCreate(&e));
    int i = 0;
    auto mark = [&]() { cudaEventRecord(ev[i++], s); };
    mark();
    enqueue_step(ctx, s, true, mark);
    ctx->launches += nk;
    int status = LSH_OK;
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaEventSynchronize(ev[nk]);
    if (e != cudaSuccess) status = fail_cuda(e, "lsh_profile_step");
    for (int k = 0; k < nk && k < cap && status == LSH_OK; ++k) cudaEventElapsedTime(&ms_out[k], ev[k], ev[k + 1]);
    for (auto& ee : ev) cudaEventDestroy(ee);
    if (n_kernels) *n_kernels = nk;
    return status;
}

int lsh_probe_fp64_peak(int device, double* gflops) {
    if (!gflops) return LSH_ERR_INVALID;
    if (lsh_check_device() != 0) return LSH_ERR_NO_DEVICE;
    if (device >= 0) LSH_CUDA(cudaSetDevice(device));
    int dev = 0, sms = 0;
    LSH_CUDA(cudaGetDevice(&dev));
    LSH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    double* out = nullptr;
    LSH_CUDA(cudaMalloc(&out, sizeof(double)));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int threads = 256, blocks = sms * 8, iters = 4096;
    k_fp64_probe<<<blocks, threads>>>(out, 64, 1.0000001, 1e-9);  // warm-up
    cudaEventRecord(e0);
    k_fp64_probe<<<blocks, threads>>>(out, iters, 1.0000001, 1e-9);
    cudaEventRecord(e1);
    cudaError_t e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    if (e != cudaSuccess) return fail_cuda(e, "lsh_probe_fp64_peak");
    const double flops = 2.0 * 8.0 * double(iters) * threads * blocks;
    *gflops = flops / (ms * 1e-3) / 1e9;
    return LSH_OK;
}

int lsh_probe_tiles(lsh_ctx* ctx, int* listed, int* total) {
    if (!ctx || !listed || !total) return LSH_ERR_INVALID;
    *listed = *total = 0;
    if (!ctx->edge_mem) return LSH_OK;
    const TileMap& m = ctx->flux.map;
    std::vector<int> rows(m.nty);
    LSH_CUDA(cudaMemcpyAsync(rows.data(), m.count, rows.size() * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    LSH_CUDA(cudaStreamSynchronize(ctx->stream));
    *total = m.ntx * m.nty;
    for (int n : rows) *listed += n;
    return LSH_OK;
}

int lsh_get_launch_count(lsh_ctx* ctx, long long* launches) {
    if (!ctx || !launches) return LSH_ERR_INVALID;
    *launches = ctx->launches;
    return LSH_OK;
}

}  // extern "C"

// ------------------------------------------------------------------ allocation-free stepping
//
// lsh_step_noalloc (include/lsh.h) runs the first-order step with all of its
// scratch in the file-scope array below instead of allocated memory.  Layout:
// the 64-byte time record and the per-row geometry (7 arrays of ny + 1, written
// by one copy per call), the wave accumulator, then either the flux pass's
// buffers with its copy of the depths, or, for grids whose edges do not fit
// there (more than LSH_NOALLOC_MAX_ROWS columns) and parameters the flux pass
// does not take, the colour passes' six other accumulators.  Host code must not
// use the array's name as an address: the device address is looked up once per
// device with cudaGetSymbolAddress (with that device current) and passed to
// the kernels.

namespace {

constexpr size_t kNaCells = LSH_NOALLOC_MAX_CELLS, kNaRows = LSH_NOALLOC_MAX_ROWS;
constexpr size_t kNaHead = (sizeof(TimeRec) + 7 * (kNaRows + 1) * sizeof(double) + 255) & ~size_t(255);
constexpr size_t kNaAccBytes = kNaCells * sizeof(double);
// two edges per cell and one more line each way, planes and kinds; two marks
// per cell; tile lists of the smallest tiles (unused here) and alignment; the
// pass counters; the copy of the depths
constexpr size_t kNaFluxBytes = 2 * (kNaCells + kNaRows) * (lsh::kEdgePlanes * sizeof(double) + 1) +
                                kNaCells * 2 * sizeof(unsigned) + (size_t(1) << 19);
constexpr size_t kNaCtrBytes = 2 * (kNaRows / kTileY + 64) * sizeof(unsigned);
constexpr size_t kNaBytes = kNaHead + kNaAccBytes + kNaFluxBytes + kNaCtrBytes + 2 * kNaAccBytes + 1024;
static_assert(kNaFluxBytes + 2 * kNaAccBytes >= 6 * kNaAccBytes, "room for the colour passes' accumulators");

__device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

constexpr int kNaMaxDevices = 64;
unsigned char* g_noalloc_base[kNaMaxDevices] = {};
std::mutex g_noalloc_mu;
// host-side staging of the time record and the geometry (no heap allocation per call)
alignas(64) unsigned char g_noalloc_head_host[kNaHead];
unsigned g_noalloc_stage = 0;  // the calls' steps so far, as the marks count them (EdgeBuf::stage)

// Move the running min of per-cell dt into dt (initial-dt pass of a no-alloc call).
__global__ void k_noalloc_take_dt(TimeRec* tm, double two_cfl) {
    tm->dt = dt_of(tm->rmax_bits, two_cfl);
    tm->rmax_bits = kRateInitBits;
}

}  // namespace

extern "C" int lsh_step_noalloc(const lsh_params* p, double* const dev_state[LSH_NVARS], int nsteps,
                                double* t_io, double* dt_io, void* cuda_stream) {
    if (int s = check_params(p)) return s;
    if (!dev_state || !t_io || !dt_io || nsteps < 0) { g_last_error = "lsh_step_noalloc: null pointer or nsteps < 0"; return LSH_ERR_INVALID; }
    for (int k = 0; k < LSH_NVARS; ++k)
        if (!dev_state[k]) { g_last_error = "lsh_step_noalloc: null state array"; return LSH_ERR_INVALID; }
    if (p->order != 1) { g_last_error = "lsh_step_noalloc: only the first-order step (order 1) runs without allocation"; return LSH_ERR_INVALID; }
    if ((long long)p->nx * p->ny > LSH_NOALLOC_MAX_CELLS || p->ny > LSH_NOALLOC_MAX_ROWS) {
        g_last_error = "lsh_step_noalloc: grid larger than LSH_NOALLOC_MAX_CELLS (65536) cells or LSH_NOALLOC_MAX_ROWS (4096) rows";
        return LSH_ERR_INVALID;
    }
    cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    int dev = 0;
    LSH_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNaMaxDevices) { g_last_error = "lsh_step_noalloc: device index out of range"; return LSH_ERR_INVALID; }
    if (!g_noalloc_base[dev]) {
        unsigned char* base = nullptr;
        cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&base), g_noalloc_scratch);
        if (e != cudaSuccess) return fail_cuda(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_base[dev] = base;
    }
    unsigned char* base = g_noalloc_base[dev];

    const int nx = p->nx, ny = p->ny;
    const size_t rows = size_t(ny) + 1;
    TimeRec init{};
    init.t = *t_io;
    init.dt = *dt_io;
    init.t_end = INFINITY;
    init.dt_min = p->dt_min;
    init.rmax_bits = kRateInitBits;
    std::memcpy(g_noalloc_head_host, &init, sizeof(init));
    lsh::fill_geo(*p, reinterpret_cast<double*>(g_noalloc_head_host + sizeof(TimeRec)), rows);
    LSH_CUDA(cudaMemcpyAsync(base, g_noalloc_head_host, sizeof(TimeRec) + 7 * rows * sizeof(double),
                             cudaMemcpyHostToDevice, s));
    TimeRec* tm = reinterpret_cast<TimeRec*>(base);

    KArgs a;
    std::memset(&a, 0, sizeof(a));
    a.c = lsh::make_consts(*p);
    a.c.track_eta = 0;
    const double* g = reinterpret_cast<const double*>(base + sizeof(TimeRec));
    a.geo.area = g;
    a.geo.len_v = g + rows;
    a.geo.len_h = g + 2 * rows;
    a.geo.tanR = g + 3 * rows;
    a.geo.wx = g + 4 * rows;
    a.geo.wy = g + 5 * rows;
    a.geo.inv_area = g + 6 * rows;
    double* acc = reinterpret_cast<double*>(base + kNaHead);
    for (int k = 0; k < 7; ++k) a.W[k] = dev_state[k];
    a.acc[6] = acc;
    for (int k = 0; k < 6; ++k) { a.acc[k] = acc + (k + 1) * kNaCells; a.Wout[k] = dev_state[k]; }
    a.tm = tm;

    const dim3 nbc = cell_grid(nx, ny);
    if (!(*dt_io > 0.0)) {
        // initial dt (ShallowWater.cu:236-257) into the time record
        launch_init_wave(a, nx, ny, s);
        k_cell_dt<<<nbc, cell_block(), 0, s>>>(a);
        k_noalloc_take_dt<<<1, 1, 0, s>>>(tm, 2.0 * p->cfl);
    }
    FluxMem fm;
    if (lsh::flux_fits(*p) && fm.layout(nullptr, nx, ny, 1) <= kNaFluxBytes) {
        // every tile, with the passes overlapped; the counters are zero at load
        // and after each step
        unsigned char* mem = base + kNaHead + kNaAccBytes;
        fm.layout(mem, nx, ny, 1);
        fm.map.count = nullptr;
        unsigned* ctr = reinterpret_cast<unsigned*>(mem + kNaFluxBytes);
        double* depth = reinterpret_cast<double*>(mem + kNaFluxBytes + ((kNaCtrBytes + 255) & ~size_t(255)));
        a.eb = fm.eb;
        a.eb.stage = g_noalloc_stage;
        g_noalloc_stage += 2u * (unsigned)nsteps;
        for (int l = 0; l < 2; ++l) a.eb.depth[l] = a.eb.depth_out[l] = depth + l * kNaCells;
        for (int i = 0; i < nsteps; ++i) enqueue_flux_step(a, a, fm.map, ctr, 2.0 * p->cfl, s, [] {});
    } else {
        const dim3 gh0 = edge_grid_h(nx, ny, 0), gh1 = edge_grid_h(nx, ny, 1);
        const dim3 gv0 = edge_grid_v(nx, ny, 0), gv1 = edge_grid_v(nx, ny, 1);
        for (int i = 0; i < nsteps; ++i) {
            k_edges_h<true, 1><<<gh0, edge_block_h(), 0, s>>>(a, 0);
            k_edges_h<false, 1><<<gh1, edge_block_h(), 0, s>>>(a, 1);
            k_edges_v<1><<<gv0, edge_block_v(), 0, s>>>(a, 0);
            k_edges_v<1><<<gv1, edge_block_v(), 0, s>>>(a, 1);
            k_volume<0><<<nbc, cell_block(), 0, s>>>(a);
            k_advance<<<1, 1, 0, s>>>(tm, 2.0 * p->cfl);
        }
    }
    LSH_CUDA(cudaGetLastError());
    TimeRec out{};
    LSH_CUDA(cudaMemcpyAsync(&out, tm, sizeof(TimeRec), cudaMemcpyDeviceToHost, s));
    LSH_CUDA(cudaStreamSynchronize(s));
    *t_io = out.t;
    *dt_io = out.dt;
    return err_bits_to_status(out.err);
}

namespace lsh {
void set_last_error(const std::string& msg) { g_last_error = msg; }
}  // namespace lsh
