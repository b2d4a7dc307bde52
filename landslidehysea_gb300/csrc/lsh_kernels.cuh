// lsh_kernels.cuh -- the step's kernels (thin launches of the per-edge and
// per-cell bodies of lsh_passes.cuh), shared by the single-grid context
// (lsh_core.cu) and the adjoint's forward recomputation (lsh_adjoint.cu), so
// both run the same device code.  Internal linkage: each translation unit
// that includes this header gets its own copy.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "../../include/lsh.h"
#include "lsh_passes.cuh"

namespace {

using lsh::KArgs;
using lsh::TimeRec;
using lsh::kCellBlock;
using lsh::kEdgeBlock;
using lsh::kRateInitBits;

// Thread-block shapes of the edge passes (x along threadIdx.x, lines along
// threadIdx.y; kEdgeTile threads, below): a warp spans LSH_EDGE_H_BX cells of an
// edge row, or LSH_EDGE_V_BX edge columns (2 LSH_EDGE_V_BX cells) of a row,
// and 32 / BX lines, so fewer warps straddle a wet/dry front than with
// one-line warps, while each row segment stays one contiguous load.
#ifndef LSH_EDGE_H_BX
#define LSH_EDGE_H_BX 16
#endif
#ifndef LSH_EDGE_V_BX
#define LSH_EDGE_V_BX 8
#endif
// Blocks per SM the edge and cell kernels are compiled for: a register cap
// of 65536 / (threads * MINB).  The FP64 unit returns results through the
// short scoreboard, and the edge passes also wait on their loads; at the
// compiler's choice (128-168 registers, 3 blocks of 128) too few warps were
// resident to cover both.  Measured on the 2048^2 fjord, ms per step
// (threads x blocks per SM: registers):
//   before the empty-edge test: 128x3 2.46, 128x4 (128) 2.33, 128x5 (96) 2.26, 128x6 2.27;
//   after it: 128x5 2.09, 128x6 (85) 2.03, 128x7 (73) 2.01, 64x12 (85) 2.03,
//   64x14 (73) 2.00, 64x16 (64) 1.98-1.99, 64x20 (48) 2.00, 64x24 (40) 2.13, 256x2 2.40.
// With the passes overlapped (programmatic dependent launches, below) the
// SMs hold blocks of two or three passes at once, and more resident warps
// pay again (steps 5-148, ms per step; edge threads x blocks, then cell
// blocks of 256 per SM): 64x12 1.814, 64x16 1.666, 64x20 1.608, 64x24 1.690,
// 64x28 1.721, 128x8 1.640, 128x10 1.611, 128x12 1.639; with 64x20: cells
// at the compiler's choice (62-64 registers) 1.608, 5 blocks 1.587,
// 6 blocks (40 registers) 1.582; 64x24 with 6 cell blocks 1.666.
// The spills stay in L1.  1: the compiler's choice.
#ifndef LSH_EDGE_MINB
#define LSH_EDGE_MINB 20
#endif
#ifndef LSH_CELL_MINB
#define LSH_CELL_MINB 6
#endif
// Threads per edge-pass block (a tile of LSH_EDGE_H_BX x threads / BX).
#ifndef LSH_EDGE_THREADS
#define LSH_EDGE_THREADS 64
#endif
constexpr int kEdgeTile = LSH_EDGE_THREADS;
#if LSH_EDGE_MINB > 1
#define LSH_EDGE_BOUNDS __launch_bounds__(kEdgeTile, LSH_EDGE_MINB)
#else
#define LSH_EDGE_BOUNDS __launch_bounds__(kEdgeTile)
#endif
#if LSH_CELL_MINB > 1
#define LSH_CELL_BOUNDS __launch_bounds__(kCellBlock, LSH_CELL_MINB)
#else
#define LSH_CELL_BOUNDS __launch_bounds__(kCellBlock)
#endif
// The reconstruction alone: 8 blocks of 256 (32 registers) hide its load
// latency best (2048^2 step: 1.940 ms at the compiler's 48 registers, 1.929
// at 6 blocks, 1.921 at 8).
#ifndef LSH_RECON_MINB
#define LSH_RECON_MINB 8
#endif
#if LSH_RECON_MINB > 1
#define LSH_RECON_BOUNDS __launch_bounds__(kCellBlock, LSH_RECON_MINB)
#else
#define LSH_RECON_BOUNDS __launch_bounds__(kCellBlock)
#endif
constexpr int kEdgeHBX = LSH_EDGE_H_BX, kEdgeHBY = kEdgeTile / LSH_EDGE_H_BX;
constexpr int kEdgeVBX = LSH_EDGE_V_BX, kEdgeVBY = kEdgeTile / LSH_EDGE_V_BX;
#ifndef LSH_CELL_BX
#define LSH_CELL_BX 16
#endif
constexpr int kCellBX = LSH_CELL_BX, kCellBY = kCellBlock / LSH_CELL_BX;

// ---------------------------------------------------------------- pass overlap
// The passes of a step run as consecutive kernels.  Each kernel's blocks end
// unevenly (wet tiles carry all the FP64 work), so a whole-grid boundary
// leaves SMs idle while the last wet tiles finish.  With `Dep` set, a pass is
// launched as a programmatic dependent of the one before it: its blocks may
// be scheduled once every block of that pass has started, and each of them
// waits only for the producer's row tiles that wrote the cell rows it reads.
// Every block of a pass adds 1 to its row tile's counter when its writes are
// done (a release add after the block's barrier); a consumer's thread 0 spins on the counters
// it needs with acquire loads, then the block synchronises.  The producer's
// blocks have all started before a consumer block can be scheduled, so a
// waiting block never keeps a producer block off the GPU.  Which rows a pass
// reads and writes:
//   horizontal edges, parity p, block row by: edge rows p + 2t,
//     t in [4 by, 4 by + 3] (kEdgeHBY = 4 lines), cells rows y - 1 and y;
//   vertical edges, block row by: cell rows [8 by, 8 by + 7];
//   cell kernels, block row by: cell rows [16 by, 16 by + 15] (the
//     reconstruction also reads the rows above and below).
// The counters are zeroed by the clock kernel at the end of the step.
enum DepKind : int { kDepH0 = 0, kDepH1 = 1, kDepV = 2, kDepCell = 3 };
struct Dep {
    const unsigned* wait = nullptr;  // producer pass's counters per block row (null: no wait)
    unsigned* done = nullptr;        // this pass's counters per block row (null: none)
    unsigned target = 0;             // producer blocks per block row (its gridDim.x)
    int kind = 0;                    // producer tiling (DepKind)
    int ntiles = 0;                  // producer block rows (its gridDim.y)
    int span = 0;                    // producer block height: cell rows, or edge lines for kDepH*
                                     // (0: the step kernels' blocks)
};

// Producer block rows that wrote cell rows [r0, r1].
__device__ __forceinline__ void dep_tiles(const Dep& d, int r0, int r1, int& t0, int& t1) {
    if (d.kind == kDepV) {
        const int b = d.span ? d.span : kEdgeVBY;
        t0 = r0 / b; t1 = r1 / b;
    } else if (d.kind == kDepCell) {
        const int b = d.span ? d.span : kCellBY;
        t0 = r0 / b; t1 = r1 / b;
    } else {
        // horizontal edge row y = p + 2 t writes cell rows y - 1 and y: the
        // edge rows touching [r0, r1] are [r0, r1 + 1]
        const int b = d.span ? d.span : kEdgeHBY;
        const int p = d.kind;
        const int lo = max(r0 - p + 1, 0) / 2, hi = (r1 + 1 - p) / 2;
        t0 = lo / b;
        t1 = max(hi, 0) / b;
    }
    t0 = max(t0, 0);
    t1 = min(t1, d.ntiles - 1);
}

// Start of a dependent pass's block: let the next pass be scheduled, then
// wait (thread 0, bounded) for the producer rows [r0, r1].  A wait that runs
// past ~2 s, or finds another block's wait already timed out, sets
// LSH_ERR_TIMEOUT in the time record and gives up (the step is then reported
// as failed and the clock kernel stops further steps).  Uniform per block.
__device__ __forceinline__ void dep_begin(const Dep& d, TimeRec* tm, int r0, int r1) {
    if (d.done) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!d.wait) return;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        int t0, t1;
        dep_tiles(d, r0, r1, t0, t1);
        const int tbit = 1 << LSH_ERR_TIMEOUT;
        volatile int* err = &tm->err;
        unsigned long long start = 0;
        for (int t = t0; t <= t1; ++t) {
            unsigned ns = 32;
            for (;;) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(d.wait + t) : "memory");
                if (v >= d.target) break;
                if (*err & tbit) { t = t1; break; }
                unsigned long long now;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                if (start == 0) start = now;
                else if (now - start > 2000000000ull) { atomicOr(&tm->err, tbit); t = t1; break; }
                __nanosleep(ns);
                if (ns < 1024) ns *= 2;
            }
        }
    }
    __syncthreads();
}

// End of a pass's block: its writes are done; count it in its block row.
// The barrier orders every thread's writes before thread 0's add, whose
// release semantics (cumulative, GPU scope) publish them with it.
__device__ __forceinline__ void dep_end(const Dep& d) {
    if (!d.done) return;
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(d.done + blockIdx.y) : "memory");
}

// Horizontal edges of parity `par`: x along threadIdx.x, edge rows par, par+2, ... along threadIdx.y / blocks.y.
// With `d` set the grid covers every line at once (gridDim.y * kEdgeHBY >= lines).
template <bool FIRST, int ORDER>
__global__ void LSH_EDGE_BOUNDS k_edges_h(KArgs a, int par, Dep d = Dep{}) {
    if (a.tm->done) return;
    const int nx = a.c.nx, ny = a.c.ny;
    if (d.done || d.wait) {
        const int y0 = par + 2 * (blockIdx.y * kEdgeHBY);
        dep_begin(d, a.tm, max(y0 - 1, 0), min(y0 + 2 * (kEdgeHBY - 1), ny - 1));
    }
    const int x = blockIdx.x * kEdgeHBX + threadIdx.x;
    if (x < nx) {
        const double dt = a.tm->dt;
        const int nlines = (ny - par) / 2 + 1;
        for (int t = blockIdx.y * kEdgeHBY + threadIdx.y; t < nlines; t += gridDim.y * kEdgeHBY)
            lsh::do_edge<0, FIRST, ORDER>(a, x, par + 2 * t, dt);
    }
    dep_end(d);
}

// Vertical edges of parity `par`: edge columns par, par+2, ... along threadIdx.x, rows along threadIdx.y / blocks.y.
template <int ORDER>
__global__ void LSH_EDGE_BOUNDS k_edges_v(KArgs a, int par, Dep d = Dep{}) {
    if (a.tm->done) return;
    const int nx = a.c.nx, ny = a.c.ny;
    if (d.done || d.wait) {
        const int y0 = blockIdx.y * kEdgeVBY;
        dep_begin(d, a.tm, y0, min(y0 + kEdgeVBY - 1, ny - 1));
    }
    const int t = blockIdx.x * kEdgeVBX + threadIdx.x;
    const int x = par + 2 * t;
    if (x <= nx) {
        const double dt = a.tm->dt;
        for (int y = blockIdx.y * kEdgeVBY + threadIdx.y; y < ny; y += gridDim.y * kEdgeVBY)
            lsh::do_edge<1, false, ORDER>(a, x, y, dt);
    }
    dep_end(d);
}

// Launch shapes of the two edge passes: one edge per thread.  (Blocks that
// walk several bands of lines measured slower, 2.19 ms per 2048^2 step with
// 2 bands against 1.98: a block holding several wet bands runs them one
// after the other.)
inline dim3 edge_block_h() { return dim3(kEdgeHBX, kEdgeHBY); }
inline dim3 edge_block_v() { return dim3(kEdgeVBX, kEdgeVBY); }
inline dim3 edge_grid_h(int nx, int ny, int par) {
    const int nlines = (ny - par) / 2 + 1;
    return dim3((nx + kEdgeHBX - 1) / kEdgeHBX, std::min((nlines + kEdgeHBY - 1) / kEdgeHBY, 65535));
}
inline dim3 edge_grid_v(int nx, int ny, int par) {
    const int nlines = (nx - par) / 2 + 1;
    return dim3((nlines + kEdgeVBX - 1) / kEdgeVBX, std::min((ny + kEdgeVBY - 1) / kEdgeVBY, 65535));
}

// Cell kernels: blocks of kCellBlock threads shaped LSH_CELL_BX x
// (kCellBlock / LSH_CELL_BX) over (x, y); LSH_CELL_BX = kCellBlock is one
// row segment per block.
inline dim3 cell_block() { return dim3(kCellBX, kCellBY); }
inline dim3 cell_grid(int nx, int ny) { return dim3((nx + kCellBX - 1) / kCellBX, (ny + kCellBY - 1) / kCellBY); }
// The cell of this thread, or -1 outside the grid.
__device__ __forceinline__ int cell_of_thread(int nx, int ny) {
    const int x = blockIdx.x * kCellBX + threadIdx.x, y = blockIdx.y * kCellBY + threadIdx.y;
    return (x < nx && y < ny) ? y * nx + x : -1;
}

// Second order: halved minmod slopes of (eta1, q1x, q1y, eta2, q2x, q2y, H)
// with a first-order fallback where a reconstructed depth would fall below
// kReconThin of the cell depth.
//
// (A variant that staged the block's 16 x 16 cells and a halo in shared
// memory, the depths first and the other variables only for tiles with a
// wet cell, measured 2.00 ms per 2048^2 step against 1.97 for this one: the
// stencil's neighbour loads already hit in L1.)
__global__ void LSH_RECON_BOUNDS k_recon(KArgs a, Dep d = Dep{}) {
    if (a.tm->done) return;
    if (d.done || d.wait) {
        const int y0 = blockIdx.y * kCellBY;
        dep_begin(d, a.tm, max(y0 - 1, 0), min(y0 + kCellBY, a.c.ny - 1));
    }
    const int id = cell_of_thread(a.c.nx, a.c.ny);
    if (id >= 0) lsh::recon_cell(a, id);
    dep_end(d);
}

// MODE 0: order 1, in place; per-cell dt min.  MODE 1: order 2 stage 1
// (W -> Wout), per-cell dt min.  MODE 2: order 2 stage 2, Wout = (Xavg + E(W)) / 2.
template <int MODE>
__global__ void LSH_CELL_BOUNDS k_volume(KArgs a, Dep d = Dep{}) {
    if (a.tm->done) return;
    if (d.done || d.wait) {
        const int y0 = blockIdx.y * kCellBY;
        dep_begin(d, a.tm, y0, min(y0 + kCellBY - 1, a.c.ny - 1));
    }
    const int id = cell_of_thread(a.c.nx, a.c.ny);
    const double dt = a.tm->dt;
    unsigned long long bits = kRateInitBits;
    if (id >= 0) bits = lsh::volume_cell<MODE>(a, id, dt);
    if (MODE != 2) lsh::block_max_bits<kCellBlock>(bits, &a.tm->rmax_bits);
    dep_end(d);
}


// Advance the device clock: t += dt, dt = min per-cell dt (ShallowWater.cu:436-442).
// One read and one write of the record: its loads do not wait for each other.
__device__ __forceinline__ void advance_clock(TimeRec* tm, double two_cfl) {
    TimeRec r = *tm;
    if (r.done) return;
    r.t += r.dt;
    r.steps += 1;
    r.dt = lsh::dt_of(r.rmax_bits, two_cfl);
    r.rmax_bits = kRateInitBits;
    if (r.t >= r.t_end) r.done = 1;
    if (r.dt_min > 0.0 && r.dt < r.dt_min) { r.err |= 1 << LSH_ERR_STALL; r.done = 1; }
    if (r.err) r.done = 1;
    *tm = r;
}

// The clock of a step of colour passes.  With `ctr`, its threads also zero the
// n_ctr pass-overlap counters of the step.
__global__ void k_advance(TimeRec* tm, double two_cfl, unsigned* ctr = nullptr, int n_ctr = 0) {
    for (int i = threadIdx.x; i < n_ctr; i += blockDim.x) ctr[i] = 0u;
    if (threadIdx.x == 0) advance_clock(tm, two_cfl);
}

// Initial-dt edge pass (procesarAristasDeltaTInicialGPU), writing acc[6]:
// the step's edge tiles (edge_block_h/v, edge_grid_h/v).
template <int DIR, bool FIRST>
__global__ void LSH_EDGE_BOUNDS k_init_wave(KArgs a, int par) {
    const int nx = a.c.nx, ny = a.c.ny;
    if (DIR == 0) {
        const int x = blockIdx.x * kEdgeHBX + threadIdx.x;
        if (x >= nx) return;
        const int nlines = (ny - par) / 2 + 1;
        for (int t = blockIdx.y * kEdgeHBY + threadIdx.y; t < nlines; t += gridDim.y * kEdgeHBY)
            lsh::init_wave_edge<0, FIRST>(a, x, par + 2 * t);
    } else {
        const int t = blockIdx.x * kEdgeVBX + threadIdx.x;
        const int x = par + 2 * t;
        if (x > nx) return;
        for (int y = blockIdx.y * kEdgeVBY + threadIdx.y; y < ny; y += gridDim.y * kEdgeVBY)
            lsh::init_wave_edge<1, FIRST>(a, x, y);
    }
}

// The four passes of the initial-dt wave sum, in the reference's order (the
// first writes acc[6], the others add).
inline void launch_init_wave(const KArgs& a, int nx, int ny, cudaStream_t s) {
    k_init_wave<0, true><<<edge_grid_h(nx, ny, 0), edge_block_h(), 0, s>>>(a, 0);
    k_init_wave<0, false><<<edge_grid_h(nx, ny, 1), edge_block_h(), 0, s>>>(a, 1);
    k_init_wave<1, false><<<edge_grid_v(nx, ny, 0), edge_block_v(), 0, s>>>(a, 0);
    k_init_wave<1, false><<<edge_grid_v(nx, ny, 1), edge_block_v(), 0, s>>>(a, 1);
}

// Per-cell rate of the initial wave pass (obtenerDeltaTVolumenesGPU) and its max.
__global__ void __launch_bounds__(kCellBlock) k_cell_dt(KArgs a) {
    const int id = cell_of_thread(a.c.nx, a.c.ny);
    unsigned long long bits = kRateInitBits;
    if (id >= 0) bits = lsh::init_cell_rate(a, id);
    lsh::block_max_bits<kCellBlock>(bits, &a.tm->rmax_bits);
}

__global__ void k_init_finish(TimeRec* tm, double two_cfl) {
    tm->dt = lsh::dt_of(tm->rmax_bits, two_cfl);
    tm->rmax_bits = kRateInitBits;
    tm->t = 0.0;
    tm->steps = 0;
    tm->done = 0;
    tm->err = 0;
}

// eta1 max initial value h1 + h2 - H, time 0 (Problema.cxx:542-546)
__global__ void __launch_bounds__(kCellBlock) k_init_eta(KArgs a) {
    const int id = cell_of_thread(a.c.nx, a.c.ny);
    if (id < 0) return;
    a.eta_max[id] = a.W[0][id] + a.W[3][id] - a.W[6][id];
    a.eta_time[id] = 0.0;
}

// ---------------------------------------------------------------- flux pass and cell update
//
// The single-grid step: per stage the reconstruction (second order), one flux
// pass over all edges and the cells' update (lsh_passes.cuh), on tiles of 16
// columns by 4 rows.  A tile is two warps of the cell passes (two rows each)
// and four of the flux pass (two rows each of its horizontal edges, between its
// rows and the rows above them, and of its vertical ones); tiles past the last
// column and row hold the outer edges.  Against the four colour passes and the
// volume kernel, an edge's faces are loaded once instead of an accumulator pass
// per colour, and a stage's chain is three passes instead of six.
//
// Tiles that nothing can reach in a step are left out: the clock kernel lists,
// per tile row, the tiles with a busy tile (TileMap::busy) at most two away.
// A tile is busy when, in the step's last update of either stage, one of its
// cells' input or output state was not all +0 or one of their edges was not
// dry.  A stage carries state one tile further at most (an edge's flux, or a
// limiter, reads two cells), so a tile left out holds +0 in both state buffers
// before and after the step, its edges' kinds are dry, its slopes are zero and
// flagged so (the reconstruction ran on it, and its neighbours, empty), and its
// maximum of eta1 has seen the empty state.  On the 2048^2 fjord, 14% wet, the
// blocks of dry tiles took 490 of the step's 1295 us (first order: 453 us with
// every tile, 250 with the lists); after a new state every tile is busy.
//
// The flux pass is launched as four consecutive ranges of its blocks, the four
// edge launches a step has always had (lsh_profile_step,
// lsh_get_launch_count); nothing orders them, so a small grid's run side by
// side and a large one's follow each other as one grid's blocks would.  One
// range instead takes a step of 24 x 17 cells from 42.5 to 39.7 us, of a 64^2
// fjord at first order from 19.9 to 16.4, at second from 131.5 to 128.9, and
// makes no difference from 200^2 up.
// Overlap as above (programmatic dependent launches), by tile rows: a block
// adds 1 to its tile row's counter, and waits for its producer's listed tiles
// in the rows around its own: the flux pass for the row itself and the one
// above (it reads the cells above its first row), the update and the
// reconstruction for one row on each side (the limiter's recursion reads edges
// and depths up to two cells away, the stencil one cell).
constexpr int kTileX = 16, kTileY = 4;
constexpr int kCellWarps = 2, kFluxWarps = 4, kFluxParts = 4;  // warps per tile, and launches of the flux pass
// Resident blocks per SM that the kernels are compiled for, [large grid, small
// grid].  A large grid wants the warps: flux pass in blocks of 128 threads, 4 /
// 6 / 8 / 10 (128 / 80 / 64 / 48 registers) ran the 1024^2 wet shelf's step in
// 916 / 852 / 872 / 975 us; the update in blocks of 64, 8 / 12 / 16 / 20: 975 /
// 902 / 876 / 886; the reconstruction 24 / 32: no difference.  A small one has
// one or two warps per SM, and wants no spills: 2, 4 and 8 blocks took the 64^2
// fjord's step from 179 to 160 us, the 200^2 shelf's from 72 to 66.
constexpr int kFluxBlocks[2] = {6, 2}, kUpdateBlocks[2] = {16, 4}, kSlopesBlocks[2] = {32, 8};
// Tiles up to which a grid is small.  All-wet shelves, large against small
// kernels, us per step: 400^2 (2626 tiles) 232 / 206 at second order, 96 / 96 at
// first; 512^2 (4257) 271 / 283 and 113 / 120.  Grids with dry land gain longer
// (fjord 523^2 234 / 219, 800^2 263 / 247), but only the step knows how much is dry.
#ifndef LSH_SMALL_TILES
#define LSH_SMALL_TILES 4000
#endif
constexpr unsigned kSmallTiles = LSH_SMALL_TILES;

inline __host__ __device__ int tiles_x(int nx) { return (nx + 1 + kTileX - 1) / kTileX; }
inline __host__ __device__ int tiles_y(int ny) { return (ny + 1 + kTileY - 1) / kTileY; }

struct TileMap {
    int ntx, nty;
    int* list;               // per tile row: the listed tiles' columns, ascending
    int* count;              // per tile row: how many (null: every tile, and no busy flags)
    // per stage (one plane serves for both at order 1) and tile, one byte for
    // each of its warps of the cell passes
    unsigned short* busy[2];
};

struct TileDep {
    const unsigned* wait = nullptr;  // producer's counters per tile row (null: no wait)
    unsigned* done = nullptr;        // this pass's (null: none)
    unsigned per = 0;                // producer blocks per listed tile
};

// The tile of unit `u` (warp number of a pass with `warps` per tile, first
// warp of the block): false when its row lists fewer.
__device__ __forceinline__ bool tile_of(const TileMap& m, unsigned u, int warps, int& tx, int& ty) {
    const unsigned t = u / (unsigned)warps;
    ty = (int)(t / (unsigned)m.ntx);
    const int k = (int)(t - (unsigned)ty * (unsigned)m.ntx);
    tx = k;
    if (ty >= m.nty) return false;
    if (!m.count) return true;
    if (k >= m.count[ty]) return false;
    tx = m.list[(size_t)ty * m.ntx + k];
    return true;
}

// Start of a block on tile row t: lets the next pass be scheduled, then waits
// for the producer's blocks on tile rows [t - 1, t + after] (one thread per
// row; bounded as dep_begin).
__device__ __forceinline__ void tile_begin(const TileDep& d, const TileMap& m, TimeRec* tm, int t, int after) {
    if (d.done) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!d.wait) return;
    const int r = max(t - 1, 0) + (int)threadIdx.x;
    if (r <= min(t + after, m.nty - 1)) {
        const unsigned target = d.per * (unsigned)(m.count ? m.count[r] : m.ntx);
        const int tbit = 1 << LSH_ERR_TIMEOUT;
        volatile int* err = &tm->err;
        unsigned long long start = 0;
        unsigned ns = 32;
        for (;;) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(d.wait + r) : "memory");
            if (v >= target) break;
            if (*err & tbit) break;
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (start == 0) start = now;
            else if (now - start > 2000000000ull) { atomicOr(&tm->err, tbit); break; }
            __nanosleep(ns);
            if (ns < 256) ns *= 2;
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void tile_end(const TileDep& d, int t) {
    if (!d.done) return;
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(d.done + t) : "memory");
}

// The warp's largest rate into *target, which only grows: most warps find it
// larger already and leave it.
__device__ __forceinline__ void warp_max_bits(unsigned long long v, unsigned long long* target) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_down_sync(0xffffffffu, v, o);
        v = (w > v) ? w : v;
    }
    if ((threadIdx.x & 31) == 0 && v > *(volatile unsigned long long*)target) atomicMax(target, v);
}

// Blocks first, first + 1, ... of the flux pass: one to four warps of a tile each.
template <int ORDER, bool SMALL>
__global__ void __launch_bounds__(32 * kFluxWarps, kFluxBlocks[SMALL])
    k_flux(const __grid_constant__ KArgs a, const __grid_constant__ TileMap m, TileDep d, unsigned first) {
    if (a.tm->done) return;
    const unsigned bw = blockDim.x / 32, u0 = (first + blockIdx.x) * bw;
    int tx, ty;
    if (!tile_of(m, u0, kFluxWarps, tx, ty)) return;
    tile_begin(d, m, a.tm, ty, 0);
    const int nx = a.c.nx, ny = a.c.ny;
    const int q = (int)((u0 + threadIdx.x / 32) % kFluxWarps), lane = threadIdx.x & 31;
    const int x = tx * kTileX + (lane & (kTileX - 1)), y = ty * kTileY + (q & 1) * 2 + lane / kTileX;
    const double dt = a.tm->dt;
    const int dir = q >> 1;
    if (dir ? (x <= nx && y < ny) : (x < nx && y <= ny)) lsh::flux_edge<ORDER>(a, dir, x, y, dt);
    tile_end(d, ty);
}

// The cell of a thread of the cell passes, or false.
__device__ __forceinline__ bool tile_cell(const KArgs& a, int tx, int ty, unsigned u0, int& half, int& i, int& j) {
    const int lane = threadIdx.x & 31;
    half = (int)((u0 + threadIdx.x / 32) % kCellWarps);
    i = tx * kTileX + (lane & (kTileX - 1));
    j = ty * kTileY + 2 * half + lane / kTileX;
    return i < a.c.nx && j < a.c.ny;
}

template <int MODE, bool SMALL>
__global__ void __launch_bounds__(32 * kCellWarps, kUpdateBlocks[SMALL])
    k_update(const __grid_constant__ KArgs a, const __grid_constant__ TileMap m, TileDep d) {
    if (a.tm->done) return;
    const unsigned u0 = blockIdx.x * (blockDim.x / 32);
    int tx, ty, half, i, j;
    if (!tile_of(m, u0, kCellWarps, tx, ty)) return;
    tile_begin(d, m, a.tm, ty, 1);
    const bool in = tile_cell(a, tx, ty, u0, half, i, j);
    unsigned long long bits = kRateInitBits;
    bool busy = false;
    if (in) bits = lsh::update_cell<MODE>(a, i, j, a.tm->dt, busy);
    __syncwarp();
    busy = __any_sync(0xffffffffu, busy);
    if (m.count && (threadIdx.x & 31) == 0)
        reinterpret_cast<unsigned char*>(m.busy[MODE == 1 ? 1 : 0] + (size_t)ty * m.ntx + tx)[half] = busy;
    if (MODE != 2) warp_max_bits(bits, &a.tm->rmax_bits);
    tile_end(d, ty);
}

template <bool SMALL>
__global__ void __launch_bounds__(32 * kCellWarps, kSlopesBlocks[SMALL])
    k_slopes(const __grid_constant__ KArgs a, const __grid_constant__ TileMap m, TileDep d) {
    if (a.tm->done) return;
    const unsigned u0 = blockIdx.x * (blockDim.x / 32);
    int tx, ty, half, i, j;
    if (!tile_of(m, u0, kCellWarps, tx, ty)) return;
    tile_begin(d, m, a.tm, ty, 1);
    if (tile_cell(a, tx, ty, u0, half, i, j)) {
        const int id = j * a.c.nx + i;
        if (SMALL) lsh::recon_cell_loaded(a, id);
        else lsh::recon_cell(a, id);
    }
    tile_end(d, ty);
}

// The clock of a step of the flux pass and cell update: t and dt advance
// (k_advance), the n_ctr pass counters go back to zero, and the next step's
// tiles are listed, one warp per tile row.  `tm` null: the list alone.
__global__ void __launch_bounds__(256) k_clock(TimeRec* tm, double two_cfl, unsigned* ctr, int n_ctr, TileMap m) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_ctr; i += gridDim.x * blockDim.x) ctr[i] = 0u;
    const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x / 32);
    for (int r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; r < m.nty; r += warps) {
        int n = 0;
        for (int c0 = 0; c0 < m.ntx; c0 += 32) {
            const int c = c0 + lane;
            unsigned v = 0;
            // the window's 50 loads at once (a loop over its part inside the
            // grid waited for each: 6 us on any grid)
#pragma unroll
            for (int dy = -2; dy <= 2; ++dy)
#pragma unroll
                for (int dx = -2; dx <= 2; ++dx) {
                    const int y = min(max(r + dy, 0), m.nty - 1), x = min(max(c + dx, 0), m.ntx - 1);
                    const size_t t = (size_t)y * m.ntx + x;
                    v |= (unsigned)m.busy[0][t] | (unsigned)m.busy[1][t];
                }
            if (c >= m.ntx) v = 0;
            const unsigned on = __ballot_sync(0xffffffffu, v != 0);
            if (v) m.list[(size_t)r * m.ntx + n + __popc(on & ((1u << lane) - 1u))] = c;
            n += __popc(on);
        }
        if (lane == 0) m.count[r] = n;
    }
    if (tm && blockIdx.x == 0 && threadIdx.x == 0) advance_clock(tm, two_cfl);
}

// ---------------------------------------------------------------- overlapped launches

// Counters per pass of a step when the passes can overlap: one per block row
// of the edge and cell kernels, rounded up; 0 when a grid would need more
// block rows than a launch holds (the passes then run fully ordered).
inline int dep_stride_for(int nx, int ny) {
    const int rows = std::max({(int)edge_grid_h(nx, ny, 0).y, (int)edge_grid_v(nx, ny, 0).y, (int)cell_grid(nx, ny).y});
    const bool fits = (long long)((ny / 2 + 1 + kEdgeHBY - 1) / kEdgeHBY) <= 65535 &&
                      (long long)((ny + kEdgeVBY - 1) / kEdgeVBY) <= 65535;
    return fits ? ((rows + 63) & ~63) : 0;
}

// Launch `kernel` on `s`; `dependent`: as a programmatic dependent of the
// kernel before it on the stream (it may start once that kernel's blocks
// have all started; its blocks order themselves through the pass counters).
template <class... P, class... A>
inline void launch_pass(bool dependent, dim3 grid, dim3 block, cudaStream_t s, void (*kernel)(P...), A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = dependent ? at : nullptr;
    cfg.numAttrs = dependent ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// The passes of one stage with overlap on an nx x ny grid: `prev` is the
// producer of the first edge pass (the reconstruction at order 2, nothing
// at order 1: then h0 is the step's first kernel); counters seg[0..4 st)
// for h0, h1, v0, v1 and the volume update (`last`: the volume's counters
// are not needed).  MODE < 0: no volume update (the stage ends after its
// edge passes).  Returns the producer description for a pass that reads
// this stage's volume output.
// snaps (may be null): for the adjoint's recomputation, the three passes
// after the first copy the partial sums they read to snaps[0], [1], [2].
template <int ORDER, int MODE>
inline Dep enqueue_stage_overlap(int nx, int ny, const KArgs& a, cudaStream_t s, Dep prev, unsigned* seg, int st,
                                 bool last, double* const (*snaps)[2] = nullptr) {
    KArgs as[3] = {a, a, a};
    if (snaps)
        for (int i = 0; i < 3; ++i) { as[i].snap[0] = snaps[i][0]; as[i].snap[1] = snaps[i][1]; }
    const dim3 gh0 = edge_grid_h(nx, ny, 0), gh1 = edge_grid_h(nx, ny, 1);
    const dim3 gv0 = edge_grid_v(nx, ny, 0), gv1 = edge_grid_v(nx, ny, 1), gc = cell_grid(nx, ny);
    Dep d0 = prev;
    d0.done = seg;
    launch_pass(prev.wait != nullptr, gh0, edge_block_h(), s, k_edges_h<true, ORDER>, a, 0, d0);
    Dep d1;
    d1.wait = seg; d1.done = seg + st; d1.target = gh0.x; d1.kind = kDepH0; d1.ntiles = (int)gh0.y;
    launch_pass(true, gh1, edge_block_h(), s, k_edges_h<false, ORDER>, as[0], 1, d1);
    Dep d2;
    d2.wait = seg + st; d2.done = seg + 2 * st; d2.target = gh1.x; d2.kind = kDepH1; d2.ntiles = (int)gh1.y;
    launch_pass(true, gv0, edge_block_v(), s, k_edges_v<ORDER>, as[1], 0, d2);
    Dep d3;
    d3.wait = seg + 2 * st; d3.done = (MODE < 0 && last) ? nullptr : seg + 3 * st; d3.target = gv0.x;
    d3.kind = kDepV; d3.ntiles = (int)gv0.y;
    launch_pass(true, gv1, edge_block_v(), s, k_edges_v<ORDER>, as[2], 1, d3);
    Dep next;
    if (MODE < 0) {
        next.wait = seg + 3 * st; next.target = gv1.x; next.kind = kDepV; next.ntiles = (int)gv1.y;
        return next;
    }
    Dep d4;
    d4.wait = seg + 3 * st; d4.done = last ? nullptr : seg + 4 * st; d4.target = gv1.x; d4.kind = kDepV;
    d4.ntiles = (int)gv1.y;
    launch_pass(true, gc, cell_block(), s, k_volume<(MODE < 0 ? 0 : MODE)>, a, d4);
    next.wait = seg + 4 * st; next.target = gc.x; next.kind = kDepCell; next.ntiles = (int)gc.y;
    return next;
}

// One whole time step with overlapped passes, counters c[0 .. 13 st):
// order 1 from a1 (in place); order 2 stage 1 from a1 (X -> Y), stage 2 from
// a2 (Y -> X with the average).  The clock kernel closes the step as a
// plain launch and zeroes the counters.  Returns the kernels launched.
inline int enqueue_step_overlap(int nx, int ny, int order, const KArgs& a1, const KArgs& a2, unsigned* c, int st,
                                TimeRec* tm, double two_cfl, cudaStream_t s) {
    const int nk = (order == 1) ? 6 : 13;
    if (order == 1) {
        enqueue_stage_overlap<1, 0>(nx, ny, a1, s, Dep{}, c, st, true);
    } else {
        const dim3 nbc = cell_grid(nx, ny);
        Dep r1;
        r1.done = c;
        launch_pass(false, nbc, cell_block(), s, k_recon, a1, r1);
        Dep pr;
        pr.wait = c; pr.target = nbc.x; pr.kind = kDepCell; pr.ntiles = (int)nbc.y;
        const Dep v1 = enqueue_stage_overlap<2, 1>(nx, ny, a1, s, pr, c + st, st, false);
        Dep r2 = v1;
        r2.done = c + 6 * st;
        launch_pass(true, nbc, cell_block(), s, k_recon, a2, r2);
        Dep pr2;
        pr2.wait = c + 6 * st; pr2.target = nbc.x; pr2.kind = kDepCell; pr2.ntiles = (int)nbc.y;
        enqueue_stage_overlap<2, 2>(nx, ny, a2, s, pr2, c + 7 * st, st, true);
    }
    // a plain launch: waits for the whole step, then zeroes the counters
    k_advance<<<1, 256, 0, s>>>(tm, two_cfl, c, nk * st);
    return nk;
}

// What the flux pass and cell update hold beside the state: edge planes and
// kinds, the cells' marks, the tile lists.  layout() places it in `mem` (256-byte
// aligned; null: the size alone) and returns the bytes; marks and busy flags lie
// next to each other in [clear, clear + clear_bytes).
struct FluxMem {
    lsh::EdgeBuf eb{};
    TileMap map{};
    unsigned char* clear = nullptr;
    size_t clear_bytes = 0;
    size_t layout(unsigned char* mem, int nx, int ny, int order) {
        const size_t tiles = size_t(tiles_x(nx)) * tiles_y(ny);
        size_t at = 0;
        auto take = [&](size_t bytes) { unsigned char* q = mem + at; at += (bytes + 255) & ~size_t(255); return q; };
        map.ntx = tiles_x(nx);
        map.nty = tiles_y(ny);
        map.list = reinterpret_cast<int*>(take(tiles * sizeof(int)));
        map.count = reinterpret_cast<int*>(take(map.nty * sizeof(int)));
        at += lsh::edge_layout(eb, mem + at, nx, ny);
        clear = reinterpret_cast<unsigned char*>(eb.mark[0]);
        for (int l = 0; l < order; ++l) map.busy[l] = reinterpret_cast<unsigned short*>(take(tiles * sizeof(unsigned short)));
        if (order == 1) map.busy[1] = map.busy[0];  // k_clock reads both
        clear_bytes = size_t(mem + at - clear);
        return at;
    }
};

inline unsigned clock_blocks(const TileMap& m) { return (unsigned)std::min((m.nty + 7) / 8, 1024); }

// A new state: every tile is busy (any byte but 0 says so).  Marks of an old
// run cost an evaluation at most.
inline void launch_all_busy(const TileMap& m, cudaStream_t s) {
    for (int l = 0; l < 2; ++l)
        (void)cudaMemsetAsync(m.busy[l], 1, size_t(m.ntx) * m.nty * sizeof(unsigned short), s);
    k_clock<<<clock_blocks(m), 256, 0, s>>>(nullptr, 0.0, nullptr, 0, m);
}

// Passes of a step before the clock, and the counters of each: one per tile
// row, rounded up.
inline int flux_step_passes(int order) { return (order == 1) ? 2 : 6; }
inline int flux_dep_stride(int ny) { return (tiles_y(ny) + 63) & ~63; }

// Launches a step's passes in order, each behind the one before through the
// counters `c` (null: one after the other); `mark` is called after each launch.
template <bool SMALL, class Mark>
struct FluxPasses {
    static constexpr unsigned cw = SMALL ? 1 : kCellWarps, fw = SMALL ? 1 : kFluxWarps;  // warps per block
    const TileMap& m;
    unsigned* c;
    const int st, last;
    const unsigned tiles;
    cudaStream_t s;
    Mark& mark;
    TileDep d;  // the pass before as producer, this pass's own counters
    int pass = 0;
    FluxPasses(const TileMap& map, unsigned* ctr, const lsh::Consts& k, cudaStream_t stream, Mark& mk)
        : m(map), c(ctr), st(flux_dep_stride(k.ny)), last(flux_step_passes(k.order) - 1),
          tiles(unsigned(map.ntx) * unsigned(map.nty)), s(stream), mark(mk) {}
    int counters() const { return c ? pass * st : 0; }
    template <class Kernel, class... X>
    void cells(Kernel kernel, const KArgs& a, const X&... x) {
        begin();
        launch_pass(d.wait != nullptr, dim3(tiles * (kCellWarps / cw)), dim3(32 * cw), s, kernel, a, m, d, x...);
        mark();
        end(kCellWarps / cw);
    }
    template <class Kernel>
    void flux(Kernel kernel, const KArgs& a) {
        begin();
        const unsigned n = tiles * (kFluxWarps / fw);
        for (int q = 0; q < kFluxParts; ++q) {
            const unsigned b0 = unsigned((unsigned long long)n * q / kFluxParts);
            const unsigned b1 = unsigned((unsigned long long)n * (q + 1) / kFluxParts);
            launch_pass(c && (q > 0 || d.wait), dim3(b1 - b0), dim3(32 * fw), s, kernel, a, m, d, b0);
            mark();
        }
        end(kFluxWarps / fw);
    }
private:
    void begin() { if (c) d.done = (pass < last) ? c + pass * st : nullptr; }
    void end(unsigned per) {
        if (c) { d.wait = d.done; d.per = per; }
        ++pass;
    }
};

// One time step: a1 the stage 1 arguments (order 1: in place), a2 stage 2's
// (with their edge buffers).  `c` (may be null: full-grid launches one after
// the other): flux_dep_stride counters for each pass, which the clock kernel
// zeroes.  `mark` is called after each launch.  Returns the kernels launched.
// A small grid takes blocks of one warp, so that every SM's FP64 unit has
// work; a large one a tile per block.
template <bool SMALL, class Mark>
inline int enqueue_flux_step_as(const KArgs& a1, const KArgs& a2, const TileMap& m, unsigned* c, double two_cfl,
                                cudaStream_t s, Mark&& mark) {
    const int order = a1.c.order;
    FluxPasses<SMALL, Mark> p(m, c, a1.c, s, mark);
    if (order == 1) {
        p.flux(k_flux<1, SMALL>, a1);
        p.cells(k_update<0, SMALL>, a1);
    } else {
        p.cells(k_slopes<SMALL>, a1);
        p.flux(k_flux<2, SMALL>, a1);
        p.cells(k_update<1, SMALL>, a1);
        p.cells(k_slopes<SMALL>, a2);
        p.flux(k_flux<2, SMALL>, a2);
        p.cells(k_update<2, SMALL>, a2);
    }
    // a plain launch: waits for the whole step, then zeroes the counters
    if (m.count) k_clock<<<clock_blocks(m), 256, 0, s>>>(a1.tm, two_cfl, c, p.counters(), m);
    else k_advance<<<1, 256, 0, s>>>(a1.tm, two_cfl, c, p.counters());
    mark();
    return (order == 1) ? 6 : 13;
}
template <class Mark>
inline int enqueue_flux_step(const KArgs& a1, const KArgs& a2, const TileMap& m, unsigned* c, double two_cfl,
                             cudaStream_t s, Mark&& mark) {
    return (unsigned(m.ntx) * unsigned(m.nty) <= kSmallTiles)
               ? enqueue_flux_step_as<true>(a1, a2, m, c, two_cfl, s, mark)
               : enqueue_flux_step_as<false>(a1, a2, m, c, two_cfl, s, mark);
}

}  // namespace
