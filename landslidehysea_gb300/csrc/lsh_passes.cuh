// lsh_passes.cuh -- per-edge and per-cell device functions of the step,
// shared by the single-grid kernels (lsh_core.cu) and the batched ensemble
// kernels (lsh_batch.cu), so both evaluate exactly the same arithmetic.
#pragma once

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#endif

#include "../../include/lsh.h"
#include "lsh_scheme.cuh"

namespace lsh {

constexpr unsigned long long kRateInitBits = 0ULL;  // +0.0
constexpr int kEdgeBlock = 128;
constexpr int kCellBlock = 256;
constexpr double kReconThin = 0.5;  // second order: least face depth / cell depth

// Sticky error bit: an atomic OR on the device, a plain OR in host code.
LSH_HD void err_or(int* word, int bit) {
#if defined(__CUDA_ARCH__)
    atomicOr(word, bit);
#else
    *word |= bit;
#endif
}

// Per-edge results of a stage's flux pass (flux_edge), read by its cells'
// update (update_cell).  Horizontal edge row y, column x: index y nx + x;
// vertical edge column x, row y: y (nx + 1) + x.  Eleven planes each: m[0..2],
// p[0..1], wave, and with a granular layer m[3..5], p[2..3] (EdgeRaw).
constexpr int kEdgePlanes = 11;
enum EdgeKind : unsigned char { kEdgeDry = 0, kEdgeSingle = 1, kEdgeBoth = 2 };
struct EdgeBuf {
    double* q[2];             // horizontal, vertical
    size_t plane[2];          // doubles between planes
    unsigned char* kind[2];   // EdgeKind of each edge
    // per cell and layer: the stage number (2 steps + stage, 32 bits) in which
    // one of its edges may empty the layer, so that the limiter has to be
    // evaluated around it; an old number that comes round again costs that
    // evaluation only
    unsigned* mark[2];
    unsigned stage;           // 0 or 1, the stage of the step
    const double* depth[2];   // the cells' depths h1, h2 as the limiter reads them
    double* depth_out[2];     // where the flux pass leaves them (null: they stay in W)
};

// An EdgeBuf's arrays placed in `mem` (256-byte aligned; null: the size alone),
// the marks last; the bytes they take.
inline size_t edge_layout(EdgeBuf& eb, unsigned char* mem, int nx, int ny) {
    const size_t N = size_t(nx) * ny;
    size_t at = 0;
    auto take = [&](size_t bytes) { unsigned char* q = mem + at; at += (bytes + 255) & ~size_t(255); return q; };
    const size_t n[2] = {(N + nx + 31) & ~size_t(31), (N + ny + 31) & ~size_t(31)};
    for (int d = 0; d < 2; ++d) {
        eb.plane[d] = n[d];
        eb.q[d] = reinterpret_cast<double*>(take(kEdgePlanes * n[d] * sizeof(double)));
        eb.kind[d] = take(n[d]);
    }
    for (int l = 0; l < 2; ++l) eb.mark[l] = reinterpret_cast<unsigned*>(take(N * sizeof(unsigned)));
    return at;
}

struct KArgs {
    Consts c;
    Geo geo;
    const double* W[7];   // input state (face values are W + slopes at order 2)
    double* Wout[6];      // output state of the volume kernel
    const double* Xavg[6];  // order 2, stage 2: the step's initial state for the average
    double* acc[7];
    const double* sx[7];
    const double* sy[7];
    double* sxw[7];       // reconstruction kernel outputs
    double* syw[7];
    double* eta_max;
    double* eta_time;
    TimeRec* tm;
    unsigned char* szero;  // per cell: 1 when the stored slopes are all zero (may be null)
    // the adjoint's recomputation (null otherwise): an edge pass after the
    // first copies acc[0], acc[3] of its non-dry edges' cells, as the pass
    // before left them, to snap[0], snap[1] -- the partial sums its limiter
    // reads, which the reverse sweep needs at exactly those cells
    double* snap[2];
    // and the cell update copies the partial sums of each cell with a wet edge
    // after the first three colours to part[colour]
    double* part[3][2];
    unsigned* tape;       // the recomputation's reconstruction branch tape (null otherwise)
    EdgeBuf eb;           // the flux pass's results (q[0] null: the colour passes run instead)
};

// Depths of a face (first order: the cell's; second order: reconstructed).
template <int ORDER>
LSH_HD void face_depths(const KArgs& a, int id, int side, double& h1, double& h2) {
    h1 = a.W[0][id];
    h2 = a.W[3][id];
    if (ORDER == 2) {
        const double* const* s = (side < 2) ? a.sx : a.sy;
        const double d1 = s[0][id] - s[3][id], d2 = s[3][id] + s[6][id];
        // side & 1: the +slope face (E or N); the sign is a sign-bit flip
        const bool neg = !(side & 1);
        h1 = h1 + lshm::neg_if(d1, neg);
        h2 = h2 + lshm::neg_if(d2, neg);
    }
}

// The rest of a face in the edge frame.  DIR 1 (vertical edge, normal
// (sg, 0)): qn = sg qx, qt = sg qy; DIR 0 (horizontal, normal (0, sg)):
// qn = sg qy, qt = -sg qx (Arista_kernel.cu:363-371, 509-525) -- selections
// and negations, no FP64 arithmetic.
template <int DIR, int ORDER>
LSH_HD void face_rest(const KArgs& a, int id, int side, bool pos_normal, lsh::Face& f) {
    double qx1 = a.W[1][id], qy1 = a.W[2][id], qx2 = a.W[4][id], qy2 = a.W[5][id], H = a.W[6][id];
    if (ORDER == 2) {
        const double* const* s = (side < 2) ? a.sx : a.sy;
        using lshm::neg_if;
        const bool neg = !(side & 1);
        qx1 = qx1 + neg_if(s[1][id], neg);
        qy1 = qy1 + neg_if(s[2][id], neg);
        qx2 = qx2 + neg_if(s[4][id], neg);
        qy2 = qy2 + neg_if(s[5][id], neg);
        H = H + neg_if(s[6][id], neg);
    }
    using lshm::neg_if;
    if (DIR == 1) {
        f.qn1 = neg_if(qx1, !pos_normal); f.qt1 = neg_if(qy1, !pos_normal);
        f.qn2 = neg_if(qx2, !pos_normal); f.qt2 = neg_if(qy2, !pos_normal);
    } else {
        f.qn1 = neg_if(qy1, !pos_normal); f.qt1 = neg_if(qx1, pos_normal);
        f.qn2 = neg_if(qy2, !pos_normal); f.qt2 = neg_if(qx2, pos_normal);
    }
    f.H = H;
}

// The accumulator update of one edge: subtract the first KL flux terms of
// each cell (KL = 3: layer 1 only, the layer-2 terms being zeros) and add the
// wave term.  The first pass of a stage writes instead of accumulating:
// every cell meets exactly one hor-even edge.
template <bool FIRST, int KL>
LSH_HD void scatter_edge(const KArgs& a, int id0, int id1, bool interior, const double d0[6], const double d1[6],
                         double wave) {
    if (FIRST) {
#pragma unroll
        for (int k = 0; k < 6; ++k) a.acc[k][id0] = (k < KL) ? lsh::minus0(d0[k]) : 0.0;
        a.acc[6][id0] = lsh::plus0(wave);
        if (interior) {
#pragma unroll
            for (int k = 0; k < 6; ++k) a.acc[k][id1] = (k < KL) ? lsh::minus0(d1[k]) : 0.0;
            a.acc[6][id1] = lsh::plus0(wave);
        }
    } else {
#pragma unroll
        for (int k = 0; k < KL; ++k) a.acc[k][id0] -= d0[k];
        a.acc[6][id0] += wave;
        if (interior) {
#pragma unroll
            for (int k = 0; k < KL; ++k) a.acc[k][id1] -= d1[k];
            a.acc[6][id1] += wave;
        }
    }
}

// The positivity limiter's inputs of one edge, loaded from the state and the
// accumulators where the limiter reads them: cell areas by row, cell depths
// h1, h2, and the depths' partial accumulators (zero in the first pass); a
// boundary edge's outer side mirrors the cell's area with zero depths.
template <bool FIRST>
struct LazyPos {
    const KArgs& a;
    int id0, id1, row0, row1;
    LSH_HD double area(int side) const { return a.geo.area[(side && id1 >= 0) ? row1 : row0]; }
    LSH_HD double inv_area(int side) const { return a.geo.inv_area[(side && id1 >= 0) ? row1 : row0]; }
    LSH_HD double hc(int side, int layer) const {
        if (side && id1 < 0) return 0.0;
        return a.W[layer ? 3 : 0][side ? id1 : id0];
    }
    LSH_HD double acch(int side, int layer) const {
        if (FIRST || (side && id1 < 0)) return 0.0;
        return a.acc[layer ? 3 : 0][side ? id1 : id0];
    }
};

// The sides of one edge.
// dir 0: horizontal edge row y between rows y-1 and y, column x.
// dir 1: vertical edge column x between columns x-1 and x, row y.
struct EdgeSides { int id0, id1, side0, row0, row1; bool interior, pos_normal; double bor, len; };
template <int DIR>
LSH_HD EdgeSides edge_sides(const KArgs& a, int x, int y) {
    const int nx = a.c.nx, ny = a.c.ny;
    EdgeSides s;
    s.id1 = -1; s.row1 = 0; s.bor = 0.0; s.pos_normal = true;
    if (DIR == 0) {
        s.len = a.geo.len_h[y];
        if (y == 0) { s.id0 = x; s.row0 = 0; s.pos_normal = false; s.bor = a.c.borde_sup; s.side0 = 2; }
        else if (y == ny) { s.id0 = (ny - 1) * nx + x; s.row0 = ny - 1; s.bor = a.c.borde_inf; s.side0 = 3; }
        else { s.id0 = (y - 1) * nx + x; s.id1 = s.id0 + nx; s.row0 = y - 1; s.row1 = y; s.side0 = 3; }
    } else {
        s.len = a.geo.len_v[y];
        s.row0 = s.row1 = y;
        if (x == 0) { s.id0 = y * nx; s.pos_normal = false; s.bor = a.c.borde_izq; s.side0 = 0; }
        else if (x == nx) { s.id0 = y * nx + nx - 1; s.bor = a.c.borde_der; s.side0 = 1; }
        else { s.id0 = y * nx + x - 1; s.id1 = s.id0 + 1; s.side0 = 1; }
    }
    s.interior = (s.id1 >= 0);
    return s;
}

// The face depths of an edge; false for a dry edge, which adds nothing.
template <int DIR, int ORDER>
LSH_HD bool edge_wet(const KArgs& a, const EdgeSides& s, Face& A, Face& B) {
    using lsh::is_zero;
    const int side1 = (DIR == 0) ? 2 : 0;
    // Both cells empty (h1 = h2 = 0) with zero stored slopes (second order:
    // the slope-zero flags): every face depth is exactly 0, so the dry test
    // below would find the edge dry.  Integer tests only, and no slope loads:
    // most edges of a flooded-coast grid are such edges.
    if (ORDER == 1 || a.szero) {
        bool empty = is_zero(a.W[0][s.id0]) && is_zero(a.W[3][s.id0]) && (ORDER == 1 || a.szero[s.id0]);
        if (empty && s.interior)
            empty = is_zero(a.W[0][s.id1]) && is_zero(a.W[3][s.id1]) && (ORDER == 1 || a.szero[s.id1]);
        if (empty) return false;
    }
    face_depths<ORDER>(a, s.id0, s.side0, A.h1, A.h2);
    if (s.interior) face_depths<ORDER>(a, s.id1, side1, B.h1, B.h2);
    else { B.h1 = A.h1; B.h2 = A.h2; }
    // dry edge (Arista_kernel.cu:397)
    return !(lshm::lt_pos(lsh::half(A.h1 + B.h1), lsh::kEps) && lshm::lt_pos(lsh::half(A.h2 + B.h2), lsh::kEps));
}

// The rest of a wet edge's faces (the ghost's at a boundary).
template <int DIR, int ORDER>
LSH_HD void edge_faces(const KArgs& a, const EdgeSides& s, Face& A, Face& B) {
    face_rest<DIR, ORDER>(a, s.id0, s.side0, s.pos_normal, A);
    if (s.interior) {
        face_rest<DIR, ORDER>(a, s.id1, (DIR == 0) ? 2 : 0, s.pos_normal, B);
    } else {
        // ghost: the cell's face with the normal discharges times the boundary factor
        B = A;
        B.qn1 = A.qn1 * s.bor;
        B.qn2 = A.qn2 * s.bor;
    }
}

// One edge of a colour pass: gather both sides, evaluate, scatter to the
// accumulators.
template <int DIR, bool FIRST, int ORDER>
LSH_HD void do_edge(const KArgs& a, int x, int y, double dt) {
    const EdgeSides s = edge_sides<DIR>(a, x, y);
    const int id0 = s.id0, id1 = s.id1, row0 = s.row0, row1 = s.row1;
    const bool pos_normal = s.pos_normal;
    lsh::EdgeIn e;
    e.len = s.len;
    e.interior = s.interior;
    if (!edge_wet<DIR, ORDER>(a, s, e.A, e.B)) {
        // nothing to add; the first pass still writes the zeros that
        // initialise the accumulators
        if (FIRST) {
#pragma unroll
            for (int k = 0; k < 7; ++k) a.acc[k][id0] = 0.0;
            if (e.interior) {
#pragma unroll
                for (int k = 0; k < 7; ++k) a.acc[k][id1] = 0.0;
            }
        }
        return;
    }
    if (!FIRST && a.snap[0]) {
        a.snap[0][id0] = a.acc[0][id0];
        a.snap[1][id0] = a.acc[3][id0];
        if (e.interior) {
            a.snap[0][id1] = a.acc[0][id1];
            a.snap[1][id1] = a.acc[3][id1];
        }
    }
    edge_faces<DIR, ORDER>(a, s, e.A, e.B);
    // the limiter's inputs are loaded where it reads them (LazyPos), not kept
    // live through the flux computation
    const LazyPos<FIRST> pos{a, id0, id1, row0, row1};
    lsh::EdgeOut o;
    using lsh::is_zero;
    const bool single = is_zero(e.A.h2) && is_zero(e.B.h2) && is_zero(e.A.qn2) && is_zero(e.B.qn2);
    if (single)
        lsh::edge_flux<false>(e, dt, a.c, o, pos);
    else
        lsh::edge_flux<true>(e, dt, a.c, o, pos);
    // back to x/y: DIR 1: (qx, qy) = sg (fn, ft); DIR 0: qx = -sg ft, qy = sg fn
    double d0[6], d1[6];
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const int k = 3 * l;
        d0[k] = o.m[k];
        d1[k] = o.p[k];
        using lshm::neg_if;
        if (DIR == 1) {
            d0[k + 1] = neg_if(o.m[k + 1], !pos_normal);
            d0[k + 2] = neg_if(o.m[k + 2], !pos_normal);
            d1[k + 1] = neg_if(o.p[k + 1], !pos_normal);
            d1[k + 2] = neg_if(o.p[k + 2], !pos_normal);
        } else {
            d0[k + 1] = neg_if(o.m[k + 2], pos_normal);
            d0[k + 2] = neg_if(o.m[k + 1], !pos_normal);
            d1[k + 1] = neg_if(o.p[k + 2], pos_normal);
            d1[k + 2] = neg_if(o.p[k + 1], !pos_normal);
        }
    }
    // A single-layer edge's layer-2 terms are zeros, and an accumulator never
    // holds -0 (the first pass writes 0 - d, which is +0 for d = +-0, and
    // x - y is -0 only for x = -0): subtracting them leaves the accumulator's
    // bits as they are.  A warp whose edges are all single-layer skips that
    // arithmetic and its loads, and the first pass stores the +0 it would
    // compute.
    if (warp_all(single)) scatter_edge<FIRST, 3>(a, id0, id1, e.interior, d0, d1, o.wave);
    else scatter_edge<FIRST, 6>(a, id0, id1, e.interior, d0, d1, o.wave);
}

// minmod: the operand of smaller magnitude when both are nonzero with one
// sign (b on a tie), else 0 -- on the bit patterns (integer pipe); for
// operands that are not NaN the same as the compares
//   a > 0 && b > 0 ? (a < b ? a : b) : a < 0 && b < 0 ? (a > b ? a : b) : 0
// `choice`: 0 for neither, 1 for a, 2 for b.
LSH_HD double minmod_choice(double a, double b, unsigned& choice) {
    // (through halves: on the plain bits the compiler finds a == 0 and b == 0)
    uint32_t alo, ahi, blo, bhi;
    lshm::halves(a, alo, ahi);
    lshm::halves(b, blo, bhi);
    const uint32_t am = ahi & 0x7fffffffu, bm = bhi & 0x7fffffffu;
    const bool nonzero = (am | alo) != 0u && (bm | blo) != 0u;
    const bool same = (int32_t)(ahi ^ bhi) >= 0;
    const bool first = (((uint64_t)am << 32) | alo) < (((uint64_t)bm << 32) | blo);
    choice = (nonzero && same) ? (first ? 1u : 2u) : 0u;
    if (!(nonzero && same)) return 0.0;
    return first ? a : b;
}
LSH_HD double minmod(double a, double b) {
    unsigned choice;
    return minmod_choice(a, b, choice);
}

// The branch tape of one cell's reconstruction, which its adjoint replays: for
// variable k and direction d (0 x, 1 y) bits 2 (7 d + k) .. +1 hold the minmod
// choice; kTapeFlat: zero slopes (a reconstructed depth below kReconThin of the
// cell's, or the dry shortcut).
constexpr unsigned kTapeFlat = 1u << 28;

// One cell of the second-order reconstruction, its inputs read through an
// accessor w(k, di, dj) = W[k] at cell (i + di, j + dj): global memory
// (recon_cell) or a shared-memory tile (k_recon).  Neighbours are read only
// inside the grid.  Returns the cell's branch tape.
template <class Acc>
LSH_HD unsigned recon_cell_from(const KArgs& a, int id, int i, int j, const Acc& w) {
    const int nx = a.c.nx, ny = a.c.ny;
    // A cell whose own and 4 neighbours' depths are all zero only meets dry
    // edges (a dry cell's faces always have zero depth: any nonzero depth
    // slope would make one face negative and trigger the fallback), so its
    // slopes are never read: store zeros and skip the FP64 work.
    {
        using lsh::is_zero;
        bool dry = is_zero(w(0, 0, 0)) && is_zero(w(3, 0, 0));
        if (dry && i > 0) dry = is_zero(w(0, -1, 0)) && is_zero(w(3, -1, 0));
        if (dry && i < nx - 1) dry = is_zero(w(0, 1, 0)) && is_zero(w(3, 1, 0));
        if (dry && j > 0) dry = is_zero(w(0, 0, -1)) && is_zero(w(3, 0, -1));
        if (dry && j < ny - 1) dry = is_zero(w(0, 0, 1)) && is_zero(w(3, 0, 1));
        if (dry) {
            // zero slopes; a cell whose stored slopes are already zero (and stays
            // dry, the common case far from the flow) skips the 14 stores
            if (a.szero && a.szero[id]) return kTapeFlat;
#pragma unroll
            for (int k = 0; k < 7; ++k) { a.sxw[k][id] = 0.0; a.syw[k][id] = 0.0; }
            if (a.szero) a.szero[id] = 1;
            return kTapeFlat;
        }
    }
    const bool inx = (i > 0 && i < nx - 1), iny = (j > 0 && j < ny - 1);
    // halved minmod slopes of variable k, rv(di, dj)
    unsigned tape = 0;
    auto slopes = [&](int k, auto rv, double& x, double& y) {
        const double pc = rv(0, 0);
        unsigned cx = 0, cy = 0;
        x = inx ? lsh::half(minmod_choice(pc - rv(-1, 0), rv(1, 0) - pc, cx)) : 0.0;
        y = iny ? lsh::half(minmod_choice(pc - rv(0, -1), rv(0, 1) - pc, cy)) : 0.0;
        tape |= (cx << (2 * k)) | (cy << (2 * (7 + k)));
    };
    // No granular layer anywhere in the stencil (h2 = q2 = 0 at the cell and
    // the neighbours it reads): eta1 = (h1 + 0) - H is h1 - H (but for the sign
    // of a zero, which minmod does not see); eta2 = 0 - H, whose differences
    // are exactly the negated differences of H, so its slope is the negated H
    // slope, or +0 where minmod gives 0; the q2 slopes are minmod's 0, so +0;
    // and the fallback's h2 tests, 0 +- 0 against 0.5 * 0, never fire.  A warp
    // whose cells all qualify skips that FP64 work and gets the same bits: 23
    // FP64 instructions instead of 56.
    bool one = true;
    {
        using lsh::is_zero;
        auto nolayer = [&](int di, int dj) {
            return is_zero(w(3, di, dj)) && is_zero(w(4, di, dj)) && is_zero(w(5, di, dj));
        };
        one = nolayer(0, 0);
        if (one && i > 0) one = nolayer(-1, 0);
        if (one && i < nx - 1) one = nolayer(1, 0);
        if (one && j > 0) one = nolayer(0, -1);
        if (one && j < ny - 1) one = nolayer(0, 1);
    }
    double sx[7], sy[7];
    const double h1 = w(0, 0, 0);
    bool bad = false;
    slopes(1, [&](int di, int dj) { return w(1, di, dj); }, sx[1], sy[1]);
    slopes(2, [&](int di, int dj) { return w(2, di, dj); }, sx[2], sy[2]);
    slopes(6, [&](int di, int dj) { return w(6, di, dj); }, sx[6], sy[6]);
    const bool fast = warp_all(one);
    if (fast) {
        slopes(0, [&](int di, int dj) { return w(0, di, dj) - w(6, di, dj); }, sx[0], sy[0]);
        sx[3] = lsh::is_zero(sx[6]) ? 0.0 : lshm::neg_if(sx[6], true);
        sy[3] = lsh::is_zero(sy[6]) ? 0.0 : lshm::neg_if(sy[6], true);
        sx[4] = sx[5] = sy[4] = sy[5] = 0.0;
        tape |= ((tape >> 12) & 3u) << 6 | ((tape >> 26) & 3u) << 20;  // eta2's choices are H's
    } else {
        lshm::rare();
        slopes(0, [&](int di, int dj) { return (w(0, di, dj) + w(3, di, dj)) - w(6, di, dj); }, sx[0], sy[0]);
        slopes(3, [&](int di, int dj) { return w(3, di, dj) - w(6, di, dj); }, sx[3], sy[3]);
        slopes(4, [&](int di, int dj) { return w(4, di, dj); }, sx[4], sy[4]);
        slopes(5, [&](int di, int dj) { return w(5, di, dj); }, sx[5], sy[5]);
    }
    // first order where a reconstructed depth would fall below kReconThin of
    // the cell's: a thin face with a finite discharge has an unbounded
    // velocity, whose wave speed would collapse dt (the compares on the
    // integer pipe).  Where every depth slope is at most a quarter of the
    // depth (by the exponents) no face of layer 1 falls below it.
    const double dh1x = sx[0] - sx[3], dh1y = sy[0] - sy[3];
    using lshm::okey;
    // (a depth of -0 or below fails the sign test: its pattern less two
    // exponents would wrap round to a large one)
    const int64_t quarter = (int64_t)(lshm::bits_of(h1) - ((uint64_t)2 << 52));
    const bool deep = lsh::gt0(h1) && quarter > ((int64_t)1 << 52) &&
                      (int64_t)lshm::bits_of(lshm::abs_bits(dh1x)) <= quarter &&
                      (int64_t)lshm::bits_of(lshm::abs_bits(dh1y)) <= quarter;
    if (!warp_all(deep)) {
        lshm::rare();
        static_assert(kReconThin == 0.5, "half() below gives kReconThin h");
        const int64_t k1 = okey(lsh::half(h1));
        bad = okey(h1 + dh1x) < k1 || okey(h1 - dh1x) < k1 || okey(h1 + dh1y) < k1 || okey(h1 - dh1y) < k1;
    }
    if (!fast) {
        lshm::rare();
        const double h2 = w(3, 0, 0);
        const double dh2x = sx[3] + sx[6], dh2y = sy[3] + sy[6];
        const int64_t k2 = okey(lsh::half(h2));
        bad = bad || okey(h2 + dh2x) < k2 || okey(h2 - dh2x) < k2 || okey(h2 + dh2y) < k2 || okey(h2 - dh2y) < k2;
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        a.sxw[k][id] = bad ? 0.0 : sx[k];
        a.syw[k][id] = bad ? 0.0 : sy[k];
    }
    if (a.szero) a.szero[id] = 0;  // conservative: only the dry path marks zeros
    return bad ? kTapeFlat : tape;
}

// One cell of the second-order reconstruction from global memory.
LSH_HD unsigned recon_cell(const KArgs& a, int id) {
    const int nx = a.c.nx;
    const int j = id / nx, i = id - j * nx;
    return recon_cell_from(a, id, i, j, [&](int k, int di, int dj) -> double { return a.W[k][id + di + dj * nx]; });
}

// The same with its 35 values loaded at once (a neighbour outside the grid is
// the cell itself, and not read): for a small grid, whose warps cannot hide
// loads that wait for the tests of others (64^2: 15.5 -> 10.5 us a launch, 156
// -> 141 us a step; it needs 84 registers, so a large grid keeps the chain).
LSH_HD unsigned recon_cell_loaded(const KArgs& a, int id) {
    const int nx = a.c.nx, ny = a.c.ny;
    const int j = id / nx, i = id - j * nx;
    const int at[5] = {id, id - (i > 0), id + (i < nx - 1), id - (j > 0 ? nx : 0), id + (j < ny - 1 ? nx : 0)};
    double v[7][5];
#pragma unroll
    for (int k = 0; k < 7; ++k)
#pragma unroll
        for (int n = 0; n < 5; ++n) v[k][n] = a.W[k][at[n]];
    return recon_cell_from(a, id, i, j, [&](int k, int di, int dj) -> double {
        return v[k][di < 0 ? 1 : di > 0 ? 2 : dj < 0 ? 3 : dj > 0 ? 4 : 0];
    });
}

#if defined(__CUDACC__)
// Block max of the per-cell rates (non-negative doubles order like their bit
// patterns), then one 64-bit atomicMax per block.
template <int BLOCK>
__device__ __forceinline__ void block_max_bits(unsigned long long v, unsigned long long* target) {
    __shared__ unsigned long long red[BLOCK / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_down_sync(0xffffffffu, v, o);
        v = (w > v) ? w : v;
    }
    // linear thread index (blocks may be 2-D; warps are x-fastest)
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = (lane < BLOCK / 32) ? red[lane] : kRateInitBits;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long w = __shfl_down_sync(0xffffffffu, v, o);
            v = (w > v) ? w : v;
        }
        if (lane == 0) atomicMax(target, v);
    }
}
#endif

// One cell of the Euler-stage update given its state wo and accumulators acc
// (changed); returns the bits of the cell's acc_w / area for the dt reduction.
// MODE 0: order 1, in place.  MODE 1: order 2 stage 1 (W -> Wout).
// MODE 2: order 2 stage 2, Wout = (Xavg + E(W)) / 2.
// `busy` (may be null): set where the input or the output state is not all +0.
// PESO1: the caller knows that peso is 1.
template <int MODE, bool PESO1 = false>
LSH_HD unsigned long long volume_finish(const KArgs& a, int id, int j, double dt, const double wo[6], double acc[7],
                                        bool* busy = nullptr) {
    double w[6], rate;
    if (MODE != 2 && a.c.track_eta) {
        // actualizarEta1MaximaGPU (Volumen_kernel.cu:182-213): state before the step
        const double v = wo[0] - a.W[6][id];
        if (lshm::lt(a.eta_max[id], v)) { a.eta_max[id] = v; a.eta_time[id] = a.tm->t; }
    }
    // a dry, still cell with nothing flowing in maps to itself through the
    // whole update (dt contribution 1e30; its second-order pressure
    // integral is g*0*... = 0): skip the FP64 work
    bool still = true;
#pragma unroll
    for (int k = 0; k < 6; ++k) still &= lsh::is_zero(wo[k]);
#pragma unroll
    for (int k = 0; k < 7; ++k) still &= lsh::is_zero(acc[k]);
    if (still) {
#pragma unroll
        for (int k = 0; k < 6; ++k) w[k] = wo[k];
        rate = 0.0;
    } else {
        // The cell has no granular layer and receives none: wo[3..5] zero and
        // acc[3..5] +0 (bit patterns).  With finite slopes its layer-2
        // pressure term is g (+-0) (finite) = +-0, leaving acc[4], acc[5] at
        // +0, and volume_update<true> gives the general path's bits.  A warp
        // whose cells all qualify takes that path (if-converted per-lane
        // selects would still issue the FP64 work).
        using lsh::is_zero;
        bool one = is_zero(wo[3]) && is_zero(wo[4]) && is_zero(wo[5]) && lshm::bits_of(acc[3]) == 0 &&
                   lshm::bits_of(acc[4]) == 0 && lshm::bits_of(acc[5]) == 0;
        auto times_peso = [&](double v) { return PESO1 ? v : a.c.peso * v; };
        double s0x = 0.0, s3x = 0.0, s0y = 0.0, s3y = 0.0;
        if (a.c.order == 2) {
            s0x = a.sx[0][id]; s3x = a.sx[3][id]; s0y = a.sy[0][id]; s3y = a.sy[3][id];
            one = one && !lsh::is_bad(s0x) && !lsh::is_bad(s3x) && !lsh::is_bad(s0y) && !lsh::is_bad(s3y);
        }
        if (warp_all(one)) {
            if (a.c.order == 2) {
                const double gh1 = a.c.g * wo[0];
                const double wx = a.geo.wx[j], wy = a.geo.wy[j];
                acc[1] -= times_peso((gh1 * lsh::twice(s0x)) * wx);
                acc[2] -= times_peso((gh1 * lsh::twice(s0y)) * wy);
            }
            lsh::volume_update<true>(wo, acc, w, rate, a.geo.inv_area[j], a.geo.tanR[j], dt, a.c);
        } else {
            if (a.c.order == 2) {
                // cell-midpoint integral of g h d(eta) over the reconstructed cell
                const double gh1 = a.c.g * wo[0], gh2 = a.c.g * wo[3];
                const double e1x = lsh::twice(s0x), e2x = lsh::twice(s3x);
                const double e1y = lsh::twice(s0y), e2y = lsh::twice(s3y);
                const double wx = a.geo.wx[j], wy = a.geo.wy[j];
                acc[1] -= times_peso((gh1 * e1x) * wx);
                acc[4] -= times_peso((gh2 * lsh::fmad(a.c.omr, e2x, a.c.r * e1x)) * wx);
                acc[2] -= times_peso((gh1 * e1y) * wy);
                acc[5] -= times_peso((gh2 * lsh::fmad(a.c.omr, e2y, a.c.r * e1y)) * wy);
            }
            lsh::volume_update(wo, acc, w, rate, a.geo.inv_area[j], a.geo.tanR[j], dt, a.c);
        }
    }
    // A still cell whose output is the very bits already stored where it goes
    // skips the stores: order 1 updates in place (w == wo); stage 2 writes back
    // into the step's initial state, and the average of two equal zeros is
    // that zero.
    bool keep = false;
    if (MODE == 0 && still) {
        keep = true;
#pragma unroll
        for (int k = 0; k < 6; ++k) keep &= (a.Wout[k] == a.W[k]);
    }
    if (MODE == 2) {
        // the TVD-RK2 average 0.5 (x + w).  Where both terms are zero (every dry
        // cell) it is the AND of their patterns (+0 unless both are -0: the sum
        // of opposite zeros is +0).  A warp whose cells all have only zero terms
        // takes the AND as a whole: a per-variable select is if-converted, and
        // its predicated-off FP64 instructions still hold the FP64 pipe.
        double x[6];
        bool z[2] = {true, true};  // per layer
        keep = still;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            x[k] = a.Xavg[k][id];
            z[k / 3] &= lsh::is_zero(x[k]) && lsh::is_zero(w[k]);
            keep &= (a.Wout[k] == a.Xavg[k]) && (lshm::bits_of(x[k]) == lshm::bits_of(w[k]));
        }
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            if (warp_all(z[l])) {
#pragma unroll
                for (int k = 3 * l; k < 3 * l + 3; ++k) w[k] = lshm::from_bits(lshm::bits_of(x[k]) & lshm::bits_of(w[k]));
            } else {
                lshm::rare();
#pragma unroll
                for (int k = 3 * l; k < 3 * l + 3; ++k) w[k] = lsh::half(x[k] + w[k]);
            }
        }
    }
    if (busy) {
        uint64_t u = 0;
#pragma unroll
        for (int k = 0; k < 6; ++k) u |= lshm::bits_of(wo[k]) | lshm::bits_of(w[k]);
        *busy |= (u != 0);
    }
    if (keep) return (unsigned long long)lshm::bits_of(rate);
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 6; ++k) { a.Wout[k][id] = w[k]; bad |= lsh::is_bad(w[k]); }
    if (bad) err_or(&a.tm->err, 1 << LSH_ERR_NUMERIC);
    return (unsigned long long)lshm::bits_of(rate);
}

// One cell of the Euler-stage update after the colour passes.
template <int MODE>
LSH_HD unsigned long long volume_cell(const KArgs& a, int id, double dt) {
    double wo[6], acc[7];
#pragma unroll
    for (int k = 0; k < 6; ++k) wo[k] = a.W[k][id];
#pragma unroll
    for (int k = 0; k < 7; ++k) acc[k] = a.acc[k][id];
    return volume_finish<MODE>(a, id, id / a.c.nx, dt, wo, acc);
}

// ---------------------------------------------------------------- flux pass and cell update
//
// An edge's flux needs nothing that another edge computes: only the
// positivity limiter reads the partial sums of the edges before it in the
// reference's colour order (even rows, odd rows, even columns, odd columns;
// ShallowWater.cu:391-427).  So one pass evaluates every edge at once, without
// the limiter (flux_edge), and the cells' update (update_cell) sums each cell's
// four edges in colour order, which gives the colour passes' bits.  Where the
// limiter cannot act (far_from_empty on every side of the edge's two cells) the
// sums are all there is; around a marked cell the limiter's factors are
// evaluated as the colour passes would, edge by edge (partial_mass).
//
// That an unmarked cell is never limited needs its partial sums not to fall
// below what its own edges take, so the limiter's factors must not be
// negative: a limited edge takes at most peso / beta of a cell's content, and
// flux_fits asks for peso = 1 and beta >= 1 (the reference's values, both 1).
// The colour passes take the other parameters.
inline bool flux_fits(const lsh_params& p) { return p.peso == 1.0 && p.beta >= 1.0; }

LSH_HD unsigned stage_mark(const KArgs& a) { return 2u * (unsigned)a.tm->steps + a.eb.stage + 1u; }

// x + y is exactly 0 (opposite values, or zeros), by the bits
LSH_HD bool cancel(double x, double y) {
    return lshm::bits_of(x) == (lshm::bits_of(y) ^ ~lshm::kMag) || (is_zero(x) && is_zero(y));
}

// A cell's state and, at second order, its slopes across an edge.
template <int ORDER>
struct CellSide { double w[7], s[ORDER == 2 ? 7 : 1]; bool zero; };
template <int DIR, int ORDER>
LSH_HD void load_side(const KArgs& a, int id, CellSide<ORDER>& c) {
#pragma unroll
    for (int k = 0; k < 7; ++k) c.w[k] = a.W[k][id];
    c.zero = true;
    if constexpr (ORDER == 2) {
        c.zero = a.szero[id] != 0;
#pragma unroll
        for (int k = 0; k < 7; ++k) c.s[k] = (DIR == 0 ? a.sy : a.sx)[k][id];
    }
}

// The face of a cell toward its +slope side (`neg`: the other one) in the edge
// frame (face_depths, face_rest).  BARE: layer 1 alone, zeros for layer 2.
template <int ORDER>
LSH_HD double side_depth(const CellSide<ORDER>& c, bool neg, int layer) {
    double h = c.w[3 * layer];
    if constexpr (ORDER == 2) h = h + lshm::neg_if(layer ? c.s[3] + c.s[6] : c.s[0] - c.s[3], neg);
    return h;
}
template <int DIR, int ORDER, bool BARE>
LSH_HD void side_rest(const CellSide<ORDER>& c, bool neg, bool pos_normal, Face& f) {
    using lshm::neg_if;
    double q[4] = {c.w[1], c.w[2], c.w[4], c.w[5]};
    f.H = c.w[6];
    if constexpr (ORDER == 2) {
        q[0] = q[0] + neg_if(c.s[1], neg);
        q[1] = q[1] + neg_if(c.s[2], neg);
        if (!BARE) {
            q[2] = q[2] + neg_if(c.s[4], neg);
            q[3] = q[3] + neg_if(c.s[5], neg);
        }
        f.H = f.H + neg_if(c.s[6], neg);
    }
    f.qn1 = neg_if(q[1 - DIR], !pos_normal);
    f.qt1 = neg_if(q[DIR], DIR == 1 ? !pos_normal : pos_normal);
    if (BARE) {
        f.h2 = f.qn2 = f.qt2 = 0.0;
    } else {
        f.qn2 = neg_if(q[3 - DIR], !pos_normal);
        f.qt2 = neg_if(q[2 + DIR], DIR == 1 ? !pos_normal : pos_normal);
    }
}

// No granular layer at the cell and its faces: h2, q2 and, at second order,
// what their slopes add (eta2's and H's slopes cancel) are zeros.
template <int ORDER>
LSH_HD bool bare_side(const CellSide<ORDER>& c) {
    bool b = is_zero(c.w[3]) & is_zero(c.w[4]) & is_zero(c.w[5]);
    if constexpr (ORDER == 2) b = b & is_zero(c.s[4]) & is_zero(c.s[5]) & cancel(c.s[3], c.s[6]);
    return b;
}

// The faces of an edge and its kind, as edge_wet and edge_faces give them.
// Both cells' values are loaded at once, whatever the edge turns out to be: a
// load behind a test of another costs an L2 round trip (700 cycles), which a
// small grid's lone warps cannot hide.  A warp whose edges all lie between cells
// without a granular layer takes their layer-1 faces alone: 10 FP64
// instructions instead of 24 at second order.
template <int DIR, int ORDER>
LSH_HD EdgeKind flux_faces(const KArgs& a, const EdgeSides& s, Face& A, Face& B) {
    CellSide<ORDER> ca, cb;
    load_side<DIR, ORDER>(a, s.id0, ca);
    load_side<DIR, ORDER>(a, s.interior ? s.id1 : s.id0, cb);
    // both cells empty with zero slopes (edge_wet)
    const bool empty = is_zero(ca.w[0]) & is_zero(ca.w[3]) & ca.zero & is_zero(cb.w[0]) & is_zero(cb.w[3]) & cb.zero;
    if (empty) return kEdgeDry;
    const bool na = !(s.side0 & 1);
    const bool bare = bare_side<ORDER>(ca) & bare_side<ORDER>(cb);
    if (warp_all(bare)) {
        A.h1 = side_depth<ORDER>(ca, na, 0);
        B.h1 = A.h1;
        if (s.interior) { lshm::rare(); B.h1 = side_depth<ORDER>(cb, true, 0); }
        if (lshm::lt_pos(half(A.h1 + B.h1), kEps)) return kEdgeDry;
        side_rest<DIR, ORDER, true>(ca, na, s.pos_normal, A);
        if (s.interior) {
            lshm::rare();
            side_rest<DIR, ORDER, true>(cb, true, s.pos_normal, B);
        } else {
            lshm::rare();
            B = A;
            B.qn1 = A.qn1 * s.bor;
        }
        return kEdgeSingle;
    }
    A.h1 = side_depth<ORDER>(ca, na, 0);
    A.h2 = side_depth<ORDER>(ca, na, 1);
    B.h1 = s.interior ? side_depth<ORDER>(cb, true, 0) : A.h1;
    B.h2 = s.interior ? side_depth<ORDER>(cb, true, 1) : A.h2;
    // dry edge (Arista_kernel.cu:397)
    if (lshm::lt_pos(half(A.h1 + B.h1), kEps) && lshm::lt_pos(half(A.h2 + B.h2), kEps)) return kEdgeDry;
    side_rest<DIR, ORDER, false>(ca, na, s.pos_normal, A);
    if (s.interior) {
        side_rest<DIR, ORDER, false>(cb, true, s.pos_normal, B);
    } else {
        // ghost: the cell's face with the normal discharges times the boundary factor
        B = A;
        B.qn1 = A.qn1 * s.bor;
        B.qn2 = A.qn2 * s.bor;
    }
    return (is_zero(A.h2) && is_zero(B.h2) && is_zero(A.qn2) && is_zero(B.qn2)) ? kEdgeSingle : kEdgeBoth;
}

// One edge of the flux pass: dir 0 horizontal, 1 vertical.  The direction is a
// value so that both share one copy of the flux's code (two filled the
// instruction cache: 5.7 of 41 stall cycles per issue waited for it).
template <int ORDER>
LSH_HD void flux_edge(const KArgs& a, int dir, int x, int y, double dt) {
    if (dir == 0 && a.eb.depth_out[0] && y < a.c.ny) {
        // order 1 updates in place: the limiter reads this copy, since a
        // neighbour may already hold its new depth
        const int id = y * a.c.nx + x;
        a.eb.depth_out[0][id] = a.W[0][id];
        a.eb.depth_out[1][id] = a.W[3][id];
    }
    EdgeSides s;
    Face A, B;
    EdgeKind kind;
    if (dir) {
        s = edge_sides<1>(a, x, y);
        kind = flux_faces<1, ORDER>(a, s, A, B);
    } else {
        s = edge_sides<0>(a, x, y);
        kind = flux_faces<0, ORDER>(a, s, A, B);
    }
    const size_t e = (size_t)y * (a.c.nx + dir) + x, np = dir ? a.eb.plane[1] : a.eb.plane[0];
    (dir ? a.eb.kind[1] : a.eb.kind[0])[e] = kind;
    if (kind == kEdgeDry) return;
    const bool single = (kind == kEdgeSingle);
    EdgeRaw r;
    if (single) edge_raw1(A, B, s.len, a.c, r);
    else edge_raw2(A, B, s.len, dt, a.c, r);
    double* const q = (dir ? a.eb.q[1] : a.eb.q[0]) + e;
    q[0] = r.m[0]; q[np] = r.m[1]; q[2 * np] = r.m[2];
    q[3 * np] = r.p[0]; q[4 * np] = r.p[1]; q[5 * np] = r.wave;
    if (!single) {
        q[6 * np] = r.m[3]; q[7 * np] = r.m[4]; q[8 * np] = r.m[5];
        q[9 * np] = r.p[2]; q[10 * np] = r.p[3];
    }
    const double scale = a.c.beta;  // >= peso = 1 (flux_fits)
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        if (l == 1 && single) break;
        const double m = l ? r.m[3] : r.m[0], p = l ? r.p[2] : r.p[0];
        if (gt0(m) && !far_from_empty(m, a.W[3 * l][s.id0], a.geo.area[s.row0], dt, scale))
            a.eb.mark[l][s.id0] = stage_mark(a);
        if (s.interior && gt0(p) && !far_from_empty(p, a.W[3 * l][s.id1], a.geo.area[s.row1], dt, scale))
            a.eb.mark[l][s.id1] = stage_mark(a);
    }
}

#if defined(__CUDACC__)
#define LSH_RECURSE static __host__ __device__ __noinline__
#else
#define LSH_RECURSE static
#endif

// The colour-C edge of cell (i, j): its direction, place, and whether the cell
// is its second one.
struct CellEdge { int x, y; bool second, boundary; };
template <int C>
LSH_HD CellEdge cell_edge(int i, int j) {
    CellEdge e;
    if (C < 2) {
        e.x = i;
        e.y = ((j & 1) == C) ? j : j + 1;
        e.second = (e.y == j) && j > 0;
        e.boundary = (e.y == 0);
    } else {
        e.y = j;
        e.x = ((i & 1) == C - 2) ? i : i + 1;
        e.second = (e.x == i) && i > 0;
        e.boundary = (e.x == 0);
    }
    return e;
}

// Whether all that the four edges take from layer `layer` of cell (i, j) in dt,
// with the limiter's beta and eps, is less than its content: then, as for an
// unmarked cell, the limiter's test is false on each of its sides.
LSH_HD bool holds_all(const KArgs& a, int i, int j, int layer, double dt) {
    double out = 0.0;
    auto edge = [&](int dir, size_t at, bool second) {
        const double v = a.eb.q[dir][at + (layer ? (second ? 9 : 6) : (second ? 3 : 0)) * a.eb.plane[dir]];
        const bool loses = a.eb.kind[dir][at] > layer && gt0(v);
        out = out + (loses ? v : 0.0);
    };
    const int nx = a.c.nx;
    edge(0, (size_t)j * nx + i, j > 0);
    edge(0, (size_t)(j + 1) * nx + i, false);
    edge(1, (size_t)j * (nx + 1) + i, i > 0);
    edge(1, (size_t)j * (nx + 1) + i + 1, false);
    const double need = dt * fmad(a.c.beta, out, 4.0 * kEps);
    return lt_pos(need, (a.eb.depth[layer][(size_t)j * nx + i] * a.geo.area[j]) * (1.0 - 0x1p-30));
}

// Whether the limiter may act on an edge of cell (i, j): one of the edges' cells
// is marked and may be emptied.
LSH_RECURSE bool limit_near(const KArgs& a, int i, int j, int layer, double dt) {
    const unsigned now = stage_mark(a);
    const unsigned* mk = a.eb.mark[layer];
    const int nx = a.c.nx, ny = a.c.ny;
    bool near = false;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int ci = i + (k == 1) - (k == 2), cj = j + (k == 3) - (k == 4);
        if (near || ci < 0 || ci >= nx || cj < 0 || cj >= ny) continue;
        if (mk[(size_t)cj * nx + ci] == now && !holds_all(a, ci, cj, layer, dt)) near = true;
    }
    return near;
}

// The limiter's factors on the edges of cell (i, j) before colour C, in colour
// order (factors[0 .. C), may be null), and the mass terms that those edges
// leave in the cell's accumulator of `layer` -- what the colour passes' limiter
// reads.  An edge with neither cell marked has factor 1.  The other cell's
// partial sum comes from the same function with the edge's colour, so at most
// 2^C - 1 edges are visited, and few where marked cells are.
template <int C>
LSH_RECURSE double partial_mass(const KArgs& a, int i, int j, int layer, double dt, double* factors);
template <>
LSH_HD double partial_mass<0>(const KArgs&, int, int, int, double, double*) { return 0.0; }

// One colour of partial_mass: the mass the colour-P edge takes from the cell
// whose partial sum before it is acc.
template <int P>
LSH_HD double limited_mass(const KArgs& a, int i, int j, int layer, double dt, double acc, double* factor) {
    constexpr int DIR = P / 2;
    const CellEdge e = cell_edge<P>(i, j);
    const size_t at = (size_t)e.y * (a.c.nx + DIR) + e.x, np = a.eb.plane[DIR];
    if (factor) *factor = 1.0;
    const EdgeSides s = edge_sides<DIR>(a, e.x, e.y);
    const int id1 = s.interior ? s.id1 : s.id0, row1 = s.interior ? s.row1 : s.row0;
    const unsigned now = stage_mark(a);
    // all that the edge may need, at once (behind each other's tests: 1024^2
    // fjord 357 against 350 us a step)
    int kind = a.eb.kind[DIR][at];
    double m = a.eb.q[DIR][at + (layer ? 6 : 0) * np], p = a.eb.q[DIR][at + (layer ? 9 : 3) * np];
    unsigned mark0 = a.eb.mark[layer][s.id0], mark1 = a.eb.mark[layer][id1];
    double h0 = a.eb.depth[layer][s.id0], h1 = a.eb.depth[layer][id1];
    lshm::together(kind, m, p, mark0, mark1, h0, h1);
    if (kind <= layer) return 0.0;
    const double own = e.second ? p : m;
    // An unmarked cell's test is false, and its quotient never the smaller one:
    // before its last edge it holds 5/8 of its content, and the denominator
    // times dt is at most 1/4 (far_from_empty), so the quotient is at least
    // 2.5 dt, a limiting side's at most dt.  Only a marked cell's partial sum is
    // read (64^2 fjord 138 -> 135 us a step, 1024^2 347 -> 340).
    const bool lose0 = gt0(m) && mark0 == now, lose1 = s.interior && gt0(p) && mark1 == now;
    if (!lose0 && !lose1) return own;
    double other = 0.0;
    if (e.second ? lose0 : lose1) {
        const int io = e.second ? s.id0 - s.row0 * a.c.nx : s.id1 - s.row1 * a.c.nx;
        other = partial_mass<P>(a, io, e.second ? s.row0 : s.row1, layer, dt, nullptr);
    }
    const double f = limiter_sides(lose0, lose1, m, p, h0, e.second ? other : acc, a.geo.area[s.row0],
                                   a.geo.inv_area[s.row0], h1, e.second ? acc : other, a.geo.area[row1],
                                   a.geo.inv_area[row1], dt, a.c);
    if (factor) *factor = f;
    return (lshm::bits_of(f) != lshm::bits_of(1.0)) ? f * own : own;
}

template <int C>
LSH_RECURSE double partial_mass(const KArgs& a, int i, int j, int layer, double dt, double* factors) {
    const double acc = partial_mass<C - 1>(a, i, j, layer, dt, factors);
    const double d = limited_mass<C - 1>(a, i, j, layer, dt, acc, factors ? factors + (C - 1) : nullptr);
    return acc - d;
}

// Subtracts the colour-C edge's terms from the cell's accumulators (the first
// colour writes them), as do_edge's scatter does.  A dry edge's planes are
// loaded like the others', so that no load waits for the kinds, and taken as
// +0: an accumulator never holds -0, so subtracting zeros leaves its bits.
// LIMIT: with the limiter's factors f1, f2 of the layers' edges by colour (null:
// all 1).
template <int C, bool LIMIT>
LSH_HD void add_edge(const KArgs& a, int i, int j, int kind, const double* f1, const double* f2, double acc[7]) {
    constexpr int DIR = C / 2;
    const CellEdge e = cell_edge<C>(i, j);
    const size_t at = (size_t)e.y * (a.c.nx + DIR) + e.x, np = a.eb.plane[DIR];
    const double* q = a.eb.q[DIR] + at;
    // back to x/y: DIR 1: (qx, qy) = sg (fn, ft); DIR 0: qx = -sg ft, qy = sg fn
    const bool neg = e.boundary;  // normal toward -x, -y
    auto take = [&](int l, const double* f, double v0, double v1, double v2) {
        if (LIMIT && f && lshm::bits_of(f[C]) != lshm::bits_of(1.0)) { v0 = f[C] * v0; v1 = f[C] * v1; v2 = f[C] * v2; }
        const double dn = lshm::neg_if(v1, neg), dq = lshm::neg_if(v2, (DIR == 1) ? neg : !neg);
        const double dx = (DIR == 1) ? dn : dq, dy = (DIR == 1) ? dq : dn;
        const int k = 3 * l;
        if (C == 0) { acc[k] = minus0(v0); acc[k + 1] = minus0(dx); acc[k + 2] = minus0(dy); }
        else { acc[k] = acc[k] - v0; acc[k + 1] = acc[k + 1] - dx; acc[k + 2] = acc[k + 2] - dy; }
    };
    const bool wet = (kind != kEdgeDry);
    const double q0 = q[(e.second ? 3 : 0) * np], q1 = q[(e.second ? 4 : 1) * np], q2 = q[2 * np], w = q[5 * np];
    // the second cell's tangential momentum is the first's, negated
    take(0, f1, wet ? q0 : 0.0, wet ? q1 : 0.0, wet ? lshm::neg_if(q2, e.second) : 0.0);
    if (kind == kEdgeBoth) {
        lshm::rare();
        take(1, f2, q[(e.second ? 9 : 6) * np], q[(e.second ? 10 : 7) * np], lshm::neg_if(q[8 * np], e.second));
    }
    acc[6] = (C == 0) ? (wet ? plus0(w) : 0.0) : acc[6] + (wet ? w : 0.0);
}

// One cell of the Euler-stage update after the flux pass (MODE as volume_finish).
// `busy` is set where the cell's input or output state is not all +0 or one of
// its edges is not dry.
// KEEP (the adjoint's recomputation): the accumulators go to a.acc and, at cells
// with a wet edge, the partial sums acc[0], acc[3] after the first three colours
// to a.part; MODE < 0 ends there.
template <int MODE, bool KEEP = false>
LSH_HD unsigned long long update_cell(const KArgs& a, int i, int j, double dt, bool& busy) {
    const int nx = a.c.nx, ny = a.c.ny, id = j * nx + i;
    const unsigned char* kh = a.eb.kind[0] + id;
    const unsigned char* kv = a.eb.kind[1] + (size_t)j * (nx + 1) + i;
    const int kb = kh[0], kt = kh[nx], kl = kv[0], kr = kv[1], any = kb | kt | kl | kr;
    const int k0 = (j & 1) ? kt : kb, k1 = (j & 1) ? kb : kt, k2 = (i & 1) ? kr : kl, k3 = (i & 1) ? kl : kr;
    busy |= (any != 0);
    double wo[6], acc[7];
#pragma unroll
    for (int k = 0; k < 6; ++k) wo[k] = a.W[k][id];
#pragma unroll
    for (int k = 3; k < 6; ++k) acc[k] = 0.0;
    if (KEEP && !warp_any(any)) {
        // nothing but dry edges: +0 all round (the recomputation visits every
        // tile; in the listed ones of a step the test cost more than it saved,
        // 104 against 108 us at 2048^2)
#pragma unroll
        for (int k = 0; k < 7; ++k) a.acc[k][id] = acc[k] = 0.0;
        if constexpr (MODE < 0) return 0;
        else return volume_finish<MODE, true>(a, id, j, dt, wo, acc, &busy);
    }
    // an edge is limited only where one of its two cells is marked
    bool limit[2];
    const unsigned now = stage_mark(a);
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const unsigned* mk = a.eb.mark[l] + id;
        limit[l] = (mk[0] == now) | (mk[j > 0 ? -nx : 0] == now) | (mk[j < ny - 1 ? nx : 0] == now) |
                   (mk[i > 0 ? -1 : 0] == now) | (mk[i < nx - 1 ? 1 : 0] == now);
        if (l == 1) limit[l] = limit[l] && (any & kEdgeBoth);
    }
    if (warp_any(any && (limit[0] || limit[1]))) {
        lshm::rare();
        limit[0] = any && limit[0] && limit_near(a, i, j, 0, dt);
        limit[1] = any && limit[1] && limit_near(a, i, j, 1, dt);
    }
    auto partial = [&](int c) {
        if (!KEEP || !any) return;
        a.part[c][0][id] = acc[0];
        a.part[c][1][id] = acc[3];
    };
    if (warp_any(any && (limit[0] || limit[1]))) {
        double f[8];
        if (limit[0]) partial_mass<4>(a, i, j, 0, dt, f);
        if (limit[1]) partial_mass<4>(a, i, j, 1, dt, f + 4);
        const double* f1 = limit[0] ? f : nullptr;
        const double* f2 = limit[1] ? f + 4 : nullptr;
        add_edge<0, true>(a, i, j, k0, f1, f2, acc);
        partial(0);
        add_edge<1, true>(a, i, j, k1, f1, f2, acc);
        partial(1);
        add_edge<2, true>(a, i, j, k2, f1, f2, acc);
        partial(2);
        add_edge<3, true>(a, i, j, k3, f1, f2, acc);
    } else {
        add_edge<0, false>(a, i, j, k0, nullptr, nullptr, acc);
        partial(0);
        add_edge<1, false>(a, i, j, k1, nullptr, nullptr, acc);
        partial(1);
        add_edge<2, false>(a, i, j, k2, nullptr, nullptr, acc);
        partial(2);
        add_edge<3, false>(a, i, j, k3, nullptr, nullptr, acc);
    }
    if (KEEP) {
#pragma unroll
        for (int k = 0; k < 7; ++k) a.acc[k][id] = acc[k];
    }
    if constexpr (MODE < 0) return 0;
    else return volume_finish<MODE, true>(a, id, j, dt, wo, acc, &busy);
}

// dt from the largest acc_w / area: 2 CFL / max rate, 1e30 when no cell has a wave speed
LSH_HD double dt_of(unsigned long long rmax_bits, double two_cfl) {
    const double m = lshm::from_bits(rmax_bits);
    return (m > 0.0) ? lsh::div(two_cfl, m) : lsh::kBig;
}

// One edge of the initial-dt pass (procesarAristasDeltaTInicialGPU,
// Arista_kernel.cu:1129-1308): its wave-speed bound into acc[6].
template <int DIR, bool FIRST>
LSH_HD void init_wave_edge(const KArgs& a, int x, int y) {
    const int nx = a.c.nx, ny = a.c.ny;
    int id0, id1 = -1;
    double bor = 0.0, len;
    bool pos_normal = true;
    if (DIR == 0) {
        len = a.geo.len_h[y];
        if (y == 0) { id0 = x; pos_normal = false; bor = a.c.borde_sup; }
        else if (y == ny) { id0 = (ny - 1) * nx + x; bor = a.c.borde_inf; }
        else { id0 = (y - 1) * nx + x; id1 = id0 + nx; }
    } else {
        len = a.geo.len_v[y];
        if (x == 0) { id0 = y * nx; pos_normal = false; bor = a.c.borde_izq; }
        else if (x == nx) { id0 = y * nx + nx - 1; bor = a.c.borde_der; }
        else { id0 = y * nx + x - 1; id1 = id0 + 1; }
    }
    lsh::Face A, B;
    A.h1 = a.W[0][id0];
    A.h2 = a.W[3][id0];
    face_rest<DIR, 1>(a, id0, 0, pos_normal, A);
    if (id1 >= 0) {
        B.h1 = a.W[0][id1];
        B.h2 = a.W[3][id1];
        face_rest<DIR, 1>(a, id1, 0, pos_normal, B);
    } else {
        B = A;
        B.qn1 = A.qn1 * bor;
        B.qn2 = A.qn2 * bor;
    }
    // both faces empty and still: every term of the bound is an exact zero and
    // lmax = 0 + eps_h, so the wave is len * eps_h without the FP64 work
    using lsh::is_zero;
    const bool empty = is_zero(A.h1) && is_zero(A.h2) && is_zero(B.h1) && is_zero(B.h2) && is_zero(A.qn1) &&
                       is_zero(A.qn2) && is_zero(B.qn1) && is_zero(B.qn2);
    const double wv = empty ? len * (0.0 + a.c.eps_h) : lsh::edge_initial_wave(A, B, len, a.c);
    if (FIRST) {
        a.acc[6][id0] = 0.0 + wv;
        if (id1 >= 0) a.acc[6][id1] = 0.0 + wv;
    } else {
        a.acc[6][id0] += wv;
        if (id1 >= 0) a.acc[6][id1] += wv;
    }

}

// acc_w / area of one cell after the initial wave pass (obtenerDeltaTVolumenesGPU)
LSH_HD unsigned long long init_cell_rate(const KArgs& a, int id) {
    const int j = id / a.c.nx;
    const double w = a.acc[6][id];
    const double rate = (w < lsh::kEps) ? 0.0 : w * a.geo.inv_area[j];
    return (unsigned long long)lshm::bits_of(rate);
}

}  // namespace lsh
