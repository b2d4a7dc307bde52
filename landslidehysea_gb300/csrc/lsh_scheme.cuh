// lsh_scheme.cuh -- FP64 device math of the two-layer time step.
//
// One thread evaluates one edge (edge functions) or one cell (volume
// functions).  The arithmetic is the LandSlide-HySEA scheme:
//   edge flux            src/GPU/Arista_kernel.cu:324-645 (procesarArista)
//   wet/dry fix          src/GPU/Arista_kernel.cu:301-321
//   hydrostatic terms    src/GPU/Arista_kernel.cu:94-150
//   eigenvalue bounds    src/GPU/Arista_kernel.cu:152-237
//   identity mod.        src/GPU/Arista_kernel.cu:239-276
//   initial-dt wave      src/GPU/Arista_kernel.cu:1040-1127
//   state update         src/GPU/Volumen_kernel.cu:7-180, 231-284
// evaluated in double precision on structure-of-arrays state.  Conventions
// (kept identical in the CPU oracle so both are one FP64 scheme up to
// rounding): EPSILON keeps FLT_EPSILON's value; u = vfac(h) * q with
// vfac(h) = sqrt(2) h / sqrt(h^4 + max(h, eps_h)^4), h^4 = (h*h)*(h*h);
// exp, cbrt and log come from lsh_fpmath.h (IEEE basic operations only, so
// host and device give identical bits); h^(4/3) = h * cbrt(h).  The library
// is compiled with --fmad=false: no implicit a*b+c contraction, so the FP64
// operation sequence here is exactly the oracle's and results match it bit
// for bit.
#pragma once

#include <cstdint>

#include "lsh_fpmath.h"
#include "lsh_ieee.h"

namespace lsh {

#if !defined(__CUDA_ARCH__)
using std::fabs;
#endif

constexpr double kEps = 1.1920928955078125e-07;  // FLT_EPSILON (Constantes.hxx:13)
constexpr double kSqrt2 = 1.41421356237309504880;
constexpr double kBig = 1e30;

// Scalars every kernel needs; passed by value (kernel parameter space).
struct Consts {
    double g, r, gp, eps_h, peso, beta, cfl, mu, mfc, mf0, mfs, vmax1, vmax2, L, H;
    double tan1, tan2, tan3, tan4;
    // host-derived, with the same formulas as the CPU oracle's make_consts
    double omr, inv_gp, inv_eps, inv_peso, eps_1r, g_mf02, g_mfs2, sqrt_g;
    double borde_sup, borde_inf, borde_izq, borde_der;
    int law;
    int order;
    int nx, ny;
    int track_eta;
    int eig_sort;
};

// Per-row geometry (device arrays, ny or ny+1 entries).
struct Geo {
    const double* area;   // [ny]
    const double* inv_area;  // [ny]
    const double* len_v;  // [ny]
    const double* len_h;  // [ny+1]
    const double* tanR;   // [ny]
    const double* wx;     // [ny]
    const double* wy;     // [ny]
};

// Device-resident time record: dt and t never leave the device between steps.
struct TimeRec {
    double t;                        // simulated time
    double dt;                       // dt of the next step
    double t_end;                    // stop once t >= t_end
    double dt_min;                   // stall guard (0: off)
    unsigned long long rmax_bits;    // running max of per-cell acc_w / area (bits of a double >= 0)
    long long steps;                 // steps taken
    int done;                        // 1 once t >= t_end (kernels then return at once)
    int err;                         // sticky error bits (LSH status values as bits)
};

struct V4 { double x, y, z, w; };

// p on every active lane of the warp (the thread's own p in host code).
LSH_HD bool warp_all(bool p) {
#if defined(__CUDA_ARCH__)
    return __all_sync(__activemask(), p);
#else
    return p;
#endif
}

// p on some active lane of the warp (the thread's own p in host code).
LSH_HD bool warp_any(bool p) {
#if defined(__CUDA_ARCH__)
    return __any_sync(__activemask(), p);
#else
    return p;
#endif
}

// Compares run on the integer pipe (lsh_fpmath.h: exact for non-NaN
// operands): lt_pos / gt_pos against the positive thresholds EPSILON, eps_h,
// vmax, lt / okey for operands of either sign.
using lshm::abs_bits;
using lshm::abs_lt;
using lshm::gt0;
using lshm::gt_pos;
using lshm::lt;
using lshm::lt0;
using lshm::lt_pos;
using lshm::okey;
// IEEE division, reciprocal and square root on the integer pipe (lsh_ieee.h)
using lshm::div;
using lshm::div_call;
using lshm::rcp;
using lshm::rcp_call;
using lshm::root;
using lshm::root_call;

LSH_HD double tmin(double a, double b) { return lt(b, a) ? b : a; }
LSH_HD double tmax(double a, double b) { return lt(a, b) ? b : a; }
LSH_HD double max0(double a) { return gt0(a) ? a : 0.0; }
LSH_HD double fmad(double a, double b, double c) { return lshm::fmad(a, b, c); }
LSH_HD double exp_neg(double x) { return lshm::exp_neg(x); }

// x == +0 or -0, by bit pattern (integer pipe)
LSH_HD bool is_zero(double x) {
    uint32_t lo, hi;
    lshm::halves(x, lo, hi);
    return ((hi << 1) | lo) == 0u;
}

// sqrt(2) h / sqrt(h^4 + max(h, eps_h)^4); exactly 1/h for h > eps_h
LSH_HD double vfac(double h, double eps_h) {
    if (gt_pos(h, eps_h)) return rcp(h);
    if (is_zero(h)) return h;  // an empty layer: the quotient below is that zero
    const double h2 = h * h, m2 = eps_h * eps_h;
    return div(kSqrt2 * h, root(fmad(h2, h2, m2 * m2)));
}

// x / 2 and 2 x on the integer pipe (no FP64 instruction even for special
// values: a rarely taken one would be predicated into every warp's stream, and
// one predicated off still holds the FP64 unit).  Subnormal results round to
// even; infinities and NaN stay.
LSH_HD double half(double x) {
    uint32_t lo, hi;
    lshm::halves(x, lo, hi);
    const uint32_t e = (hi >> 20) & 0x7ffu;
    if (e - 2u < 2045u) return lshm::from_halves(lo, hi - 0x00100000u);
    if (e >= 2u) return x;
    // the magnitude is m 2^-1074 (exponent 1 included): m / 2, ties to even
    const uint64_t m = ((uint64_t)(hi & 0x7fffffffu) << 32) | lo;
    const uint64_t h = (m >> 1) + (m & (m >> 1) & 1u);
    return lshm::from_halves((uint32_t)h, (uint32_t)(h >> 32) | (hi & 0x80000000u));
}
LSH_HD double twice(double x) {
    uint32_t lo, hi;
    lshm::halves(x, lo, hi);
    const uint32_t e = (hi >> 20) & 0x7ffu;
    if (e - 1u < 2045u) return lshm::from_halves(lo, hi + 0x00100000u);
    if (e == 0x7ffu) return x;
    if (e != 0u) return lshm::from_halves(0u, (hi & 0x80000000u) | 0x7ff00000u);
    return lshm::from_halves(lo << 1, (hi & 0x80000000u) | (hi << 1) | (lo >> 31));
}

// 0 + x and 0 - x on the integer pipe: x and -x, with +0 for either zero (NaN
// keeps its sign, which steers integer compares)
LSH_HD double plus0(double x) {
    uint32_t lo, hi;
    lshm::halves(x, lo, hi);
    return lshm::from_halves(lo, (lo == 0u && hi == 0x80000000u) ? 0u : hi);
}
LSH_HD double minus0(double x) {
    uint32_t lo, hi;
    lshm::halves(x, lo, hi);
    const uint32_t mag = hi & 0x7fffffffu;
    const bool nan = mag > 0x7ff00000u || (mag == 0x7ff00000u && lo != 0u);
    return lshm::from_halves(lo, ((mag | lo) == 0u) ? 0u : (nan ? hi : (hi ^ 0x80000000u)));
}

// log2 x of a positive normal x in units of 2^-20, low by at most 0.0861
// (the significand taken as its own logarithm): the high word, rebased
LSH_HD int32_t log2_low(double x) {
    uint32_t lo, hi;
    lshm::halves(x, lo, hi);
    return (int32_t)(hi & 0x7fffffffu) - 0x3ff00000;
}
constexpr int32_t kLog2One = 1 << 20;

LSH_HD double pow43(double h) { return h * lshm::cbrt_pos(h); }

LSH_HD int sgn(double x) { return abs_lt(x, kEps) ? 0 : (gt0(x) ? 1 : -1); }

// NaN or Inf, by the exponent bits (integer pipe)
LSH_HD bool is_bad(double x) {
    uint32_t lo, hi;
    lshm::halves(x, lo, hi);
    return (hi & 0x7ff00000u) == 0x7ff00000u;
}

// Bounds of the four eigenvalue estimates as the compare-and-swap sequence of
// Arista_kernel.cu:193-234 leaves them (with its (2,1) compare, or with `full`
// the same sequence made a true sort): its first and last value and the
// larger magnitude of the two between.  The estimates are a = u - c, b = u' -
// c', c = u' + c', d = u + c with a <= d and b <= c (rounding is monotone), so
// of its seven compares three can swap:
//   first (a, b); then the larger of those against d, which is above d only
//   when b is.  Last: the (2,1) form leaves max(b, d) and between it
//   {c, d or max(a, b)}; the true sort max(c, d), with {max(a, b), min(c, d)}.
struct EigBounds { double lo, hi, mid; };
LSH_HD EigBounds eig_bounds(double a, double b, double c, double d, int full) {
    EigBounds e;
    const bool ab = lt(b, a);
    e.lo = ab ? b : a;
    const double top = ab ? a : b;
    double m1, m2;
    if (full) {
        const bool cd = lt(d, c);
        e.hi = cd ? c : d;
        m1 = top;
        m2 = cd ? d : c;
    } else {
        const bool bd = lt(d, b);
        e.hi = bd ? b : d;
        m1 = bd ? d : top;
        m2 = c;
    }
    m1 = abs_bits(m1);
    m2 = abs_bits(m2);
    e.mid = lt_pos(m1, m2) ? m2 : m1;
    return e;
}

// aproximarAutovalores1D (Arista_kernel.cu:152-237), both layers.
LSH_HD EigBounds eig_edge(double h1, double h2, double u1, double u2, double q, const Consts& c, double sqrt_h = -1.0,
                          bool mean_u = false) {
    const double h = h1 + h2;
    const double F = vfac(h, c.eps_h);
    // mean_u (the edge average, q = h1 u1 + h2 u2): with no granular layer and
    // h > eps_h, u = q vfac(h) = (h1 u1) / h1 is u1 itself -- an exact
    // restatement the CPU oracle makes too
    const double u = (mean_u && is_zero(h2) && gt_pos(h, c.eps_h)) ? u1 : q * F;
    // sqrt_h >= 0: sqrt(h1) is known and h2 == 0, so sqrt(g h) = sqrt(g) sqrt(h1)
    const double cg = !lt0(sqrt_h) ? c.sqrt_g * sqrt_h : root(c.g * h);
    const double uu = fmad(u1, h2, u2 * h1) * F;
    const double du = u1 - u2;
    const double aux = fmad(-((du * du) * F), c.inv_gp, 1.0);
    const double ci = root((((c.gp * h1) * h2) * F) * abs_bits(aux));
    return eig_bounds(u - cg, uu - ci, uu + ci, u + cg, c.eig_sort);
}

// defTerminoFriccion (Arista_kernel.cu:11-58)
LSH_HD double friction_mu(double h1, double u1, double h2, double u2, const Consts& c) {
    if (c.law == 0) return c.mu;
    const double a = (10.0 * h1) * c.inv_eps;
    const double rr = 1.0 - c.r * (1.0 - exp_neg(a * a));
    const double gp = c.g * rr;
    const double fr1 = div((u1 * u1) * vfac(h1, c.eps_h), gp);
    const double fr2 = div((u2 * u2) * vfac(h2, c.eps_h), gp);
    const double fr = root(fmad((1.0 - rr) * fr1, fr2, fr1 + fr2));
    const double beta = 0.136, L2c = 8.0e-4, chi = 1.0e-3;
    const double mustop = c.tan1 + div(c.tan2 - c.tan1, 1.0 + div(h2, L2c));
    const double mustart = c.tan3 + div(c.tan4 - c.tan3, 1.0 + div(h2, L2c));
    double muf;
    if (gt_pos(fr, beta)) muf = c.tan1 + div(c.tan2 - c.tan1, 1.0 + div(beta * h2, fr * L2c));
    else if (abs_lt(fr, kEps)) muf = c.tan3 + div(c.tan4 - c.tan3, 1.0 + div(h2, L2c));
    else muf = fmad(lshm::pow_pos(div(fr, beta), chi), mustop - mustart, mustart);
    return div(muf * c.L, c.H);
}

LSH_HD double fsc_of(double h1, const Consts& c) {
    // logarithms 3 apart (each low by at most 0.0861) put h1 above 7.5 eps_h: the
    // exponent is beyond 75^2, exp_neg gives 0 from 746 on, so this is
    // 1 - r (1 - 0) = 1 - r
    if (log2_low(h1) - log2_low(c.eps_h) > 3 * kLog2One && gt0(h1)) return 1.0 - c.r;
    const double a = (10.0 * h1) * c.inv_eps;
    return 1.0 - c.r * (1.0 - exp_neg(a * a));
}

// One face state in the edge's normal frame: depth, normal and tangential
// discharge of each layer, bottom depth.
struct Face { double h1, qn1, qt1, h2, qn2, qt2, H; };

// Inputs of one edge (the CPU oracle's EdgeIn): the two facing states A, B,
// cell-average depths and partial accumulators for the positivity limiter.
struct EdgeIn {
    Face A, B;
    double len, area0, area1, inv_area0, inv_area1;
    double hc0[2], hc1[2];
    double acc0h[2], acc1h[2];
    bool interior;
};

// Normal-frame output: per layer (mass, normal momentum, tangential
// momentum) to subtract from cell 0 (m) and cell 1 (p), and the wave term.
struct EdgeOut { double m[6], p[6]; double wave; };

// The positivity limiter's inputs, read from an EdgeIn that holds them.
struct EdgeInPos {
    const EdgeIn& e;
    LSH_HD double area(int side) const { return side ? e.area1 : e.area0; }
    LSH_HD double inv_area(int side) const { return side ? e.inv_area1 : e.inv_area0; }
    LSH_HD double hc(int side, int layer) const { return side ? e.hc1[layer] : e.hc0[layer]; }
    LSH_HD double acch(int side, int layer) const { return side ? e.acc1h[layer] : e.acc0h[layer]; }
};

// The flux of one edge before the positivity limiter, in the normal frame and
// times the edge length: m (mass, normal and tangential momentum of each
// layer, for cell 0) and p (mass and normal momentum, for cell 1; its
// tangential momentum is -m[3 l + 2]), and the wave term.
struct EdgeRaw { double m[6], p[4], wave; };

// A single-layer edge: edge_raw where both faces have no granular layer (h2 =
// qn2 = 0; tangential terms of layer 2 unused), whose layer-1 values are the
// same as in the general path, and its layer-2 outputs zeros.
//
// The FP64 unit bounds every pass (16 cycles per instruction and SM, 55 of
// latency), so what gives the same bits off it runs on the integer pipe, and
// what only some edges need sits in blocks that a warp votes on: an
// instruction predicated off still holds the unit.  63 FP64 instructions of
// the 200 that the plain statement takes (10 of them the second-order faces').
LSH_HD void edge_raw1(const Face& A, const Face& B, double len, const Consts& c, EdgeRaw& o) {
    const double eps = c.eps_h;
    double Aq = A.qn1, Bq = B.qn1;
    const double h = half(A.h1 + B.h1);
    const double tA = A.h1 - A.H, tB = B.h1 - B.H;
    // tratamientoSecoMojado (Arista_kernel.cu:301-321); H - h is -(h - H)
    if (lt_pos(A.h1, eps) && lt(A.H, lshm::neg_if(tB, true))) Bq = 0.0;
    if (lt_pos(B.h1, eps) && lt(B.H, lshm::neg_if(tA, true))) Aq = 0.0;
    const double fA = vfac(A.h1, eps), fB = vfac(B.h1, eps);
    const double sA = root(A.h1), sB = root(B.h1);
    const double uA = fA * Aq, uB = fB * Bq;
    const double u = div(fmad(sA, uA, sB * uB), sA + sB + kEps);

    const double Hm = tmin(A.H, B.H);
    const double deta = max0(tB + Hm) - max0(tA + Hm);
    const double gh = c.g * h;

    // eigenvalue bounds (eig_edge, its single-layer form): min(u - c, 0) and
    // max(u + c, 0) of the average and of both faces
    double ue = u;
    if (!gt_pos(h, eps)) ue = (h * u) * vfac(h, eps);  // else q vfac(h) = (h u) / h restated as u
    const double cg = root(gh);
    const double lo = ue - cg, hi = ue + cg;
    const double cA = c.sqrt_g * sA, cB = c.sqrt_g * sB;
    const double eA = uA - cA, wA = uA + cA, eB = uB - cB, wB = uB + cB;
    // (least of values <= 0 and greatest of values >= 0: by their magnitudes)
    auto larger = [](double x, double y) { return abs_lt(x, y) ? y : x; };
    const double aut1 = larger(gt0(lo) ? 0.0 : lo, larger(gt0(eA) ? 0.0 : eA, gt0(eB) ? 0.0 : eB));
    const double aut3 = larger(lt0(hi) ? 0.0 : hi, larger(lt0(wA) ? 0.0 : wA, lt0(wB) ? 0.0 : wB));
    const double b1 = abs_bits(aut1), b3 = abs_bits(aut3);
    double lmax = lt_pos(b3, b1) ? b1 : b3;
    if (lt_pos(lmax, abs_bits(u))) lmax = abs_bits(u);
    const double d13 = aut1 - aut3;
    // IFCP coefficients.  Subcritical average (its middle eigenvalues 0), waves
    // to both sides: aut3 |aut1| - aut1 |aut3| is -2 p for the rounded product p
    // = aut1 aut3 (the fma's sum -2 p + (p - exact) is within half an ulp of
    // -2 p), and the middle gaps are aut1 and -aut3.
    double n0, n1;
    bool wide;
    const bool sub = !gt0(lo) && !lt0(hi) && lt0(aut1) && gt0(aut3) && !lt_pos(b1, 0x1p-400) && !lt_pos(b3, 0x1p-400);
    if (warp_all(sub)) {
        lshm::rare();
        n0 = lshm::neg_if(twice(aut1 * aut3), true);
        n1 = aut3 + aut1;
        wide = !lt_pos(b1, kEps) && !lt_pos(b3, kEps);
    } else {
        lshm::rare();
        double aut2 = gt0(lo) ? lo : (lt0(hi) ? abs_bits(hi) : 0.0);
        aut2 = lshm::neg_if(aut2, sgn(aut1 + aut3) < 0);
        n0 = fmad(aut3, b1, -(aut1 * b3));
        n1 = b3 - b1;
        wide = !abs_lt(aut1 - aut2, kEps) && !abs_lt(aut2 - aut3, kEps);
    }
    double a0 = lmax, a1 = 0.0;
    if (wide && !abs_lt(d13, kEps)) {
        const double inv = rcp(lshm::neg_if(d13, true));  // 1 / (aut3 - aut1)
        a0 = n0 * inv;
        a1 = n1 * inv;
    }

    const double FA = lt_pos(A.h1, kEps) ? 0.0 : uA * Aq, FB = lt_pos(B.h1, kEps) ? 0.0 : uB * Bq;
    const double dF = Bq - Aq;
    const double tx = plus0(dF), ty = gh * deta + (FB - FA);
    const double half_x = half(tx), half_y = half(ty);
    const double Qx = half(fmad(a0, deta, a1 * tx));
    const double Qy = half(fmad(a0, dF, a1 * ty));
    const double Fm = half_x + (Aq - Qx);
    const bool out = gt0(Fm);
    const double ut = abs_lt(Fm, kEps) ? 0.0 : (out ? fA : fB) * (out ? A.qt1 : B.qt1);
    o.m[0] = len * Fm;
    o.m[1] = len * (half_y + (FA - Qy));
    o.m[2] = len * (Fm * ut);
    o.p[0] = len * (half_x + (Qx - Bq));
    o.p[1] = len * (half_y + (Qy - FB));
    o.m[3] = o.m[4] = o.m[5] = o.p[2] = o.p[3] = 0.0;
    if (lt_pos(lmax, eps)) { lshm::rare(); lmax = lmax + eps; }
    o.wave = len * lmax;
}

// procesarArista (Arista_kernel.cu:324-645) up to the limiter, the depths
// already known to be wet (the caller skips dry edges, :397): both layers.
LSH_HD void edge_raw2(const Face& A, const Face& B, double len, double dt, const Consts& c, EdgeRaw& o) {
    const double eps = c.eps_h;
    double Aq1 = A.qn1, Aq2 = A.qn2, Bq1 = B.qn1, Bq2 = B.qn2;
    const double Ah1 = A.h1, Bh1 = B.h1;
    const double Ah2 = A.h2, Bh2 = B.h2;
    const double H0 = A.H, H1 = B.H;
    const double h1ij = half(Ah1 + Bh1);
    const double h2ij = half(Ah2 + Bh2);

    // tratamientoSecoMojado (Arista_kernel.cu:301-321): the conditions on
    // layer 1 need its depth below eps_h on one side (or a negative h2)
    if (lt_pos(Ah2, eps) || lt_pos(Bh2, eps)) {
        lshm::rare();
        if (lt_pos(Ah2, eps) && lt(H0, H1 - Bh2)) Bq2 = 0.0;
        if (lt_pos(Bh2, eps) && lt(H1, H0 - Ah2)) Aq2 = 0.0;
    }
    if (lt_pos(Ah1, eps) || lt_pos(Bh1, eps) || lt0(Ah2) || lt0(Bh2)) {
        lshm::rare();
        if (lt_pos(Ah1, eps) && lt(H0 - Ah2, H1 - Bh1 - Bh2)) Bq1 = 0.0;
        if (lt_pos(Bh1, eps) && lt(H1 - Bh2, H0 - Ah1 - Ah2)) Aq1 = 0.0;
        if (lt_pos(Ah2 + Ah1, eps) && lt(H0, H1 - Bh1 - Bh2)) { Bq1 = 0.0; Bq2 = 0.0; }
        if (lt_pos(Bh2 + Bh1, eps) && lt(H1, H0 - Ah1 - Ah2)) { Aq1 = 0.0; Aq2 = 0.0; }
    }

    const double fA1 = vfac(Ah1, eps), fB1 = vfac(Bh1, eps);
    const double sa1 = root(Ah1), sb1 = root(Bh1);
    const double uA1 = fA1 * Aq1, uB1 = fB1 * Bq1;
    const double u1ij = div(fmad(sa1, uA1, sb1 * uB1), sa1 + sb1 + kEps);
    const double fA2 = vfac(Ah2, eps), fB2 = vfac(Bh2, eps);
    const double sa2 = root(Ah2), sb2 = root(Bh2);
    const double uA2 = fA2 * Aq2, uB2 = fB2 * Bq2;
    const double u2ij = div(fmad(sa2, uA2, sb2 * uB2), sa2 + sb2 + kEps);
    // a face's celerity sqrt(g h) is sqrt(g) sqrt(h1) when its granular layer is empty
    const bool oneA = is_zero(Ah2), oneB = is_zero(Bh2);

    const double Hm = tmin(H0, H1);
    const double deta1 = max0(Bh1 + Bh2 - H1 + Hm) - max0(Ah1 + Ah2 - H0 + Hm);
    const double deta2 = max0(Bh2 - H1 + Hm) - max0(Ah2 - H0 + Hm);
    const double gh1 = c.g * h1ij, gh2 = c.g * h2ij;
    // pressure terms, and layer 2's below the Coulomb threshold
    const double p1 = gh1 * deta1;
    const double p2 = gh2 * fmad(c.omr, deta2, c.r * deta1);
    const double mu = friction_mu(h1ij, u1ij, h2ij, u2ij, c);
    const double sc = ((fsc_of(h1ij, c) * mu) * c.g) * h2ij;
    const bool coul = lt_pos(abs_bits(h2ij * u2ij), (c.peso * sc) * dt);
    const double p2c = coul ? (gh2 * c.r) * deta1 : p2;

    const EigBounds D = eig_edge(h1ij, h2ij, u1ij, u2ij, fmad(h1ij, u1ij, h2ij * u2ij), c, -1.0, true);
    const EigBounds E0 = eig_edge(Ah1, Ah2, uA1, uA2, Aq1 + Aq2, c, oneA ? sa1 : -1.0);
    const EigBounds E1 = eig_edge(Bh1, Bh2, uB1, uB2, Bq1 + Bq2, c, oneB ? sb1 : -1.0);
    const double aut1 = tmin(D.lo, tmin(E0.lo, E1.lo));
    const double aut3 = tmax(D.hi, tmax(E0.hi, E1.hi));
    const double b1 = abs_bits(aut1), b3 = abs_bits(aut3);
    double lmax = lt_pos(b3, b1) ? b1 : b3;
    if (lt_pos(lmax, abs_bits(u1ij))) lmax = abs_bits(u1ij);
    if (lt_pos(lmax, abs_bits(u2ij))) lmax = abs_bits(u2ij);
    const double aut2 = lshm::neg_if(D.mid, sgn(aut1 + aut3) < 0);
    const double d12 = aut1 - aut2, d13 = aut1 - aut3, d23 = aut2 - aut3;

    double a0, a1, a2 = 0.0;
    if (!abs_lt(d13, kEps) && !abs_lt(d12, kEps) && !abs_lt(d23, kEps)) {
        if (!lt_pos(h1ij, eps) && !lt_pos(h2ij, eps)) {
            const double inv = rcp((d12 * d13) * d23);
            const double a = (b1 * d23) * inv;
            const double b = -((abs_bits(aut2) * d13) * inv);
            const double cc = (b3 * d12) * inv;
            a0 = fmad(a * aut2, aut3, fmad(b * aut1, aut3, (cc * aut1) * aut2));
            a1 = -fmad(a, aut2 + aut3, fmad(b, aut1 + aut3, cc * (aut1 + aut2)));
            a2 = a + b + cc;
        } else {
            const double inv = rcp(lshm::neg_if(d13, true));  // 1 / (aut3 - aut1), not 0
            a0 = fmad(aut3, b1, -(aut1 * b3)) * inv;
            a1 = (b3 - b1) * inv;
        }
    } else {
        a0 = lmax; a1 = 0.0;
    }

    const double FAy = lt_pos(Ah1, kEps) ? 0.0 : uA1 * Aq1, FBy = lt_pos(Bh1, kEps) ? 0.0 : uB1 * Bq1;
    const double dFx = Bq1 - Aq1, dFy = FBy - FAy;
    const double tx = plus0(dFx), ty = p1 + dFy;
    const double half_x = half(tx), half_y = half(ty);  // dF + pressure is ty with the terms exchanged

    const double Ix = (!coul && gt_pos(Ah1, eps) && gt_pos(Bh1, eps)) ? deta1 - deta2 : deta1;
    const double dFz = Bq2 - Aq2;
    const double tz = plus0(dFz);
    const double FAw = lt_pos(Ah2, kEps) ? 0.0 : uA2 * Aq2, FBw = lt_pos(Bh2, kEps) ? 0.0 : uB2 * Bq2;
    const double dFw = FBw - FAw;
    const double tw = p2c + dFw;
    const double Aty = fmad(gh1, tz, fmad(u1ij + u1ij, ty, fmad(-u1ij, u1ij, gh1) * tx));
    const double Qx = half(fmad(a0, Ix, fmad(a1, tx, a2 * ty)));
    const double Qy = half(fmad(a0, dFx, fmad(a1, ty, a2 * Aty)));
    const double Iz = coul ? 0.0 : deta2;
    const double Atw = fmad(c.r * gh2, tx, fmad(fmad(-u2ij, u2ij, gh2), tz, (u2ij + u2ij) * tw));
    const double Qz = half(fmad(a0, Iz, fmad(a1, tz, a2 * tw)));
    const double Qw = half(fmad(a0, dFz, fmad(a1, tw, a2 * Atw)));
    const double half_z = half(tz), half_w = half(dFw + p2);
    const double Fmz = half_z + (Aq2 - Qz), Fmw = half_w + (FAw - Qw);
    const double Fpz = half_z + (Qz - Bq2), Fpw = half_w + (Qw - FBw);
    const double u2t = abs_lt(Fmz, kEps) ? 0.0 : (gt0(Fmz) ? fA2 * A.qt2 : fB2 * B.qt2);
    o.m[3] = len * Fmz; o.m[4] = len * Fmw; o.m[5] = len * (Fmz * u2t);
    o.p[2] = len * Fpz; o.p[3] = len * Fpw;
    const double Fmx = half_x + (Aq1 - Qx), Fmy = half_y + (FAy - Qy);
    const double Fpx = half_x + (Qx - Bq1), Fpy = half_y + (Qy - FBy);
    const double u1t = abs_lt(Fmx, kEps) ? 0.0 : (gt0(Fmx) ? fA1 * A.qt1 : fB1 * B.qt1);
    o.m[0] = len * Fmx; o.m[1] = len * Fmy; o.m[2] = len * (Fmx * u1t);
    o.p[0] = len * Fpx; o.p[1] = len * Fpy;
    if (lt_pos(lmax, eps)) { lshm::rare(); lmax = lmax + eps; }
    o.wave = len * lmax;
}

// The positivity limiter's factor of one layer of an edge (Arista_kernel.cu:
// 554-609), 1 where it does not act: m and p are the mass terms of cells 0 and
// 1, h the cells' depths and acc the partial sums before this edge.  A side
// limits when dt exceeds the time it takes to empty its layer, hp area /
// (beta out + eps): tested as dt (beta out + eps) > hp area (the denominator
// is positive), so the divisions run only on limited edges.  oa, ob: whether
// cell 0, 1 loses mass and may be emptied.
LSH_HD double limiter_sides(bool oa, bool ob, double m, double p, double h0, double acc0, double area0,
                            double inv_area0, double h1, double acc1, double area1, double inv_area1, double dt,
                            const Consts& c) {
    double ha = 0.0, hb = 0.0, da = 1.0, db = 1.0;
    bool lim = false;
    if (oa) {
        ha = fmad(dt * inv_area0, acc0, h0) * area0;
        da = fmad(c.beta, m, kEps);
        lim = lt(ha, dt * da);
    }
    if (ob) {
        hb = fmad(dt * inv_area1, acc1, h1) * area1;
        db = fmad(c.beta, p, kEps);
        lim = lim || lt(hb, dt * db);
    }
    if (!lim) return 1.0;
    const double dta = oa ? div(ha, da) : kBig, dtb = ob ? div(hb, db) : kBig;
    return div(tmin(dta, dtb), dt + kEps);
}
LSH_HD double limiter(double m, double p, bool interior, double h0, double acc0, double area0, double inv_area0,
                      double h1, double acc1, double area1, double inv_area1, double dt, const Consts& c) {
    return limiter_sides(gt0(m), interior && gt0(p), m, p, h0, acc0, area0, inv_area0, h1, acc1, area1, inv_area1, dt, c);
}

// Whether a loss `out` (> 0) is far from emptying a layer of depth h: both
// dt scale out and dt eps at most an eighth of h area, by the operands'
// logarithms (log2_low is low by at most 0.0861: 3 + 3 x 0.0861 < 3.5; in half
// units, so that four of them add up in 32 bits).  With scale >= 1, beta and
// peso, a cell all of whose losses pass keeps at least a quarter of its
// content whatever the order of its edges and the others' limiter, so the
// limiter's test is false on each of its sides.
LSH_HD bool far_from_empty(double out, double h, double area, double dt, double scale) {
    const int32_t room = (log2_low(h) >> 1) + (log2_low(area) >> 1) - (log2_low(dt) >> 1) - 7 * (kLog2One / 4);
    return gt_pos(h, 0x1p-900) && (log2_low(out) >> 1) + (log2_low(scale) >> 1) <= room &&
           (log2_low(kEps) >> 1) <= room;
}

// procesarArista with the positivity limiter: the edge's terms to subtract
// from its cells' accumulators and to add to their wave sums.
// `pos` supplies the limiter's inputs (cell areas, cell depths and the partial
// accumulators of the cells' depths; EdgeInPos reads them from `e`): a caller
// may load them only where the limiter needs them, so they do not stay live
// through the flux computation.
template <bool L2, class Pos>
LSH_HD void edge_flux(const EdgeIn& e, double dt, const Consts& c, EdgeOut& o, const Pos& pos) {
    EdgeRaw w;
    if (L2) edge_raw2(e.A, e.B, e.len, dt, c, w);
    else edge_raw1(e.A, e.B, e.len, c, w);
    o.wave = w.wave;
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const int k = 3 * l;
        o.m[k] = w.m[k]; o.m[k + 1] = w.m[k + 1]; o.m[k + 2] = w.m[k + 2];
        o.p[k] = w.p[2 * l]; o.p[k + 1] = w.p[2 * l + 1]; o.p[k + 2] = lshm::neg_if(w.m[k + 2], true);
        if (l == 1 && !L2) break;
        if (gt0(o.m[k]) || (e.interior && gt0(o.p[k]))) {
            const double alpha = limiter(o.m[k], o.p[k], e.interior, pos.hc(0, l), pos.acch(0, l), pos.area(0),
                                         pos.inv_area(0), pos.hc(1, l), pos.acch(1, l), pos.area(1), pos.inv_area(1),
                                         dt, c);
            if (lshm::bits_of(alpha) != lshm::bits_of(1.0)) {
#pragma unroll
                for (int q = 0; q < 3; ++q) { o.m[k + q] = alpha * o.m[k + q]; o.p[k + q] = alpha * o.p[k + q]; }
            }
        }
    }
    if (!L2) { o.p[3] = o.p[4] = o.p[5] = 0.0; }
    if (lshm::bits_of(c.peso) != lshm::bits_of(1.0)) {
        o.wave = o.wave * c.inv_peso;
#pragma unroll
        for (int k = 0; k < 6; ++k) { o.m[k] = c.peso * o.m[k]; o.p[k] = c.peso * o.p[k]; }
    }
}

template <bool L2>
LSH_HD void edge_flux(const EdgeIn& e, double dt, const Consts& c, EdgeOut& o) {
    edge_flux<L2>(e, dt, c, o, EdgeInPos{e});
}

// procesarAristaDeltaTInicial: wave-speed bound for the initial dt.
LSH_HD double edge_initial_wave(const Face& A, const Face& B, double len, const Consts& c) {
    const double eps = c.eps_h;
    const double h1ij = half(A.h1 + B.h1);
    const double fA1 = vfac(A.h1, eps), fB1 = vfac(B.h1, eps);
    double sa = root(A.h1), sb = root(B.h1);
    const double u1ij = div(fmad(sa, fA1 * A.qn1, sb * (fB1 * B.qn1)), sa + sb + kEps);
    const double h2ij = half(A.h2 + B.h2);
    const double fA2 = vfac(A.h2, eps), fB2 = vfac(B.h2, eps);
    sa = root(A.h2); sb = root(B.h2);
    const double u2ij = div(fmad(sa, fA2 * A.qn2, sb * (fB2 * B.qn2)), sa + sb + kEps);
    const EigBounds D = eig_edge(h1ij, h2ij, u1ij, u2ij, fmad(h1ij, u1ij, h2ij * u2ij), c);
    double lmax = tmax(D.lo, D.hi);
    const double b = tmax(abs_bits(u1ij), abs_bits(u2ij));
    if (lt(lmax, b)) lmax = b;
    if (lt_pos(lmax, eps)) lmax = lmax + eps;
    return len * lmax;
}

// filtroEstado (Volumen_kernel.cu:92-180).  L2 == false: h2 = q2 = 0, so
// the layer-2 damping (0 times a factor) is skipped.
template <bool L2>
LSH_HD void filtro(double w[6], double dt, const Consts& c) {
    if (lt0(w[0])) w[0] = 0.0;
    if (lt0(w[3])) w[3] = 0.0;
#pragma unroll
    for (int layer = 0; layer < (L2 ? 2 : 1); ++layer) {
        const int k = 3 * layer;
        // exp(-dt/d), d = (w/eps_h)^4 + EPSILON, is exactly 1 once dt/d < 2^-54:
        // skipped by the operands' logarithms (log2_low: 4 log2(w/eps_h) above
        // log2 dt + 54 + 0.1 with a margin of 0.4 for the roundings)
        if ((log2_low(dt) >> 2) + 13 * kLog2One + 5 * (kLog2One / 8) < log2_low(w[k]) + log2_low(c.inv_eps)) continue;
        const double x = w[k] * c.inv_eps;
        const double x2 = x * x;
        const double d = fmad(x2, x2, kEps);
        const double aux = exp_neg(dt * rcp(d));
        w[k + 1] = w[k + 1] * aux;
        w[k + 2] = w[k + 2] * aux;
    }
#pragma unroll
    for (int layer = 0; layer < 2; ++layer) {
        const double vmax = layer ? c.vmax2 : c.vmax1;
        if (gt0(vmax)) {
            const int k = 3 * layer;
            const double h = w[k];
            const double f = vfac(h, c.eps_h);
            double ux = f * w[k + 1], uy = f * w[k + 2];
            const double u = root(fmad(ux, ux, uy * uy));
            if (gt_pos(u, vmax)) {
                const double s = div(vmax, u);
                ux = ux * s; uy = uy * s;
                w[k + 1] = ux * h; w[k + 2] = uy * h;
            }
        }
    }
}

// X < 2^-55 max(h, EPSILON) for h >= 1, X < 2^-55 EPSILON below, by the
// operands' logarithms (log2_low)
LSH_HD bool still_water(double X, double h) {
    const int32_t lh = log2_low(h), le = log2_low(kEps);
    return log2_low(X) + kLog2One / 8 < ((lh > 0) ? lh : le) - 55 * kLog2One;
}

// disImplicita (Volumen_kernel.cu:31-90).  L2 == false: the new and the old
// granular layer are empty (h2 = q2 = 0): only the water-bottom branch can run.
// fo1 = vfac(wo[0]), the old state's water factor, computed by the caller.
template <bool L2>
LSH_HD void dis_implicita(const double wo[6], double w[6], double dt, const Consts& c,
                                              double fo1) {
    if (lt0(w[0])) w[0] = 0.0;
    if (lt0(w[3])) w[3] = 0.0;
    const double eps = c.eps_h;
    const double h1 = w[0], h2 = L2 ? w[3] : 0.0;
    const double uo1x = fo1 * wo[1], uo1y = fo1 * wo[2];
    const double u1 = root(fmad(uo1x, uo1x, uo1y * uo1y));
    if (!L2) {
        // bottom friction h u / (1 + c1), 1/(1 + X/Y) = Y/(Y + X); above
        // eps_h, h u is q itself
        if (gt0(h1)) {
            const double X = (dt * c.g_mf02) * u1;
            // X below 2^-54 of Y >= max(min(h, h^(4/3)), EPSILON): Y + X is Y and
            // inv is 1 (h at least 1 there, so h <= h^(4/3))
            if (gt_pos(h1, eps) && still_water(X, h1)) return;
            const double Y = pow43(h1) + kEps;
            const double inv = div(Y, Y + X);
            if (gt_pos(h1, eps)) { w[1] = w[1] * inv; w[2] = w[2] * inv; }
            else {
                const double f1 = vfac(h1, eps);
                w[1] = (h1 * (f1 * w[1])) * inv;
                w[2] = (h1 * (f1 * w[2])) * inv;
            }
        }
        return;
    }
    const double f1 = vfac(h1, eps);
    double u1x = f1 * w[1], u1y = f1 * w[2];
    const double f2 = vfac(h2, eps);
    double u2x = f2 * w[4], u2y = f2 * w[5];
    const double fo2 = vfac(wo[3], eps);
    const double uo2x = fo2 * wo[4], uo2y = fo2 * wo[5];
    const double u2 = root(fmad(uo2x, uo2x, uo2y * uo2y));
    if (gt0(h1) && gt0(h2)) {
        // interlayer friction; without it (mfc = 0) its coefficient is +0 for
        // any finite depths and velocities
        double k12 = 0.0;
        if (lshm::bits_of(c.mfc) != 0) {
            const double dx = uo1x - uo2x, dy = uo1y - uo2y;
            const double du = root(fmad(dx, dx, dy * dy));
            const double hmod = fmad(c.r, h1, h2);
            const double m = gt_pos(hmod, c.eps_1r) ? hmod : c.eps_1r;
            const double hm2 = hmod * hmod, m2 = m * m;
            const double hh = div(hmod, root(fmad(hm2, hm2, m2 * m2)));
            k12 = ((dt * kSqrt2) * hh) * (c.mfc * du);
        }
        const double c1 = k12 * h2;
        const double c2 = (k12 * c.r) * h1;
        const double c3 = div((dt * c.g_mfs2) * u2, pow43(h2) + kEps);
        const double e1 = 1.0 + c1, e2 = 1.0 + c2 + c3;
        const double det = rcp(fmad(e1, e2, -(c1 * c2)));
        w[1] = (h1 * fmad(u1x, e2, c1 * u2x)) * det;
        w[4] = (h2 * fmad(u2x, e1, c2 * u1x)) * det;
        w[2] = (h1 * fmad(u1y, e2, c1 * u2y)) * det;
        w[5] = (h2 * fmad(u2y, e1, c2 * u1y)) * det;
    }
    if (gt0(h1) && lt_pos(h2, eps)) {
        const double Y = pow43(h1) + kEps, X = (dt * c.g_mf02) * u1;
        const double inv = div(Y, Y + X);
        if (gt_pos(h1, eps)) { w[1] = w[1] * inv; w[2] = w[2] * inv; }
        else { w[1] = (h1 * (f1 * w[1])) * inv; w[2] = (h1 * (f1 * w[2])) * inv; }
    }
    if (gt0(h2) && lt_pos(h1, eps)) {
        const double Y = pow43(h2) + kEps, X = (dt * c.g_mfs2) * u2;
        const double inv = div(Y, Y + X);
        if (gt_pos(h2, eps)) { w[4] = w[4] * inv; w[5] = w[5] * inv; }
        else { w[4] = (h2 * (f2 * w[4])) * inv; w[5] = (h2 * (f2 * w[5])) * inv; }
    }
}

// coulomb (Volumen_kernel.cu:7-26)
LSH_HD void coulomb(double w[6], double dt, const Consts& c) {
    if (!gt0(w[3])) {
        w[4] = w[4] * 0.0;
        w[5] = w[5] * 0.0;
        return;
    }
    double mu = c.mu;
    if (c.law != 0) {
        const double u1 = root(fmad(w[1], w[1], w[2] * w[2])) * vfac(w[0], c.eps_h);
        const double u2 = root(fmad(w[4], w[4], w[5] * w[5])) * vfac(w[3], c.eps_h);
        mu = friction_mu(w[0], u1, w[3], u2, c);
    }
    const double sc = ((((fsc_of(w[0], c) * mu) * c.g) * w[3]) * dt);
    const double normq = root(fmad(w[4], w[4], w[5] * w[5]));
    double aux = 0.0;
    if (!lt_pos(normq + sc, kEps) && !lt(normq, sc)) aux = div(normq, normq + sc);
    w[4] = w[4] * aux;
    w[5] = w[5] * aux;
}

// One cell of obtenerEstadoYDeltaTVolumenesGPU (Volumen_kernel.cu:231-284),
// plus the spherical metric source (tanR = tan(lat)/R, 0 for Cartesian).
// `rate` gets acc_w / area (0 below EPSILON): the step's dt is
// 2 CFL / max(rate), the min over cells of 2 CFL area / acc_w
// (Volumen_kernel.cu:256) with one division per step.
// ONE: the caller has checked that the cell's granular state wo[3..5] is
// zero and its layer-2 accumulators are +0 (an accumulator never holds -0).
// Then every layer-2 value below is the +0 the general path computes
// (b * (+0) + (+-0) = +0; Coulomb's +0 * 0 = +0), so that arithmetic is
// skipped and the single-layer branch taken.
template <bool ONE = false>
LSH_HD void volume_update(const double wo[6], const double acc[7], double w[6], double& rate,
                                              double inv_area, double tanR, double dt, const Consts& c) {
    rate = lt_pos(acc[6], kEps) ? 0.0 : acc[6] * inv_area;
    const double b = dt * inv_area;
#pragma unroll
    for (int k = 0; k < (ONE ? 3 : 6); ++k) w[k] = fmad(b, acc[k], wo[k]);
    if (ONE) { w[3] = 0.0; w[4] = 0.0; w[5] = 0.0; }
    const double fo1 = vfac(wo[0], c.eps_h);
    if (!is_zero(tanR)) {
#pragma unroll
        for (int layer = 0; layer < (ONE ? 1 : 2); ++layer) {
            const int k = 3 * layer;
            if (is_zero(wo[k]) && is_zero(wo[k + 1]) && is_zero(wo[k + 2])) continue;  // adds exactly 0
            const double ux = (layer ? vfac(wo[k], c.eps_h) : fo1) * wo[k + 1];
            const double s = dt * (ux * tanR);
            w[k + 1] = fmad(s, wo[k + 2], w[k + 1]);
            w[k + 2] = fmad(-s, wo[k + 1], w[k + 2]);
        }
    }
    // single layer: the granular layer is empty before and after the Euler
    // update (h2 = q2 = 0 in both), so its friction and Coulomb terms are zeros
    if (ONE) {
        filtro<false>(w, dt, c);
        dis_implicita<false>(wo, w, dt, c, fo1);
    } else if (is_zero(wo[3]) && is_zero(wo[4]) && is_zero(wo[5]) && is_zero(w[3]) && is_zero(w[4]) && is_zero(w[5])) {
        filtro<false>(w, dt, c);
        dis_implicita<false>(wo, w, dt, c, fo1);
        w[4] = w[4] * 0.0;  // coulomb() with h2 = 0
        w[5] = w[5] * 0.0;
    } else {
        filtro<true>(w, dt, c);
        dis_implicita<true>(wo, w, dt, c, fo1);
        coulomb(w, dt, c);
    }
}

}  // namespace lsh
