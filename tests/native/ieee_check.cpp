// Host check of the integer division, reciprocal and square root steps
// (lsh_ieee.h) against the host's IEEE operations, with the approximation
// instruction replaced by any value inside its documented error bound.
#include <cstdint>
#include <cstring>

#include "../../landslidehysea_gb300/csrc/lsh_ieee.h"

namespace {

double g_err = 0.0;  // relative error of the seed, set by the caller

struct Seed {
    static float rcp(float x) { return (float)((1.0 / (double)x) * (1.0 + g_err)); }
    static float rsqrt(float x) { return (float)((1.0 / std::sqrt((double)x)) * (1.0 + g_err)); }
};

void split(double x, uint32_t& lo, uint32_t& hi) { lshm::halves(x, lo, hi); }

bool differ(double a, double b) { return lshm::bits_of(a) != lshm::bits_of(b); }

}  // namespace

extern "C" {

// Mismatches of op (0: a / b, 1: 1 / b, 2: sqrt(b)) over n operand pairs of
// positive or negative normal values, with the seed's relative error `err`
// on top of its rounding to FP32.
long long ieeec_check(int op, const double* a, const double* b, long long n, double err) {
    g_err = err;
    long long bad = 0;
    for (long long i = 0; i < n; ++i) {
        uint32_t alo, ahi, blo, bhi;
        split(a[i], alo, ahi);
        split(b[i], blo, bhi);
        const uint32_t ea = (ahi >> 20) & 0x7ffu, eb = (bhi >> 20) & 0x7ffu;
        if (op == 0) {
            if (ea - 1u >= 2046u || eb - 1u >= 2046u || ea - eb + 1021u > 2043u) continue;
            bad += differ(lshm::div_normal<Seed>(alo, ahi, blo, bhi), a[i] / b[i]);
        } else if (op == 1) {
            if (eb - 1u >= 2044u) continue;
            bad += differ(lshm::rcp_normal<Seed>(blo, bhi), 1.0 / b[i]);
        } else {
            if (bhi - 0x00100000u >= 0x7fe00000u) continue;
            bad += differ(lshm::sqrt_normal<Seed>(blo, bhi), std::sqrt(b[i]));
        }
    }
    return bad;
}

}  // extern "C"
