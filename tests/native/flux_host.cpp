// TEST INFRASTRUCTURE: the flux pass and cell update (flux_edge, update_cell)
// against the colour passes (do_edge, volume_cell), both compiled for the
// host: the same steps from the same state, every field and rate bit for bit.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../landslidehysea_gb300/csrc/lsh_adjoint.cuh"
#include "../../landslidehysea_gb300/csrc/lsh_setup.h"

using namespace lsh;

namespace lsh { void set_last_error(const std::string&) {} }

namespace {

using Vec = std::vector<double>;

struct Grid {
    lsh_params p;
    size_t N;
    Vec geo, X[7], Y[6], acc[7], sx[7], sy[7], eh, ev, em, et;
    std::vector<unsigned char> zero, kh, kv;
    std::vector<unsigned> mark, mark2;
    TimeRec tm{};
    explicit Grid(const lsh_params& q, const double* const* W) : p(q), N(size_t(q.nx) * q.ny) {
        const size_t st = size_t(p.ny) + 1;
        geo.assign(7 * st, 0.0);
        fill_geo(p, geo.data(), st);
        for (int k = 0; k < 7; ++k) { X[k].assign(W[k], W[k] + N); acc[k].assign(N, 0.0); sx[k].assign(N, 0.0); sy[k].assign(N, 0.0); }
        for (auto& y : Y) y.assign(N, 0.0);
        // garbage where an edge's planes are not written
        eh.assign(kEdgePlanes * (N + p.nx), 1e300);
        ev.assign(kEdgePlanes * (N + p.ny), 1e300);
        kh.assign(N + p.nx, 77);
        kv.assign(N + p.ny, 77);
        mark.assign(N, 0u);
        mark2.assign(N, 0u);
        zero.assign(N, 0);
        em.assign(N, -1e300);
        et.assign(N, 0.0);
    }
    KArgs args(int stage) {
        KArgs a;
        std::memset(&a, 0, sizeof(a));
        a.c = make_consts(p);
        const size_t st = size_t(p.ny) + 1;
        const double* g = geo.data();
        a.geo = Geo{g, g + 6 * st, g + st, g + 2 * st, g + 3 * st, g + 4 * st, g + 5 * st};
        for (int k = 0; k < 7; ++k) { a.acc[k] = acc[k].data(); a.sx[k] = a.sxw[k] = sx[k].data(); a.sy[k] = a.syw[k] = sy[k].data(); }
        for (int k = 0; k < 6; ++k) {
            a.W[k] = stage ? Y[k].data() : X[k].data();
            a.Wout[k] = (p.order == 2 && !stage) ? Y[k].data() : X[k].data();
            a.Xavg[k] = X[k].data();
        }
        a.W[6] = X[6].data();
        a.tm = &tm;
        a.szero = (p.order == 2) ? zero.data() : nullptr;
        a.eta_max = em.data();
        a.eta_time = et.data();
        a.eb.q[0] = eh.data(); a.eb.q[1] = ev.data();
        a.eb.plane[0] = N + p.nx; a.eb.plane[1] = N + p.ny;
        a.eb.kind[0] = kh.data(); a.eb.kind[1] = kv.data();
        a.eb.mark[0] = mark.data(); a.eb.mark[1] = mark2.data();
        a.eb.stage = unsigned(stage);
        if (p.order == 1) {
            a.eb.depth[0] = a.eb.depth_out[0] = Y[0].data();
            a.eb.depth[1] = a.eb.depth_out[1] = Y[3].data();
        } else {
            a.eb.depth[0] = a.W[0]; a.eb.depth[1] = a.W[3];
        }
        return a;
    }
};

template <int ORDER, int MODE>
unsigned long long stage(Grid& g, int st, bool flux, double dt, long long* marked) {
    KArgs a = g.args(st);
    const int nx = g.p.nx, ny = g.p.ny;
    if (ORDER == 2) for (size_t id = 0; id < g.N; ++id) recon_cell(a, int(id));
    unsigned long long r = 0;
    if (flux) {
        for (int y = 0; y <= ny; ++y) for (int x = 0; x < nx; ++x) flux_edge<ORDER>(a, 0, x, y, dt);
        for (int y = 0; y < ny; ++y) for (int x = 0; x <= nx; ++x) flux_edge<ORDER>(a, 1, x, y, dt);
        for (size_t id = 0; id < g.N; ++id) *marked += (g.mark[id] == stage_mark(a)) + (g.mark2[id] == stage_mark(a));
        for (int j = 0; j < ny; ++j) for (int i = 0; i < nx; ++i) { bool busy = false; const unsigned long long b = update_cell<MODE>(a, i, j, dt, busy); r = b > r ? b : r; }
    } else {
        for (int y = 0; y <= ny; y += 2) for (int x = 0; x < nx; ++x) do_edge<0, true, ORDER>(a, x, y, dt);
        for (int y = 1; y <= ny; y += 2) for (int x = 0; x < nx; ++x) do_edge<0, false, ORDER>(a, x, y, dt);
        for (int y = 0; y < ny; ++y) for (int x = 0; x <= nx; x += 2) do_edge<1, false, ORDER>(a, x, y, dt);
        for (int y = 0; y < ny; ++y) for (int x = 1; x <= nx; x += 2) do_edge<1, false, ORDER>(a, x, y, dt);
        for (size_t id = 0; id < g.N; ++id) { const unsigned long long b = volume_cell<MODE>(a, int(id), dt); r = b > r ? b : r; }
    }
    return r;
}

unsigned long long step(Grid& g, bool flux, double dt, long long* marked) {
    unsigned long long r;
    if (g.p.order == 1) r = stage<1, 0>(g, 0, flux, dt, marked);
    else { r = stage<2, 1>(g, 0, flux, dt, marked); stage<2, 2>(g, 1, flux, dt, marked); }
    g.tm.steps += 1;
    g.tm.t += dt;
    return r;
}

}  // namespace

extern "C" {

// One recomputed stage of step dt from W both ways (update_cell keeping its accumulators; the colour passes, copied
// between): the number of accumulators, partial sums at cells with a wet edge, and branch tapes that differ.
long long fluxc_keep(const lsh_params* p, const double* const* W, double dt) {
    Grid a(*p, W), b(*p, W);
    const int nx = p->nx, ny = p->ny, order = p->order;
    const size_t N = a.N;
    KArgs ka = a.args(0), kb = b.args(0);
    ka.eb.depth[0] = ka.W[0]; ka.eb.depth[1] = ka.W[3];  // nothing is updated in place
    ka.eb.depth_out[0] = ka.eb.depth_out[1] = nullptr;
    long long bad = 0;
    Vec sa[3][2], sb[3][2];
    for (int c = 0; c < 3; ++c)
        for (int l = 0; l < 2; ++l) { sa[c][l].assign(N, 7.0); sb[c][l].assign(N, 0.0); ka.part[c][l] = sa[c][l].data(); }
    for (int k = 0; k < 7; ++k) std::fill(a.acc[k].begin(), a.acc[k].end(), 7.0);
    if (order == 2)
        for (size_t id = 0; id < N; ++id) {
            bad += recon_cell(ka, int(id)) != recon_tape_cell(kb.W, nx, ny, int(id));
            bad += recon_cell_loaded(kb, int(id)) != recon_tape_cell(kb.W, nx, ny, int(id));
        }
    auto flux = [&](int dir, int x, int y) { order == 2 ? flux_edge<2>(ka, dir, x, y, dt) : flux_edge<1>(ka, dir, x, y, dt); };
    for (int y = 0; y <= ny; ++y) for (int x = 0; x < nx; ++x) flux(0, x, y);
    for (int y = 0; y < ny; ++y) for (int x = 0; x <= nx; ++x) flux(1, x, y);
    for (int j = 0; j < ny; ++j) for (int i = 0; i < nx; ++i) { bool busy = false; update_cell<-1, true>(ka, i, j, dt, busy); }
    auto copy = [&](int c) { for (int l = 0; l < 2; ++l) sb[c][l] = b.acc[3 * l]; };
    for (int y = 0; y <= ny; y += 2) for (int x = 0; x < nx; ++x) order == 2 ? do_edge<0, true, 2>(kb, x, y, dt) : do_edge<0, true, 1>(kb, x, y, dt);
    copy(0);
    for (int y = 1; y <= ny; y += 2) for (int x = 0; x < nx; ++x) order == 2 ? do_edge<0, false, 2>(kb, x, y, dt) : do_edge<0, false, 1>(kb, x, y, dt);
    copy(1);
    for (int y = 0; y < ny; ++y) for (int x = 0; x <= nx; x += 2) order == 2 ? do_edge<1, false, 2>(kb, x, y, dt) : do_edge<1, false, 1>(kb, x, y, dt);
    copy(2);
    for (int y = 0; y < ny; ++y) for (int x = 1; x <= nx; x += 2) order == 2 ? do_edge<1, false, 2>(kb, x, y, dt) : do_edge<1, false, 1>(kb, x, y, dt);
    for (size_t id = 0; id < N; ++id) {
        const size_t j = id / nx;
        const bool wet = a.kh[id] | a.kh[id + nx] | a.kv[id + j] | a.kv[id + j + 1];
        for (int k = 0; k < 7; ++k) bad += lshm::bits_of(a.acc[k][id]) != lshm::bits_of(b.acc[k][id]);
        for (int c = 0; c < 3 && wet; ++c)
            for (int l = 0; l < 2; ++l) bad += lshm::bits_of(sa[c][l][id]) != lshm::bits_of(sb[c][l][id]);
    }
    return bad;
}

// Runs `nsteps` steps of size dt (the lagged CFL step when dt <= 0) both ways from W (7 arrays); returns the number of
// values that differ in their bits; *marked: cells around which the limiter was evaluated.  A run ends with its first
// value that is not finite, as the product's does (LSH_ERR_NUMERIC).
long long fluxc_compare(const lsh_params* p, const double* const* W, int nsteps, double dt0, double dt_fixed,
                        long long* marked) {
    Grid a(*p, W), b(*p, W);
    long long bad = 0, none = 0;
    *marked = 0;
    double dt = dt0;
    for (int n = 0; n < nsteps; ++n) {
        const unsigned long long ra = step(a, true, dt, marked), rb = step(b, false, dt, &none);
        if (b.tm.err) return bad + (a.tm.err != b.tm.err);
        bad += (ra != rb);
        for (int k = 0; k < 6; ++k)
            for (size_t i = 0; i < a.N; ++i) {
                const double u = a.X[k][i], v = b.X[k][i];
                bad += (lshm::bits_of(u) != lshm::bits_of(v)) && !(u != u && v != v);
            }
        for (size_t i = 0; i < a.N; ++i) bad += (a.em[i] != b.em[i]) + (a.et[i] != b.et[i]);
        dt = (dt_fixed > 0.0) ? dt_fixed : dt_of(rb, 2.0 * p->cfl);
        if (bad) break;
    }
    return bad;
}

}  // extern "C"
