// TEST INFRASTRUCTURE: the loop of lsh_run_until over a clock that fails on request.
#include "../../landslidehysea_gb300/csrc/lsh_scheme.cuh"
#include "../../landslidehysea_gb300/csrc/lsh_run_until.h"

namespace {

// The device's record beside the host's copy.  The step call `fail_step` (counted from 1; 0: none) launches half of its
// steps and reports 7; so does the reading `fail_read`, which changes nothing.
struct Fake {
    lsh::TimeRec dev{}, host{};
    int steps_called = 0, reads = 0, fail_step = 0, fail_read = 0, stuck = 0;
    long long launched = 0;
    lsh::TimeRec& rec() { return host; }
    int read() {
        if (++reads == fail_read || (stuck && reads >= fail_read)) return 7;
        host = dev;
        return 0;
    }
    int put(double t_end) {
        host.t_end = t_end;
        host.done = host.t >= t_end || host.err;
        dev = host;
        return 0;
    }
    void one() {
        ++launched;
        if (dev.done) return;
        dev.t += dev.dt;
        dev.steps += 1;
        dev.done = dev.t >= dev.t_end;
    }
    int step(int n) {
        const bool bad = (++steps_called == fail_step);
        for (int i = 0; i < (bad ? (n + 1) / 2 : n); ++i) one();
        return bad ? 7 : 0;
    }
    int failed() { return host.err; }
};

}  // namespace

// out: device t, steps, t_end, done; steps_done; steps launched
extern "C" int rununtil(double dt, double t_end, long long max_steps, int most, int fail_step, int fail_read, int stuck,
                        double out[6]) {
    Fake f;
    f.dev.dt = dt;
    f.dev.t_end = INFINITY;
    f.fail_step = fail_step;
    f.fail_read = fail_read;
    f.stuck = stuck;
    long long done = -1;
    const int status = lsh::run_until(f, t_end, max_steps, most, &done);
    out[0] = f.dev.t; out[1] = (double)f.dev.steps; out[2] = f.dev.t_end; out[3] = f.dev.done; out[4] = (double)done;
    out[5] = (double)f.launched;
    return status;
}
