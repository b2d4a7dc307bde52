// lsh_run_until.h -- the loop of lsh_run_until (include/lsh.h), apart from the
// device so that a host test can make its calls fail.
#pragma once

#include <algorithm>
#include <cmath>

namespace lsh {

// Clock: read() fetches the device's time record into rec() and waits for the
// work before it; put(t_end) writes rec() back with that t_end; step(n) launches
// n steps; failed() is the record's own error as a status.
// `most`: steps launched between two readings at most.
template <class Clock>
int run_until(Clock& c, double t_end, long long max_steps, int most, long long* steps_done) {
    if (int s = c.read()) return s;
    if (int s = c.put(t_end)) return s;
    const long long start = c.rec().steps;
    int status = 0;
    while (!c.rec().done) {
        const long long left = (max_steps > 0) ? max_steps - (c.rec().steps - start) : (1LL << 40);
        if (left <= 0) break;
        // Steps past t_end find the record done and do nothing, but are launched
        // all the same: as many as the next step's dt needs to get there (6
        // readings 8 steps apart on a 512^2 fjord: 47 ms with batches of 128).
        const double need = std::ceil((t_end - c.rec().t) / c.rec().dt);
        int batch = (int)std::min<long long>(left, most);
        if (need < batch) batch = std::max(1, (int)need);
        if ((status = c.step(batch))) break;
        if ((status = c.read())) break;
    }
    // After a failure the record that the host holds may be older than the
    // state, some of the steps having been launched: written back it would take
    // the clock to before them.
    const bool current = (status == 0) || c.read() == 0;
    if (steps_done) *steps_done = c.rec().steps - start;
    if (status == 0) status = c.failed();
    if (!current) return status;
    // step-count mode again for later steps
    const int s2 = c.put(INFINITY);
    return status ? status : s2;
}

}  // namespace lsh
