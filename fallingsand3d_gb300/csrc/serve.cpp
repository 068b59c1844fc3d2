// The request stream of the serving loop: seeded Poisson arrivals of worlds of
// seeded sizes and step counts.
#include <math.h>
#include <string.h>

#include "fs3d_common.h"
#include "pcg.h"

using namespace fs3d;

extern "C" {

fs3d_status fs3d_serve_plan(const fs3d_serve_params* p, int64_t capacity, fs3d_serve_request* reqs,
                            int64_t* n_reqs) {
    if (!p || !n_reqs || p->lambda <= 0.0 || p->duration_s <= 0.0 || capacity < 0 || (capacity > 0 && !reqs))
        return set_error(FS3D_ERR_INVALID_ARG, "fs3d_serve_plan: bad args");
    static const int kDims[7] = {16, 24, 32, 48, 64, 96, 128};
    const int lo = p->min_steps > 0 ? p->min_steps : 10, hi = p->max_steps > 0 ? p->max_steps : 1000;
    if (hi < lo) return set_error(FS3D_ERR_INVALID_ARG, "fs3d_serve_plan: max_steps < min_steps");
    Pcg32 r(p->master_seed, 0xC4u);
    double t = 0.0;
    int64_t n = 0;
    const int64_t cap = p->max_requests > 0 ? p->max_requests : INT64_MAX;
    for (;;) {
        // exponential inter-arrival time from a 32-bit draw in (0, 1)
        const double u = ((double)r.next() + 0.5) / 4294967296.0;
        t += -log(u) / p->lambda;
        if (t > p->duration_s || n >= cap) break;
        int d[3];
        for (int& v : d) v = kDims[r.bounded(7u)];
        const double v = ((double)r.next() + 0.5) / 4294967296.0;
        int steps = (int)floor(exp(log((double)lo) + v * (log((double)hi) - log((double)lo))));
        steps = steps < lo ? lo : (steps > hi ? hi : steps);
        if (n < capacity) {
            fs3d_serve_request& q = reqs[n];
            memset(&q, 0, sizeof(q));
            q.arrival_s = t;
            q.X = d[0];
            q.Y = d[1];
            q.Z = d[2];
            q.n_steps = steps;
            q.seed = fmix64(p->master_seed ^ (0x5E7E000000000000ull + (uint64_t)n));
        }
        ++n;
    }
    *n_reqs = n;
    return FS3D_OK;
}

}  // extern "C"
