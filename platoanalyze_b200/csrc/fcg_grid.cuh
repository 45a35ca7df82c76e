// Cooperative form of the flexible-CG iterations (fcg_grid.cu), used by fcg_poly (mixed.cu).
#pragma once

#include "grid.cuh"
#include "plato_internal.cuh"

namespace plato {

struct ChebCoef {
    float c0;      // first step: d = c0 Dinv r
    float c1[64];  // step k: d_k = c1[k] d_(k-1) + c2[k] Dinv res
    float c2[64];
};

// Whether this system's iterations can run in cooperative launches: the device has them, every slice has a warp, nothing
// wants a look between the stages (sampled timings, deflation), and no earlier launch gave up.
bool fcg_grid_ok(const plato_problem* h);

// Enqueues one launch: up to some hundred iterations from "p and p.r are there", with the coarse
// correction when coarse = 1.  Returns at once on the device when the scalars say done.
int fcg_grid_iterations(plato_problem* h, int entry_bytes, bool half_entries, const void* vin, const ChebCoef& cc, int degree,
                        int coarse, double* x, const float* scale, int32_t max_it);

// Whether a wait ran out in a launch since the last call (synchronises the stream).
int fcg_grid_gave_up(plato_problem* h, int* gave_up);

}  // namespace plato
