// The coarse box grid of the two-level preconditioner, as its kernels see it (coarse.cu, fcg_grid.cu).
#pragma once

#include "plato_internal.cuh"

namespace plato {

struct CoarseView {
    int nc0, nc1, nc2;
    double x0, y0, z0, hx, hy, hz;
    double ihx, ihy, ihz;  // 1 / h: local coordinates of the hot kernels are (x - lo) * ih
};

__host__ __device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ void cell_of(const CoarseView& cv, double x, double y, double z, int& cx, int& cy,
                                        int& cz) {
    cx = clampi(int(floor((x - cv.x0) / cv.hx)), 0, cv.nc0 - 1);
    cy = clampi(int(floor((y - cv.y0) / cv.hy)), 0, cv.nc1 - 1);
    cz = clampi(int(floor((z - cv.z0) / cv.hz)), 0, cv.nc2 - 1);
}

__device__ __forceinline__ int cell_id(const CoarseView& cv, int cx, int cy, int cz) {
    return (cx * cv.nc1 + cy) * cv.nc2 + cz;
}

__device__ __forceinline__ int coarse_node(const CoarseView& cv, int ix, int iy, int iz) {
    return (ix * (cv.nc1 + 1) + iy) * (cv.nc2 + 1) + iz;
}

// trilinear weight of corner (bx,by,bz) at local coordinates (u,v,w)
__device__ __forceinline__ double corner_weight(int b, double u, double v, double w) {
    return ((b & 4) ? u : 1.0 - u) * ((b & 2) ? v : 1.0 - v) * ((b & 1) ? w : 1.0 - w);
}

// Sums 24 values per lane over a warp; lanes with (lane & 3) == 0 get three sums each, values
// warp_sum24_first(lane) to + 2.
__device__ __forceinline__ void warp_sum24(const double (&s)[24], int lane, double (&t3)[3]) {
    // warp sums of the 24 values by halving: each exchange hands half of a lane's values to its
    // partner, so after offsets 16, 8, 4 a lane holds 3 of the 24 sums (which 3 set by lane bits
    // 4..2) and offsets 2, 1 finish them -- 27 shuffles instead of 24 x 5
    double t12[12], t6[6];
    {
        const bool hi = (lane & 16) != 0;
#pragma unroll
        for (int i = 0; i < 12; ++i) {
            const double send = hi ? s[i] : s[12 + i];
            t12[i] = (hi ? s[12 + i] : s[i]) + __shfl_xor_sync(0xffffffffu, send, 16);
        }
    }
    {
        const bool hi = (lane & 8) != 0;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const double send = hi ? t12[i] : t12[6 + i];
            t6[i] = (hi ? t12[6 + i] : t12[i]) + __shfl_xor_sync(0xffffffffu, send, 8);
        }
    }
    {
        const bool hi = (lane & 4) != 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double send = hi ? t6[i] : t6[3 + i];
            t3[i] = (hi ? t6[3 + i] : t6[i]) + __shfl_xor_sync(0xffffffffu, send, 4);
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        t3[i] += __shfl_xor_sync(0xffffffffu, t3[i], 2);
        t3[i] += __shfl_xor_sync(0xffffffffu, t3[i], 1);
    }
}
__device__ __forceinline__ int warp_sum24_first(int lane) {
    return ((lane & 16) ? 12 : 0) + ((lane & 8) ? 6 : 0) + ((lane & 4) ? 3 : 0);
}

CoarseView coarse_view(const plato_problem* h);

}  // namespace plato
