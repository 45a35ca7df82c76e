// Grid-wide sums and barriers of the cooperative Krylov kernels (pcg_grid.cu, fcg_grid.cu).
#pragma once

#include "solver_common.cuh"

namespace plato {

// A grid-wide sum: every CTA writes its block sums to its place of a box, adds one to a counter
// (release), and one of its threads waits until the counter has reached the number of CTAs times the
// number of this barrier (acquire); then all CTAs read the box and add it in CTA order, so all of
// them get the same bits.  Two boxes alternate: a CTA that writes barrier n + 2 has seen everyone at
// n + 1, hence done with reading n.  One waiting thread per CTA keeps the counter's cache line free for
// the arrivals; with every CTA polling every other's place, 80 CTAs took 2.6 us longer per barrier
// than 8.  Every wait has a limit; when one runs out the CTA raises `abort`, all CTAs leave, and the
// host goes on with the launch-per-stage loop from the x that is there.
constexpr uint32_t kGridPolls = 1u << 22;  // a second or two
constexpr int kGridValues = 2;             // values of one sum at most
constexpr int kGridSmemMax = 224 * 1024;   // dynamic shared memory: the opt-in limit less the static arrays

struct GridBox {
    double*   box;    // [2][kGridValues][gridDim.x]
    uint32_t* count;  // arrivals in this launch
    int32_t*  abort;
    uint32_t  polls;  // limit of a wait
    int32_t   stall_cta;      // test hook: this CTA's wait at this barrier is for arrivals that never come
    uint32_t  stall_barrier;  // (0: none)
};

// acquire-release at GPU scope; __threadfence() is the sequentially consistent one, which costs more
__device__ __forceinline__ void grid_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Thread 0 of a CTA whose other threads' writes a __syncthreads() has put before this.
__device__ __forceinline__ bool grid_arrive_and_wait(const GridBox& a, uint32_t barrier) {
    uint32_t target = barrier * gridDim.x;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.count) : "memory");
    if (barrier == a.stall_barrier && int(blockIdx.x) == a.stall_cta) target += 1u << 30;
    for (uint32_t polls = 1;; ++polls) {
        uint32_t v;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.count) : "memory");
        if (int32_t(v - target) >= 0) break;
        if ((polls & 1023u) == 0 && (polls >= a.polls || *reinterpret_cast<volatile int32_t*>(a.abort))) {
            *reinterpret_cast<volatile int32_t*>(a.abort) = 1;
            return false;
        }
    }
    grid_fence();
    return true;
}

// Sums NV values over the grid (the same bits in every thread) and orders all global writes before
// it ahead of all reads after it.  `barrier` counts the barriers of the launch from 1.  False when a wait
// ran out or another CTA gave up.
template <int NV>
__device__ __forceinline__ bool grid_sum(double (&v)[NV], const GridBox& a, uint32_t barrier, double (*sh_cta)[32],
                                         double (*sh_grid)[32]) {
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31, G = gridDim.x;
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = warp_sum(v[q]);
    if (l == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) sh_cta[q][w] = v[q];
    __syncthreads();
    double* box = a.box + (barrier & 1u) * kGridValues * G;
    bool ok = true;
    if (w == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = warp_sum(l < nw ? sh_cta[q][l] : 0.0);
        if (l == 0) {
#pragma unroll
            for (int q = 0; q < NV; ++q) *reinterpret_cast<volatile double*>(box + q * G + blockIdx.x) = v[q];
            ok = grid_arrive_and_wait(a, barrier);
        }
    }
    if (__syncthreads_or(!ok)) return false;
    double got[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) got[q] = warp_sum(tid < G ? *reinterpret_cast<volatile double*>(box + q * G + tid) : 0.0);
    if (l == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) sh_grid[q][w] = got[q];
    __syncthreads();
    const int nw = (G + 31) >> 5;  // the grid has no more CTAs than a CTA has threads
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        v[q] = 0.0;
        for (int i = 0; i < nw; ++i) v[q] += sh_grid[q][i];
    }
    return true;
}

// The same without values: every write before it in the grid is seen by every read after it.
__device__ __forceinline__ bool grid_barrier(const GridBox& a, uint32_t barrier) {
    __syncthreads();
    const bool ok = threadIdx.x != 0 || grid_arrive_and_wait(a, barrier);
    return !__syncthreads_or(!ok);
}

// The same sum over the CTAs of one cluster (at most 16, the whole grid): each CTA writes its block sums
// into every CTA's box through distributed shared memory, and the cluster's hardware barrier is the only
// wait (an iteration with two sums of a 12x6x6 system 7 -> 4.8 us).  The CTAs' threads call it in step; the first
// call comes after a cluster_barrier(), since a CTA's shared memory exists only once it runs.
constexpr int kClusterMax = 16;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

template <int NV>
__device__ __forceinline__ void cluster_sum(double (&v)[NV], uint32_t barrier, double (*sh_cta)[32],
                                            double (*box)[kGridValues][kClusterMax]) {
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31, G = gridDim.x;
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = warp_sum(v[q]);
    if (l == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) sh_cta[q][w] = v[q];
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const double s = warp_sum(l < nw ? sh_cta[q][l] : 0.0);  // in all lanes
            if (l < G) {
                const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(&box[barrier & 1u][q][blockIdx.x]));
                uint32_t peer;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(mine), "r"(l));
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(peer), "d"(s) : "memory");
            }
        }
    }
    cluster_barrier();
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        v[q] = 0.0;
        for (int i = 0; i < G; ++i) v[q] += box[barrier & 1u][q][i];
    }
}

// Cooperative launch of one CTA per SM.
template <typename Args>
inline cudaError_t launch_cooperative(void (*kernel)(Args), int grid, int block, size_t smem, cudaStream_t stream,
                                      const Args& args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(unsigned(block));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args);
}

// What a warp does in a CTA whose `warps` warps form groups of `parts`, a group per slice: its part of the
// slice and its group.  Where `parts` does not divide `warps`, the warps that are left over belong to no
// group and lead none.
struct WarpRole {
    int  part, group;
    bool leader;  // keeps the rows' vectors and adds the other parts' sums to its own
};
__host__ __device__ __forceinline__ WarpRole warp_role(int warp, int parts, int warps) {
    const int group = warp / parts, part = warp - group * parts;
    return {part, group, part == 0 && group < warps / parts};
}

// The boxes, counter and abort flag of a handle for its next launch: the counter is cleared, and a stall that the
// test hook asked for is taken up (pcg_grid.cu).
int grid_box(plato_problem* h, GridBox* box);

}  // namespace plato
