// The Jacobi-PCG iterations of systems that fit on the chip, in one cooperative launch.
//
// A system of a few thousand to some hundred thousand rows leaves a kernel of the launch-per-stage
// loop (solver.cu) idle most of the time: its launch, its last-block reduction and the gap to
// the next one cost far more than the arithmetic (20x10x10 cantilever, 455 iterations: 31.5 us
// an iteration for three kernels over a 2.4 MB matrix).  Here one CTA per SM owns a run of SELL
// slices for the whole solve: its part of the matrix stays in shared memory when it fits (else it
// is read from L2), its rows' x, r, p, A p and inverse diagonal stay in registers, and an
// iteration is
//   A p with p = z + beta p formed at each gathered column   -> sum p.Ap over the grid -> alpha
//   x += alpha p, r -= alpha A p, z = Dinv r                 -> sums r.z, r.r          -> beta
// so two grid-wide sums per iteration, which are also its two barriers.  Only z and p leave the SM.
// Bound by the two sums (1.5 to 3 us each).  Solve of a cantilever with a random density to 1e-8, launch per stage
// against this: 12x6x6 6.9 -> 1.2 ms and 20x10x10 12.7 -> 2.2 (as one cluster, see pcg_split), 30x16x16 19.7 -> 4.6, 40x20x20
// 24.6 -> 6.3, 60x30x30 42.0 -> 18.1, 64x32x32 70.9 -> 19.6, 72x31x31 (2,336 of the 2,368 slices that qualify) 75.5 ->
// 28.0.  Density filter (one unknown per row) to 1e-12: 20x10x10 0.74 -> 0.25 ms, 80x40x40 2.77 -> 1.45, 100x50x50 5.34
// -> 2.57, 106x52x51 (9,217 of 9,472 slices, two to a warp) 5.58 -> 3.17.
#include <algorithm>
#include <utility>

#include "grid.cuh"
#include "plato_internal.cuh"

namespace plato {

int ensure_smem_attribute(plato_problem* h, const void* kernel, int bytes);
SellView sell_view(const plato_problem* h);

namespace {

constexpr int kLaunchIters = 2048;         // iterations per launch: some ten milliseconds
static_assert(kLaunchIters % 2 == 0, "the direction buffers swap once per iteration");

struct GridPcg {
    SellView      A;
    int32_t       nslices;
    int32_t       ks;        // warps per slice group
    const double* vals;
    const double* dinv;
    double*       x;
    double*       r;
    double*       z;
    double*       p[2];
    int32_t       pcur;      // buffer that holds the current direction
    int32_t       max_it;
    int32_t       smem_bytes;
    GridBox       box;
    PcgScalars*   S;
};

// NB unknowns per row (3: block SELL, 1: scalar SELL), T slices per group of ks warps.
// CLUSTER: the grid is one cluster.
template <int NB, int T, int THREADS, bool CLUSTER>
__global__ void __launch_bounds__(THREADS, 1) k_pcg_grid(GridPcg a) {
    extern __shared__ __align__(16) unsigned char grid_smem[];
    __shared__ double sh_cta[2][32], sh_grid[2][32];
    __shared__ double box[CLUSTER ? 2 : 1][kGridValues][kClusterMax];
    __shared__ double part[NB][THREADS];
    constexpr int NE = NB * NB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s0 = int((int64_t)a.nslices * blockIdx.x / gridDim.x), s1 = int((int64_t)a.nslices * (blockIdx.x + 1) / gridDim.x);
    const WarpRole role = warp_role(warp, a.ks, THREADS / 32);
    const int kg = role.part, group = role.group, groups = (THREADS / 32) / a.ks;
    const bool leader = role.leader;

    // this CTA's slots in shared memory, when they fit
    const int64_t first = a.A.ptr[s0], slots = a.A.ptr[s1] - first;
    const double* vals = a.vals + NE * first;
    const int32_t* cols = a.A.cols + first;
    if (slots * (8 * NE + 4) <= a.smem_bytes) {
        double* sv = reinterpret_cast<double*>(grid_smem);
        int32_t* sc = reinterpret_cast<int32_t*>(sv + NE * slots);
        for (int64_t i = tid; i < NE * slots; i += THREADS) sv[i] = __ldg(vals + i);
        for (int64_t i = tid; i < slots; i += THREADS) sc[i] = __ldg(cols + i);
        vals = sv;
        cols = sc;
    }

    double x[T][NB], r[T][NB], p[T][NB], ap[T][NB], di[T][NB];
    int32_t width[T];
    int32_t base[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int s = s0 + group + t * groups;
        const int64_t row = 32 * int64_t(s) + lane;
        width[t] = s < s1 ? a.A.width[s] : 0;
        base[t] = s < s1 ? int32_t(a.A.ptr[s] - first) : 0;
        const bool own = leader && s < s1 && row < a.A.num_rows;
#pragma unroll
        for (int d = 0; d < NB; ++d) {
            x[t][d] = own ? a.x[NB * row + d] : 0.0;
            r[t][d] = own ? a.r[NB * row + d] : 0.0;
            p[t][d] = own ? a.p[a.pcur][NB * row + d] : 0.0;
            di[t][d] = own ? a.dinv[NB * row + d] : 0.0;
        }
    }
    double rz = a.S->rz, rr = a.S->rr, beta = a.S->beta, pap = 0.0, alpha = 0.0;
    const double tol2 = a.S->tol2;
    int32_t iter = a.S->iter, done = a.S->done, nonfinite = a.S->nonfinite;
    uint32_t epoch = 0;  // barriers of this launch
    int pcur = a.pcur;
    if constexpr (CLUSTER) cluster_barrier();
    else __syncthreads();

    for (int it = 0; it < kLaunchIters && !done; ++it) {
        const double* pold = a.p[pcur];
        double* pnew = a.p[pcur ^ 1];
        double s2[2] = {0.0, 0.0};
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int s = s0 + group + t * groups;
            double acc[NB];
#pragma unroll
            for (int d = 0; d < NB; ++d) acc[d] = 0.0;
            const int32_t* c0 = cols + base[t] + lane;
            const double* v0 = vals + NE * base[t] + lane;
#pragma unroll 4
            for (int k = kg; k < width[t]; k += a.ks) {
                const int64_t c = c0[32 * k];
                double pc[NB];
#pragma unroll
                for (int d = 0; d < NB; ++d) pc[d] = a.z[NB * c + d] + beta * pold[NB * c + d];
#pragma unroll
                for (int i = 0; i < NB; ++i)
#pragma unroll
                    for (int j = 0; j < NB; ++j) acc[i] += v0[32 * (NE * k + NB * i + j)] * pc[j];
            }
            if (a.ks > 1) {
                if (t > 0) __syncthreads();  // the leaders have read the slice before
#pragma unroll
                for (int d = 0; d < NB; ++d) part[d][tid] = acc[d];
                __syncthreads();
                if (leader)
#pragma unroll
                    for (int d = 0; d < NB; ++d)
                        for (int q = 1; q < a.ks; ++q) acc[d] += part[d][tid + 32 * q];
            }
            const int64_t row = 32 * int64_t(s) + lane;
            if (leader && s < s1 && row < a.A.num_rows) {
#pragma unroll
                for (int d = 0; d < NB; ++d) {
                    p[t][d] = di[t][d] * r[t][d] + beta * p[t][d];
                    pnew[NB * row + d] = p[t][d];
                    ap[t][d] = acc[d];
                    s2[0] += p[t][d] * acc[d];
                }
            }
        }
        pcur ^= 1;
        double s1v[1] = {s2[0]};
        if constexpr (CLUSTER) cluster_sum<1>(s1v, ++epoch, sh_cta, box);
        else if (!grid_sum<1>(s1v, a.box, ++epoch, sh_cta, sh_grid)) break;
        pap = s1v[0];
        alpha = rz / pap;
        if (!isfinite(alpha) || pap <= 0.0) {
            nonfinite = 1;
            done = 1;
            break;
        }
        s2[0] = s2[1] = 0.0;
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int s = s0 + group + t * groups;
            const int64_t row = 32 * int64_t(s) + lane;
            if (leader && s < s1 && row < a.A.num_rows) {
#pragma unroll
                for (int d = 0; d < NB; ++d) {
                    x[t][d] += alpha * p[t][d];
                    r[t][d] -= alpha * ap[t][d];
                    const double zi = di[t][d] * r[t][d];
                    a.z[NB * row + d] = zi;
                    s2[0] += r[t][d] * zi;
                    s2[1] += r[t][d] * r[t][d];
                }
            }
        }
        if constexpr (CLUSTER) cluster_sum<2>(s2, ++epoch, sh_cta, box);
        else if (!grid_sum<2>(s2, a.box, ++epoch, sh_cta, sh_grid)) break;
        beta = s2[0] / rz;
        rz = s2[0];
        rr = s2[1];
        ++iter;
        if (!isfinite(rz) || !isfinite(rr)) nonfinite = 1;
        if (nonfinite || rr <= tol2 || iter >= a.max_it) done = 1;
    }
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int s = s0 + group + t * groups;
        const int64_t row = 32 * int64_t(s) + lane;
        if (leader && s < s1 && row < a.A.num_rows)
#pragma unroll
            for (int d = 0; d < NB; ++d) {
                a.x[NB * row + d] = x[t][d];
                a.r[NB * row + d] = r[t][d];
            }
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.S->rz = rz;
        a.S->rz_new = rz;
        a.S->rr = rr;
        a.S->pAp = pap;
        a.S->alpha = alpha;
        a.S->beta = beta;
        a.S->iter = iter;
        a.S->nonfinite = nonfinite;
        a.S->done = done;
    }
}

template <int NB>
constexpr int grid_threads() { return NB == 3 ? 512 : 1024; }

template <int NB, int T>
int launch_grid(plato_problem* h, GridPcg& a, int grid) {
    constexpr int THREADS = grid_threads<NB>();
    const auto kernel = k_pcg_grid<NB, T, THREADS, false>;
    PLATO_RC(ensure_smem_attribute(h, reinterpret_cast<const void*>(kernel), a.smem_bytes));
    PLATO_CUDA(h, launch_cooperative(kernel, grid, THREADS, size_t(a.smem_bytes), h->stream, a));
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

// The launch as one cluster of `grid` CTAs; *ok is cleared, and nothing launched, where the device has no
// place for it.
template <int NB>
int launch_cluster(plato_problem* h, GridPcg& a, int grid, int* ok) {
    constexpr int THREADS = grid_threads<NB>();
    const auto kernel = k_pcg_grid<NB, 1, THREADS, true>;
    PLATO_RC(ensure_smem_attribute(h, reinterpret_cast<const void*>(kernel), a.smem_bytes));
    PLATO_CUDA(h, cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = size_t(a.smem_bytes);
    cfg.stream = h->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(grid);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
        (void)cudaGetLastError();
        *ok = 0;
        return PLATO_OK;
    }
    PLATO_CUDA(h, cudaLaunchKernelEx(&cfg, kernel, a));
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

}  // namespace

int grid_box(plato_problem* h, GridBox* box) {
    const size_t bytes = sizeof(double) * 2 * kGridValues * size_t(h->coop_sms);
    if (!h->grid_box) {
        PLATO_CUDA(h, cudaMalloc(&h->grid_box, bytes + 128));
        PLATO_CUDA(h, cudaMemsetAsync(h->grid_box, 0, bytes + 128, h->stream));
    }
    box->count = static_cast<uint32_t*>(h->grid_box);  // a cache line of its own
    box->abort = reinterpret_cast<int32_t*>(static_cast<char*>(h->grid_box) + 64);
    box->box = reinterpret_cast<double*>(static_cast<char*>(h->grid_box) + 128);
    PLATO_CUDA(h, cudaMemsetAsync(box->count, 0, sizeof(uint32_t), h->stream));
    const GridStall stall = std::exchange(h->grid_stall, GridStall{});
    box->polls = stall.barrier ? kGridPolls >> 6 : kGridPolls;
    box->stall_cta = stall.cta;
    box->stall_barrier = stall.barrier;
    return PLATO_OK;
}

// Whether the iterations of this system run in cooperative launches: the device has them, every slice has a
// group of warps (one slice a group for block systems, at most two for scalar ones), nothing else wants a
// look between iterations (sampled timings, a deflated direction), and no earlier launch gave up.
//
// A scalar system with 17 to 26 slices per SM gives each a warp and leaves the other 6 to 15 of the CTA idle.  With
// rows as narrow as a box's (15 blocks a slot row) the matrix is in shared memory and that does not matter (72x36x36, 22 slices,
// shuffled: 28.0 -> 18.6 us an iteration); Delaunay rows (27) are read from L2, and the launch per stage is the steadier
// one: 17 slices 20.6 us against 23.8, 20 shuffled 30.6 against 36.3, 22 RCM 22.8 against 28.0, shuffled 31.3 against 42, 26 23.8
// against 25.8 (RCM 26.3 against 23.4).  With 28 and 36 the loop wins again (36.2 -> 31.2, 41.6 -> 35.8 us), as with 16.
bool pcg_grid_ok(const plato_problem* h, int nb) {
    if (h->grid_off || h->timing || h->ritz_deflating) return false;
    const int64_t warps = (nb == 3 ? grid_threads<3>() : grid_threads<1>()) / 32, n = h->sell.nslices;
    if (n > int64_t(h->coop_sms) * warps * (nb == 3 ? 1 : 2)) return false;
    const bool wide = h->sell.total_slots > 20 * 32 * n;
    return !(nb == 1 && wide && n > 16 * int64_t(h->coop_sms) && n <= 26 * int64_t(h->coop_sms));
}

namespace {

// How a system of nslices slices with total_slots slots is laid over the SMs.
struct PcgSplit {
    int     grid, clustered;
    int     per_cta;     // slices of the largest share
    int     ks;          // warps per slice
    int     turns;       // slices a group of warps takes one after the other
    int64_t smem_bytes;  // dynamic shared memory (0: the matrix is read from L2)
};

PcgSplit pcg_split(int nslices, int64_t total_slots, int nb, int sms, bool may_cluster) {
    const int warps = (nb == 3 ? grid_threads<3>() : grid_threads<1>()) / 32;
    const int64_t room = kGridSmemMax - (nb == 3 ? 512 * 24 : 1024 * 8) - 2048;
    // shared memory for the average CTA's slots and a tenth more; a CTA with more reads L2
    const auto smem_for = [&](int ctas) { return (total_slots / ctas + 32) * (8 * nb * nb + 4) * 11 / 10; };
    // A system that gives each of 16 SMs its part in shared memory and each slice 3 warps (scalar: one) runs
    // as one cluster, whose barrier is a hardware one.  One grid-wide counter against this (densities of 0.01 to 1, to 1e-10): 12x6x6 2.0 -> 1.4 ms,
    // 18x9x9 3.0 -> 2.3, 20x10x10 (80 slices, 3 warps each) 3.2 -> 2.5; with 2 warps a slice 21x10x10 3.38 -> 3.41,
    // so the line lies there.  Filter: 16x8x8 0.49 -> 0.38 ms, 37x20x18 (474 slices, a warp each) 0.97 -> 0.86.
    int cluster = 1;
    while (2 * cluster <= std::min<int>(kClusterMax, nslices)) cluster *= 2;
    PcgSplit p{};
    p.clustered = may_cluster && (nslices + cluster - 1) / cluster * (nb == 3 ? 3 : 1) <= warps && smem_for(cluster) <= room;
    p.grid = p.clustered ? cluster : std::min({sms, nslices, 32 * warps});
    p.per_cta = (nslices + p.grid - 1) / p.grid;
    p.ks = std::max(1, warps / p.per_cta);
    p.turns = (p.per_cta + warps / p.ks - 1) / (warps / p.ks);
    const int64_t want = smem_for(p.grid);
    p.smem_bytes = want <= room ? (want + 15) / 16 * 16 : 0;
    return p;
}

}  // namespace

// The split of a system and the highest index that its kernel's leaders read of the array of partial sums
// (a CTA has as many entries as threads).
void pcg_split_info(int nslices, int64_t total_slots, int nb, int sms, bool may_cluster, int32_t out[6]) {
    const PcgSplit p = pcg_split(nslices, total_slots, nb, sms, may_cluster);
    const int warps = (nb == 3 ? grid_threads<3>() : grid_threads<1>()) / 32;
    int top = -1;
    if (p.ks > 1)
        for (int w = 0; w < warps; ++w)
            if (warp_role(w, p.ks, warps).leader) top = 32 * (w + p.ks - 1) + 31;
    out[0] = p.grid;
    out[1] = p.per_cta;
    out[2] = p.ks;
    out[3] = p.turns;
    out[4] = p.smem_bytes > 0;
    out[5] = top;
}

// Runs the iterations from the state that k_pcg_start left (r, z, p = z, the scalars) until the scalars
// say done; *gave_up is set when a launch gave up.  p2 is the second direction buffer.
int pcg_grid(plato_problem* h, int nb, const double* vals, const double* dinv, double* x, double* p2, int32_t max_it,
             PcgScalars* fin, int* gave_up) {
    *gave_up = 0;
    PcgSplit split = pcg_split(h->sell.nslices, h->sell.total_slots, nb, h->coop_sms, true);
    GridPcg a{};
    a.A = sell_view(h);
    a.nslices = h->sell.nslices;
    a.vals = vals;
    a.dinv = dinv;
    a.x = x;
    a.r = h->v_r;
    a.z = h->v_z;
    a.p[0] = h->v_p;
    a.p[1] = p2;
    a.max_it = max_it;
    a.S = h->scal;
    for (;;) {
        a.ks = split.ks;
        a.smem_bytes = int(split.smem_bytes);
        PLATO_RC(grid_box(h, &a.box));
        if (split.clustered) {
            int ok = 1;
            if (nb == 3) PLATO_RC(launch_cluster<3>(h, a, split.grid, &ok));
            else PLATO_RC(launch_cluster<1>(h, a, split.grid, &ok));
            if (!ok) {
                split = pcg_split(h->sell.nslices, h->sell.total_slots, nb, h->coop_sms, false);
                continue;
            }
        } else if (nb == 3) PLATO_RC((launch_grid<3, 1>(h, a, split.grid)));
        else if (split.turns == 1) PLATO_RC((launch_grid<1, 1>(h, a, split.grid)));
        else PLATO_RC((launch_grid<1, 2>(h, a, split.grid)));
        int32_t abort = 0;
        PLATO_CUDA(h, cudaMemcpyAsync(h->scal_host, h->scal, sizeof(PcgScalars), cudaMemcpyDeviceToHost, h->stream));
        PLATO_CUDA(h, cudaMemcpyAsync(&abort, a.box.abort, sizeof(abort), cudaMemcpyDeviceToHost, h->stream));
        PLATO_CUDA(h, cudaStreamSynchronize(h->stream));
        *fin = h->scal_host[0];
        if (abort) {
            PLATO_CUDA(h, cudaMemsetAsync(a.box.abort, 0, sizeof(abort), h->stream));
            *gave_up = 1;
            return PLATO_OK;
        }
        if (fin->done) return PLATO_OK;
        // after an even number of iterations the current direction is in the same buffer again
    }
}

}  // namespace plato
