// Flexible CG with the Chebyshev preconditioner in cooperative launches, for block systems that
// give every SELL slice a group of warps (fcg_poly in mixed.cu is the launch-per-stage form and has
// the formulas).  One CTA per SM owns a run of slices: their rows' vectors stay in registers, the
// low-precision matrix in shared memory when it fits (else it is read from L2), and only the search
// direction p and the Chebyshev directions leave the SM.  An iteration is
//   q = A p                                            sum p.q -> alpha
//   x += alpha p, r -= alpha q, first direction        sum r.r -> stop test
//   degree - 1 Chebyshev steps                         a barrier each
//   z.q -> beta, p = z + beta p, p.r                   two sums
// so degree + 3 grid-wide sums or barriers (grid.cuh) instead of as many kernels with a launch, a
// ramp and a tail each.  With a coarse space the sweep ends with the residual step of the two-level
// form, and the correction Z E^-1 Z^T of it takes five more barriers: restriction per coarse cell (a
// warp each), its sums, the two triangular products (a warp per row), and the prolongation onto the
// CTA's own rows.  Bound by these barriers (1.5 to 3 us each) and, beyond what shared memory holds, by L2.
// Solve to 1e-8, launch per stage against this: FP32 Chebyshev 20x10x10 6.9 -> 2.5 ms, 64x32x32 30.1 -> 17.3;
// two-level FP32 4.0 -> 1.7 and 8.3 -> 4.9 ms; two-level FP16 3.9 -> 1.7 and 7.6 -> 4.0 ms.  64x32x32 has 2,213 slices and
// 72x31x31 2,336; larger systems have more slices than the 2,368 warps and keep the launch per stage,
// whose streams from HBM hide its gaps.
#include <algorithm>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "coarse_view.cuh"
#include "fcg_grid.cuh"

namespace plato {

int ensure_smem_attribute(plato_problem* h, const void* kernel, int bytes);
SellView sell_view(const plato_problem* h);

namespace {

constexpr int kGridThreads = 512, kGridWarps = kGridThreads / 32;
constexpr int kLaunchIters = 512;  // iterations per launch: some ten milliseconds

struct GridFcg {
    SellView      A;
    int32_t       nslices;
    int32_t       ks;          // warps per slice
    const double* v64;
    const void*   vin;         // low-precision entries
    const float*  dinv;        // inverse diagonal in the preconditioner's variables
    const float*  scale;       // D^-1/2 of the scaled preconditioner, or null
    double *      x, *r, *p;
    float *       res, *d[2];
    int32_t       degree, coarse, max_it, iters;
    int32_t       smem_bytes;
    GridBox       box;
    PcgScalars*   S;
    ChebCoef      cc;
    // coarse space (coarse = 1)
    CoarseView     cv;
    const double*  coords;
    const uint8_t* mask;
    const float*   sq;         // D^1/2 of the scaled preconditioner, or null
    const int32_t *node_ptr, *node_list;
    int32_t        split, ndof, ldf;  // warps per coarse cell; coarse dofs and the row stride of X, U
    double *       rpart, *rc, *tc, *yc;
    const float *  X, *U;      // L^-1 and its transpose
};

// out = M in for a triangular FP32 matrix (coarse.cu's k_coarse_trmv), a warp per row.
__device__ void coarse_product(const float* M, const double* in, double* out, int n, int ld, bool lower) {
    const int lane = threadIdx.x & 31;
    const int warp = blockIdx.x * (kGridThreads / 32) + (threadIdx.x >> 5), warps = gridDim.x * (kGridThreads / 32);
    for (int row = warp; row < n; row += warps) {
        const int q0 = lower ? 0 : (row >> 2), q1 = lower ? (row >> 2) + 1 : (n + 3) >> 2;
        const float4* mp = reinterpret_cast<const float4*>(M + (int64_t)row * ld);
        double s = 0.0;
#pragma unroll 4
        for (int q = q0 + lane; q < q1; q += 32) {
            const float4 v = __ldg(mp + q);
            const int c = 4 * q;
            s += double(v.x) * in[c];
            if (c + 1 < n) s += double(v.y) * in[c + 1];
            if (c + 2 < n) s += double(v.z) * in[c + 2];
            if (c + 3 < n) s += double(v.w) * in[c + 3];
        }
        s = warp_sum(s);
        if (lane == 0) out[row] = s;
    }
}

// yc = E^-1 Z^T P res (res as published by the rows' owners); false when a wait ran out.
__device__ __noinline__ bool coarse_solve(const GridFcg& a, uint32_t& epoch) {
    const int lane = threadIdx.x & 31;
    const int warp = blockIdx.x * (kGridThreads / 32) + (threadIdx.x >> 5), warps = gridDim.x * (kGridThreads / 32);
    const int ncells = a.cv.nc0 * a.cv.nc1 * a.cv.nc2;
    if (!grid_barrier(a.box, ++epoch)) return false;
    for (int item = warp; item < ncells * a.split; item += warps) {
        const int cell = item / a.split, piece = item - cell * a.split;
        const int cz = cell % a.cv.nc2, cy = (cell / a.cv.nc2) % a.cv.nc1, cx = cell / (a.cv.nc1 * a.cv.nc2);
        const double lo[3] = {a.cv.x0 + cx * a.cv.hx, a.cv.y0 + cy * a.cv.hy, a.cv.z0 + cz * a.cv.hz};
        const int q0 = __ldg(a.node_ptr + cell), q1 = __ldg(a.node_ptr + cell + 1);
        const int chunk = (q1 - q0 + a.split - 1) / a.split;
        const int a0 = q0 + piece * chunk, a1 = min(q1, a0 + chunk);
        double s[24];
#pragma unroll
        for (int t = 0; t < 24; ++t) s[t] = 0.0;
        for (int q = a0 + lane; q < a1; q += 32) {
            const int64_t p = __ldg(a.node_list + q);
            const double u = (__ldg(a.coords + 3 * p) - lo[0]) * a.cv.ihx, v = (__ldg(a.coords + 3 * p + 1) - lo[1]) * a.cv.ihy,
                         w = (__ldg(a.coords + 3 * p + 2) - lo[2]) * a.cv.ihz;
            double val[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const float r = a.res[3 * p + d];
                val[d] = __ldg(a.mask + 3 * p + d) ? 0.0 : double(a.sq ? __ldg(a.sq + 3 * p + d) * r : r);
            }
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const double wgt = corner_weight(b, u, v, w);
#pragma unroll
                for (int d = 0; d < 3; ++d) s[3 * b + d] += wgt * val[d];
            }
        }
        double t3[3];
        warp_sum24(s, lane, t3);
        if ((lane & 3) == 0)
#pragma unroll
            for (int i = 0; i < 3; ++i) a.rpart[24 * (int64_t)item + warp_sum24_first(lane) + i] = t3[i];
    }
    if (!grid_barrier(a.box, ++epoch)) return false;
    for (int t = warp; t < a.ndof; t += warps) {  // the <= 8 cells around a coarse node, all their pieces
        const int J = t / 3, d = t - 3 * J;
        const int iz = J % (a.cv.nc2 + 1), iy = (J / (a.cv.nc2 + 1)) % (a.cv.nc1 + 1), ix = J / ((a.cv.nc1 + 1) * (a.cv.nc2 + 1));
        double sum = 0.0;
        for (int i = lane; i < 8 * a.split; i += 32) {
            const int b = i / a.split, k = i - b * a.split;
            const int cx = ix - ((b >> 2) & 1), cy = iy - ((b >> 1) & 1), cz = iz - (b & 1);
            if (cx < 0 || cy < 0 || cz < 0 || cx >= a.cv.nc0 || cy >= a.cv.nc1 || cz >= a.cv.nc2) continue;
            sum += a.rpart[24 * ((int64_t)cell_id(a.cv, cx, cy, cz) * a.split + k) + 3 * b + d];
        }
        sum = warp_sum(sum);
        if (lane == 0) a.rc[t] = sum;
    }
    if (!grid_barrier(a.box, ++epoch)) return false;
    coarse_product(a.X, a.rc, a.tc, a.ndof, a.ldf, true);
    if (!grid_barrier(a.box, ++epoch)) return false;
    coarse_product(a.U, a.tc, a.yc, a.ndof, a.ldf, false);
    return grid_barrier(a.box, ++epoch);
}

__device__ __forceinline__ float entry(float v) { return v; }
__device__ __forceinline__ float entry(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float entry(__half v) { return __half2float(v); }
__device__ __forceinline__ double entry(double v) { return v; }

// FP64 product: this lane's share (slots kg, kg + ks, ...) of its row; v points at entry 0 of slot 0.
__device__ __forceinline__ void row_share(const double* v, const int32_t* cols, int width, int kg, int ks, const double* x,
                                          double acc[3]) {
    acc[0] = acc[1] = acc[2] = 0.0;
#pragma unroll 4
    for (int k = kg; k < width; k += ks) {
        const int64_t c = cols[32 * k];
        const double x0 = x[3 * c], x1 = x[3 * c + 1], x2 = x[3 * c + 2];
        const double* e = v + 288 * k;
        acc[0] += e[0] * x0 + e[32] * x1 + e[64] * x2;
        acc[1] += e[96] * x0 + e[128] * x1 + e[160] * x2;
        acc[2] += e[192] * x0 + e[224] * x1 + e[256] * x2;
    }
}

// Preconditioner product: CW components of the row from component c0 on, slot after slot -- the sums
// of the launch-per-stage kernels, bit for bit (a low-precision preconditioner carries a changed last
// bit through a whole solve).
template <int CW, typename TA, typename TV>
__device__ __forceinline__ void row_components(const TV* v, const int32_t* cols, int width, int c0, const float* x, TA acc[CW]) {
#pragma unroll
    for (int i = 0; i < CW; ++i) acc[i] = TA(0);
#pragma unroll 4
    for (int k = 0; k < width; ++k) {
        const int64_t c = cols[32 * k];
        const TA x0 = TA(x[3 * c]), x1 = TA(x[3 * c + 1]), x2 = TA(x[3 * c + 2]);
        const TV* e = v + 288 * k + 96 * c0;
#pragma unroll
        for (int i = 0; i < CW; ++i)
            acc[i] += TA(entry(e[96 * i])) * x0 + TA(entry(e[96 * i + 32])) * x1 + TA(entry(e[96 * i + 64])) * x2;
    }
}

// TV: entries of the preconditioner's matrix; its sums are FP32 (FP64 for FP64 entries).  CW = 3: the
// first of a slice's ks warps owns its rows' vectors; CW = 1 (ks >= 4): warps 0, 1, 2 own a
// component each.
template <typename TV, int CW>
__global__ void __launch_bounds__(kGridThreads, 1) k_fcg_grid(const __grid_constant__ GridFcg a) {
    using TA = decltype(entry(TV()));
    extern __shared__ __align__(16) unsigned char fcg_smem[];
    __shared__ double sh_cta[kGridValues][32], sh_grid[kGridValues][32];
    __shared__ double part[3][kGridThreads];
    int32_t done = a.S->done;
    if (done || *reinterpret_cast<volatile int32_t*>(a.box.abort)) {
        // an abort that CTA 0 did not see in its own launch (another CTA's wait ran out at the last barrier) ends
        // the host's loop here: it looks at done
        if (!done && blockIdx.x == 0 && threadIdx.x == 0) a.S->done = 1;
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s0 = int((int64_t)a.nslices * blockIdx.x / gridDim.x), s1 = int((int64_t)a.nslices * (blockIdx.x + 1) / gridDim.x);
    const int kg = warp % a.ks, s = s0 + warp / a.ks;
    const int c0 = CW == 3 ? 0 : kg;  // first component of this thread
    const int64_t row = 32 * int64_t(s) + lane;
    const bool owner = s < s1 && kg < 3 / CW, own = owner && row < a.A.num_rows;
    const int64_t first = a.A.ptr[s0], slots = a.A.ptr[s1] - first;
    const int width = s < s1 ? a.A.width[s] : 0;
    const int64_t base = s < s1 ? a.A.ptr[s] - first : 0;
    const int32_t* gcols = a.A.cols + first + base + lane;  // for the FP64 product
    const double* v64 = a.v64 + 9 * (first + base) + lane;
    const TV* vin = static_cast<const TV*>(a.vin) + 9 * first;
    const int32_t* cols = a.A.cols + first;
    if (a.degree + a.coarse > 1 && slots * int64_t(9 * sizeof(TV) + 4) <= a.smem_bytes) {
        int32_t* sc = reinterpret_cast<int32_t*>(fcg_smem);
        TV* sv = reinterpret_cast<TV*>(fcg_smem + 4 * slots);  // slots is a multiple of 32
        for (int64_t i = tid; i < slots; i += kGridThreads) sc[i] = __ldg(cols + i);
        const uint4* from = reinterpret_cast<const uint4*>(vin);  // 288 sizeof(TV) bytes a slot row: 16-byte pieces
        uint4* to = reinterpret_cast<uint4*>(sv);
        for (int64_t i = tid; i < 9 * slots * int64_t(sizeof(TV)) / 16; i += kGridThreads) to[i] = __ldg(from + i);
        vin = sv;
        cols = sc;
    }
    vin += 9 * base + lane;
    cols += base + lane;

    double x[CW], r[CW], p[CW], q[CW];
    float res[CW], y[CW], d[CW], di[CW], sc3[CW];
#pragma unroll
    for (int i = 0; i < CW; ++i) {
        const int64_t k = 3 * row + c0 + i;
        x[i] = own ? a.x[k] : 0.0;
        r[i] = own ? a.r[k] : 0.0;
        p[i] = own ? a.p[k] : 0.0;
        q[i] = 0.0;
        y[i] = 0.f;
        di[i] = own ? a.dinv[k] : 0.f;
        sc3[i] = own && a.scale ? a.scale[k] : 1.f;
        res[i] = d[i] = 0.f;
    }
    double pr = a.S->rz, rr = a.S->rr, pq = a.S->pAp, alpha = a.S->alpha, beta = a.S->beta, zq = a.S->zq;
    const double tol2 = a.S->tol2;
    int32_t iter = a.S->iter, nonfinite = a.S->nonfinite;
    uint32_t epoch = 0;  // barriers of this launch
    bool gave_up = false;
    __syncthreads();

    for (int it = 0; it < a.iters; ++it) {
        // q = A p, alpha
        double acc[3];
        row_share(v64, gcols, width, kg, a.ks, const_cast<const double*>(a.p), acc);
        if (a.ks > 1) {
#pragma unroll
            for (int i = 0; i < 3; ++i) part[i][tid] = acc[i];
            __syncthreads();
        }
        double v1[1] = {0.0};
        if (own)
#pragma unroll
            for (int i = 0; i < CW; ++i) {
                q[i] = acc[CW == 3 ? i : 0];
                if (a.ks > 1) {
                    const double* mine = &part[c0 + i][tid - 32 * kg];
                    q[i] = mine[0];
                    for (int k = 1; k < a.ks; ++k) q[i] += mine[32 * k];
                }
                v1[0] += p[i] * q[i];
            }
        if (!grid_sum<1>(v1, a.box, ++epoch, sh_cta, sh_grid)) { gave_up = true; break; }
        pq = v1[0];
        alpha = pr / pq;
        if (!isfinite(alpha) || pq <= 0.0) { nonfinite = 1; done = 1; break; }
        // x, r, the first Chebyshev direction
        v1[0] = 0.0;
        if (own)
#pragma unroll
            for (int i = 0; i < CW; ++i) {
                x[i] += alpha * p[i];
                r[i] -= alpha * q[i];
                v1[0] += r[i] * r[i];
                res[i] = a.scale ? sc3[i] * float(r[i]) : float(r[i]);
                d[i] = a.cc.c0 * di[i] * res[i];
                y[i] = d[i];
                a.d[0][3 * row + c0 + i] = d[i];
            }
        if (!grid_sum<1>(v1, a.box, ++epoch, sh_cta, sh_grid)) { gave_up = true; break; }
        rr = v1[0];
        ++iter;
        if (!isfinite(rr)) nonfinite = 1;
        if (nonfinite || rr <= tol2 || iter >= a.max_it) { done = 1; break; }
        // Chebyshev steps; with a coarse space a last step that only updates the residual
        bool ok = true;
        for (int k = 1; k < a.degree + a.coarse; ++k) {
            const bool more = k < a.degree, publish = k + 1 < a.degree + a.coarse;
            if (owner) {
                TA w[CW];
                row_components<CW, TA>(vin, cols, width, c0, const_cast<const float*>(a.d[(k - 1) & 1]), w);
                if (own)
#pragma unroll
                    for (int i = 0; i < CW; ++i) {
                        const float rs = res[i] - float(w[i]);
                        res[i] = rs;
                        if (more) {
                            // the scaled variables have a unit diagonal
                            const float dn = a.scale ? a.cc.c1[k] * d[i] + a.cc.c2[k] * rs
                                                     : a.cc.c1[k] * d[i] + a.cc.c2[k] * di[i] * rs;
                            d[i] = dn;
                            y[i] += dn;
                            if (publish) a.d[k & 1][3 * row + c0 + i] = dn;
                        }
                    }
            }
            if (publish) {
                ok = grid_barrier(a.box, ++epoch);
                if (!ok) break;
            }
        }
        if (!ok) { gave_up = true; break; }
        if (a.coarse) {
            if (own)
#pragma unroll
                for (int i = 0; i < CW; ++i) a.res[3 * row + c0 + i] = res[i];
            if (!coarse_solve(a, epoch)) { gave_up = true; break; }
            if (own) {  // y += P Z yc on the own rows (times D^1/2)
                const double px = __ldg(a.coords + 3 * row), py = __ldg(a.coords + 3 * row + 1), pz = __ldg(a.coords + 3 * row + 2);
                int cx, cy, cz;
                cell_of(a.cv, px, py, pz, cx, cy, cz);
                const double u = (px - (a.cv.x0 + cx * a.cv.hx)) * a.cv.ihx, v = (py - (a.cv.y0 + cy * a.cv.hy)) * a.cv.ihy,
                             w = (pz - (a.cv.z0 + cz * a.cv.hz)) * a.cv.ihz;
                double c[CW];
#pragma unroll
                for (int i = 0; i < CW; ++i) c[i] = 0.0;
                for (int b = 0; b < 8; ++b) {
                    const double wgt = corner_weight(b, u, v, w);
                    const int J = coarse_node(a.cv, cx + ((b >> 2) & 1), cy + ((b >> 1) & 1), cz + (b & 1));
#pragma unroll
                    for (int i = 0; i < CW; ++i) c[i] += wgt * a.yc[3 * J + c0 + i];
                }
#pragma unroll
                for (int i = 0; i < CW; ++i) {
                    const int64_t k = 3 * row + c0 + i;
                    y[i] += __ldg(a.mask + k) ? 0.f : (a.sq ? __ldg(a.sq + k) * float(c[i]) : float(c[i]));
                }
            }
        }
        // z = y (times D^-1/2), beta, the next direction and p.r
        double z[CW];
        v1[0] = 0.0;
#pragma unroll
        for (int i = 0; i < CW; ++i) {
            z[i] = double(a.scale ? sc3[i] * y[i] : y[i]);
            if (own) v1[0] += z[i] * q[i];
        }
        if (!grid_sum<1>(v1, a.box, ++epoch, sh_cta, sh_grid)) { gave_up = true; break; }
        zq = v1[0];
        beta = -zq / pq;
        if (!isfinite(beta)) { nonfinite = 1; done = 1; break; }
        v1[0] = 0.0;
        if (own)
#pragma unroll
            for (int i = 0; i < CW; ++i) {
                p[i] = z[i] + beta * p[i];
                a.p[3 * row + c0 + i] = p[i];
                v1[0] += p[i] * r[i];
            }
        if (!grid_sum<1>(v1, a.box, ++epoch, sh_cta, sh_grid)) { gave_up = true; break; }
        pr = v1[0];
        if (!isfinite(pr)) { nonfinite = 1; done = 1; break; }
    }
    if (own)
#pragma unroll
        for (int i = 0; i < CW; ++i) {
            a.x[3 * row + c0 + i] = x[i];
            a.r[3 * row + c0 + i] = r[i];
        }
    if (blockIdx.x == 0 && tid == 0) {
        a.S->rz = pr;
        a.S->rr = rr;
        a.S->pAp = pq;
        a.S->alpha = alpha;
        a.S->beta = beta;
        a.S->zq = zq;
        a.S->iter = iter;
        a.S->nonfinite = nonfinite;
        a.S->done = done || gave_up ? 1 : 0;
    }
}

template <typename TV>
int launch(plato_problem* h, const GridFcg& a, int grid) {
    auto kernel = a.ks >= 4 ? k_fcg_grid<TV, 1> : k_fcg_grid<TV, 3>;
    PLATO_RC(ensure_smem_attribute(h, reinterpret_cast<const void*>(kernel), a.smem_bytes));
    PLATO_CUDA(h, launch_cooperative(kernel, grid, kGridThreads, size_t(a.smem_bytes), h->stream, a));
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

}  // namespace

bool fcg_grid_ok(const plato_problem* h) {
    return !h->grid_off && !h->timing && !h->ritz_deflating && h->sell.nslices <= int64_t(h->coop_sms) * kGridWarps;
}

int fcg_grid_iterations(plato_problem* h, int entry_bytes, bool half_entries, const void* vin, const ChebCoef& cc, int degree,
                        int coarse, double* x, const float* scale, int32_t max_it) {
    const int grid = std::min(h->coop_sms, h->sell.nslices);
    const int per_cta = (h->sell.nslices + grid - 1) / grid;  // at most kGridWarps (fcg_grid_ok)
    GridFcg a{};
    a.A = sell_view(h);
    a.nslices = h->sell.nslices;
    a.ks = 1;
    while (2 * a.ks * per_cta <= kGridWarps) a.ks *= 2;
    a.v64 = h->sell64;
    a.vin = vin;
    a.dinv = h->f_dinv;
    a.scale = scale;
    a.x = x;
    a.r = h->v_r;
    a.p = h->v_p;
    a.res = h->f_res;
    a.d[0] = h->f_d0;
    a.d[1] = h->f_d1;
    a.degree = degree;
    a.coarse = coarse;
    a.max_it = max_it;
    a.iters = h->grid_stall.iterations > 0 ? h->grid_stall.iterations : kLaunchIters;
    a.S = h->scal;
    a.cc = cc;
    if (coarse) {
        const CoarseSpace& c = h->coarse;
        a.cv = coarse_view(h);
        a.coords = h->coords;
        a.mask = h->bc_mask;
        a.sq = scale ? h->f_sq : nullptr;
        a.node_ptr = c.node_ptr;
        a.node_list = c.node_list;
        a.split = c.rsplit;
        a.ndof = c.ndof;
        a.ldf = c.ldf;
        a.rpart = c.rpart;
        a.rc = c.rc;
        a.tc = c.tc;
        a.yc = c.yc;
        a.X = c.Xf;
        a.U = c.Uf;
    }
    // shared memory for the average CTA's slots and a tenth more; a CTA with more reads L2
    const int64_t want = (h->sell.total_slots / grid + 32) * (9 * entry_bytes + 4) * 11 / 10;
    a.smem_bytes = want <= kGridSmemMax - 3 * kGridThreads * 8 - 2048 ? int((want + 15) / 16 * 16) : 0;
    PLATO_RC(grid_box(h, &a.box));
    if (entry_bytes == 8) return launch<double>(h, a, grid);
    if (entry_bytes == 4) return launch<float>(h, a, grid);
    return half_entries ? launch<__half>(h, a, grid) : launch<__nv_bfloat16>(h, a, grid);
}

int fcg_grid_gave_up(plato_problem* h, int* gave_up) {
    GridBox m;
    PLATO_RC(grid_box(h, &m));  // (no stall is pending: the loop's first launch has taken it)
    int32_t abort = 0;
    PLATO_CUDA(h, cudaMemcpyAsync(&abort, m.abort, sizeof(abort), cudaMemcpyDeviceToHost, h->stream));
    PLATO_CUDA(h, cudaStreamSynchronize(h->stream));
    if (abort) PLATO_CUDA(h, cudaMemsetAsync(m.abort, 0, sizeof(abort), h->stream));
    *gave_up = abort ? 1 : 0;
    return PLATO_OK;
}

}  // namespace plato
