// Element kernels that run once per handle or per batch member: the traction load and the
// members' energies.  (The residual, the criteria and their derivatives over a whole mesh are
// in fan_kernels.cu.)
#include <algorithm>

#include "plato_internal.cuh"

namespace plato {
namespace {

constexpr int kThreads = 256;

struct CellState {
    int4   n;
    TetGeom<double> G;
    double rho;  // mean nodal control, ApplyWeighting (src/ApplyWeighting.hpp:55-60)
};

__device__ __forceinline__ void load_cell(const MeshView& m, const Material& mat, const double* __restrict__ z,
                                          int64_t c, CellState& cs) {
    cs.n = m.conn[c];
    double x[4][3];
    load_cell_coords(m.coords, cs.n, x);
    tet_geometry(x, cs.G);
    cs.rho = cell_rho(mat, z, c, cs.n);
}

__device__ __forceinline__ void gather_state(const double* __restrict__ u, int4 n, double ue[4][3]) {
    const int ids[4] = {n.x, n.y, n.z, n.w};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const double* p = u + 3 * (int64_t)ids[a];
        ue[a][0] = __ldg(p + 0);
        ue[a][1] = __ldg(p + 1);
        ue[a][2] = __ldg(p + 2);
    }
}

// Cell energy 1/2 vol s(rho) eps.C.eps (InternalElasticEnergy::evaluate,
// src/elliptic/InternalElasticEnergy.hpp:169-192).
__device__ __forceinline__ double cell_energy(const MeshView& m, const Material& mat, const double* __restrict__ u,
                                              const double* __restrict__ z, int64_t c) {
    CellState cs;
    load_cell(m, mat, z, c, cs);
    double ue[4][3], e[6], s[6];
    gather_state(u, cs.n, ue);
    strain_voigt(cs.G.g, ue, e);
    stress_voigt(mat, e, s);
    const double ese = s[0] * e[0] + s[1] * e[1] + s[2] * e[2] + s[3] * e[3] + s[4] * e[4] + s[5] * e[5];
    return 0.5 * ese * cs.G.vol * simp(mat, cs.rho);
}

__device__ __forceinline__ double block_sum(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 32) {
        r = (l < (int)(blockDim.x >> 5)) ? sh[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    __syncthreads();
    return r;  // valid in thread 0
}

// Traction load F: SurfaceLoadIntegral<3> (src/SurfaceLoadIntegral.hpp:97-150) with the
// triangle degree-one rule (weight 1/2, basis 1/3 each), area from
// CalculateSurfaceArea<3> (src/SurfaceIntegralUtilities.hpp:217-227).
__global__ void k_traction(int32_t nfaces, const int32_t* __restrict__ fcell,
                           const int32_t* __restrict__ floc, double tx, double ty, double tz,
                           MeshView m, double* __restrict__ F) {
    for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nfaces;
         f += (int64_t)gridDim.x * blockDim.x) {
        const int4 n = m.conn[fcell[f]];
        int id[3];
        for (int a = 0; a < 3; ++a) id[a] = node_of(n, floc[3 * f + a]);
        double J[2][3];
        for (int a = 0; a < 2; ++a)
            for (int d = 0; d < 3; ++d) J[a][d] = m.coords[3 * (int64_t)id[a] + d] - m.coords[3 * (int64_t)id[2] + d];
        const double J23 = J[0][1] * J[1][2] - J[0][2] * J[1][1];
        const double J31 = J[0][2] * J[1][0] - J[0][0] * J[1][2];
        const double J12 = J[0][0] * J[1][1] - J[0][1] * J[1][0];
        const double area = 0.5 * sqrt(J23 * J23 + J31 * J31 + J12 * J12);
        const double c = 1.0 / 3.0;
        const double basis[3] = {1.0 - c - c, c, c};
        const double t[3] = {tx, ty, tz};
        for (int a = 0; a < 3; ++a)
            for (int d = 0; d < 3; ++d) atomicAdd(&F[3 * (int64_t)id[a] + d], basis[a] * t[d] * area);
    }
}

__global__ void k_coords_soa(int64_t N, const double* __restrict__ x, double* __restrict__ planes) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
        for (int d = 0; d < 3; ++d) planes[d * N + i] = x[3 * i + d];
}

__global__ void k_axpby(int64_t n, double a, const double* __restrict__ x, double b,
                        double* __restrict__ y) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        y[i] = a * x[i] + (b == 0.0 ? 0.0 : b * y[i]);
}

}  // namespace

MeshView mesh_view(const plato_problem* h) { return MeshView{h->N, h->C, h->conn, h->coords}; }
GraphView graph_view(const plato_problem* h) {
    return GraphView{h->N, h->nblocks, h->row_map, h->cols, h->diag, h->n2c_ptr, h->n2c};
}

int launch_coords_soa(plato_problem* h) {
    k_coords_soa<<<grid_for(h->N, kThreads), kThreads, 0, h->stream>>>(h->N, h->coords, h->coords_soa);
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

int launch_axpby(plato_problem* h, int64_t n, double a, const double* x, double b, double* y) {
    k_axpby<<<grid_for(n, kThreads), kThreads, 0, h->stream>>>(n, a, x, b, y);
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

int launch_traction(plato_problem* h, int32_t nfaces, const int32_t* fcell, const int32_t* floc,
                    const double t[3]) {
    if (nfaces == 0) return PLATO_OK;
    k_traction<<<grid_for(nfaces, kThreads), kThreads, 0, h->stream>>>(nfaces, fcell, floc, t[0], t[1],
                                                                        t[2], mesh_view(h), h->F);
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

// Internal elastic energy of each member of a batch: CTA (member, piece) sums its share of
// the member's cells, then one thread per member adds the pieces in order (deterministic).
__global__ void __launch_bounds__(kThreads) k_energy_pieces(MeshView m, Material mat, const double* __restrict__ u,
                                                            const double* __restrict__ z,
                                                            const int32_t* __restrict__ cell_off,
                                                            double* __restrict__ pieces) {
    __shared__ double sh[32];
    const int s = blockIdx.x / kEnergySplit, piece = blockIdx.x - s * kEnergySplit;
    const int64_t c0 = cell_off[s], c1 = cell_off[s + 1];
    const int64_t len = (c1 - c0 + kEnergySplit - 1) / kEnergySplit;
    const int64_t a = c0 + piece * len, e = a + len < c1 ? a + len : c1;
    double v = 0.0;
    for (int64_t c = a + threadIdx.x; c < e; c += blockDim.x) v += cell_energy(m, mat, u, z, c);
    v = block_sum(v, sh);
    if (threadIdx.x == 0) pieces[blockIdx.x] = v;
}

__global__ void k_sum_pieces(int32_t nseg, const double* __restrict__ pieces, double* __restrict__ values) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x) {
        double t = 0.0;
        for (int k = 0; k < kEnergySplit; ++k) t += pieces[(int64_t)s * kEnergySplit + k];
        values[s] = t;
    }
}

// Energy of every batch member into values[nseg] (device).
int launch_energy_segments(plato_problem* h, const double* u, const double* z, double* values) {
    const int nseg = h->batch.nseg;
    k_energy_pieces<<<nseg * kEnergySplit, kThreads, 0, h->stream>>>(mesh_view(h), h->material, u, z,
                                                                      h->batch.cell_off_d, h->batch.values);
    PLATO_LAUNCH_CHECK(h);
    k_sum_pieces<<<grid_for(nseg, 128), 128, 0, h->stream>>>(nseg, h->batch.values, values);
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

}  // namespace plato
