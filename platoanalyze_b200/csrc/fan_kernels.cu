// Element kernels of the elastostatic residual, the internal-energy and volume criteria, their
// control derivatives and the matrix-free operator, walking the mesh fan by fan (fans.cu).
//
// One thread walks a fan: for every cell kinematics, strain, stress or a scalar in registers, with
// the data of the ring node after the next one already on its way.  It leaves its sums for the fan's
// nodes in shared memory; the CTA, which holds a tile of fans, adds them per node and writes each
// sum to part[slot], the place of that (tile, node) pair in node order.  k_fan_nodes then adds each
// node's few contiguous sums.  No atomics: the order of every sum is fixed, so results repeat
// bit for bit.
//
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "fans.cuh"
#include "solver_common.cuh"

namespace plato {

int ensure_smem_attribute(plato_problem* h, const void* kernel, int bytes);

namespace {

enum FanOp { FAN_FORCE, FAN_EBE, FAN_DIAG, FAN_QUANT, FAN_VOLUME };

constexpr int kFanThreads = 128;  // most fans in a tile

template <int OP> constexpr int fan_values() { return OP == FAN_FORCE || OP == FAN_EBE || OP == FAN_DIAG ? 3 : 1; }
template <int OP> constexpr bool fan_has_u() { return OP != FAN_DIAG && OP != FAN_VOLUME; }
template <int OP> constexpr bool fan_has_z() { return OP == FAN_FORCE || OP == FAN_QUANT || OP == FAN_VOLUME; }
template <int OP, int MODE> constexpr bool fan_has_lam() { return OP == FAN_QUANT && (MODE == 3 || MODE == 4); }
// MODE of FAN_QUANT: 0 energy sum; 1 energy derivative; 2 self-adjoint compliance derivative;
// 3 (dR/dz)^T lambda; 4 modes 1 + 3; 5 energy sum and mode 2.  Of FAN_VOLUME: 0 sum, 1 derivative.
template <int OP, int MODE> constexpr bool fan_sums() {
    return (OP == FAN_QUANT && (MODE == 0 || MODE == 5)) || (OP == FAN_VOLUME && MODE == 0);
}
template <int OP, int MODE> constexpr bool fan_nodes() { return !(OP == FAN_QUANT && MODE == 0) && !(OP == FAN_VOLUME && MODE == 0); }

template <typename T>
struct Vec3 {
    T x, y, z;
};
template <typename T>
__device__ __forceinline__ Vec3<T> operator-(const Vec3<T>& a, const Vec3<T>& b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <typename T>
__device__ __forceinline__ Vec3<T> cross(const Vec3<T>& a, const Vec3<T>& b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
template <typename T>
__device__ __forceinline__ T dot(const Vec3<T>& a, const Vec3<T>& b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// det(J) times the Voigt strain (engineering shear, Strain<3>, src/Strain.hpp:70-95) of the field with
// differences db, dp, dn to node a: sum of du (x) cofactor over the three other nodes.
template <typename T>
__device__ __forceinline__ void fan_strain(const Vec3<T>& db, const Vec3<T>& dp, const Vec3<T>& dn, const Vec3<T>& cb,
                                           const Vec3<T>& cp, const Vec3<T>& cn, T e[6]) {
    e[0] = db.x * cb.x + dp.x * cp.x + dn.x * cn.x;
    e[1] = db.y * cb.y + dp.y * cp.y + dn.y * cn.y;
    e[2] = db.z * cb.z + dp.z * cp.z + dn.z * cn.z;
    e[3] = db.z * cb.y + dp.z * cp.y + dn.z * cn.y + db.y * cb.z + dp.y * cp.z + dn.y * cn.z;
    e[4] = db.z * cb.x + dp.z * cp.x + dn.z * cn.x + db.x * cb.z + dp.x * cp.z + dn.x * cn.z;
    e[5] = db.y * cb.x + dp.y * cp.x + dn.y * cn.x + db.x * cb.y + dp.x * cp.y + dn.x * cn.y;
}

template <typename T>
struct FanArgs {
    const T*       coords;   // x, y, z planes of n values
    int64_t        n;
    const T*       u;        // state, or the operator's input
    const T*       lam;
    const double*  z;
    const T*       w;        // [6 nfans] SIMP weight of each cell (FAN_EBE, FAN_DIAG)
    const uint8_t* mask;     // constrained dofs of u read as zero (may be null)
    T*             part;     // [entries * values]
    double*        sums;     // [gridDim.x] sum of each CTA
    uint32_t*      ticket;
    double*        result;
    double*        cell_out; // element control: the derivative itself
    int            accumulate;
};

// What a cell needs of one of its nodes.
template <typename T>
struct FanNode {
    Vec3<T> x, u, l;
    T       z;
};

template <int OP, int MODE, typename T>
__global__ void __launch_bounds__(kFanThreads, 3)
k_fans(FanView fv, Material mat, FanArgs<T> A, const PcgScalars* S) {
    if (S && S->done) return;
    constexpr int NV = fan_values<OP>();
    constexpr bool U = fan_has_u<OP>(), Z = fan_has_z<OP>(), L = fan_has_lam<OP, MODE>();
    constexpr bool NODES = fan_nodes<OP, MODE>(), SUMS = fan_sums<OP, MODE>();
    extern __shared__ __align__(16) unsigned char fan_smem[];
    const int W = blockDim.x, tid = threadIdx.x;
    T* st = reinterpret_cast<T*>(fan_smem);  // [NV][8][W] sums of each fan for its nodes
    uint4* uses = reinterpret_cast<uint4*>(fan_smem + (NODES ? sizeof(T) * NV * 8 * W : 0));
    const bool cells = Z && mat.cell_control != 0;       // one density per cell
    const bool direct = cells && OP != FAN_FORCE;        // and the derivative per cell
    double total = 0.0;

    auto load = [&](int64_t a) {
        FanNode<T> n{};
        n.x = {__ldg(A.coords + a), __ldg(A.coords + A.n + a), __ldg(A.coords + 2 * A.n + a)};
        if (U) {
            n.u = {__ldg(A.u + 3 * a), __ldg(A.u + 3 * a + 1), __ldg(A.u + 3 * a + 2)};
            if (OP != FAN_QUANT && A.mask) {
                if (__ldg(A.mask + 3 * a)) n.u.x = T(0);
                if (__ldg(A.mask + 3 * a + 1)) n.u.y = T(0);
                if (__ldg(A.mask + 3 * a + 2)) n.u.z = T(0);
            }
        }
        if (L) n.l = {__ldg(A.lam + 3 * a), __ldg(A.lam + 3 * a + 1), __ldg(A.lam + 3 * a + 2)};
        if (Z && !cells) n.z = T(__ldg(A.z + a));
        return n;
    };

    const int4 none = make_int4(-1, -1, -1, -1);
    int4 next0 = none, next1 = none;  // the next tile's record
    auto fetch = [&](int t) {
        const int64_t f = int64_t(t) * W + tid;
        next0 = next1 = none;
        if (t < fv.ntiles && f < fv.nfans) {
            next0 = __ldg(fv.rec + 2 * f);
            next1 = __ldg(fv.rec + 2 * f + 1);
        }
    };
    fetch(blockIdx.x);
    for (int tile = blockIdx.x; tile < fv.ntiles; tile += gridDim.x) {
        const int64_t fan = int64_t(tile) * W + tid;
        const int4 rec = next0;
        const int ring[6] = {next0.z, next0.w, next1.x, next1.y, next1.z, next1.w};
        fetch(tile + gridDim.x);
        // where this tile's sums go: read now, used after the walk
        int e0 = 0, nn = 0;
        uint32_t place0 = 0;
        int32_t slot0 = 0;
        uint4 mine_uses = make_uint4(0, 0, 0, 0);
        if (NODES && !direct) {
            mine_uses = __ldg(fv.inc + fan);
            e0 = __ldg(fv.tile_ptr + tile);
            nn = __ldg(fv.tile_ptr + tile + 1) - e0;
            if (tid < nn) {
                place0 = __ldg(fv.place + e0 + tid);
                slot0 = __ldg(fv.slot + e0 + tid);
            }
        }

        // a warp whose fans are all closed rings of six cells takes the walk without their ends
        auto walk = [&](auto full) {
            constexpr bool FULL = decltype(full)::value;  // six cells, closed: no ends to look for
            const bool closed = FULL || (rec.x & kFanClosed) != 0;
            const FanNode<T> na = load(rec.x & ~kFanClosed), nb = load(rec.y);
            const FanNode<T> np = load(ring[0]);
            FanNode<T> ahead = load(ring[1]);  // the ring node of the next cell
            const Vec3<T> eb = nb.x - na.x, db = nb.u - na.u, lb = nb.l - na.l;
            const T zab = na.z + nb.z;
            Vec3<T> ep = np.x - na.x, dp = np.u - na.u, lp = np.l - na.l;
            T zp = np.z;
            Vec3<T> cbp = cross(eb, ep);
            T va[3] = {T(0), T(0), T(0)}, vb[3] = {T(0), T(0), T(0)}, vp[3] = {T(0), T(0), T(0)};
            T* slot = st + tid;
            int last = 0;
            bool shut = false;  // the cell at hand closes the ring
            // unrolled, so that the ring stays in registers and nothing is moved from one cell to the next
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const FanNode<T> cur = ahead;
                const int q = i + 2 < 6 ? ring[i + 2] : -1;
                const int after = FULL ? (i < 5 ? ring[(i + 2) % 6] : -1) : (q < 0 && closed && !shut ? ring[0] : q);
                if (FULL ? i < 5 : after >= 0 && !shut) ahead = load(after);
                const Vec3<T> en = cur.x - na.x;
                // cofactors of b, p (= r_i) and n (= r_(i+1)): det(J) times their basis gradients
                // (ComputeGradientWorkset<3>, src/ImplicitFunctors.hpp:169-221); a has minus their sum
                const Vec3<T> cb = cross(ep, en), cbn = cross(eb, en), cp = {-cbn.x, -cbn.y, -cbn.z};
                const Vec3<T>& cn = cbp;
                const T det = fabs(dot(eb, cb));
                const T zn = cur.z;
                T weight = T(0), dweight = T(0);
                const int64_t cell = cells ? __ldg(fv.cells + 6 * fan + i) : 0;
                if (Z) {
                    const T rho = cells ? T(__ldg(A.z + cell)) : (zab + zp + zn) * T(0.25);
                    if (OP == FAN_FORCE || SUMS) weight = simp(mat, rho);
                    if (!(OP == FAN_FORCE) && NODES) dweight = simp_dx(mat, rho) * T(rho_dz(mat));
                } else {
                    weight = __ldg(A.w + 6 * fan + i);
                }
                T n[3] = {T(0), T(0), T(0)};     // this cell's share for the next ring node
                T mine[3] = {T(0), T(0), T(0)};  // and for p
                if (OP == FAN_VOLUME) {
                    const T vol = det * (T(1) / T(6));
                    if (SUMS) total += double(vol * weight);
                    n[0] = vol * dweight;
                } else if (OP == FAN_DIAG) {
                    const T k = weight / (T(6) * det), lm = T(mat.c01) + T(mat.c33), mu = T(mat.c33);
                    const Vec3<T> ca = {-(cb.x + cp.x + cn.x), -(cb.y + cp.y + cn.y), -(cb.z + cp.z + cn.z)};
                    auto diag = [&](const Vec3<T>& c, T out[3]) {
                        const T cc = mu * dot(c, c);
                        out[0] += k * (lm * c.x * c.x + cc);
                        out[1] += k * (lm * c.y * c.y + cc);
                        out[2] += k * (lm * c.z * c.z + cc);
                    };
                    diag(ca, va);
                    diag(cb, vb);
                    diag(cp, mine);
                    diag(cn, n);
                } else {
                    const Vec3<T> dn = cur.u - na.u;
                    T e[6], s[6];
                    fan_strain(db, dp, dn, cb, cp, cn, e);
                    stress_voigt(mat, e, s);
                    const T k = T(1) / (T(6) * det);
                    if (OP == FAN_FORCE || OP == FAN_EBE) {
                        // vol B^T sigma of b, p and n; a takes minus the total of the others
#pragma unroll
                        for (int d = 0; d < 6; ++d) s[d] *= weight * k;
                        vb[0] += s[0] * cb.x + s[5] * cb.y + s[4] * cb.z;
                        vb[1] += s[5] * cb.x + s[1] * cb.y + s[3] * cb.z;
                        vb[2] += s[4] * cb.x + s[3] * cb.y + s[2] * cb.z;
                        mine[0] = s[0] * cp.x + s[5] * cp.y + s[4] * cp.z;
                        mine[1] = s[5] * cp.x + s[1] * cp.y + s[3] * cp.z;
                        mine[2] = s[4] * cp.x + s[3] * cp.y + s[2] * cp.z;
                        n[0] = s[0] * cn.x + s[5] * cn.y + s[4] * cn.z;
                        n[1] = s[5] * cn.x + s[1] * cn.y + s[3] * cn.z;
                        n[2] = s[4] * cn.x + s[3] * cn.y + s[2] * cn.z;
#pragma unroll
                        for (int d = 0; d < 3; ++d) va[d] -= mine[d] + n[d];
                    } else {
                        // vol eps(u).C.eps(u), and with lambda vol eps(lambda).C.eps(u)
                        const T ese = k * (s[0] * e[0] + s[1] * e[1] + s[2] * e[2] + s[3] * e[3] + s[4] * e[4] + s[5] * e[5]);
                        if (SUMS) total += double(T(0.5) * ese * weight);
                        if (MODE == 1) n[0] = T(0.5) * ese * dweight;
                        if (MODE == 2 || MODE == 5) n[0] = -(T(0.5) * ese * dweight);
                        if (L) {
                            const Vec3<T> ln = cur.l - na.l;
                            T el[6];
                            fan_strain(lb, lp, ln, cb, cp, cn, el);
                            lp = ln;
                            const T esl = k * (s[0] * el[0] + s[1] * el[1] + s[2] * el[2] + s[3] * el[3] + s[4] * el[4] + s[5] * el[5]);
                            n[0] = (MODE == 3 ? esl : T(0.5) * ese + esl) * dweight;
                        }
                    }
                    dp = dn;
                }
                if (NODES) {
                    if (direct) {
                        A.cell_out[cell] = A.accumulate ? A.cell_out[cell] + double(n[0]) : double(n[0]);
                    } else {
                        if (NV == 1) { va[0] += n[0]; vb[0] += n[0]; mine[0] = n[0]; }
#pragma unroll
                        for (int d = 0; d < NV; ++d) {
                            slot[(8 * d + 2 + i) * W] = vp[d] + mine[d];
                            vp[d] = n[d];
                        }
                    }
                }
                last = i + 1;
                if (FULL ? i == 5 : shut || after < 0) break;
                shut = FULL ? i == 4 : q < 0;
                ep = en;
                cbp = cbn;
                zp = zn;
            }
            if (NODES && !direct) {
                // the last ring node of an open fan; of a closed one that is the first again
#pragma unroll
                for (int d = 0; d < NV; ++d) {
                    if (shut) slot[(8 * d + 2) * W] += vp[d];
                    else slot[(8 * d + 2 + last) * W] = vp[d];
                    slot[8 * d * W] = (OP == FAN_FORCE || OP == FAN_EBE) ? va[d] - vb[d] : va[d];
                    slot[(8 * d + 1) * W] = vb[d];
                }
            }
        };
        const bool six = rec.x >= 0 && (rec.x & kFanClosed) != 0 && ring[5] >= 0;
        if (__all_sync(0xffffffffu, six)) walk(std::true_type{});
        else if (rec.x >= 0) walk(std::false_type{});
        if (NODES && !direct) {
            uses[tid] = mine_uses;
            __syncthreads();
            const uint16_t* use = reinterpret_cast<const uint16_t*>(uses);
            for (int i = tid; i < nn; i += W) {
                const uint32_t place = i == tid ? place0 : __ldg(fv.place + e0 + i);
                const int64_t to = i == tid ? slot0 : __ldg(fv.slot + e0 + i);
                const int k0 = int(place >> 16), k1 = k0 + int(place & 0xffffu);
                T sum[3] = {T(0), T(0), T(0)};
#pragma unroll 4
                for (int k = k0; k < k1; ++k) {
                    const int j = use[k];
#pragma unroll
                    for (int d = 0; d < NV; ++d) sum[d] += st[8 * d * W + j];
                }
#pragma unroll
                for (int d = 0; d < NV; ++d) A.part[NV * to + d] = sum[d];
            }
            __syncthreads();  // the next tile's walk refills the sums
        }
    }
    pdl_trigger();
    if (SUMS) {
        __shared__ double sh[1][32];
        __shared__ bool last;
        double v[1] = {total};
        block_sum_n<1>(v, sh);
        if (publish_partials<1>(v, A.sums, A.ticket, &last)) {
            const double t = final_sum_narrow(A.sums, sh);
            if (tid == 0) {
                *A.result = t;
                *A.ticket = 0u;
            }
        }
    }
}

// A scalar quantity cell by cell, a thread each, where the fans are short (cells_win in fans.cu): the derivative per
// cell goes to cell_out (one density per cell) or to part, from where k_cell_nodes sums it per node.  Four CTAs an SM at 64
// registers (three with lambda, where four spill: 35.5 -> 33.8 us) hide the 14 to 40 gathers of a cell, which bound it.  `corners` has each cell's nodes in an order that suits the
// rounding and the gathers (fans.cu).  Kernels of 1.1 M Delaunay cells: dC/dz 23.2 + 17.0 us, (dR/dz)^T lambda 33.5 + 17.3 us (a
// fan with its 168 registers: 55 and 77 us together), energy 24.6 us (36).
constexpr int kCellThreads = 256;
template <int OP, int MODE>
__global__ void __launch_bounds__(kCellThreads, fan_has_lam<OP, MODE>() ? 3 : 4)
k_cells(int32_t C, const int4* __restrict__ corners, const double* __restrict__ coords, Material mat, FanArgs<double> A) {
    constexpr bool U = fan_has_u<OP>(), L = fan_has_lam<OP, MODE>();
    constexpr bool NODES = fan_nodes<OP, MODE>(), SUMS = fan_sums<OP, MODE>();
    double total = 0.0;
    double* out = mat.cell_control ? A.cell_out : A.part;
    const bool add = mat.cell_control && A.accumulate;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C; c += (int64_t)gridDim.x * blockDim.x) {
        const int4 n = __ldg(corners + c);
        auto at = [](const double* v, int64_t a) { return Vec3<double>{__ldg(v + 3 * a), __ldg(v + 3 * a + 1), __ldg(v + 3 * a + 2)}; };
        const Vec3<double> xa = at(coords, n.x);
        const Vec3<double> eb = at(coords, n.y) - xa, ep = at(coords, n.z) - xa, en = at(coords, n.w) - xa;
        const Vec3<double> cb = cross(ep, en), cp = cross(en, eb), cn = cross(eb, ep);
        const double det = fabs(dot(eb, cb));
        const double rho = cell_rho(mat, A.z, c, n);
        double q = det * (1.0 / 6.0);  // the volume, or vol eps(u).C.eps(u) and with lambda vol eps(lambda).C.eps(u)
        if (U) {
            const double k = 1.0 / (6.0 * det);
            const Vec3<double> ua = at(A.u, n.x);
            double e[6], s[6], esl = 0.0;
            fan_strain(at(A.u, n.y) - ua, at(A.u, n.z) - ua, at(A.u, n.w) - ua, cb, cp, cn, e);
            stress_voigt(mat, e, s);
            if (MODE != 3) q = k * (s[0] * e[0] + s[1] * e[1] + s[2] * e[2] + s[3] * e[3] + s[4] * e[4] + s[5] * e[5]);
            if (L) {
                const Vec3<double> la = at(A.lam, n.x);
                fan_strain(at(A.lam, n.y) - la, at(A.lam, n.z) - la, at(A.lam, n.w) - la, cb, cp, cn, e);
                esl = k * (s[0] * e[0] + s[1] * e[1] + s[2] * e[2] + s[3] * e[3] + s[4] * e[4] + s[5] * e[5]);
            }
            if (SUMS) total += 0.5 * q * simp(mat, rho);
            q = MODE == 3 ? esl : 0.5 * q + esl;
            if (MODE == 2 || MODE == 5) q = -q;
        } else if (SUMS) {
            total += q * simp(mat, rho);
        }
        if (NODES) {
            q *= simp_dx(mat, rho) * rho_dz(mat);
            out[c] = add ? out[c] + q : q;
        }
    }
    pdl_trigger();
    if (SUMS) {
        __shared__ double sh[1][32];
        __shared__ bool last;
        double v[1] = {total};
        block_sum_n<1>(v, sh);
        if (publish_partials<1>(v, A.sums, A.ticket, &last)) {
            double t[1];
            final_sums<1>(t, A.sums, sh);
            if (threadIdx.x == 0) {
                *A.result = t[0];
                *A.ticket = 0u;
            }
        }
    }
}

// out[a] = sum of the quantity over the node's cells in cell order, or added to out.
__global__ void __launch_bounds__(kThreads)
k_cell_nodes(int32_t N, const int32_t* __restrict__ n2c_ptr, const int32_t* __restrict__ n2c, const double* __restrict__ part,
             double* __restrict__ out, int accumulate) {
    pdl_wait();
    for (int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; a < N; a += (int64_t)gridDim.x * blockDim.x) {
        double sum = 0.0;
        const int32_t k1 = __ldg(n2c_ptr + a + 1);
        for (int32_t k = __ldg(n2c_ptr + a); k < k1; ++k) sum += part[__ldg(n2c + k) >> 2];
        out[a] = accumulate ? out[a] + sum : sum;
    }
}

// out[a] = sum of the node's tile sums in slot order, plus scale * F[a] (F != null), or added to
// out (accumulate).  copy != null: constrained dofs take copy's value instead (identity rows).
template <int NV, typename T>
__global__ void __launch_bounds__(kThreads)
k_fan_nodes(int32_t N, const int32_t* __restrict__ node_ptr, const T* __restrict__ part, T* __restrict__ out,
            const T* __restrict__ F, T scale, int accumulate, const uint8_t* __restrict__ mask,
            const T* __restrict__ copy, const PcgScalars* S) {
    pdl_wait();
    if (S && S->done) return;
    for (int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; a < N; a += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k0 = __ldg(node_ptr + a), k1 = __ldg(node_ptr + a + 1);
        T sum[NV];
#pragma unroll
        for (int d = 0; d < NV; ++d) sum[d] = T(0);
        for (int64_t k = k0; k < k1; ++k)
#pragma unroll
            for (int d = 0; d < NV; ++d) sum[d] += part[NV * k + d];
#pragma unroll
        for (int d = 0; d < NV; ++d) {
            const int64_t i = NV * a + d;
            T v = sum[d];
            if (F) v += scale * F[i];
            if (accumulate) v += out[i];
            if (copy && mask[i]) v = copy[i];
            out[i] = v;
        }
    }
}

// Inverse diagonal of the constrained operator from the node sums; 1 on constrained dofs.
__global__ void __launch_bounds__(kThreads)
k_fan_diag_nodes(int32_t N, const int32_t* __restrict__ node_ptr, const double* __restrict__ part,
                 const uint8_t* __restrict__ mask, double* __restrict__ dinv64, float* __restrict__ dinv32) {
    pdl_wait();
    for (int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; a < N; a += (int64_t)gridDim.x * blockDim.x) {
        double sum[3] = {0.0, 0.0, 0.0};
        for (int64_t k = __ldg(node_ptr + a); k < __ldg(node_ptr + a + 1); ++k)
#pragma unroll
            for (int d = 0; d < 3; ++d) sum[d] += part[3 * k + d];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double v = mask[3 * a + d] ? 1.0 : 1.0 / sum[d];
            if (dinv64) dinv64[3 * a + d] = v;
            if (dinv32) dinv32[3 * a + d] = float(v);
        }
    }
}

// SIMP weight s(rho_e) of each cell (ApplyWeighting, src/ApplyWeighting.hpp:55-64) in fan order.
__global__ void __launch_bounds__(kThreads)
k_fan_weights(int64_t n, const int32_t* __restrict__ cells, const int4* __restrict__ conn, const double* __restrict__ z,
              Material mat, double* __restrict__ w64, float* __restrict__ w32) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t c = cells[i];
        if (c < 0) continue;
        const double w = simp(mat, cell_rho(mat, z, c, conn[c]));
        w64[i] = w;
        w32[i] = float(w);
    }
}

__global__ void k_to_float(int64_t n, const double* __restrict__ a, float* __restrict__ b) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = float(a[i]);
}

// y_free += a x_free
__global__ void k_masked_axpy(int64_t n, const uint8_t* __restrict__ mask, double a, const double* __restrict__ x,
                              double* __restrict__ y) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (!mask[i]) y[i] += a * x[i];
}

// CTAs of one resident wave of a kernel, asked of the runtime once per (device, kernel, launch shape).
int resident_ctas(plato_problem* h, const void* kernel, int threads, int smem, int* ctas) {
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, int, int>, int> known;
    std::lock_guard<std::mutex> lock(mu);
    int& have = known[{h->device, kernel, threads, smem}];
    if (have == 0) {
        int per_sm = 0, sms = 0;
        PLATO_CUDA(h, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device));
        PLATO_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
        have = std::min(kFanMaxCtas, std::max(1, per_sm) * std::max(1, sms));
    }
    *ctas = have;
    return PLATO_OK;
}

// One handle has one `part`, so a call on another stream than the last one's first waits for that call there.
// On the legacy stream, which always exists, the end is recorded only when another stream has to wait for it; a
// stream of the caller's may be gone by then, so its end is recorded after each call (0.4 us of host time).
// Inside a capture nothing is waited for or recorded: the order of a graph's replays is its owner's.
bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) == cudaSuccess) return st != cudaStreamCaptureStatusNone;
    (void)cudaGetLastError();  // the legacy stream while a blocking stream is being captured
    return true;
}

int fan_begin(plato_problem* h) {
    FanPlan& P = h->fans;
    if (!P.pending || P.last == h->stream || capturing(h->stream)) return PLATO_OK;
    if (P.pending == 1) {
        if (capturing(P.last)) return PLATO_OK;
        PLATO_CUDA(h, cudaEventRecord(P.end, P.last));
    }
    PLATO_CUDA(h, cudaStreamWaitEvent(h->stream, P.end, 0));
    return PLATO_OK;
}

int fan_end(plato_problem* h) {
    FanPlan& P = h->fans;
    const bool legacy = h->stream == nullptr || h->stream == cudaStreamLegacy;
    if (!legacy) {
        if (capturing(h->stream)) return PLATO_OK;
        PLATO_CUDA(h, cudaEventRecord(P.end, h->stream));
    }
    P.last = h->stream;
    P.pending = legacy ? 1 : 2;
    return PLATO_OK;
}

template <int OP, int MODE, typename T>
int launch_fans(plato_problem* h, const Material& mat, FanArgs<T> A, const PcgScalars* S) {
    PLATO_RC(fan_plan(h));
    PLATO_RC(fan_begin(h));
    FanView fv = fan_view(h);
    A.n = h->N;
    A.part = reinterpret_cast<T*>(h->fans.part);
    A.sums = h->fans.sums;
    A.ticket = h->red_ticket;
    constexpr int NV = fan_values<OP>();
    const bool nodes = fan_nodes<OP, MODE>();
    if (!nodes) {  // a sum over all cells has no use for the tiles: as many small tiles as there are on a small mesh leave the
                   // last CTA's 32 threads hundreds of sums to add (energy of 12,000 cells 28 -> 21 us)
        fv.width = kFanThreads;
        fv.ntiles = (fv.nfans + kFanThreads - 1) / kFanThreads;
    }
    const int smem = nodes ? int(sizeof(T) * NV * 8 * fv.width + sizeof(uint4) * fv.width) : 0;
    // one resident wave; a small mesh has fewer tiles than that, and its calls are short of host time
    int ctas = fv.ntiles;
    if (fv.ntiles > kNumSMs) {
        const void* kernel = reinterpret_cast<const void*>(k_fans<OP, MODE, T>);
        PLATO_RC(ensure_smem_attribute(h, kernel, smem));
        int wave = 0;
        PLATO_RC(resident_ctas(h, kernel, fv.width, smem, &wave));
        ctas = std::min(ctas, wave);
    }
    k_fans<OP, MODE, T><<<ctas, fv.width, smem, h->stream>>>(fv, mat, A, S);
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

template <int NV, typename T>
int launch_fan_nodes(plato_problem* h, T* out, const T* F, T scale, int accumulate, const T* copy, const PcgScalars* S) {
    PLATO_CUDA(h, launch_pdl(k_fan_nodes<NV, T>, grid_for(h->N, kThreads, 148 * 16), kThreads, h->stream, h->N,
                             (const int32_t*)h->fans.node_ptr, reinterpret_cast<const T*>(h->fans.part), out, F, scale,
                             accumulate, (const uint8_t*)h->bc_mask, copy, S));
    PLATO_LAUNCH_CHECK(h);
    return S ? PLATO_OK : fan_end(h);  // a solver's products: the solve ends with the stream waited for
}

// A scalar quantity, by fans or by cells; with one density per node its nodal sums go to `out`, or are added to it.
template <int OP, int MODE>
int launch_scalar(plato_problem* h, const Material& mat, FanArgs<double> A, double* out) {
    constexpr bool nodes = fan_nodes<OP, MODE>();
    PLATO_RC(fan_plan(h));
    if (!h->fans.by_cell) {
        PLATO_RC((launch_fans<OP, MODE, double>(h, mat, A, nullptr)));
        if (!nodes || mat.cell_control) return PLATO_OK;
        return launch_fan_nodes<1, double>(h, out, nullptr, 0.0, A.accumulate, nullptr, nullptr);
    }
    PLATO_RC(fan_begin(h));
    A.part = h->fans.part;
    A.sums = h->fans.sums;
    A.ticket = h->red_ticket;
    // a sum takes one resident wave, whose last CTA then has few block sums to add (energy of 1.1 M cells 25 us, 36 with
    // a CTA for every 256 cells)
    int wave = kFanMaxCtas;
    if (fan_sums<OP, MODE>())
        PLATO_RC(resident_ctas(h, reinterpret_cast<const void*>(k_cells<OP, MODE>), kCellThreads, 0, &wave));
    k_cells<OP, MODE><<<grid_for(h->C, kCellThreads, wave), kCellThreads, 0, h->stream>>>(h->C, reinterpret_cast<const int4*>(h->fans.corners), h->coords, mat, A);
    PLATO_LAUNCH_CHECK(h);
    if (nodes && !mat.cell_control) {
        PLATO_CUDA(h, launch_pdl(k_cell_nodes, grid_for(h->N, kThreads, 148 * 16), kThreads, h->stream, h->N,
                                 (const int32_t*)h->n2c_ptr, (const int32_t*)h->n2c, (const double*)h->fans.part, out,
                                 A.accumulate));
        PLATO_LAUNCH_CHECK(h);
    }
    return fan_end(h);
}

}  // namespace

// R = K(z) u + scale_F * F: ElastostaticResidual::evaluate (src/elliptic/ElastostaticResidual.hpp:
// 165-234) and assemble_residual (src/Assembly.hpp:1222-1281); scale_F = -1 gives
// VectorFunction::value, 0 gives df/du.
int launch_internal_force(plato_problem* h, const double* u, const double* z, double* R, double scale_F) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.u = u;
    A.z = z;
    PLATO_RC((launch_fans<FAN_FORCE, 0, double>(h, h->material, A, nullptr)));
    return launch_fan_nodes<3, double>(h, R, scale_F != 0.0 ? h->F : nullptr, scale_F, 0, nullptr, nullptr);
}

// Control derivative: mode 1 the energy's d/dz (PhysicsScalarFunction::gradient_z,
// src/elliptic/PhysicsScalarFunction.hpp:432-495), 2 the compliance sensitivity with lambda = -u
// (Problem::criterionGradient, src/elliptic/Problem.hpp:423-448), 3 (dR/dz)^T lambda
// (VectorFunction::gradient_z, src/elliptic/VectorFunction.hpp:618-710, times lambda), 4 = 1 + 3.
int launch_nodal_control_derivative(plato_problem* h, int mode, const double* u, const double* z, const double* lam,
                                    double* out, int accumulate) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.u = u;
    A.z = z;
    A.lam = lam;
    A.cell_out = out;
    A.accumulate = accumulate;
    switch (mode) {
        case 1: return launch_scalar<FAN_QUANT, 1>(h, h->material, A, out);
        case 2: return launch_scalar<FAN_QUANT, 2>(h, h->material, A, out);
        case 3: return launch_scalar<FAN_QUANT, 3>(h, h->material, A, out);
        case 4: return launch_scalar<FAN_QUANT, 4>(h, h->material, A, out);
        default: return plato_fail(h, PLATO_BAD_INPUT, "unknown control-derivative mode");
    }
}

// Internal elastic energy into *result (device scalar).
int launch_energy(plato_problem* h, const double* u, const double* z, double* result) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.u = u;
    A.z = z;
    A.result = result;
    return launch_scalar<FAN_QUANT, 0>(h, h->material, A, nullptr);
}

// Compliance into *result (device scalar) and the self-adjoint dC/dz into dfdz, one pass (what an
// MPMD ComputeCriterion operation asks for together, src/Analyze_App.cpp:727-1014).
int launch_energy_and_gradient(plato_problem* h, const double* u, const double* z, double* result, double* dfdz) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.u = u;
    A.z = z;
    A.result = result;
    A.cell_out = dfdz;
    return launch_scalar<FAN_QUANT, 5>(h, h->material, A, dfdz);
}

// Geometric "Volume" criterion (src/geometric/Volume.hpp:83-110) with its own penalty, and its derivative.
int launch_volume(plato_problem* h, const Material& pen, const double* z, double* result) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.z = z;
    A.result = result;
    return launch_scalar<FAN_VOLUME, 0>(h, pen, A, nullptr);
}

int launch_volume_gradient(plato_problem* h, const Material& pen, const double* z, double* dvdz) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.z = z;
    A.cell_out = dvdz;
    return launch_scalar<FAN_VOLUME, 1>(h, pen, A, dvdz);
}

// ---- matrix-free operator ---------------------------------------------------------------------
//
// K(z) = sum_e s(rho_e) vol_e B_e^T C B_e applied element by element.  The constrained operator
// is the one applyBlockConstraints produces (src/ApplyConstraints.hpp:40-112): y = P K P x +
// (I - P) x with P the free-dof mask.  FP64 for the outer Krylov operator, FP32 (with FP32
// coordinates) for the mixed-precision preconditioner.

// Cell weights (FP64 and FP32, fan order) and the inverse diagonal (FP64 into h->v_dinv, FP32 into
// h->f_dinv) for control z.
int matfree_setup(plato_problem* h, const double* z) {
    const int64_t n = 3 * (int64_t)h->N;
    PLATO_RC(fan_plan(h));
    FanPlan& P = h->fans;
    const int64_t nw = 6 * (int64_t)P.nfans;
    if (!P.w64) PLATO_CUDA(h, cudaMalloc(&P.w64, sizeof(double) * nw));
    if (!P.w32) PLATO_CUDA(h, cudaMalloc(&P.w32, sizeof(float) * nw));
    if (!h->f_dinv) PLATO_CUDA(h, cudaMalloc(&h->f_dinv, sizeof(float) * n));
    if (!h->f_coords) {
        PLATO_CUDA(h, cudaMalloc(&h->f_coords, sizeof(float) * n));
        k_to_float<<<grid_for(n, kThreads), kThreads, 0, h->stream>>>(n, h->coords_soa, h->f_coords);
        PLATO_LAUNCH_CHECK(h);
    }
    k_fan_weights<<<grid_for(nw, kThreads), kThreads, 0, h->stream>>>(nw, P.cells, h->conn, z, h->material, P.w64, P.w32);
    PLATO_LAUNCH_CHECK(h);
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.w = P.w64;
    PLATO_RC((launch_fans<FAN_DIAG, 0, double>(h, h->material, A, nullptr)));
    PLATO_CUDA(h, launch_pdl(k_fan_diag_nodes, grid_for(h->N, kThreads, 148 * 16), kThreads, h->stream, h->N,
                             (const int32_t*)P.node_ptr, (const double*)P.part, (const uint8_t*)h->bc_mask, h->v_dinv,
                             h->f_dinv));
    PLATO_LAUNCH_CHECK(h);
    return fan_end(h);
}

// y = P K P x + (I - P) x with the weights of matfree_setup.  With S != nullptr both kernels return at
// once after the solver has converged.
int launch_ebe_apply64(plato_problem* h, const double* x, double* y, const PcgScalars* S) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.u = x;
    A.w = h->fans.w64;
    A.mask = h->bc_mask;
    PLATO_RC((launch_fans<FAN_EBE, 0, double>(h, h->material, A, S)));
    return launch_fan_nodes<3, double>(h, y, nullptr, 0.0, 0, x, S);
}

int launch_ebe_apply32(plato_problem* h, const float* x, float* y, const PcgScalars* S) {
    FanArgs<float> A{};
    A.coords = h->f_coords;
    A.u = x;
    A.w = h->fans.w32;
    A.mask = h->bc_mask;
    PLATO_RC((launch_fans<FAN_EBE, 0, float>(h, h->material, A, S)));
    return launch_fan_nodes<3, float>(h, y, nullptr, 0.f, 0, x, S);
}

// K x without the constraint mask (for the Dirichlet lift of inhomogeneous values).
int launch_ebe_apply64_unmasked(plato_problem* h, const double* x, double* y) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.u = x;
    A.w = h->fans.w64;
    PLATO_RC((launch_fans<FAN_EBE, 0, double>(h, h->material, A, nullptr)));
    return launch_fan_nodes<3, double>(h, y, nullptr, 0.0, 0, nullptr, nullptr);
}

int launch_masked_axpy(plato_problem* h, double a, const double* x, double* y) {
    const int64_t n = 3 * (int64_t)h->N;
    k_masked_axpy<<<grid_for(n, kThreads), kThreads, 0, h->stream>>>(n, h->bc_mask, a, x, y);
    PLATO_LAUNCH_CHECK(h);
    return PLATO_OK;
}

// y = P K(z) P x + (I - P) x for one product with a given control: the weights come from z on the
// way, without matfree_setup's weight and diagonal passes.
int launch_constrained_apply(plato_problem* h, const double* z, const double* x, double* y) {
    FanArgs<double> A{};
    A.coords = h->coords_soa;
    A.u = x;
    A.z = z;
    A.mask = h->bc_mask;
    PLATO_RC((launch_fans<FAN_FORCE, 0, double>(h, h->material, A, nullptr)));
    return launch_fan_nodes<3, double>(h, y, nullptr, 0.0, 0, x, nullptr);
}

}  // namespace plato
