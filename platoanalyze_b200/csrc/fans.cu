// Grouping of a mesh's cells into fans and tiles, built once per mesh on the device.
//
// An element kernel that gives every tetrahedron its own thread loads four nodes and adds to
// four nodes per cell.  Cells around a common edge share most of that: a fan of m cells
// {a, b, r_i, r_(i+1)} walked by one thread loads a, b and the ring r once, carries r_(i+1) and
// its cross product with the edge from one cell to the next, and adds to m + 2 or m + 3 nodes
// instead of 4 m.  Each cell joins the group of its longest edge -- the hex diagonal of a Kuhn
// box, which six cells share; on general meshes the groups are smaller -- and a group is cut
// into chains of adjacent cells of at most kFanRing ring nodes.  Whatever the mesh (cells that
// share an edge but no face, repeated cells, hundreds of cells around an edge), every cell ends
// in exactly one fan.
//
// The fans are sorted by blocks of space, and within a block by node number: a block is about 32
// fans long in the direction in which the node numbers run and 2 x 2 fans across, and the blocks
// follow a Morton curve (batch members one after the other).  So a tile of 128 consecutive fans
// touches about 300 distinct nodes instead of 1024, and the 32 lanes of a warp, a run of neighbours
// with consecutive node numbers, read a node quantity from 7 cache lines; with cubic blocks they
// touch nearly 32, and the L1 cache, which looks up one line after the other, bounds the kernels
// (residual of 6.1 M cells: 144 against 192 us).  The fans' sums meet in shared memory, and
// each (tile, node) sum is written to its place in node order; a second kernel adds a node's one to
// eight sums in a fixed order (fan_kernels.cu).
//
// On small meshes the fans are cut shorter, down to single cells: there the parallelism of more
// threads is worth more than the sharing.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <utility>

#include "fans.cuh"

namespace plato {
namespace {

constexpr int kRing = 6;     // most ring nodes of a fan
constexpr int kWindow = 32;  // cells of a group that are chained together
constexpr int kT = 256;

int bits_for(int64_t max_value) {
    int bits = 1;
    while (bits < 63 && (int64_t(1) << bits) <= max_value) ++bits;
    return bits;
}

// Key (smaller node, larger node) of each cell's longest edge; equal lengths go to the smaller key,
// and a length is always computed from the smaller to the larger node, so that every cell around an
// edge sees the same number.
__global__ void k_longest_edge(int32_t C, const int4* __restrict__ conn, const double* __restrict__ x,
                               uint64_t* __restrict__ key, int32_t* __restrict__ cell) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C; c += (int64_t)gridDim.x * blockDim.x) {
        const int4 n = conn[c];
        const int32_t id[4] = {n.x, n.y, n.z, n.w};
        uint64_t best = ~uint64_t(0);
        double len = -1.0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = i + 1; j < 4; ++j) {
                const int32_t p = min(id[i], id[j]), q = max(id[i], id[j]);
                double l = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double t = x[3 * (int64_t)q + d] - x[3 * (int64_t)p + d];
                    l = fma(t, t, l);
                }
                const uint64_t k = (uint64_t(uint32_t(p)) << 32) | uint32_t(q);
                if (l > len || (l == len && k < best)) {
                    len = l;
                    best = k;
                }
            }
        key[c] = best;
        cell[c] = int32_t(c);
    }
}

// The two nodes of a cell that are not on the edge.
__device__ __forceinline__ int2 opposite(int4 n, int32_t a, int32_t b) {
    const int32_t id[4] = {n.x, n.y, n.z, n.w};
    int32_t o[2] = {-1, -1};
    int k = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (id[i] != a && id[i] != b && k < 2) o[k++] = id[i];
    return make_int2(o[0], o[1]);
}

// Cuts each group's cells (edge `key[g]`, cells start[g] .. start[g] + count[g]) into fans.  FILL = 0
// counts them; FILL = 1 writes fan f0[g] + k: its 8 nodes (-1: none), cells and closed flag.  A fan has
// at most ring_max ring nodes.
template <int FILL>
__global__ void k_chain(int32_t ngroups, int ring_max, const uint64_t* __restrict__ key, const int32_t* __restrict__ start,
                        const int32_t* __restrict__ count, const int32_t* __restrict__ cell,
                        const int4* __restrict__ conn, const int32_t* __restrict__ f0, int32_t* __restrict__ nf,
                        int32_t* __restrict__ nodes, int32_t* __restrict__ cells, uint8_t* __restrict__ closed) {
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < ngroups;
         g += (int64_t)gridDim.x * blockDim.x) {
        const int32_t a = int32_t(key[g] >> 32), b = int32_t(key[g] & 0xffffffffu);
        int32_t made = 0;
        for (int32_t w0 = 0; w0 < count[g]; w0 += kWindow) {
            const int m = min(kWindow, count[g] - w0);
            const int32_t* mine = cell + start[g] + w0;
            uint32_t left = m == 32 ? 0xffffffffu : (1u << m) - 1u;
            while (left) {
                // start at an end of a chain (a ring node that only one remaining cell has), else anywhere
                int first = __ffs(left) - 1;
                int2 o = opposite(conn[mine[first]], a, b);
                bool found = false;
                for (int i = 0; i < m && !found; ++i) {
                    if (!((left >> i) & 1u)) continue;
                    const int2 oi = opposite(conn[mine[i]], a, b);
                    int sx = 0, sy = 0;
                    for (int j = 0; j < m; ++j) {
                        if (j == i || !((left >> j) & 1u)) continue;
                        const int2 oj = opposite(conn[mine[j]], a, b);
                        sx |= oj.x == oi.x || oj.y == oi.x;
                        sy |= oj.x == oi.y || oj.y == oi.y;
                    }
                    if (!sx || !sy) {
                        first = i;
                        o = sx ? make_int2(oi.y, oi.x) : oi;  // the free end comes first
                        found = true;
                    }
                }
                int32_t ring[kRing], cl[kRing];
                ring[0] = o.x;
                ring[1] = o.y;
                cl[0] = mine[first];
                int nr = 2, nt = 1;
                bool shut = false;
                left &= ~(1u << first);
                while (left && !shut && nt < ring_max) {
                    int next = -1;
                    int32_t far = -1;
                    for (int j = 0; j < m && next < 0; ++j) {
                        if (!((left >> j) & 1u)) continue;
                        const int2 oj = opposite(conn[mine[j]], a, b);
                        if (oj.x == ring[nr - 1]) { next = j; far = oj.y; }
                        else if (oj.y == ring[nr - 1]) { next = j; far = oj.x; }
                    }
                    if (next < 0) break;
                    if (far == ring[0]) shut = true;
                    else if (nr == ring_max) break;
                    else ring[nr++] = far;
                    cl[nt++] = mine[next];
                    left &= ~(1u << next);
                }
                if (FILL) {
                    const int64_t f = int64_t(f0[g]) + made;
                    nodes[8 * f] = a;
                    nodes[8 * f + 1] = b;
                    for (int i = 0; i < kRing; ++i) {
                        nodes[8 * f + 2 + i] = i < nr ? ring[i] : -1;
                        cells[6 * f + i] = i < nt ? cl[i] : -1;
                    }
                    closed[f] = shut ? 1 : 0;
                }
                ++made;
            }
        }
        if (!FILL) nf[g] = made;
    }
}

__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // 10 bits to every third bit
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    return (v | (v << 2)) & 0x09249249u;
}

// The axis along which consecutive node numbers lie most often: count[d] of the pairs (i, i + 1) that
// differ most in coordinate d.
__global__ void k_number_axis(int32_t N, const double* __restrict__ x, unsigned long long* __restrict__ count) {
    unsigned int mine[3] = {0, 0, 0};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i + 1 < N; i += (int64_t)gridDim.x * blockDim.x) {
        const double d0 = fabs(x[3 * i + 3] - x[3 * i]), d1 = fabs(x[3 * i + 4] - x[3 * i + 1]), d2 = fabs(x[3 * i + 5] - x[3 * i + 2]);
        mine[0] += d0 > d1 && d0 > d2;
        mine[1] += d1 >= d0 && d1 > d2;
        mine[2] += d2 >= d0 && d2 >= d1;
    }
    for (int d = 0; d < 3; ++d) {
        const unsigned int w = __reduce_add_sync(0xffffffffu, mine[d]);
        if ((threadIdx.x & 31) == 0 && w) atomicAdd(count + d, (unsigned long long)w);
    }
}

// *count += the cells whose smallest node number is within 64 of the cell before's
__global__ void k_cell_steps(int32_t C, const int4* __restrict__ conn, unsigned long long* __restrict__ count) {
    unsigned int mine = 0;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c + 1 < C; c += (int64_t)gridDim.x * blockDim.x) {
        const int4 a = conn[c], b = conn[c + 1];
        mine += abs(min(min(a.x, a.y), min(a.z, a.w)) - min(min(b.x, b.y), min(b.z, b.w))) <= 64;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(count, (unsigned long long)mine);
}

// Sort key of each fan: batch member, then the Morton code of the block its edge midpoint lies in.
__global__ void k_morton(int32_t nf, const int32_t* __restrict__ nodes, const double* __restrict__ x, double x0,
                         double x1, double x2, double s0, double s1, double s2, const int32_t* __restrict__ member_off,
                         int nmembers, uint64_t* __restrict__ key, int32_t* __restrict__ id) {
    for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nf; f += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = nodes[8 * f], b = nodes[8 * f + 1];
        const double lo[3] = {x0, x1, x2}, scale[3] = {s0, s1, s2};
        uint32_t q[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double t = (0.5 * (x[3 * a + d] + x[3 * b + d]) - lo[d]) * scale[d];
            q[d] = uint32_t(fmin(fmax(t, 0.0), 1023.0));
        }
        int lo_m = 0, hi_m = nmembers - 1;  // the last member whose first node is <= a
        while (lo_m < hi_m) {
            const int mid = (lo_m + hi_m + 1) >> 1;
            if (member_off[mid] <= a) lo_m = mid; else hi_m = mid - 1;
        }
        key[f] = (uint64_t(lo_m) << 30) | (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
        id[f] = int32_t(f);
    }
}

// Final order of the fans: records and cells, and the (tile, node) reference of every node position,
// value = position * width + fan within the tile.  Absent ring nodes get the key (ntiles, 0) behind
// all others.
__global__ void k_place(int32_t nf, int32_t width, int32_t ntiles, const int32_t* __restrict__ order,
                        const int32_t* __restrict__ nodes, const int32_t* __restrict__ cells_in,
                        const uint8_t* __restrict__ closed, int32_t* __restrict__ rec, int32_t* __restrict__ cells,
                        uint64_t* __restrict__ key, uint32_t* __restrict__ ref) {
    for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nf; f += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = order[f];
        const uint32_t tile = uint32_t(f / width), lf = uint32_t(f % width);
        for (int p = 0; p < 8; ++p) {
            const int32_t n = nodes[8 * o + p];
            rec[8 * f + p] = p == 0 && closed[o] ? n | kFanClosed : n;
            key[8 * f + p] = n < 0 ? (uint64_t(ntiles) << 32) : ((uint64_t(tile) << 32) | uint32_t(n));
            ref[8 * f + p] = (uint32_t(p) * uint32_t(width)) + lf;
        }
        for (int i = 0; i < 6; ++i) cells[6 * f + i] = cells_in[6 * o + i];
    }
}

// The cells' nodes for the cell-by-cell kernels: first the corner whose three edges are shortest -- a sliver's determinant
// loses the fewest digits from there (error of a lambda product on eight Delaunay meshes against extended precision, geometric
// mean: 1.3e-15, from the end of the longest edge 4.3e-15) -- then the others by number, so that neighbouring cells' nodes
// lie side by side (energy of 1.1 M cells 28.3 -> 24.6 us).
__global__ void k_corners(int32_t C, const int4* __restrict__ conn, const double* __restrict__ x, int4* __restrict__ corners) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C; c += (int64_t)gridDim.x * blockDim.x) {
        int32_t id[4] = {conn[c].x, conn[c].y, conn[c].z, conn[c].w};
        auto swap_if = [&](int p, int q) {
            if (id[p] > id[q]) { const int32_t t = id[p]; id[p] = id[q]; id[q] = t; }
        };
        swap_if(0, 1); swap_if(2, 3); swap_if(0, 2); swap_if(1, 3); swap_if(1, 2);
        double sum[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int q = p + 1; q < 4; ++q) {
                double l = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double t = x[3 * (int64_t)id[q] + d] - x[3 * (int64_t)id[p] + d];
                    l = fma(t, t, l);
                }
                sum[p] += l;
                sum[q] += l;
            }
        int best = 0;
#pragma unroll
        for (int p = 1; p < 4; ++p)
            if (sum[p] < sum[best]) best = p;
        corners[c] = best == 0 ? make_int4(id[0], id[1], id[2], id[3]) : best == 1 ? make_int4(id[1], id[0], id[2], id[3])
                   : best == 2 ? make_int4(id[2], id[0], id[1], id[3]) : make_int4(id[3], id[0], id[1], id[2]);
    }
}

__global__ void k_heads(int64_t nref, const uint64_t* __restrict__ key, int32_t ntiles, int32_t* __restrict__ head,
                        unsigned long long* __restrict__ nvalid) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nref; i += (int64_t)gridDim.x * blockDim.x) {
        const bool valid = int32_t(key[i] >> 32) < ntiles;
        head[i] = valid && (i == 0 || key[i] != key[i - 1]) ? 1 : 0;
        if (valid && (i == nref - 1 || int32_t(key[i + 1] >> 32) >= ntiles)) *nvalid = (unsigned long long)(i + 1);
    }
}

// entry = scan - 1 of each valid reference: its node, its first reference, the tile's first entry
__global__ void k_entries(int64_t nvalid, const uint64_t* __restrict__ key, const int32_t* __restrict__ head,
                          const int32_t* __restrict__ scan, int32_t ntiles, int32_t* __restrict__ tile_ptr,
                          int32_t* __restrict__ node, int32_t* __restrict__ first, int32_t* __restrict__ count) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nvalid; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t e = scan[i] - 1;
        if (head[i]) {
            const int32_t n = int32_t(key[i] & 0xffffffffu);
            node[e] = n;
            first[e] = int32_t(i);
            atomicAdd(count + n, 1);
            const int32_t t = int32_t(key[i] >> 32);
            if (i == 0 || int32_t(key[i - 1] >> 32) != t) tile_ptr[t] = e;  // every tile holds a fan
        }
        if (i == nvalid - 1) {
            tile_ptr[ntiles] = e + 1;
            first[e + 1] = int32_t(nvalid);
        }
    }
}

// a tile's references stand side by side in `inc` from the tile's start, 8 per fan
__global__ void k_uses(int64_t nvalid, int32_t width, const uint64_t* __restrict__ key, const uint32_t* __restrict__ ref,
                       const int32_t* __restrict__ head, const int32_t* __restrict__ scan,
                       const int32_t* __restrict__ tile_ptr, const int32_t* __restrict__ first,
                       uint32_t* __restrict__ place, uint16_t* __restrict__ inc) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nvalid; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t t = int32_t(key[i] >> 32), e = scan[i] - 1;
        const int32_t k = int32_t(i) - first[tile_ptr[t]];
        inc[8 * int64_t(t) * width + k] = uint16_t(ref[i]);
        if (head[i]) place[e] = (uint32_t(k) << 16) | uint32_t(first[e + 1] - first[e]);
    }
}

__global__ void k_entry_keys(int32_t ne, const int32_t* __restrict__ node, uint32_t* __restrict__ key,
                             int32_t* __restrict__ id) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
        key[e] = uint32_t(node[e]);
        id[e] = int32_t(e);
    }
}

__global__ void k_slots(int32_t ne, const int32_t* __restrict__ sorted, int32_t* __restrict__ slot) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ne; i += (int64_t)gridDim.x * blockDim.x)
        slot[sorted[i]] = int32_t(i);
}

// Stream-ordered scratch that is given back at the end of its scope.
struct Scratch {
    plato_problem* h;
    cudaStream_t s;
    std::vector<void*> held;
    explicit Scratch(plato_problem* handle) : h(handle), s(handle->stream) {}
    ~Scratch() { release(); }
    void release() {
        for (void* p : held) cudaFreeAsync(p, s);
        held.clear();
    }
    template <typename T>
    cudaError_t get(T** p, int64_t count) {
        void* q = nullptr;
        const cudaError_t e = plan_alloc(h, &q, sizeof(T) * size_t(std::max<int64_t>(count, 1)), s);
        if (e == cudaSuccess) held.push_back(q);
        *p = static_cast<T*>(q);
        return e;
    }
};

template <typename K, typename V>
cudaError_t sort_pairs(Scratch& mem, const K* kin, K* kout, const V* vin, V* vout, int64_t n, int bits) {
    size_t bytes = 0;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, bytes, kin, kout, vin, vout, n, 0, bits, mem.s);
    char* tmp = nullptr;
    if (e == cudaSuccess) e = mem.get(&tmp, int64_t(bytes));
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(tmp, bytes, kin, kout, vin, vout, n, 0, bits, mem.s);
    return e;
}

template <bool INCLUSIVE>
cudaError_t scan(Scratch& mem, const int32_t* in, int32_t* out, int64_t n) {
    size_t bytes = 0;
    char* tmp = nullptr;
    cudaError_t e = INCLUSIVE ? cub::DeviceScan::InclusiveSum(nullptr, bytes, in, out, n, mem.s)
                              : cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, n, mem.s);
    if (e == cudaSuccess) e = mem.get(&tmp, int64_t(bytes));
    if (e == cudaSuccess)
        e = INCLUSIVE ? cub::DeviceScan::InclusiveSum(tmp, bytes, in, out, n, mem.s)
                      : cub::DeviceScan::ExclusiveSum(tmp, bytes, in, out, n, mem.s);
    return e;
}

// Arrays of the plan that share one allocation: add() each, then allocate(), which sets their pointers.
// A cudaMalloc and its cudaFree cost 0.2 to 0.4 ms, a tenth of the creation of a 60x30x30 handle for eleven.
struct Arena {
    std::vector<std::pair<void**, size_t>> parts;
    size_t total = 0;
    template <typename T>
    void add(T** p, int64_t count) {
        parts.emplace_back(reinterpret_cast<void**>(p), total);
        total += (sizeof(T) * size_t(std::max<int64_t>(count, 1)) + 255) & ~size_t(255);
    }
    cudaError_t allocate(void** base) {
        const cudaError_t e = cudaMalloc(base, total);
        if (e == cudaSuccess)
            for (auto& [p, offset] : parts) *p = static_cast<char*>(*base) + offset;
        return e;
    }
};

// Fans per tile: the wider the tile the fewer (tile, node) sums, as long as every SM gets
// about four tiles (the residual of 12,000 cells takes 5 us in tiles of 32, one CTA on each SM, against
// 11 us in 63 tiles of full-length fans).
int32_t tile_width(int64_t nfans) {
    for (int32_t w : {128, 64})
        if (nfans >= int64_t(w) * 4 * kNumSMs) return w;
    return 32;
}

// Ring nodes of a fan: single cells below about 200 cells per SM, pairs below 400, then the full six.
int ring_nodes(int64_t cells) {
    if (cells < 200 * int64_t(kNumSMs)) return 2;
    return cells < 400 * int64_t(kNumSMs) ? 3 : kRing;
}

// Whether the scalar quantities (energy, volume, control derivatives) run cell by cell.  On a box cut into Kuhn's six cells,
// jittered or not, a fan has 5 to 6 cells and shares more than the walk costs; on a general mesh it has about two,
// and a warp walks as long as its longest fan with a third of the warps.  Jitter of 0.3 of the spacing, 3.6 cells a fan,
// is about even (120x60x60: dC/dz 86 by fans, 79 us by cells, value and dC/dz 122 and 114, energy 66 and 68, lambda
// 125 and 96; 5.5 cells: 54 and 78, 85 and 114, 53 and 69, 78 and 96), two cells are not (1.1 M Delaunay cells: dC/dz 56 and 42,
// lambda 78 and 54, energy 35 and 27, volume gradient 41 and 33).  The cells come in the mesh's order; the
// fans are sorted by place, so where neighbours in the numbering are far apart the fans win (the same, shuffled: dC/dz 73
// and 110, lambda 102 and 133).  Below the size at which fans get their full length both take the time of two launches.
// The residual and the matrix-free product stay with the fans, which win on all of these (1.1 M cells 76 and 94).
bool cells_win(int64_t cells, int64_t nfans, int64_t close) {
    return cells >= 400 * int64_t(kNumSMs) && cells < 3 * nfans && 2 * close >= cells;
}

}  // namespace

void fan_release(plato_problem* h) {
    FanPlan& f = h->fans;
    for (void* p : {f.mem[0], f.mem[1], (void*)f.w64, (void*)f.w32})
        if (p) cudaFree(p);
    if (f.end) cudaEventDestroy(f.end);
    f = FanPlan{};
}

FanView fan_view(const plato_problem* h) {
    const FanPlan& f = h->fans;
    return FanView{f.nfans, f.ntiles, f.width, reinterpret_cast<const int4*>(f.rec), f.cells, f.tile_ptr, f.place,
                   f.slot, reinterpret_cast<const uint4*>(f.inc), f.node_ptr};
}

int fan_plan(plato_problem* h) {
    FanPlan& P = h->fans;
    if (P.ready) return PLATO_OK;
    fan_release(h);  // what an earlier attempt that failed has left
    cudaStream_t s = h->stream;
    Scratch mem(h), early(h);
    const int32_t C = h->C, N = h->N;
    constexpr int kGrid = 148 * 64;

    // groups of cells with the same longest edge
    uint64_t *key = nullptr, *key2 = nullptr, *gkey = nullptr;
    int32_t *cell = nullptr, *cell2 = nullptr, *gcount = nullptr, *gstart = nullptr, *ngroups_d = nullptr;
    PLATO_CUDA(h, early.get(&key, C));
    PLATO_CUDA(h, early.get(&key2, C));
    PLATO_CUDA(h, early.get(&gkey, C));
    PLATO_CUDA(h, early.get(&cell, C));
    PLATO_CUDA(h, early.get(&cell2, C));
    PLATO_CUDA(h, early.get(&gcount, C));
    PLATO_CUDA(h, early.get(&gstart, C));
    PLATO_CUDA(h, early.get(&ngroups_d, 1));
    k_longest_edge<<<grid_for(C, kT, kGrid), kT, 0, s>>>(C, h->conn, h->coords, key, cell);
    PLATO_LAUNCH_CHECK(h);
    PLATO_CUDA(h, sort_pairs(early, key, key2, cell, cell2, C, 32 + bits_for(N)));
    {
        size_t bytes = 0;
        char* tmp = nullptr;
        PLATO_CUDA(h, cub::DeviceRunLengthEncode::Encode(nullptr, bytes, key2, gkey, gcount, ngroups_d, C, s));
        PLATO_CUDA(h, early.get(&tmp, int64_t(bytes)));
        PLATO_CUDA(h, cub::DeviceRunLengthEncode::Encode(tmp, bytes, key2, gkey, gcount, ngroups_d, C, s));
    }
    int32_t ng = 0;
    PLATO_CUDA(h, cudaMemcpyAsync(&ng, ngroups_d, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    PLATO_CUDA(h, cudaStreamSynchronize(s));
    PLATO_CUDA(h, scan<false>(early, gcount, gstart, ng));

    // fans of each group: count, place, write
    const int ring_max = ring_nodes(C);
    int32_t *gfans = nullptr, *gfirst = nullptr, *fnodes = nullptr, *fcells = nullptr;
    uint8_t* closed = nullptr;
    PLATO_CUDA(h, early.get(&gfans, int64_t(ng) + 1));
    PLATO_CUDA(h, early.get(&gfirst, int64_t(ng) + 1));
    PLATO_CUDA(h, cudaMemsetAsync(gfans + ng, 0, sizeof(int32_t), s));
    k_chain<0><<<grid_for(ng, 128, kGrid), 128, 0, s>>>(ng, ring_max, gkey, gstart, gcount, cell2, h->conn, nullptr, gfans, nullptr,
                                                        nullptr, nullptr);
    PLATO_LAUNCH_CHECK(h);
    PLATO_CUDA(h, scan<false>(early, gfans, gfirst, int64_t(ng) + 1));
    int32_t nf = 0;
    PLATO_CUDA(h, cudaMemcpyAsync(&nf, gfirst + ng, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    PLATO_CUDA(h, cudaStreamSynchronize(s));
    PLATO_CUDA(h, mem.get(&fnodes, 8 * int64_t(nf)));
    PLATO_CUDA(h, mem.get(&fcells, 6 * int64_t(nf)));
    PLATO_CUDA(h, mem.get(&closed, nf));
    k_chain<1><<<grid_for(ng, 128, kGrid), 128, 0, s>>>(ng, ring_max, gkey, gstart, gcount, cell2, h->conn, gfirst, nullptr, fnodes,
                                                        fcells, closed);
    PLATO_LAUNCH_CHECK(h);

    // order by blocks along a Morton curve; within a block the sort keeps the groups' order, by node
    int32_t *order = nullptr, *order_in = nullptr, *members = nullptr;
    unsigned long long* axis_d = nullptr;  // pairs along each axis, and close cells
    const int nmem = h->batch.nseg > 0 ? h->batch.nseg : 1;
    PLATO_CUDA(h, mem.get(&order, nf));
    PLATO_CUDA(h, early.get(&order_in, nf));
    PLATO_CUDA(h, early.get(&members, nmem));
    PLATO_CUDA(h, early.get(&axis_d, 4));
    const int32_t zero = 0;
    PLATO_CUDA(h, cudaMemcpyAsync(members, h->batch.nseg > 0 ? h->batch.node_off.data() : &zero, sizeof(int32_t) * nmem,
                                  cudaMemcpyHostToDevice, s));
    PLATO_CUDA(h, cudaMemsetAsync(axis_d, 0, 4 * sizeof(unsigned long long), s));
    k_number_axis<<<grid_for(N, kT, 148 * 8), kT, 0, s>>>(N, h->coords, axis_d);
    PLATO_LAUNCH_CHECK(h);
    k_cell_steps<<<grid_for(C, kT, 148 * 8), kT, 0, s>>>(C, h->conn, axis_d + 3);
    PLATO_LAUNCH_CHECK(h);
    unsigned long long axis[4] = {0, 0, 0, 0};
    PLATO_CUDA(h, cudaMemcpyAsync(axis, axis_d, sizeof(axis), cudaMemcpyDeviceToHost, s));
    PLATO_CUDA(h, cudaStreamSynchronize(s));
    const int along = axis[2] >= axis[1] && axis[2] >= axis[0] ? 2 : (axis[1] >= axis[0] ? 1 : 0);
    // a fan's share of the mesh's box (of one member's, on the average) is about a cube of side `side`
    double volume = 1.0, scale[3];
    for (int d = 0; d < 3; ++d) volume *= std::max(h->bbox_max[d] - h->bbox_min[d], 0.0);
    const double side = std::cbrt(volume * nmem / std::max(nf, 1));
    for (int d = 0; d < 3; ++d) {
        const double extent = h->bbox_max[d] - h->bbox_min[d];
        const double block = std::max(side * (d == along ? 32.0 : 2.0), extent / 1023.0);
        scale[d] = block > 0.0 ? 1.0 / block : 0.0;
    }
    k_morton<<<grid_for(nf, kT, kGrid), kT, 0, s>>>(nf, fnodes, h->coords, h->bbox_min[0], h->bbox_min[1], h->bbox_min[2],
                                                    scale[0], scale[1], scale[2], members, nmem, key, order_in);
    PLATO_LAUNCH_CHECK(h);
    PLATO_CUDA(h, sort_pairs(early, key, key2, order_in, order, nf, 30 + bits_for(nmem)));
    early.release();  // a general mesh would need 60 bytes a cell more at the references' sort

    // tiles: references sorted by (tile, node), and their distinct nodes
    const int32_t W = tile_width(nf), nt = (nf + W - 1) / W;
    const int64_t nref = 8 * int64_t(nf);
    uint64_t *rkey = nullptr, *rkey2 = nullptr;
    uint32_t *ref = nullptr, *ref2 = nullptr;
    int32_t *head = nullptr, *entry = nullptr, *count = nullptr, *node = nullptr, *first = nullptr;
    unsigned long long* nvalid_d = nullptr;
    PLATO_CUDA(h, mem.get(&rkey, nref));
    PLATO_CUDA(h, mem.get(&rkey2, nref));
    PLATO_CUDA(h, mem.get(&ref, nref));
    PLATO_CUDA(h, mem.get(&ref2, nref));
    PLATO_CUDA(h, mem.get(&head, nref));
    PLATO_CUDA(h, mem.get(&entry, nref));
    PLATO_CUDA(h, mem.get(&count, int64_t(N) + 1));
    PLATO_CUDA(h, mem.get(&nvalid_d, 1));
    Arena by_fan;
    by_fan.add(&P.rec, nref);
    by_fan.add(&P.cells, 6 * int64_t(nf));
    by_fan.add(&P.tile_ptr, int64_t(nt) + 1);
    by_fan.add(&P.inc, 8 * int64_t(nt) * W);
    by_fan.add(&P.node_ptr, int64_t(N) + 1);
    by_fan.add(&P.sums, int64_t(kFanMaxCtas));  // workspace: a sum per CTA
    PLATO_CUDA(h, by_fan.allocate(&P.mem[0]));
    PLATO_CUDA(h, cudaMemsetAsync(count, 0, sizeof(int32_t) * (size_t(N) + 1), s));
    k_place<<<grid_for(nf, kT, kGrid), kT, 0, s>>>(nf, W, nt, order, fnodes, fcells, closed, P.rec, P.cells, rkey, ref);
    PLATO_LAUNCH_CHECK(h);
    PLATO_CUDA(h, sort_pairs(mem, rkey, rkey2, ref, ref2, nref, 32 + bits_for(nt)));
    k_heads<<<grid_for(nref, kT, kGrid), kT, 0, s>>>(nref, rkey2, nt, head, nvalid_d);
    PLATO_LAUNCH_CHECK(h);
    PLATO_CUDA(h, scan<true>(mem, head, entry, nref));
    unsigned long long nv = 0;
    int32_t ne = 0;
    PLATO_CUDA(h, cudaMemcpyAsync(&nv, nvalid_d, sizeof(nv), cudaMemcpyDeviceToHost, s));
    PLATO_CUDA(h, cudaMemcpyAsync(&ne, entry + nref - 1, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    PLATO_CUDA(h, cudaStreamSynchronize(s));
    PLATO_CUDA(h, mem.get(&node, ne));
    PLATO_CUDA(h, mem.get(&first, int64_t(ne) + 1));
    const int by_cell = cells_win(C, nf, int64_t(axis[3]));
    Arena by_entry;
    by_entry.add(&P.place, ne);
    by_entry.add(&P.slot, ne);
    by_entry.add(&P.corners, by_cell ? 4 * int64_t(C) : 0);
    by_entry.add(&P.part, std::max<int64_t>(3 * int64_t(ne), by_cell ? C : 0));  // workspace: three values per entry
    PLATO_CUDA(h, by_entry.allocate(&P.mem[1]));
    k_entries<<<grid_for(int64_t(nv), kT, kGrid), kT, 0, s>>>(int64_t(nv), rkey2, head, entry, nt, P.tile_ptr, node, first,
                                                              count);
    PLATO_LAUNCH_CHECK(h);
    k_uses<<<grid_for(int64_t(nv), kT, kGrid), kT, 0, s>>>(int64_t(nv), W, rkey2, ref2, head, entry, P.tile_ptr, first,
                                                           P.place, P.inc);
    PLATO_LAUNCH_CHECK(h);

    if (by_cell) {
        k_corners<<<grid_for(C, kT, kGrid), kT, 0, s>>>(C, h->conn, h->coords, reinterpret_cast<int4*>(P.corners));
        PLATO_LAUNCH_CHECK(h);
    }

    // places of the entries in node order
    uint32_t *ekey = nullptr, *ekey2 = nullptr;
    int32_t *eid = nullptr, *eid2 = nullptr;
    PLATO_CUDA(h, mem.get(&ekey, ne));
    PLATO_CUDA(h, mem.get(&ekey2, ne));
    PLATO_CUDA(h, mem.get(&eid, ne));
    PLATO_CUDA(h, mem.get(&eid2, ne));
    k_entry_keys<<<grid_for(ne, kT, kGrid), kT, 0, s>>>(ne, node, ekey, eid);
    PLATO_LAUNCH_CHECK(h);
    PLATO_CUDA(h, sort_pairs(mem, ekey, ekey2, eid, eid2, ne, bits_for(N)));
    k_slots<<<grid_for(ne, kT, kGrid), kT, 0, s>>>(ne, eid2, P.slot);
    PLATO_LAUNCH_CHECK(h);
    PLATO_CUDA(h, scan<false>(mem, count, P.node_ptr, int64_t(N) + 1));

    PLATO_CUDA(h, cudaStreamSynchronize(s));
    PLATO_CUDA(h, cudaEventCreateWithFlags(&P.end, cudaEventDisableTiming));
    P.by_cell = by_cell;
    P.nfans = nf;
    P.ntiles = nt;
    P.width = W;
    P.ready = 1;
    return PLATO_OK;
}

}  // namespace plato
