// Fans: the cell grouping that the element kernels walk (fans.cu builds it once per mesh).
#pragma once

#include "plato_internal.cuh"

namespace plato {

// A fan is up to 6 tetrahedra {a, b, r_i, r_(i+1)} around one edge (a, b): nodes a and b, then
// up to 6 ring nodes; a closed fan of m tetrahedra has m ring nodes, an open one m + 1.  A tile is
// `width` consecutive fans, one per thread of a CTA; an entry is a (tile, distinct node) pair.
constexpr int32_t kFanClosed = 1 << 30;  // flag in the record's node a (node ids stay below 2^30)
struct FanView {
    int32_t         nfans, ntiles, width;
    const int4*     rec;       // [2 * nfans] a (and the closed flag), b, ring; -1: none
    const int32_t*  cells;     // [6 * nfans] cell of each tetrahedron (-1: none)
    const int32_t*  tile_ptr;  // [ntiles + 1] first entry of each tile
    const uint32_t* place;     // [entries] uses of the entry's node in the tile: first place in inc << 16 | count
    const int32_t*  slot;      // [entries] position of the entry among all entries sorted by node
    const uint4*    inc;       // [ntiles * width] 8 uses each: position in the fan * width + fan within the tile
    const int32_t*  node_ptr;  // [num_nodes + 1] slots of each node
};

int fan_plan(plato_problem* h);      // builds the grouping (once per mesh)
void fan_release(plato_problem* h);
FanView fan_view(const plato_problem* h);

}  // namespace plato
