// demwalk.cuh -- the spheres around the fluid particles of a warp.
//
// A fluid particle near the spheres has up to ~160 of them in its window of 27
// coupling cells; a thread that walks them alone waits for four loads in a
// chain per sphere (slot -> index -> position -> constants).  Here the lanes
// of a warp, whose particles are neighbours in cell order and so have nearly
// the same window, load 32 spheres at once into shared memory, and every lane
// tests all of them.  A lane meets its spheres in slot order, as on its own.
#pragma once

#include <limits.h>

#include "common.cuh"

namespace sd {

struct DemTile {
    float4 p[32];  // x, y, z, bound of d2 (below it: in reach)
    float4 q[32], r[32];
};

// load(b, p, q, r): fields of sphere b (p.w the bound on d2; a negative one
// keeps the sphere out).  body(i, d2): sphere i of the tile is in reach of this
// lane's particle.  All lanes of the warp call it; mine = false: no particle.
template <class Load, class Body>
__device__ __forceinline__ void warp_dem_visit(const Geo& gd, bool mine, float px, float py, float pz, float rq,
                                               int inst, DemTile& sh, Load&& load, Body&& body) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned todo = __ballot_sync(kAll, mine);
    while (todo) {
        const int ins = __shfl_sync(kAll, inst, __ffs(todo) - 1);
        const bool in = mine && inst == ins;
        todo &= ~__ballot_sync(kAll, in);
        const Win o = window(gd, px, py, pz, rq);
        Win w;
        w.x0 = __reduce_min_sync(kAll, in ? o.x0 : INT_MAX);
        w.x1 = __reduce_max_sync(kAll, in ? o.x1 : INT_MIN);
        w.y0 = __reduce_min_sync(kAll, in ? o.y0 : INT_MAX);
        w.y1 = __reduce_max_sync(kAll, in ? o.y1 : INT_MIN);
        w.z0 = __reduce_min_sync(kAll, in ? o.z0 : INT_MAX);
        w.z1 = __reduce_max_sync(kAll, in ? o.z1 : INT_MIN);
        warp_candidates(gd, w, ins, [&](int slot) {
            const int n = __popc(__ballot_sync(kAll, slot >= 0));  // the first n lanes have one
            if (slot >= 0) load(gd.order[slot], sh.p[lane], sh.q[lane], sh.r[lane]);
            __syncwarp();
            for (int i = 0; i < n; ++i) {
                const float4 p = sh.p[i];
                const D2 d = d2_exact(px, py, pz, p.x, p.y, p.z);
                if (in && d.d2 < p.w) body(i, d.d2);
            }
            __syncwarp();
        });
    }
}

}  // namespace sd
