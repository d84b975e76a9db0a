// demwalk.cuh -- the spheres around the fluid particles of a warp.
//
// A fluid particle near the spheres has up to ~160 of them in its window of 27
// coupling cells; a thread that walks them alone waits for four loads in a
// chain per sphere (slot -> index -> position -> constants).  Here the lanes
// of a warp, whose particles are neighbours in cell order and so have nearly
// the same window, load 32 spheres at once into shared memory, and every lane
// tests all of them.  A lane meets its spheres in slot order, as on its own, and
// of those in reach takes the ones whose cell lies in its own window: with a
// query radius below a sphere's reach the window decides (the warp's union must
// not, or a result would depend on the particles that share the warp).
#pragma once

#include <limits.h>

#include "common.cuh"

namespace sd {

struct DemTile {
    float4 p[32];  // x, y, z, bound of d2 (below it: in reach)
    float4 q[32], r[32];
    int4 cell[32];  // cell coordinates, where some sphere's reach is beyond the query radius
};

__device__ __forceinline__ bool in_window(const Win& w, const int4& c) {
    return c.x >= w.x0 && c.x <= w.x1 && c.y >= w.y0 && c.y <= w.y1 && c.z >= w.z0 && c.z <= w.z1;
}

// load(b, p, q, r): fields of sphere b (p.w the bound on d2; a negative one
// keeps the sphere out).  body(i, d2): sphere i of the tile is in reach of this
// lane's particle.  All lanes of the warp call it; mine = false: no particle.
template <class Load, class Body>
__device__ __forceinline__ void warp_dem_visit(const Geo& gd, bool mine, float px, float py, float pz, float rq,
                                               int inst, DemTile& sh, Load&& load, Body&& body) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // reach (squared) up to which a sphere lies in the window of every particle
    // that it reaches: the query radius before its padding
    const float radius = (rq - 1.0e-6f) * (1.0f / 1.001f), within = radius * radius * 1.0001f;
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
            const bool wide = __any_sync(kAll, slot >= 0 && sh.p[lane].w > within);
            if (wide && slot >= 0) {
                const int c = __ldg(gd.key + gd.order[slot]) - ins * gd.ncl, column = c / gd.dim[2];
                sh.cell[lane] = make_int4(column / gd.dim[1], column % gd.dim[1], c % gd.dim[2], 0);
            }
            __syncwarp();
            if (!wide) {
                for (int i = 0; i < n; ++i) {
                    const float4 p = sh.p[i];
                    const D2 d = d2_exact(px, py, pz, p.x, p.y, p.z);
                    if (in && d.d2 < p.w) body(i, d.d2);
                }
            } else {
                const Win own = window(gd, px, py, pz, rq);
                for (int i = 0; i < n; ++i) {
                    const float4 p = sh.p[i];
                    const D2 d = d2_exact(px, py, pz, p.x, p.y, p.z);
                    if (in && d.d2 < p.w && in_window(own, sh.cell[i])) body(i, d.d2);
                }
            }
            __syncwarp();
        });
    }
}

}  // namespace sd
