// walk.cuh -- the neighbour walk of the SPH loops: a warp finds the members of
// its 32 / L subjects together, L lanes to a subject.
//
// A thread that walks its own cells tests ~380 candidates to find ~74 members
// (h = 1.3 dx), its loads wait on one another, and the warp pays for the
// member's arithmetic on nearly every candidate, because some lane takes it.
// Here the walk has three phases, all without divergence to speak of:
//   A  the candidates of all subjects of the warp (the subjects are neighbours
//      in cell order: ~550 candidates for 8 of them) are copied to shared
//      memory, and the lanes of each subject test them, every L-th word of 32
//      each: packed FP32 pairs, and one funnel shift that moves the sign of
//      d2 - t into the lane's mask;
//   B  the set bits become a list per subject, in slot order;
//   C  the lanes of a subject take the entries of its list in turn, so that
//      the member's arithmetic runs for 32 members at a time.
// Slot order is the order of the cell walk (columns x-major, z fastest), and
// the body sums the terms of a subject's L lanes in lane order (ordered_fma),
// so every sum has the same order and bits as one thread that walks the cells.
#pragma once

#include "common.cuh"

namespace sd {

constexpr int kWalkCap = 256;    // candidates per batch (a list entry is a byte)
constexpr int kWalkStride = 36;  // floats per word of 32: the words that L lanes read at once lie in other banks

template <int L>
struct WarpWalk {
    float x[kWalkCap / 32 * kWalkStride], y[kWalkCap / 32 * kWalkStride], z[kWalkCap / 32 * kWalkStride];
    float m[kWalkCap];
    int slot[kWalkCap];
    uint8_t list[32 / L][kWalkCap];
};

__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ unsigned long long f32x2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}

// d2 - t of two candidates (contracted operations), as the bits of two floats.
__device__ __forceinline__ void walk_d2(unsigned long long x, unsigned long long y, unsigned long long z,
                                        unsigned long long nx, unsigned long long ny, unsigned long long nz,
                                        unsigned long long nt, uint32_t& d0, uint32_t& d1) {
    asm("{\n\t.reg .b64 a, b, c, d;\n\t"
        "add.rn.ftz.f32x2 a, %2, %5;\n\t"
        "add.rn.ftz.f32x2 b, %3, %6;\n\t"
        "add.rn.ftz.f32x2 c, %4, %7;\n\t"
        "fma.rn.ftz.f32x2 d, a, a, %8;\n\t"
        "fma.rn.ftz.f32x2 d, b, b, d;\n\t"
        "fma.rn.ftz.f32x2 d, c, c, d;\n\t"
        "mov.b64 {%0, %1}, d;\n\t}"
        : "=r"(d0), "=r"(d1)
        : "l"(x), "l"(y), "l"(z), "l"(nx), "l"(ny), "l"(nz), "l"(nt));
}

// acc + a_0 b_0 + a_1 b_1 + ... over the L lanes of this lane's subject, one
// FMA after another in lane order; the same result in all of them.
template <int L>
__device__ __forceinline__ float ordered_fma(float acc, float a, float b) {
#pragma unroll
    for (int s = 0; s < L; ++s)
        acc = fmaf(L == 1 ? a : __shfl_sync(0xffffffffu, a, s, L), L == 1 ? b : __shfl_sync(0xffffffffu, b, s, L), acc);
    return acc;
}

// Calls body(ok, j, q, r), by all 32 lanes of the warp together, until every
// slot j of g with d2 < s2 has been given to one of the L lanes of its subject
// (ok; q = posm[j], r the exact difference), in slot order over the calls and,
// within a call, over the L lanes.  All lanes call warp_walk, the L lanes of a
// subject with the same arguments; mine = false where there is no subject.  rq
// is the padded query radius, w the warp's own shared memory.
//
// The subjects are taken column by column of g (mostly all of them lie in one,
// or in two that follow each other): the box of those in one column is small.
template <int L, class Body>
__device__ __forceinline__ void warp_walk(const Geo& g, const float4* __restrict__ posm, bool mine, float px, float py,
                                          float pz, float rq, float s2, int inst, WarpWalk<L>& w, Body&& body) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kRounds = kWalkCap / (32 * L);  // words per lane and batch
    const int lane = threadIdx.x & 31, sub = lane / L, sl = lane % L;
    const float t_hi = band_hi(s2);
    const unsigned long long nx = f32x2(-px, -px), ny = f32x2(-py, -py), nz = f32x2(-pz, -pz), nt = f32x2(-t_hi, -t_hi);
    const int column = (inst * g.dim[0] + coord(px, g.inv, g.lo[0], g.dim[0])) * g.dim[1] +
                       coord(py, g.inv, g.lo[1], g.dim[1]);
    unsigned todo = __ballot_sync(kAll, mine);
    while (todo) {
        const int lead = __ffs(todo) - 1;
        const int lead_column = __shfl_sync(kAll, column, lead);  // by all lanes, also those without a subject
        const bool in = mine && column == lead_column;
        todo &= ~__ballot_sync(kAll, in);
        const int ins = __shfl_sync(kAll, inst, lead);
        const float bx0 = warp_min(in ? px : INFINITY), bx1 = warp_max(in ? px : -INFINITY);
        const float by0 = warp_min(in ? py : INFINITY), by1 = warp_max(in ? py : -INFINITY);
        const float bz0 = warp_min(in ? pz : INFINITY), bz1 = warp_max(in ? pz : -INFINITY);
        // the window's columns: lanes 0-3 find x0, x1, y0, y1
        const bool ax = (lane & 2) == 0, hi = lane & 1;
        const float edge = ax ? (hi ? bx1 + rq : bx0 - rq) : (hi ? by1 + rq : by0 - rq);
        const int at = coord(edge, g.inv, ax ? g.lo[0] : g.lo[1], ax ? g.dim[0] : g.dim[1]);
        const int x0 = __shfl_sync(kAll, at, 0), x1 = __shfl_sync(kAll, at, 1);
        const int y0 = __shfl_sync(kAll, at, 2), y1 = __shfl_sync(kAll, at, 3);
        const int nyc = y1 - y0 + 1, ncols = x1 >= x0 && y1 >= y0 ? (x1 - x0 + 1) * nyc : 0;  // (NaN: none)
        const float per_y = __frcp_rn((float)nyc);
        int c0 = 0, s = 0, e = 0, cs = 0, ce = 0;
        unsigned some = 0u;  // columns of the current 32 whose slots are still to be copied
        bool done = false;
        while (!done) {
            int T = 0;
            while (T < kWalkCap) {
                if (cs < ce) {
                    const int take = min(ce - cs, kWalkCap - T);
                    for (int i = lane; i < take; i += 32) {
                        const float4 q = posm[cs + i];
                        const int u = T + i, v = u + (u >> 5) * (kWalkStride - 32);
                        w.x[v] = q.x;
                        w.y[v] = q.y;
                        w.z[v] = q.z;
                        w.m[u] = q.w;
                        w.slot[u] = cs + i;
                    }
                    T += take;
                    cs += take;
                } else if (some) {
                    const int src = __ffs(some) - 1;
                    some &= some - 1;
                    cs = __shfl_sync(kAll, s, src);
                    ce = __shfl_sync(kAll, e, src);
                } else if (c0 < ncols) {
                    // each lane trims one column to the ball around the box,
                    // as column_range_ball does around a point
                    s = e = 0;
                    const int c = c0 + lane;
                    if (c < ncols) {
                        const int dcx = (int)(((float)c + 0.5f) * per_y);  // c / nyc: exact, c < 2^20
                        const int cx = x0 + dcx, cy = y0 + (c - dcx * nyc);
                        const float margin = 0.01f * g.cell;
                        const float xa = cx == 0 ? -INFINITY : (float)(g.lo[0] + cx) * g.cell;
                        const float xb = cx == g.dim[0] - 1 ? INFINITY : (float)(g.lo[0] + cx + 1) * g.cell;
                        const float ya = cy == 0 ? -INFINITY : (float)(g.lo[1] + cy) * g.cell;
                        const float yb = cy == g.dim[1] - 1 ? INFINITY : (float)(g.lo[1] + cy + 1) * g.cell;
                        const float gx = fmaxf(0.0f, fmaxf(xa - bx1, bx0 - xb) - margin);
                        const float gy = fmaxf(0.0f, fmaxf(ya - by1, by0 - yb) - margin);
                        const float rem = rq * rq - gx * gx - gy * gy;
                        if (rem >= 0.0f) {
                            const float zr = fminf(rem * rsqrtf(fmaxf(rem, 1.0e-30f)) + margin, rq);
                            const int base = ins * g.ncl + (cx * g.dim[1] + cy) * g.dim[2];
                            s = __ldg(g.start + base + coord(bz0 - zr, g.inv, g.lo[2], g.dim[2]));
                            e = __ldg(g.start + base + coord(bz1 + zr, g.inv, g.lo[2], g.dim[2]) + 1);
                        }
                    }
                    some = __ballot_sync(kAll, e > s);
                    c0 += 32;
                } else {
                    done = true;
                    break;
                }
            }
            if (T == 0) break;
            __syncwarp();
            // A: this lane's words; t is padded (band_hi), phase C decides by
            // the exact predicate
            uint32_t m[kRounds];
#pragma unroll
            for (int r = 0; r < kRounds; ++r) {
                m[r] = 0u;
                if (32 * L * r < T) {
                    const int wd = L * r + sl;
                    const float* xs = w.x + wd * kWalkStride;
                    const float* ys = w.y + wd * kWalkStride;
                    const float* zs = w.z + wd * kWalkStride;
                    uint32_t bits = 0u;
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(xs + i);
                        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(ys + i);
                        const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(zs + i);
                        uint32_t d0, d1, d2, d3;
                        walk_d2(x.x, y.x, z.x, nx, ny, nz, nt, d0, d1);
                        walk_d2(x.y, y.y, z.y, nx, ny, nz, nt, d2, d3);
                        bits = __funnelshift_l(d0, bits, 1);
                        bits = __funnelshift_l(d1, bits, 1);
                        bits = __funnelshift_l(d2, bits, 1);
                        bits = __funnelshift_l(d3, bits, 1);
                    }
                    const int left = T - 32 * wd;  // bit 31 - i: candidate 32 wd + i; none past the end
                    m[r] = !in || left <= 0 ? 0u : (left < 32 ? bits & (0xffffffffu << (32 - left)) : bits);
                }
            }
            // B: the subject's list
            int count = 0;
#pragma unroll
            for (int r = 0; r < kRounds; ++r) {
                if (32 * L * r < T) {
                    const int c = __popc(m[r]);
                    int pos = c;
#pragma unroll
                    for (int o = 1; o < L; o <<= 1) {
                        const int v = __shfl_up_sync(kAll, pos, o, L);
                        if (sl >= o) pos += v;
                    }
                    const int all = L == 1 ? pos : __shfl_sync(kAll, pos, L - 1, L);
                    pos += count - c;
                    count += all;
                    const int trips = __reduce_max_sync(kAll, c);
                    uint32_t b = m[r];
                    uint8_t* to = &w.list[sub][pos];
                    const int first = 32 * (L * r + sl);
                    for (int t = 0; t < trips; ++t)
                        if (b) {
                            const int i = __clz(b);
                            b ^= 0x80000000u >> i;
                            *to++ = (uint8_t)(first + i);
                        }
                }
            }
            __syncwarp();
            // C: the members, L of each subject at a time
            const int trips = __reduce_max_sync(kAll, count);
            for (int t = 0; t < trips; t += L) {
                const bool has = t + sl < count;
                const int u = has ? w.list[sub][t + sl] : 0, v = u + (u >> 5) * (kWalkStride - 32);
                const int j = w.slot[u];
                const float4 q = make_float4(w.x[v], w.y[v], w.z[v], w.m[u]);
                const D2 r = d2_exact(px, py, pz, q.x, q.y, q.z);
                body(has && r.d2 < s2, j, q, r);
            }
            __syncwarp();
        }
    }
}

}  // namespace sd
