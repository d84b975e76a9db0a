// grid.cu -- neighbour grid build: counting sort of points by cell.
//
// Replaces wp.HashGrid.build (main.py:66,73,85,87).  Steps, all on one stream
// (small grids: all in one CTA, k_build_one):
//   1. bin      key[i] = cell of point i, count[key]++            (atomics)
//   2. scan     exclusive prefix sum of the counts -> cell_start, and a copy
//               of it -> cursor (per-span sums, then one scan kernel)
//   3. scatter  order[cursor[key]++] = i                          (atomics)
//   4. sort     each cell's slots by point index, so the order is stable and
//               every later sum is deterministic run to run; for the fluid
//               the same kernel writes the sorted copies of the fields that
//               the neighbour loops read
// Memory: cell_start [ncell+1], order/key [n], cursor [ncell] and scan scratch
// are caller-owned tensors; nothing is allocated here.
#include <limits.h>
#include <stdio.h>
#include <string.h>

#include "common.cuh"

namespace sd {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048 cells per tile
constexpr int kScanSpans = 1024;                      // at most this many CTAs, each a span of whole tiles
constexpr int kScanScratchTile = 1024;                // the scratch holds a word per 1024 cells (>= one per span)

__global__ void k_bin(const float* __restrict__ pos, int n, const int* __restrict__ inst, int lo0, int lo1,
                      int lo2, int d0, int d1, int d2, float inv, int ncl, int* __restrict__ key,
                      int* __restrict__ count, sphdem_ctl_t* ctl) {
    pdl_wait();
    pdl_launch();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    if (!isfinite(x) || !isfinite(y) || !isfinite(z)) flag(ctl, SPHDEM_FLAG_NONFINITE);
    int cx = coord(x, inv, lo0, d0), cy = coord(y, inv, lo1, d1), cz = coord(z, inv, lo2, d2);
    int k = (inst ? inst[i] : 0) * ncl + (cx * d1 + cy) * d2 + cz;
    key[i] = k;
    atomicAdd(count + k, 1);
}

// Exclusive scan in two launches: every CTA sums its span of tiles, then every
// CTA adds up the sums of the spans before its own (at most 1023 words, read
// from L2 by all threads) and scans its span.  A look-back chain would save
// the first launch and need a spin wait; a one-CTA scan of the sums between
// the two (the earlier form) is a third launch that one CTA runs alone.
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const int* __restrict__ data, int n, int span,
                                                            int* __restrict__ sums) {
    pdl_wait();
    pdl_launch();
    __shared__ int warp_tot[kScanThreads / 32];
    const int c0 = blockIdx.x * span, c1 = min(n, c0 + span);
    int s = 0;
    for (int c = c0 + threadIdx.x; c < c1; c += kScanThreads) s += data[c];
    int total;
    block_exclusive_scan(s, warp_tot, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// data[0..n) scanned in place, data[n] = the total; copy (optional) receives
// data[0..n) too (the cursors of the scatter).
__global__ void __launch_bounds__(kScanThreads) k_scan_write(int* __restrict__ data, int n, int span,
                                                             const int* __restrict__ sums, int* __restrict__ copy) {
    pdl_wait();
    pdl_launch();
    __shared__ int warp_tot[kScanThreads / 32];
    // the threads stride over a tile to load it and each scan kScanItems
    // consecutive cells of it; one pad word per 8 keeps both free of conflicts
    __shared__ int tile[kScanTile + kScanTile / kScanItems];
    int before = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += kScanThreads) before += sums[b];
    int carry;
    block_exclusive_scan(before, warp_tot, carry);
    const int c0 = blockIdx.x * span, c1 = min(n, c0 + span);
    for (int base = c0; base < c1; base += kScanTile) {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            const int i = k * kScanThreads + threadIdx.x;
            tile[i + i / kScanItems] = base + i < c1 ? data[base + i] : 0;
        }
        __syncthreads();
        int v[kScanItems], s = 0;
        const int t0 = threadIdx.x * (kScanItems + 1);
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = tile[t0 + k];
            s += v[k];
        }
        int total;
        int run = carry + block_exclusive_scan(s, warp_tot, total);
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            tile[t0 + k] = run;
            run += v[k];
        }
        carry += total;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            const int i = k * kScanThreads + threadIdx.x;
            if (base + i < c1) {
                const int w = tile[i + i / kScanItems];
                data[base + i] = w;
                if (copy) copy[base + i] = w;
            }
        }
        __syncthreads();
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) data[n] = carry;
}

__global__ void k_scatter(const int* __restrict__ key, int n, int* __restrict__ cursor, int* __restrict__ order) {
    pdl_wait();
    pdl_launch();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    order[atomicAdd(cursor + key[i], 1)] = i;
}

// Sorted copies of the fluid fields that the neighbour loops read.
struct FluidCopy {
    const float* __restrict__ pos;
    const float* __restrict__ m;
    const float* __restrict__ vel;
    const float* __restrict__ rho;
    float4* __restrict__ posm;
    float4* __restrict__ velo;
    float* __restrict__ vprev;
    __device__ __forceinline__ void operator()(int k, int o) const {
        const float mo = m[o];
        posm[k] = make_float4(pos[3 * o], pos[3 * o + 1], pos[3 * o + 2], mo);
        velo[k] = make_float4(vel[3 * o], vel[3 * o + 1], vel[3 * o + 2], 0.0f);
        vprev[k] = mo / rho[o];
    }
};

// Sorts v[0..len) ascending in place, all threads of the CTA (blockDim.x
// compare-exchanges at a time): the bitonic network whose merges start with a
// reversed step, so that a length that is no power of two needs no padding.
__device__ __forceinline__ void block_sort(int* v, int len) {
    for (int size = 2; size < 2 * len; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const bool flip = stride == size >> 1;
            for (int t = threadIdx.x; t < (len + 1) / 2 + stride; t += blockDim.x) {
                const int off = t & (stride - 1), base = (t - off) * 2;
                const int a = base + off, b = flip ? base + 2 * stride - 1 - off : a + stride;
                if (b < len) {
                    const int x = v[a], y = v[b];
                    if (x > y) {
                        v[a] = y;
                        v[b] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// Stable order inside each cell: the slots of a cell sorted by point index.
// A CTA owns the cells that start in its window of 256 slots (so work is
// balanced by points, not by cells: most cells of a tank are empty).  It
// loads their slots into shared memory; each thread finds the rank of its
// points among those of their cell (17 points in a fluid cell) and writes
// them, and with COPY the point's sorted copies, at their place.  A cell that
// reaches more than 768 slots past the window is sorted by the whole CTA.
// A warp that sorts one cell after another in registers (an insertion sort by
// one lane beyond 32 points), with a separate copy kernel after it, took 20 +
// 4 us at 100k points and 32 + 12 at 792k; this one takes 8.7 and 21 us.
constexpr int kSortThreads = 256;
constexpr int kSortCap = 1024;   // slots ranked together
constexpr int kSortLong = 4096;  // points of a long cell sorted in shared memory (else in place)

template <bool COPY>
__global__ void __launch_bounds__(kSortThreads) k_sort_slots(const int* __restrict__ start, const int* __restrict__ key,
                                                             int n, int* __restrict__ order, FluidCopy copy) {
    pdl_wait();
    pdl_launch();
    __shared__ int v[kSortLong];
    __shared__ int range[2];
    if (threadIdx.x < 2) {
        // first slot, from this window edge on, that starts a cell.  A
        // neighbour may be permuting the cell of this slot: any point of it
        // names the same cell.
        const int b = min(n, (int)(blockIdx.x + threadIdx.x) * kSortThreads);
        int r = n;
        if (b < n) {
            const int k = key[*(volatile int*)(order + b)];
            r = start[k];
            if (r != b) r = start[k + 1];
        }
        range[threadIdx.x] = r;
    }
    __syncthreads();
    const int lo = range[0];
    int hi = range[1];
    if (hi - lo > kSortCap) {  // the last cell is a long one
        const int k = key[order[hi - 1]];
        __syncthreads();
        const int s = start[k], len = hi - s;
        int* w = order + s;
        if (len <= kSortLong) {
            for (int t = threadIdx.x; t < len; t += kSortThreads) v[t] = w[t];
            __syncthreads();
            block_sort(v, len);
            for (int t = threadIdx.x; t < len; t += kSortThreads) w[t] = v[t];
        } else {
            block_sort(w, len);
        }
        __syncthreads();
        if (COPY)
            for (int t = threadIdx.x; t < len; t += kSortThreads) copy(s + t, w[t]);
        __syncthreads();
        hi = s;
    }
    for (int t = threadIdx.x; t < hi - lo; t += kSortThreads) v[t] = order[lo + t];
    __syncthreads();
    for (int t = threadIdx.x; t < hi - lo; t += kSortThreads) {
        const int o = v[t], k = key[o];
        const int s = start[k], e = start[k + 1];
        int r = s;
        for (int j = s - lo; j < e - lo; ++j) r += v[j] < o;
        order[r] = o;
        if (COPY) copy(r, o);
    }
}

// The whole build in one CTA, for small grids (at most kOneMaxPoints points
// and kOneMaxCells cells): the same bin, exclusive scan, scatter and per-cell
// sort as the multi-kernel path, phase after phase behind __syncthreads, so
// the cell starts and the order are the same; one launch instead of six
// (small systems are bound by launch latency, not by these loops).
constexpr int kOneThreads = 1024;
constexpr int kOneMaxPoints = 4096;
constexpr int kOneMaxCells = 65536;
constexpr int kOneItems = 4;     // consecutive cells a thread scans per tile
constexpr int kOneRankMax = 64;  // longest cell that is sorted by ranks

__global__ void __launch_bounds__(kOneThreads) k_build_one(const float* __restrict__ pos, int n,
                                                          const int* __restrict__ inst, int lo0, int lo1, int lo2,
                                                          int d0, int d1, int d2, float inv, int ncl, int ncell,
                                                          int* __restrict__ key, int* __restrict__ start,
                                                          int* __restrict__ cursor, int* __restrict__ order,
                                                          sphdem_ctl_t* ctl) {
    pdl_wait();
    pdl_launch();
    __shared__ int warp_tot[kOneThreads / 32];
    __shared__ int v[kOneMaxPoints];
    const int tid = threadIdx.x;
    for (int c = tid; c <= ncell; c += kOneThreads) start[c] = 0;
    __syncthreads();
    for (int i = tid; i < n; i += kOneThreads) {
        const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
        if (!isfinite(x) || !isfinite(y) || !isfinite(z)) flag(ctl, SPHDEM_FLAG_NONFINITE);
        const int cx = coord(x, inv, lo0, d0), cy = coord(y, inv, lo1, d1), cz = coord(z, inv, lo2, d2);
        const int k = (inst ? inst[i] : 0) * ncl + (cx * d1 + cy) * d2 + cz;
        key[i] = k;
        atomicAdd(start + k, 1);
    }
    __syncthreads();
    // exclusive scan, tile after tile of neighbouring cells (a contiguous
    // chunk of all cells per thread strides the loads by the chunk: 25 us for
    // the whole build of 2,000 spheres in the large tank against 12)
    int carry = 0, longest = 0;
    for (int base = 0; base < ncell; base += kOneThreads * kOneItems) {
        const int c0 = base + tid * kOneItems;
        int w[kOneItems], sum = 0;
#pragma unroll
        for (int u = 0; u < kOneItems; ++u) {
            w[u] = c0 + u < ncell ? start[c0 + u] : 0;
            sum += w[u];
            longest = max(longest, w[u]);
        }
        int total;
        int run = carry + block_exclusive_scan(sum, warp_tot, total);
#pragma unroll
        for (int u = 0; u < kOneItems; ++u) {
            if (c0 + u < ncell) start[c0 + u] = cursor[c0 + u] = run;
            run += w[u];
        }
        carry += total;
    }
    if (tid == 0) start[ncell] = n;
    if (__syncthreads_or(longest > kOneRankMax)) {
        // a crowded grid: all points by (cell, index) at once, packed in 28
        // bits (2,000 spheres in a few cells: 22 us; 35 ms as an insertion
        // sort by one lane per cell)
        for (int i = tid; i < n; i += kOneThreads) v[i] = key[i] * kOneMaxPoints + i;
        __syncthreads();
        block_sort(v, n);
        for (int k = tid; k < n; k += kOneThreads) order[k] = v[k] & (kOneMaxPoints - 1);
        return;
    }
    for (int i = tid; i < n; i += kOneThreads) v[atomicAdd(cursor + key[i], 1)] = i;
    __syncthreads();
    for (int t = tid; t < n; t += kOneThreads) {
        const int o = v[t], k = key[o];
        const int s = start[k], e = start[k + 1];
        int r = s;
        for (int j = s; j < e; ++j) r += v[j] < o;
        order[r] = o;
    }
}

__global__ void k_gather_fluid(const int* __restrict__ order, int n, FluidCopy copy) {
    pdl_wait();
    pdl_launch();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) copy(k, order[k]);
}

__global__ void k_gather_vol(const int* __restrict__ order, int n, const float* __restrict__ m,
                             const float* __restrict__ rho, float* __restrict__ out) {
    pdl_wait();
    pdl_launch();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) {
        int o = order[k];
        out[k] = m[o] / rho[o];
    }
}

// Wall-only part of the wall density, sum_{wall j, d2 < s^2} m_j W(r, h)
// (the second loop of Kernel_density_bnd, kernel/KERNEL_rho.py:119-125).  Walls
// never move, so this sum is a constant of the wall grid and is cached here.
__global__ void k_wall_self(Geo gb, const float4* __restrict__ posm, int n, float s2, float rq, Kern kern,
                            float* __restrict__ self) {
    pdl_wait();
    pdl_launch();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float4 p = posm[k];
    int inst = inst_of(gb, gb.order[k]);
    float acc = 0.0f;
    for_each_range_ball(gb, p.x, p.y, p.z, rq, inst, [&](int s, int e) {
        for (int j = s; j < e; ++j) {
            float4 q = posm[j];
            D2 r = d2_exact(p.x, p.y, p.z, q.x, q.y, q.z);
            if (r.d2 < s2) acc += q.w * kern_w(kern, fast_sqrt(r.d2));
        }
    });
    self[k] = acc;
}

FluidCopy fluid_copy(const sphdem_ctx_t* c) {
    return {c->sph.pos,  c->sph.m, c->sph.vel, c->sph.rho, (float4*)c->work.f_posm, (float4*)c->work.f_vel,
            c->work.f_vprev};
}

// Exclusive scan of n counts in place, data[n] = their total; copy: see k_scan_write.
int scan_launch(int* data, int n, int* sums, int* copy, cudaStream_t st) {
    const int tiles = n > 0 ? (n + kScanTile - 1) / kScanTile : 1;
    const int span = (tiles + kScanSpans - 1) / kScanSpans * kScanTile;
    const int nb = n > 0 ? (n + span - 1) / span : 1;
    launch_pdl(k_scan_sums, nb, kScanThreads, 0, st, data, n, span, sums);
    launch_pdl(k_scan_write, nb, kScanThreads, 0, st, data, n, span, sums, copy);
    return launch_status("scan");
}

// Bin + scan + scatter + stable per-cell sort of the points of one grid; with
// copy, the fluid's sorted copies too.
int build(sphdem_grid_t* g, const float* pos, sphdem_ctl_t* ctl, const FluidCopy* copy, cudaStream_t st) {
    const int ncell = g->ninst * g->ncell_local;
    if (ncell <= 0 || g->n < 0) {
        set_error_msg("grid: empty cell box");
        return SPHDEM_ERR_INVALID;
    }
    const int n = g->n;
    if (n <= kOneMaxPoints && ncell <= kOneMaxCells) {
        launch_pdl(k_build_one, 1, kOneThreads, 0, st, pos, n, g->inst, g->lo[0], g->lo[1], g->lo[2], g->dim[0], g->dim[1],
                                               g->dim[2], g->inv_cell, g->ncell_local, ncell, g->key, g->cell_start,
                                               g->cursor, g->order, ctl);
        if (copy && n > 0) launch_pdl(k_gather_fluid, blocks_for(n, 256), 256, 0, st, g->order, n, *copy);
        return launch_status("build_grid");
    }
    cudaError_t e = zero_words(g->cell_start, (long)ncell, st);
    if (e != cudaSuccess) {
        set_error("grid memset", e);
        return SPHDEM_ERR_CUDA;
    }
    if (n > 0)
        launch_pdl(k_bin, blocks_for(n, 256), 256, 0, st, pos, n, g->inst, g->lo[0], g->lo[1], g->lo[2], g->dim[0],
                                                  g->dim[1], g->dim[2], g->inv_cell, g->ncell_local, g->key,
                                                  g->cell_start, ctl);
    const int rc = scan_launch(g->cell_start, ncell, g->block_sums, g->cursor, st);
    if (rc) return rc;
    if (n > 0) {
        launch_pdl(k_scatter, blocks_for(n, 256), 256, 0, st, g->key, n, g->cursor, g->order);
        if (copy)
            launch_pdl(k_sort_slots<true>, blocks_for(n, kSortThreads), kSortThreads, 0, st, g->cell_start, g->key, n,
                       g->order, *copy);
        else
            launch_pdl(k_sort_slots<false>, blocks_for(n, kSortThreads), kSortThreads, 0, st, g->cell_start, g->key, n,
                       g->order, FluidCopy{});
    }
    return launch_status("build_grid");
}

}  // namespace

// Exclusive scan of n counts in place, data[n] = their total (device side).
int scan_counts(int* data, int n, int* sums, cudaStream_t st) { return scan_launch(data, n, sums, nullptr, st); }

int build_grid(sphdem_grid_t* g, const float* pos, sphdem_ctl_t* ctl, cudaStream_t st) {
    return build(g, pos, ctl, nullptr, st);
}

// The fluid grid and the fluid's sorted copies.
int build_fluid(sphdem_ctx_t* c, cudaStream_t st) {
    const FluidCopy copy = fluid_copy(c);
    return build(&c->grid_sph, c->sph.pos, c->ctl, &copy, st);
}

int gather_fluid(const sphdem_ctx_t* c, cudaStream_t st) {
    const int n = c->sph.n;
    if (n <= 0) return SPHDEM_OK;
    launch_pdl(k_gather_fluid, blocks_for(n, 256), 256, 0, st, c->grid_sph.order, n, fluid_copy(c));
    return launch_status("gather_fluid");
}

int gather_wall(const sphdem_ctx_t* c, float support, float h, cudaStream_t st) {
    const int n = c->bnd.n;
    if (n <= 0) return SPHDEM_OK;
    // Same gather as the fluid (x, y, z, m), then the wall self density.
    const FluidCopy copy{c->bnd.pos, c->bnd.m, c->bnd.vel, c->bnd.rho, (float4*)c->work.b_posm,
                         (float4*)c->work.b_vel, c->work.b_vprev};
    launch_pdl(k_gather_fluid, blocks_for(n, 256), 256, 0, st, c->grid_bnd.order, n, copy);
    Geo gb = make_geo(c->grid_bnd);
    launch_pdl(k_wall_self, blocks_for(n, 128), 128, 0, st, gb, (const float4*)c->work.b_posm, n, support * support,
                                                    pad_radius(support), make_kern(h), c->work.b_self);
    return launch_status("gather_wall");
}

int gather_wall_rho(const sphdem_ctx_t* c, cudaStream_t st) {
    const int n = c->bnd.n;
    if (n <= 0) return SPHDEM_OK;
    launch_pdl(k_gather_vol, blocks_for(n, 256), 256, 0, st, c->grid_bnd.order, n, c->bnd.m, c->bnd.rho, c->work.b_vprev);
    return launch_status("gather_wall_rho");
}

int64_t scan_scratch_words(int64_t ncell) { return (ncell + kScanScratchTile - 1) / kScanScratchTile + 2; }

}  // namespace sd

extern "C" int64_t sphdem_scan_scratch(int64_t ncell) { return sd::scan_scratch_words(ncell); }
