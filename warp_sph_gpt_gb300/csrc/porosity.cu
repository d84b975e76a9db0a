// porosity.cu -- the porosity pass of Kernel_prep_sphdem
// (kernel/KERNEL_SPHDEM_interaction.py:43-95) for a uniform DEM coupling
// length h, with the fluid normaliser's pair distances on the tensor cores.
//
// The normaliser of a fluid particle i near a sphere is
//     flt_i = 21/(16 pi h^3) sum_j V_j w(|x_i - x_j|^2 / h^2),
//     w(s) = (1 - q/2)^4 (1 + 2q),  q = sqrt(s), s clamped to 4,
// over every fluid j (w vanishes from q = 2 on, so candidates beyond the
// coupling support add exact zeros and no membership test is needed).  At
// the large dam break a listed particle has ~54k neighbours, so the pass is
// ~4.5e9 pair evaluations per step.  Here the squared distances of a tile of
// 128 subjects against a chunk of 128 candidates come from one tcgen05 MMA:
//     s_ij = |p_i|^2 + |q_j|^2 - 2 p_i . q_j
// with p, q in units of h relative to a common centre, every FP32 operand
// split exactly into three BF16 pieces (a = a0 + a1 + a2) and all products of
// p . q but p2 q2 (below 2^-32 of |p| |q|), plus the pieces of |p|^2 and |q|^2
// times ones, laid along K = 32: the FP32 accumulation of exact BF16 products
// gives s to ~1e-6 of the ball radius squared.  The CUDA cores then evaluate only
// w(s) (one MUFU square root, the polynomial on packed FP32 pairs) and the
// V_j-weighted sums.
//
// Every subject's sum is canonical -- the same bits whatever the tiling, the
// launch shape or the other members of a batched state:
//   * the centre of a tile is the centre of a world-anchored frame block of
//     F x F x F fluid-grid cells, and a tile holds listed particles of one
//     frame block only, so p_i and q_j depend only on (i, j);
//   * candidate ranges are padded to slot offsets aligned to 8 within their
//     instance (padding carries V = 0), so candidate j always lands in
//     accumulator (slot - instance start) mod 8 of the eight per subject: the
//     two epilogue warps of a TMEM lane quarter own classes 0-3 and 4-7
//     (staging puts them in chunk columns 0-63 and 64-127);
//   * the window is cut into world-anchored column slabs of Wx columns; each
//     (tile, slab) work unit writes a partial sum per subject, and the finish
//     kernel adds a subject's slab partials in slab order.
// Candidates outside a subject's own ball add +0 exactly, so the extra
// candidates of a tile's wider window change nothing.
//
// Kernels (one porosity pass):
//   k_pnear      a warp per 32 fluid slots: a DEM within 2 h_b?  Dry particles
//                get clamp(1); listed ones are counted per frame block, and a
//                frame block's first listed particle puts it on a list.
//   k_plist      one warp per listed frame block: reserves its segment of the
//                near list and of the tile table (atomics: segment placement
//                varies, results do not), writes its listed slots along
//                pencils of 2 x 2 cells (so a tile of 128 is compact) and its
//                tiles.
//   k_porosity_mma  persistent, 2 CTAs per SM: work units (tile, slab);
//                warps 0-7 epilogue (TMEM lane = subject; warp w reads lane
//                quarter w mod 4, chunk half w / 4), warps 8-11 stage
//                candidate rows (each thread loads its next chunk's candidate
//                while it builds the current chunk's row); warp 8 also issues
//                the MMAs and owns tensor memory.
//   k_pfinish    a warp per 32 listed particles: slab partials -> flt, solid
//                fraction over the DEM neighbours, porosity.
// Every wait is bounded; a timeout raises SPHDEM_FLAG_TIMEOUT, the CTA drains
// its MMAs (bounded) and frees its tensor memory.
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"
#include "demwalk.cuh"
#include "umma.cuh"

namespace sd {

namespace {

constexpr int kPM = 128;            // subjects per tile (MMA M, TMEM lanes)
constexpr int kPN = 128;            // candidates per chunk (MMA N, TMEM columns)
constexpr int kPK = 32;             // BF16 K of the distance MMA (30 used)
constexpr int kPStages = 6;         // candidate-row stages in shared memory
constexpr int kPSlabs = SPHDEM_POROSITY_SLABS;
constexpr int kPMaxRanges = 512;    // candidate ranges per column batch
constexpr int kPMaxChunks = 2048;   // chunks per column batch with a precomputed first range
constexpr int kPEpiWarps = 8;       // two per TMEM lane quarter, one per half of each chunk
constexpr int kPStageWarps = 4;     // one thread per candidate of a chunk; the first also issues the MMAs
constexpr int kPMmaWarp = kPEpiWarps;
constexpr int kPThreads = 32 * (kPEpiWarps + kPStageWarps);  // 384
constexpr int kPAlign = 8;          // candidate class = slot offset in the instance mod 8
constexpr uint32_t kPRowBytes = kPK * 2;
constexpr uint32_t kPTileBytes = kPM * kPRowBytes;  // = kPN * kPRowBytes
constexpr uint32_t kPTmemCols = 2 * kPN;            // two accumulator buffers
constexpr int kPPolls = 1 << 20;

struct PorSmem {
    uint8_t A[kPTileBytes];               // subjects (1024-aligned)
    uint8_t B[kPStages][kPTileBytes];     // candidate rows
    float V[kPStages][kPN];               // candidate volumes (0: padding)
    int rs[kPMaxRanges];                  // aligned first slot of each range
    int info[kPMaxRanges];                // leading pad | (true length << 3)
    int pre[kPMaxRanges + 1];             // exclusive prefix of aligned lengths
    int cr[kPMaxChunks + 1];              // range holding each chunk's first candidate
    uint64_t full[kPStages], empty[kPStages], afull[2], aempty[2], drain;
    float red[6][4];
    float hsum[kPM];                      // second-half sums of each subject
    int wtot[kPThreads / 32];
    int unit, abort_flag;
    int tstart, tcount, slab;             // the current work unit's tile and slab
    uint32_t tmem;
};
// Dynamic shared memory per CTA: the struct, its 1024-byte alignment, and a
// floor that keeps at most two CTAs (2 x 256 TMEM columns) on an SM.
constexpr uint32_t kPSmemBytes = (sizeof(PorSmem) + 1024 > 80u * 1024u) ? (uint32_t)sizeof(PorSmem) + 1024u
                                                                         : 80u * 1024u;

struct PorArgs {
    Geo gs, gd;
    const float4* __restrict__ f_posm;  // x, y, z, m (fluid, grid order; the near flags read these)
    const float4* __restrict__ f_posv;  // x, y, z, m/rho (fluid, grid order)
    const float4* __restrict__ aux;     // per DEM: 1/h, cw, sqrt bound of 2h, 2h
    sphdem_sph_t P;
    sphdem_dem_t D;
    int* near_list;
    int* flag;      // [n_sph] near flag per slot
    int* cnt;       // [nfb] listed particles per frame block
    int* fbl;       // [nfb] frame blocks with listed particles
    int4* tiles;    // (near start, count, frame block, 0)
    float* part;    // [n_sph * kPSlabs]
    sphdem_ctl_t* ctl;
    float rq;       // padded coupling support (2 h, world units)
    float inv_h, cw, eps_min, eps_max;
    int F;          // frame-block edge in cells
    int f0[3], nf[3], nfb_local, nfb;
    int Wx;         // slab width in columns
};

__device__ __forceinline__ int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

__device__ __forceinline__ float sqrt_apx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Exact three-piece BF16 split of an FP32 value, a = a0 + a1 + a2, by truncation
// (8 of its 24 significant bits each): the bits of a piece are a float's upper
// half, so a pair of them is one byte permute.  (Pieces rounded by conversion
// instructions, two per piece and one per pair, made a row twice as long and
// kept the unit busy that the square roots need: with two staging warps and
// those, 3.00 ms at 800k and 0.99 at 100k with submerged spheres; with four
// staging warps and this, 2.71 and 0.90.)
__device__ __forceinline__ void split3(float a, uint32_t* t) {
    t[0] = __float_as_uint(a) & 0xffff0000u;
    const float r1 = a - __uint_as_float(t[0]);
    t[1] = __float_as_uint(r1) & 0xffff0000u;
    t[2] = __float_as_uint(r1 - __uint_as_float(t[1]));
}

// BF16 pair (lo, hi) of two pieces.
__device__ __forceinline__ uint32_t pk(uint32_t lo, uint32_t hi) { return __byte_perm(lo, hi, 0x7632); }

// One 64-byte operand row (32 BF16 along K) at row r of a K-major tile, from
// the pieces of x, y, z and of the square n.  K holds per coordinate the
// products a0b0, a0b1, a1b0, a0b2, a1b1, a2b0, a1b2, a2b1, with n against ones
// on either side; SUBJECT: the a (and n before ones), else the b.
template <bool SUBJECT>
__device__ __forceinline__ void store_row(uint8_t* tile, int r, const uint32_t (*x)[3], const uint32_t* n) {
    constexpr int i1 = SUBJECT ? 0 : 1, i2 = SUBJECT ? 1 : 0, i3 = SUBJECT ? 0 : 2, i5 = SUBJECT ? 2 : 0;
    constexpr uint32_t kOne = 0x3f800000u;
    const uint32_t m0 = SUBJECT ? n[0] : kOne, m1 = SUBJECT ? n[1] : kOne, m2 = SUBJECT ? n[2] : kOne;
    const uint32_t l0 = SUBJECT ? kOne : n[0], l1 = SUBJECT ? kOne : n[1], l2 = SUBJECT ? kOne : n[2];
    auto put = [&](int k, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
        *reinterpret_cast<uint4*>(tile + umma::tile_off(r, k, kPK)) = make_uint4(a, b, c, d);
    };
    // (x y z) of a0b0, a0b1, a1b0, a0b2, a1b1, a2b0, then n, then a1b2, a2b1
    put(0, pk(x[0][0], x[1][0]), pk(x[2][0], x[0][i1]), pk(x[1][i1], x[2][i1]), pk(x[0][i2], x[1][i2]));
    put(8, pk(x[2][i2], x[0][i3]), pk(x[1][i3], x[2][i3]), pk(x[0][1], x[1][1]), pk(x[2][1], x[0][i5]));
    put(16, pk(x[1][i5], x[2][i5]), pk(m0, m1), pk(m2, l0), pk(l1, l2));
    constexpr int i6 = SUBJECT ? 1 : 2, i7 = SUBJECT ? 2 : 1;
    put(24, pk(x[0][i6], x[1][i6]), pk(x[2][i6], x[0][i7]), pk(x[1][i7], x[2][i7]), 0u);
}

// Subject row: p pieces, |p|^2 pieces against ones, ones against |q|^2 pieces;
// candidate row: -2 q pieces, ones, |q|^2 pieces.
template <bool SUBJECT>
__device__ __forceinline__ void make_row(uint8_t* tile, int r, float px, float py, float pz) {
    uint32_t x[3][3], n[3];
    const float f = SUBJECT ? 1.0f : -2.0f;
    split3(f * px, x[0]);
    split3(f * py, x[1]);
    split3(f * pz, x[2]);
    split3(fmaf(pz, pz, fmaf(py, py, px * px)), n);
    store_row<SUBJECT>(tile, r, x, n);
}

// Frame block of local cell (cx, cy, cz) of instance inst.
__device__ __forceinline__ int frame_of(const PorArgs& a, int inst, int cx, int cy, int cz) {
    const int fx = floor_div(a.gs.lo[0] + cx, a.F) - a.f0[0];
    const int fy = floor_div(a.gs.lo[1] + cy, a.F) - a.f0[1];
    const int fz = floor_div(a.gs.lo[2] + cz, a.F) - a.f0[2];
    return inst * a.nfb_local + (fx * a.nf[1] + fy) * a.nf[2] + fz;
}

// Local cell range [c0, c1] of frame block coordinate f along axis d.
__device__ __forceinline__ void frame_cells(const PorArgs& a, int d, int f, int& c0, int& c1) {
    const int w0 = (a.f0[d] + f) * a.F;
    c0 = max(w0 - a.gs.lo[d], 0);
    c1 = min(w0 + a.F - 1 - a.gs.lo[d], a.gs.dim[d] - 1);
}

// ---------------------------------------------------------------------------
// near flags, dry particles, per-frame-block counts
// ---------------------------------------------------------------------------
constexpr int kNearThreads = 128;

__global__ void __launch_bounds__(kNearThreads) k_pnear(PorArgs a) {
    pdl_wait();
    pdl_launch();
    __shared__ DemTile tiles[kNearThreads / 32];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = k < a.P.n;
    const int o = mine ? a.gs.order[k] : 0;
    const float4 p = mine ? a.f_posm[k] : make_float4(0.f, 0.f, 0.f, 0.f);  // positions only: runs before the density pass is done
    const int key = mine ? a.gs.key[o] : 0;
    const int inst = a.gs.ncl > 0 ? key / a.gs.ncl : 0;
    bool near = false;
    if (a.D.n > 0)
        warp_dem_visit(
            a.gd, mine, p.x, p.y, p.z, a.rq, inst, tiles[threadIdx.x >> 5],
            [&](int b, float4& q, float4&, float4&) {
                const float3 x = ld3(a.D.pos, b);
                q = make_float4(x.x, x.y, x.z, a.aux[b].z);  // len < 2 h_b, :87-88
            },
            [&](int, float) { near = true; });
    if (!mine) return;
    a.flag[k] = near ? 1 : 0;
    if (near) {
        const int local = key - inst * a.gs.ncl;
        const int cz = local % a.gs.dim[2], cy = (local / a.gs.dim[2]) % a.gs.dim[1];
        const int cx = local / (a.gs.dim[2] * a.gs.dim[1]);
        const int fb = frame_of(a, inst, cx, cy, cz);
        if (atomicAdd(&a.cnt[fb], 1) == 0) a.fbl[atomicAdd(&a.ctl->n_pfb, 1)] = fb;
    } else {
        a.P.porosity[o] = fminf(fmaxf(1.0f, a.eps_min), a.eps_max);
    }
}

// ---------------------------------------------------------------------------
// listed slots of each frame block, and its tiles: the cells in pencils of 2 x 2
// columns, up one pencil and down the next, so that 128 consecutive particles
// (7 cells) lie in a box of about 2 x 2 x 2 cells wherever a tile begins.  Each
// lane counts and then writes the listed slots of one cell (one cell piece
// after another per warp, 32 slots at a time, took 25-31 us, this form 14:
// a frame block's 64 pieces are one chain of loads each).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_plist(PorArgs a) {
    pdl_wait();
    pdl_launch();
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int n_pfb = a.ctl->n_pfb;
    for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n_pfb; i += nw) {
        const int fb = a.fbl[i];
        const int c = a.cnt[fb];
        const int nt = (c + kPM - 1) / kPM;
        int n0 = 0, t0 = 0;
        if (lane == 0) {
            n0 = atomicAdd(&a.ctl->n_near, c);
            t0 = atomicAdd(&a.ctl->n_ptiles, nt);
        }
        n0 = __shfl_sync(kAll, n0, 0);
        t0 = __shfl_sync(kAll, t0, 0);
        const int inst = fb / a.nfb_local;
        const int l = fb - inst * a.nfb_local;
        const int fz = l % a.nf[2], fy = (l / a.nf[2]) % a.nf[1], fx = l / (a.nf[2] * a.nf[1]);
        int x0, x1, y0, y1, z0, z1;
        frame_cells(a, 0, fx, x0, x1);
        frame_cells(a, 1, fy, y0, y1);
        frame_cells(a, 2, fz, z0, z1);
        const int npy = (y1 - y0) / 2 + 1, nz = z1 - z0 + 1, pieces = ((x1 - x0) / 2 + 1) * npy * nz * 4;
        int pos = n0;
        for (int p0 = 0; p0 < pieces; p0 += 32) {
            const int p = p0 + lane, q = p >> 2, pencil = q / nz;
            const int px = pencil / npy, py = (px & 1) ? npy - 1 - pencil % npy : pencil % npy;
            const int cx = x0 + 2 * px + ((p >> 1) & 1), cy = y0 + 2 * py + (p & 1);
            const int cz = (pencil & 1) ? z1 - q % nz : z0 + q % nz;
            int s = 0, e = 0;
            if (p < pieces && cx <= x1 && cy <= y1) {
                const int base = inst * a.gs.ncl + (cx * a.gs.dim[1] + cy) * a.gs.dim[2] + cz;
                s = a.gs.start[base];
                e = a.gs.start[base + 1];
            }
            int count = 0;
#pragma unroll 8
            for (int k = s; k < e; ++k) count += a.flag[k] != 0;
            int end = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(kAll, end, o);
                if (lane >= o) end += v;
            }
            int to = pos + end - count;
            pos += __shfl_sync(kAll, end, 31);
            if (count > 0)
                for (int k = s; k < e; ++k)
                    if (a.flag[k] != 0) a.near_list[to++] = k;
        }
        for (int t = lane; t < nt; t += 32) a.tiles[t0 + t] = make_int4(n0 + kPM * t, min(kPM, c - kPM * t), fb, 0);
    }
}

// ---------------------------------------------------------------------------
// the normaliser on the tensor cores
// ---------------------------------------------------------------------------
// Bounded wait; on a timeout, or when another warp has given up, the CTA's abort
// flag is set and false returned.
__device__ __forceinline__ bool bwait(uint64_t* bar, uint32_t parity, PorSmem& sh, sphdem_ctl_t* ctl) {
    if (*(volatile int*)&sh.abort_flag == 0) {
        if (mbar_wait(bar, parity, kPPolls)) return true;
        sh.abort_flag = 1;
        flag(ctl, SPHDEM_FLAG_TIMEOUT);
    }
    return false;
}
// The same for a whole warp: every lane returns the same.
__device__ __forceinline__ bool bwait_warp(uint64_t* bar, uint32_t parity, PorSmem& sh, sphdem_ctl_t* ctl) {
    return __all_sync(0xffffffffu, bwait(bar, parity, sh, ctl));
}

// 16 columns of this thread's TMEM lane, loaded and waited for in one statement.
__device__ __forceinline__ void ld16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// The polynomial's packed constants as 64-bit register pairs.
struct Kpk {
    unsigned long long k0, k1, k2, k3, one;
};
__device__ __forceinline__ unsigned long long pk2(float a) {
    return ((unsigned long long)__float_as_uint(a) << 32) | __float_as_uint(a);
}

// The weighted sums of 16 chunk columns r (s_ij bits of this thread's
// subject): column 4i + c holds a candidate of class c (or c + 4 in the second
// half of the chunk) and goes to accumulator c (a01 holds classes 0-1, a23
// classes 2-3, as FP32 pairs).  u^4 (1 + 2q), u = 1 - q/2, is evaluated as the
// expanded polynomial 1 + s (-5/2 + q (5/2 + q (-15/16 + q/8))) with s = q^2
// clamped to [0, 4] (|s| first: the MMA's rounding can leave a coincident pair
// slightly negative): every Horner step is exact at q = 2, so the weight there
// is exactly 0.  The polynomial and the sums run on packed FP32 pairs
// (fma.rn.ftz.f32x2: two independent round-to-nearest FMAs); V (candidate
// volumes, 0 for padding) is read from shared memory at vaddr.
//
// sums16_next is one statement that first issues the load of the lane's next
// 16 columns into s and ends with the wait for it: the arithmetic reads only
// registers that are not the load's destination, and nothing outside the
// statement sees s before the data has landed, so the load's latency hides
// behind the arithmetic without a register of a load in flight ever being
// read, moved or spilled.
// PTX of four columns: operands R0..R3 hold their s bits, V the shared-memory
// address of the chunk's volumes, OFF the byte offset of these four, A01/A23
// the accumulators, K0..K3/ONE the packed polynomial constants.
#define POR_SUMS4(R0, R1, R2, R3, V, OFF, A01, A23, K0, K1, K2, K3, ONE)                              \
    "mov.b32 s0, %" #R0 ";\n\tmov.b32 s1, %" #R1 ";\n\tmov.b32 s2, %" #R2 ";\n\tmov.b32 s3, %" #R3 ";\n\t" \
    "abs.ftz.f32 s0, s0;\n\tabs.ftz.f32 s1, s1;\n\tabs.ftz.f32 s2, s2;\n\tabs.ftz.f32 s3, s3;\n\t"        \
    "min.ftz.f32 s0, s0, 0f40800000;\n\tmin.ftz.f32 s1, s1, 0f40800000;\n\t"                           \
    "min.ftz.f32 s2, s2, 0f40800000;\n\tmin.ftz.f32 s3, s3, 0f40800000;\n\t"                           \
    "sqrt.approx.ftz.f32 q0, s0;\n\tsqrt.approx.ftz.f32 q1, s1;\n\t"                                    \
    "sqrt.approx.ftz.f32 q2, s2;\n\tsqrt.approx.ftz.f32 q3, s3;\n\t"                                    \
    "mov.b64 sa, {s0, s1};\n\tmov.b64 sb, {s2, s3};\n\tmov.b64 qa, {q0, q1};\n\tmov.b64 qb, {q2, q3};\n\t" \
    "fma.rn.ftz.f32x2 ca, %" #K0 ", qa, %" #K1 ";\n\tfma.rn.ftz.f32x2 cb, %" #K0 ", qb, %" #K1 ";\n\t"   \
    "fma.rn.ftz.f32x2 ca, ca, qa, %" #K2 ";\n\tfma.rn.ftz.f32x2 cb, cb, qb, %" #K2 ";\n\t"               \
    "fma.rn.ftz.f32x2 ca, ca, qa, %" #K3 ";\n\tfma.rn.ftz.f32x2 cb, cb, qb, %" #K3 ";\n\t"               \
    "fma.rn.ftz.f32x2 wa, ca, sa, %" #ONE ";\n\tfma.rn.ftz.f32x2 wb, cb, sb, %" #ONE ";\n\t"             \
    "ld.shared.v4.f32 {v0, v1, v2, v3}, [%" #V "+" #OFF "];\n\t"                                         \
    "mov.b64 va, {v0, v1};\n\tmov.b64 vb, {v2, v3};\n\t"                                                \
    "fma.rn.ftz.f32x2 %" #A01 ", va, wa, %" #A01 ";\n\tfma.rn.ftz.f32x2 %" #A23 ", vb, wb, %" #A23 ";\n\t"
#define POR_REGS                          \
    ".reg .f32 s<4>, q<4>, v<4>;\n\t"     \
    ".reg .b64 sa, sb, qa, qb, ca, cb, va, vb, wa, wb;\n\t"

// Operands: %0-%15 s (next columns), %16/%17 a01/a23, %18-%33 r, %34 vaddr,
// %35 the next columns' TMEM address, %36-%40 the constants.
__device__ __forceinline__ void sums16_next(const uint32_t* r, uint32_t vaddr, uint32_t tnext, uint32_t* s,
                                            unsigned long long& a01, unsigned long long& a23, const Kpk& K) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%35];\n\t"
        "{\n\t" POR_REGS
        POR_SUMS4(18, 19, 20, 21, 34, 0, 16, 17, 36, 37, 38, 39, 40)
        POR_SUMS4(22, 23, 24, 25, 34, 16, 16, 17, 36, 37, 38, 39, 40)
        POR_SUMS4(26, 27, 28, 29, 34, 32, 16, 17, 36, 37, 38, 39, 40)
        POR_SUMS4(30, 31, 32, 33, 34, 48, 16, 17, 36, 37, 38, 39, 40)
        "}\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]),
          "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]), "=r"(s[14]), "=r"(s[15]),
          "+l"(a01), "+l"(a23)
        : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(vaddr),
          "r"(tnext), "l"(K.k0), "l"(K.k1), "l"(K.k2), "l"(K.k3), "l"(K.one)
        : "memory");
}

// The same arithmetic on the last 16 columns of a chunk half (no load behind
// it).  Operands: %0/%1 a01/a23, %2-%17 r, %18 vaddr, %19-%23 the constants.
__device__ __forceinline__ void sums16(const uint32_t* r, uint32_t vaddr, unsigned long long& a01,
                                       unsigned long long& a23, const Kpk& K) {
    asm volatile(
        "{\n\t" POR_REGS
        POR_SUMS4(2, 3, 4, 5, 18, 0, 0, 1, 19, 20, 21, 22, 23)
        POR_SUMS4(6, 7, 8, 9, 18, 16, 0, 1, 19, 20, 21, 22, 23)
        POR_SUMS4(10, 11, 12, 13, 18, 32, 0, 1, 19, 20, 21, 22, 23)
        POR_SUMS4(14, 15, 16, 17, 18, 48, 0, 1, 19, 20, 21, 22, 23)
        "}"
        : "+l"(a01), "+l"(a23)
        : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(vaddr),
          "l"(K.k0), "l"(K.k1), "l"(K.k2), "l"(K.k3), "l"(K.one)
        : "memory");
}
#undef POR_SUMS4
#undef POR_REGS

__global__ void __launch_bounds__(kPThreads, 2) k_porosity_mma(PorArgs a) {
    pdl_wait();
    pdl_launch();
    extern __shared__ uint8_t raw[];
    PorSmem& sh = *reinterpret_cast<PorSmem*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < kPStages; ++s) {
            mbar_init(&sh.full[s], kPStageWarps);
            mbar_init(&sh.empty[s], 1 + kPEpiWarps);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh.afull[b], 1);
            mbar_init(&sh.aempty[b], kPEpiWarps);
        }
        mbar_init(&sh.drain, 1);
        fence_mbar_init();
        sh.abort_flag = 0;
    }
    if (warp == kPMmaWarp) umma::tmem_alloc(&sh.tmem, kPTmemCols);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = sh.tmem;
    const Geo& G = a.gs;
    const int n_units = a.ctl->n_ptiles * kPSlabs;
    constexpr uint32_t idesc = umma::idesc_bf16(kPM, kPN);
    // chunks run so far by this CTA, the same in every role: candidate stage and
    // its phase, accumulator and its phase
    uint32_t stage = 0, sphase = 0, buf = 0, bphase = 0;
    auto next_chunk = [&]() {
        if (++stage == kPStages) {
            stage = 0;
            sphase ^= 1u;
        }
        buf ^= 1u;
        bphase ^= buf ^ 1u;
    };
    bool issued = false;     // this CTA issued MMAs (drained before freeing TMEM)

    for (;;) {
        __syncthreads();
        if (tid == 0) {
            const int u0 = sh.abort_flag ? n_units : atomicAdd(&a.ctl->near_next, 1);
            sh.unit = u0;
            if (u0 < n_units) {
                const int4 T0 = a.tiles[u0 / kPSlabs];
                sh.tstart = T0.x;
                sh.tcount = T0.y;
                sh.slab = u0 % kPSlabs;
            }
        }
        __syncthreads();
        const int u = sh.unit;
        if (u >= n_units) break;
        const int tile = u / kPSlabs, slab = u - tile * kPSlabs;
        const int4 T = a.tiles[tile];
        const int fb = T.z;
        const int inst = fb / a.nfb_local;
        const int l = fb - inst * a.nfb_local;
        const int fzl = l % a.nf[2], fyl = (l / a.nf[2]) % a.nf[1], fxl = l / (a.nf[2] * a.nf[1]);
        // canonical centre: the frame block's centre (world units)
        const float half = 0.5f * (float)a.F * G.cell;
        const float cxw = (float)((a.f0[0] + fxl) * a.F) * G.cell + half;
        const float cyw = (float)((a.f0[1] + fyl) * a.F) * G.cell + half;
        const float czw = (float)((a.f0[2] + fzl) * a.F) * G.cell + half;
        // subjects: A rows and the tile's world box (warps 0-3; row = tid)
        float2 acc01 = make_float2(0.f, 0.f), acc23 = make_float2(0.f, 0.f);
        if (warp < 4) {
            float px = 0.f, py = 0.f, pz = 0.f;
            float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
            if (tid < T.y) {
                const float4 x = a.f_posv[a.near_list[T.x + tid]];
                px = (x.x - cxw) * a.inv_h;
                py = (x.y - cyw) * a.inv_h;
                pz = (x.z - czw) * a.inv_h;
                lo[0] = hi[0] = x.x;
                lo[1] = hi[1] = x.y;
                lo[2] = hi[2] = x.z;
            }
            make_row<true>(sh.A, tid, px, py, pz);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                    hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
                }
            if (lane == 0)
                for (int d = 0; d < 3; ++d) {
                    sh.red[d][warp] = lo[d];
                    sh.red[3 + d][warp] = hi[d];
                }
            fence_proxy_async_smem();  // A is read by the MMA (async proxy)
        }
        __syncthreads();
        float bb[6];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bb[d] = fminf(fminf(sh.red[d][0], sh.red[d][1]), fminf(sh.red[d][2], sh.red[d][3]));
            bb[3 + d] = fmaxf(fmaxf(sh.red[3 + d][0], sh.red[3 + d][1]), fmaxf(sh.red[3 + d][2], sh.red[3 + d][3]));
        }
        // window columns of the tile, cut to this unit's world-anchored slab
        const float rq = a.rq;
        const int wx0 = coord(bb[0] - rq, G.inv, G.lo[0], G.dim[0]), wx1 = coord(bb[3] + rq, G.inv, G.lo[0], G.dim[0]);
        const int wy0 = coord(bb[1] - rq, G.inv, G.lo[1], G.dim[1]), wy1 = coord(bb[4] + rq, G.inv, G.lo[1], G.dim[1]);
        const int sw = floor_div(G.lo[0] + wx0, a.Wx) + slab;
        const int sx0 = max(wx0, sw * a.Wx - G.lo[0]), sx1 = min(wx1, sw * a.Wx + a.Wx - 1 - G.lo[0]);
        const int ny = wy1 - wy0 + 1;
        const int ncols = sx1 >= sx0 ? (sx1 - sx0 + 1) * ny : 0;
        const int S_m = G.start[inst * G.ncl];  // first slot of the instance (slot alignment origin)
        const float margin = 0.01f * G.cell;
        for (int c0 = 0; c0 < ncols; c0 += kPMaxRanges) {
            // trim each column of the batch to the ball around the bounding box,
            // pad to 8-aligned instance slot offsets, compact in column order
            constexpr int kPer = (kPMaxRanges + kPThreads - 1) / kPThreads;
            int ls[kPer], li[kPer], ln[kPer], cnt = 0, len_sum = 0;
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                const int c = c0 + tid * kPer + q;
                ln[q] = 0;
                if (c >= ncols || tid * kPer + q >= kPMaxRanges) continue;
                const int cx = sx0 + c / ny, cy = wy0 + c % ny;
                const float xa = cx == 0 ? -INFINITY : (float)(G.lo[0] + cx) * G.cell;
                const float xb = cx == G.dim[0] - 1 ? INFINITY : (float)(G.lo[0] + cx + 1) * G.cell;
                const float ya = cy == 0 ? -INFINITY : (float)(G.lo[1] + cy) * G.cell;
                const float yb = cy == G.dim[1] - 1 ? INFINITY : (float)(G.lo[1] + cy + 1) * G.cell;
                const float gx = fmaxf(0.0f, fmaxf(xa - bb[3], bb[0] - xb) - margin);
                const float gy = fmaxf(0.0f, fmaxf(ya - bb[4], bb[1] - yb) - margin);
                const float rem = rq * rq - gx * gx - gy * gy;
                if (rem < 0.0f) continue;
                const float zr = sqrtf(rem) + margin;
                const int z0 = coord(bb[2] - zr, G.inv, G.lo[2], G.dim[2]);
                const int z1 = coord(bb[5] + zr, G.inv, G.lo[2], G.dim[2]);
                const int base = inst * G.ncl + (cx * G.dim[1] + cy) * G.dim[2];
                const int s = __ldg(G.start + base + z0), e = __ldg(G.start + base + z1 + 1);
                if (e <= s) continue;
                const int al = s - ((s - S_m) & (kPAlign - 1));
                const int ae = e + ((kPAlign - ((e - S_m) & (kPAlign - 1))) & (kPAlign - 1));
                ls[q] = al;
                li[q] = (s - al) | ((e - s) << 3);
                ln[q] = ae - al;
                ++cnt;
                len_sum += ae - al;
            }
            int m, tot;
            int off = block_exclusive_scan(cnt, sh.wtot, m);
            int loff = block_exclusive_scan(len_sum, sh.wtot, tot);
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if (ln[q] > 0) {
                    sh.rs[off] = ls[q];
                    sh.info[off] = li[q];
                    sh.pre[off] = loff;
                    loff += ln[q];
                    ++off;
                }
            if (tid == 0) sh.pre[m] = tot;
            __syncthreads();
            const int nchunks = (tot + kPN - 1) / kPN;
            if (tid == 0 && nchunks > 0) atomicAdd(&a.ctl->n_pchunks, nchunks);
            const bool crs = nchunks <= kPMaxChunks;  // else each candidate searches all ranges
            if (crs) {
                for (int c = tid; c < nchunks; c += kPThreads) {
                    const int u0 = c * kPN;
                    int lo = 0, hi = m - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (sh.pre[mid] <= u0) lo = mid;
                        else hi = mid - 1;
                    }
                    sh.cr[c] = lo;
                }
                if (tid == 0) sh.cr[nchunks] = m - 1;
                __syncthreads();
            }
            if (warp >= kPEpiWarps) {
                // ---- staging: a candidate row and volume per thread; the next
                // chunk's candidate is loaded while this one's row is built.
                // Warp kPMmaWarp then issues the chunk's MMA (it waits for the
                // accumulator there, at most two chunks ahead of the epilogue).
                const int t = tid - 32 * kPEpiWarps;
                // chunk position t (= slot offset mod 8 in its low bits) -> column:
                // classes 0-3 fill columns 0-63, classes 4-7 columns 64-127
                const int col = (t & 4) * 16 + (t >> 3) * 4 + (t & 3);
                auto fetch = [&](int c) {
                    const int uu = c * kPN + t;
                    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);  // V = 0: padding and past the end
                    if (uu >= tot) return x;
                    int lo = crs ? sh.cr[c] : 0, hi = crs ? sh.cr[c + 1] : m - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (sh.pre[mid] <= uu) lo = mid;
                        else hi = mid - 1;
                    }
                    const int off2 = uu - sh.pre[lo];
                    const int inf = sh.info[lo];
                    const int pf = inf & (kPAlign - 1), len = inf >> 3;
                    if (off2 >= pf && off2 < pf + len) x = __ldg(a.f_posv + sh.rs[lo] + off2);
                    return x;
                };
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (nchunks > 0) x = fetch(0);
                for (int c = 0; c < nchunks; ++c) {
                    if (!bwait_warp(&sh.empty[stage], sphase ^ 1u, sh, a.ctl)) break;
                    const float4 y = x;
                    if (c + 1 < nchunks) x = fetch(c + 1);
                    make_row<false>(sh.B[stage], col, (y.x - cxw) * a.inv_h, (y.y - cyw) * a.inv_h,
                                    (y.z - czw) * a.inv_h);
                    sh.V[stage][col] = y.w;
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.full[stage]);  // one arrival per staging warp
                    if (warp == kPMmaWarp) {
                        if (lane == 0 && bwait(&sh.full[stage], sphase, sh, a.ctl) &&
                            bwait(&sh.aempty[buf], bphase ^ 1u, sh, a.ctl)) {
                            umma::fence_after();
                            umma::mma_tile(tmem + buf * kPN, sh.A, sh.B[stage], kPK, idesc, false);
                            umma::commit(&sh.afull[buf]);
                            umma::commit(&sh.empty[stage]);
                            issued = true;
                        }
                        __syncwarp();
                    }
                    next_chunk();
                }
            } else {
                // ---- epilogue: w(s) and the volume-weighted sums ----
                for (int c = 0; c < nchunks; ++c) {
                    if (!bwait_warp(&sh.afull[buf], bphase, sh, a.ctl)) break;
                    umma::fence_after();
                    // this warp's half of the chunk, 16 columns per step, the
                    // load of the next 16 behind the arithmetic; the other
                    // epilogue warps of the sub-partition hide the first load
                    const int h0 = (warp >> 2) * (kPN / 2);
                    const uint32_t tcol = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + buf * kPN + h0;
                    {
                        const Kpk K{pk2(0.125f), pk2(-0.9375f), pk2(2.5f), pk2(-2.5f), pk2(1.0f)};
                        const uint32_t va = (uint32_t)__cvta_generic_to_shared(&sh.V[stage][h0]);
                        unsigned long long u01, u23;
                        memcpy(&u01, &acc01, 8);
                        memcpy(&u23, &acc23, 8);
                        uint32_t r0[16], r1[16];
                        ld16(tcol, r0);
                        sums16_next(r0, va, tcol + 16, r1, u01, u23, K);
                        sums16_next(r1, va + 64, tcol + 32, r0, u01, u23, K);
                        sums16_next(r0, va + 128, tcol + 48, r1, u01, u23, K);
                        sums16(r1, va + 192, u01, u23, K);
                        memcpy(&acc01, &u01, 8);
                        memcpy(&acc23, &u23, 8);
                    }
                    umma::fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&sh.aempty[buf]);
                        mbar_arrive(&sh.empty[stage]);
                    }
                    next_chunk();
                }
            }
            __syncthreads();
        }
        // classes 4-7 (warps 4-7) are added to classes 0-3 (warps 0-3) of the same subject
        if (warp >= 4 && warp < kPEpiWarps) sh.hsum[tid - 128] = (acc01.x + acc01.y) + (acc23.x + acc23.y);
        __syncthreads();
        if (warp < 4 && tid < sh.tcount)
            a.part[(size_t)(sh.tstart + tid) * kPSlabs + sh.slab] =
                ((acc01.x + acc01.y) + (acc23.x + acc23.y)) + sh.hsum[tid];
    }
    // drain this CTA's MMAs, then free tensor memory
    __syncthreads();
    if (warp == kPMmaWarp) {
        if (lane == 0 && issued) {
            umma::commit(&sh.drain);
            if (!mbar_wait(&sh.drain, 0, kPPolls)) flag(a.ctl, SPHDEM_FLAG_TIMEOUT);
        }
        __syncwarp();
    }
    umma::fence_before();
    __syncthreads();
    if (warp == kPMmaWarp) {
        umma::fence_after();
        umma::tmem_dealloc(tmem, kPTmemCols);
    }
}

// ---------------------------------------------------------------------------
// slab partials -> normaliser -> solid fraction -> porosity
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kNearThreads) k_pfinish(PorArgs a) {
    pdl_wait();
    pdl_launch();
    __shared__ DemTile tiles[kNearThreads / 32];
    DemTile& sh = tiles[threadIdx.x >> 5];
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int n_near = a.ctl->n_near;
    if ((idx & ~31) >= n_near) return;  // the warp has no entry
    const bool mine = idx < n_near;
    const int k = mine ? a.near_list[idx] : 0;
    const int o = a.gs.order[k];
    float f = 0.0f;
    if (mine)
#pragma unroll
        for (int s = 0; s < kPSlabs; ++s) f += a.part[(size_t)idx * kPSlabs + s];
    const float flt = f * a.cw;
    const float4 p = a.f_posv[k];
    const int inst = a.gs.ncl > 0 ? a.gs.key[o] / a.gs.ncl : 0;
    float solid = 0.0f;
    warp_dem_visit(
        a.gd, mine, p.x, p.y, p.z, a.rq, inst, sh,
        [&](int b, float4& x, float4& q, float4&) {
            const float3 pb = ld3(a.D.pos, b);
            const float4 ab = a.aux[b];
            x = make_float4(pb.x, pb.y, pb.z, ab.z);  // len < 2 h_b, :87-88
            q = make_float4(ab.x, ab.y, a.D.volume[b], 0.0f);
        },
        [&](int t, float d2) {
            const float4 ab = sh.q[t];
            const float q = fast_sqrt(d2) * ab.x;
            const float uu = 1.0f - 0.5f * q;
            const float u2 = uu * uu;
            const float wb = q < 2.0f ? ab.y * u2 * u2 * (1.0f + 2.0f * q) : 0.0f;
            solid += ab.z * wb / (flt + 1.0e-20f);
        });
    if (mine) a.P.porosity[o] = fminf(fmaxf(1.0f - solid, a.eps_min), a.eps_max);
}

// Frame-block lattice of the fluid grid (world-anchored), per axis.
void frame_lattice(const sphdem_grid_t& g, int F, int* f0, int* nf) {
    for (int d = 0; d < 3; ++d) {
        auto fdiv = [&](int x) { return x >= 0 ? x / F : -((-x + F - 1) / F); };
        f0[d] = fdiv(g.lo[d]);
        nf[d] = fdiv(g.lo[d] + g.dim[d] - 1) - f0[d] + 1;
    }
}

int smem_opt_in_porosity() {
    static std::mutex mu;
    static std::map<int, bool> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev]) return SPHDEM_OK;
    cudaError_t e = cudaFuncSetAttribute(k_porosity_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPSmemBytes);
    if (e != cudaSuccess) {
        set_error("porosity: shared memory opt-in", e);
        return SPHDEM_ERR_CUDA;
    }
    done[dev] = true;
    return SPHDEM_OK;
}

}  // namespace

int porosity_frame_edge(int frame) { return frame > 0 ? frame : 4; }

int64_t porosity_frames(const sphdem_grid_t& g, int F) {
    if (F <= 0 || g.ncell_local <= 0) return 0;
    int f0[3], nf[3];
    frame_lattice(g, F, f0, nf);
    return (int64_t)nf[0] * nf[1] * nf[2] * (g.ninst > 0 ? g.ninst : 1);
}

// Kernel attributes of the tensor-core porosity pass; called eagerly (outside
// any stream capture) before its first launch on a device.
int porosity_setup() { return smem_opt_in_porosity(); }

// The tensor-core porosity pass (uniform DEM h > 0) with the frame-block
// edge its scratch was sized for.  Returns SPHDEM_ERR_INVALID when the
// context lacks those buffers.
// part 0: the whole pass; 1: the near flags and tiles (k_pnear, k_plist: they
// read positions only, so they may run while the density pass runs); 2: the
// normaliser and the finish (after the density pass and part 1).
int run_porosity_mma(const sphdem_ctx_t* c, float support, float h, float eps_min, float eps_max, cudaStream_t st,
                     int part) {
    const int n = c->sph.n;
    if (n <= 0) return SPHDEM_OK;
    const sphdem_work_t& w = c->work;
    const int F = porosity_frame_edge(w.pframe);
    const int64_t nfb = porosity_frames(c->grid_sph, F);
    if (!w.pfb || !w.ptiles || !w.ppart || !w.pflag || nfb <= 0 || 2 * (nfb + 1) > w.pfb_words ||
        nfb > (1 << 30)) {
        set_error_msg("porosity (tensor cores): frame-block scratch missing or too small for the fluid grid");
        return SPHDEM_ERR_INVALID;
    }
    const int rc = porosity_setup();
    if (rc) return rc;
    PorArgs a;
    a.gs = make_geo(c->grid_sph);
    a.gd = make_geo(c->grid_dem);
    a.f_posm = (const float4*)w.f_posm;
    a.f_posv = (const float4*)w.f_posv;
    a.aux = (const float4*)w.dem_aux;
    a.P = c->sph;
    a.D = c->dem;
    a.near_list = w.near_list;
    a.flag = w.pflag;
    a.nfb = (int)nfb;
    a.cnt = w.pfb;
    a.fbl = w.pfb + (nfb + 1);
    a.tiles = (int4*)w.ptiles;
    a.part = w.ppart;
    a.ctl = c->ctl;
    a.rq = pad_radius(support);
    const Kern k = make_kern(h);
    a.inv_h = k.inv_h;
    a.cw = k.cw;
    a.eps_min = eps_min;
    a.eps_max = eps_max;
    a.F = F;
    frame_lattice(c->grid_sph, F, a.f0, a.nf);
    a.nfb_local = a.nf[0] * a.nf[1] * a.nf[2];
    // slab width: kPSlabs slabs cover any tile window (frame block + 2 rq + clamping slack)
    const float cell = c->grid_sph.cell > 0.0f ? c->grid_sph.cell : 1.0f;
    const int span = (int)ceilf(2.0f * a.rq / cell) + F + 3;
    a.Wx = (span + kPSlabs - 2) / (kPSlabs - 1);
    if (a.Wx < 1) a.Wx = 1;
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (part != 2) {
        // counters: listed particles, work units, tiles, listed frame blocks,
        // evaluated chunks (control words 6..10)
        cudaError_t e = zero_words(&c->ctl->n_near, 5, st);
        if (e == cudaSuccess) e = zero_words(a.cnt, nfb, st);
        if (e != cudaSuccess) {
            set_error("porosity memset", e);
            return SPHDEM_ERR_CUDA;
        }
        launch_pdl(k_pnear, blocks_for(n, kNearThreads), kNearThreads, 0, st, a);
        launch_pdl(k_plist, 8 * sms, 256, 0, st, a);
    }
    if (part != 1) {
        launch_pdl(k_porosity_mma, 2 * sms, kPThreads, kPSmemBytes, st, a);
        launch_pdl(k_pfinish, blocks_for(n, kNearThreads), kNearThreads, 0, st, a);
    }
    return launch_status("porosity (tensor cores)");
}

}  // namespace sd
