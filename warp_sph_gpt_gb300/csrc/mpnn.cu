// mpnn.cu -- learned K-step surrogate: a message-passing network over the
// radius graph of all particles, trained and evaluated by tensor-core
// (tcgen05, BF16 operands, FP32 accumulation in tensor memory) kernels.
//
// Kernels (persistent, 512 threads: four per TMEM lane):
//   k_rows     node MLP layers: Y = X W^T (+ bias, SiLU), one 128-row tile per
//              MMA group; the weight image is bulk-copied (TMA) into shared
//              memory once per CTA.
//   k_edges    the fused edge pass: edge features -> layer 1 (edges x 128,
//              TMEM lane = edge) -> ReLU -> layer 2 computed transposed
//              (TMEM lane = feature, columns = edges) -> per-feature segmented
//              sums over the receiver-sorted edges: aggregation (forward) or
//              the scatter to senders (backward of the second round).
//   k_edges_bwd  backward of the first round and of the edge MLP: recomputes
//              both layers, forms dF, scatters dh0, and accumulates dW2 and
//              dW1 across all of the CTA's tiles in TMEM.
//   k_wgrad    weight gradients of the node layers, reduction over rows in
//              TMEM, per-CTA partials reduced in a fixed order; the training
//              pass runs them, and the node layers, on the receivers and the
//              nodes that send (29k of 80k rows for a dam break member).
// Every wait on an MMA or a bulk copy is bounded; on timeout the CTA raises
// SPHDEM_FLAG_TIMEOUT, waits once more (bounded), frees its tensor memory and
// returns.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <stdio.h>

#include <map>
#include <initializer_list>
#include <mutex>
#include <utility>

#include "cluster.cuh"
#include "common.cuh"
#include "sphdem_mpnn.h"
#include "umma.cuh"

namespace sd {

int build_grid(sphdem_grid_t* g, const float* pos, sphdem_ctl_t* ctl, cudaStream_t st);
int scan_counts(int* data, int n, int* sums, cudaStream_t st);

namespace {

using umma::tile_off;

constexpr int kH = SPHDEM_MPNN_HIDDEN;
constexpr int kT = 128;  // threads per CTA = rows per tile
constexpr int kRT = 4;   // node layers: threads per row (kRT x kT threads per CTA)
constexpr int kPolls = 1 << 20;
constexpr int kMaxCtas = 512;
constexpr int kBwdStride = 128 * 128 + 128 * 16 + 256;  // per-CTA partials of k_edges_bwd

// BF16 image offsets (halves) inside `packed`.
constexpr int P_E1 = 0, P_E2 = 2048, P_E2T = 18432, P_N1 = 34816, P_N2 = 36864, P_N2T = 53248, P_N3 = 69632,
              P_N3T = 71680;
static_assert(P_N3T + 2048 == SPHDEM_MPNN_PACKED, "packed layout");

enum { EPI_F32 = 0, EPI_SILU = 1 };
// Edge-input column 7 is the constant 1 and the layer-1 image holds the bias
// there, so the first edge MMA adds the bias itself.
constexpr int kBiasCol = 7;
enum { MODE_AGG = 0, MODE_SCATTER = 1 };

// SiLU z * sigmoid(z) with the fast exponential and reciprocal (relative
// error far below the BF16 rounding of the activations it feeds).
__device__ __forceinline__ float sigmoid(float z) { return __frcp_rn(1.0f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigmoid(z); }
__device__ __forceinline__ float silu_grad(float z) {
    const float s = sigmoid(z);
    return s * (1.0f + z * (1.0f - s));
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
// max(a, 0), max(b, 0) rounded to BF16 and packed (a in the low half), one
// instruction.
__device__ __forceinline__ uint32_t pack2_relu(float a, float b) {
    uint32_t r;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
__device__ __forceinline__ uint16_t bf16_bits(float a) {
    __nv_bfloat16 h = __float2bfloat16_rn(a);
    return *reinterpret_cast<uint16_t*>(&h);
}
__device__ __forceinline__ float bf(uint16_t u) { return __uint_as_float((uint32_t)u << 16); }

__device__ __forceinline__ void raise_flag(int32_t* status, int bits) {
    if (status) atomicOr(status, bits);
}

// CTA prologue: mbarriers ([0] MMA completion, [1] bulk copies) and tensor memory.
__device__ __forceinline__ uint32_t cta_begin(uint64_t* bars, uint32_t* slot, uint32_t ncols) {
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    if ((threadIdx.x >> 5) == 0) umma::tmem_alloc(slot, ncols);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    return *slot;
}

// The same prologue when thread 0 has already initialised the barriers.
__device__ __forceinline__ uint32_t cta_tmem(uint32_t* slot, uint32_t ncols) {
    if ((threadIdx.x >> 5) == 0) umma::tmem_alloc(slot, ncols);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    return *slot;
}

// Issue (thread 0) after the operand tiles were written and fenced by all.
__device__ __forceinline__ void operands_ready() {
    fence_proxy_async_smem();
    umma::fence_before();
    __syncthreads();
}

// Wait for the MMA group with `phase`; returns false on a CTA-wide timeout.
__device__ __forceinline__ bool mma_done(uint64_t* bars, uint32_t& phase, bool& mine) {
    mine = mbar_wait(&bars[0], phase, kPolls);
    const bool bad = __syncthreads_or(!mine);
    if (!bad) phase ^= 1u;
    umma::fence_after();
    return !bad;
}

__device__ __forceinline__ void cta_end(uint64_t* bars, uint32_t phase, bool pending, uint32_t tmem, uint32_t ncols,
                                        int32_t* status, bool failed) {
    if (failed) {
        if (threadIdx.x == 0) raise_flag(status, SPHDEM_FLAG_TIMEOUT);
    }
    if (pending) mbar_wait(&bars[0], phase, kPolls);
    umma::fence_before();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) {
        umma::fence_after();
        umma::tmem_dealloc(tmem, ncols);
    }
}

// ---------------------------------------------------------------------------
// weight images
// ---------------------------------------------------------------------------
struct Img {
    int dst, src, R, K, trans;
};
__constant__ Img kImgs[8] = {
    {P_E1, SPHDEM_MPNN_E1_W, 128, 16, 0},   {P_E2, SPHDEM_MPNN_E2_W, 128, 128, 0},
    {P_E2T, SPHDEM_MPNN_E2_W, 128, 128, 1}, {P_N1, SPHDEM_MPNN_N1_W, 128, 16, 0},
    {P_N2, SPHDEM_MPNN_N2_W, 128, 128, 0},  {P_N2T, SPHDEM_MPNN_N2_W, 128, 128, 1},
    {P_N3, SPHDEM_MPNN_N3_W, 16, 128, 0},   {P_N3T, SPHDEM_MPNN_N3_W, 128, 16, 1},
};

// Image element (r, k) = W[r][k], or W[k][r] for a transposed image; W is
// row-major with (trans ? R : K) columns.
__global__ void k_pack(const float* __restrict__ theta, uint16_t* __restrict__ packed) {
    const Img im = kImgs[blockIdx.y];
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= im.R * im.K) return;
    const int r = idx / im.K, k = idx % im.K;
    float w = im.trans ? theta[im.src + k * im.R + r] : theta[im.src + r * im.K + k];
    if (im.dst == P_E1 && k == kBiasCol) w = theta[SPHDEM_MPNN_E1_B + r];  // layer-1 bias rides in the MMA
    packed[im.dst + tile_off(r, k, im.K) / 2] = bf16_bits(w);
}

// ---------------------------------------------------------------------------
// node MLP layers: out = epi(A[M,K] * B[N,K]^T + bias)
// ---------------------------------------------------------------------------
// add (optional, K = 128): rows r < n_add of the A operand are A[r] + add[r]
// (the residual h + s * sum_j f_ij (.) h_j, formed while staging the tile);
// with clear, add[r] is zero afterwards (for the next round's sums).
// a_out (optional): the staged operand rows are stored there too.
// EPI_F32: z_out (optional) receives the output as well.
// list (optional): the layer runs on rows 0 .. n_direct - 1 and on the list[0]
// rows list[1 ..] (in any order: rows are independent); M bounds both.
template <int K, int N, int EPI, bool IMG>
__global__ void __launch_bounds__(kRT * kT) k_rows(const uint16_t* __restrict__ A, int M, float* add, int n_add,
                                             bool clear, const uint16_t* __restrict__ B,
                                             const float* __restrict__ bias, float* __restrict__ out_f32,
                                             uint16_t* __restrict__ out_bf, float* __restrict__ z_out,
                                             int32_t* status, const int* __restrict__ list, int n_direct,
                                             int early, uint16_t* __restrict__ a_out) {
    constexpr uint32_t kB = N * K * 2, kA = kT * K * 2;
    constexpr uint32_t kCols = N < 32 ? 32 : N;
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t* sB = sm;
    uint8_t* sA = sm + kB;
    float* sbias = reinterpret_cast<float*>(sA + kA);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sbias + (N < 2 ? 2 : N));
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2);
    // output: warps w, w + 4, ... (same TMEM lanes, rows rt) split the columns
    const int tid = threadIdx.x, warp = tid >> 5, rt = tid & (kT - 1), hh = tid / kT;

    // early (inference): the weight image is fixed, so its copy starts before
    // the previous kernel is done (no kernel of the inference chain writes it)
    const bool pre = IMG && early;
    if (pre && tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
        mbar_arrive_expect_tx(&bars[1], kB);
        tma_load_1d(sB, B, kB, &bars[1]);
    }
    pdl_wait();
    pdl_launch();
    const uint32_t tmem = pre ? cta_tmem(slot, kCols) : cta_begin(bars, slot, kCols);
    for (int i = tid; i < N; i += kRT * kT) sbias[i] = bias ? bias[i] : 0.0f;
    bool mine = true, failed = false, pending = false;
    uint32_t phase = 0;
    if (IMG) {
        if (tid == 0 && !pre) {
            mbar_arrive_expect_tx(&bars[1], kB);
            tma_load_1d(sB, B, kB, &bars[1]);
        }
        failed = __syncthreads_or(!mbar_wait(&bars[1], 0, kPolls));
    } else {
        for (int idx = tid; idx < N * (K / 8); idx += kRT * kT) {
            const int r = idx / (K / 8), q = idx % (K / 8);
            *reinterpret_cast<uint4*>(sB + tile_off(r, 8 * q, K)) =
                __ldg(reinterpret_cast<const uint4*>(B + (size_t)r * K) + q);
        }
    }
    __syncthreads();
    constexpr uint32_t idesc = umma::idesc_bf16(128, N);
    const int Mv = list ? min(M, n_direct + __ldg(list)) : M;  // rows of this launch
    for (int tile = blockIdx.x; !failed && tile * kT < Mv; tile += gridDim.x) {
        int row = tile * kT + rt;
        if (list && row >= n_direct) row = row < Mv ? __ldg(list + 1 + (row - n_direct)) : M;  // M: no row
        // staging: a warp takes 8 rows, 64 bytes of each at a time (whole
        // sectors, and no bank conflict in the tile), and loads before it
        // stores: with one thread per row share and the sums cleared between
        // the loads the layer with add took 38 us for 38k rows, now 14
        const int st = 8 * warp + (tid & 7);
        int srow = tile * kT + st;
        if (list && srow >= n_direct) srow = srow < Mv ? __ldg(list + 1 + (srow - n_direct)) : M;
        const bool plus = add != nullptr && srow < n_add;
        constexpr int QN = K / 8, NI = QN < 4 ? 1 : QN / 4;
        constexpr int BT = NI < 4 ? NI : EPI == EPI_SILU ? 4 : 2;  // 16-byte words in flight per thread
#pragma unroll
        for (int i0 = 0; i0 < NI; i0 += BT) {
            uint4 v[BT];
            float4 a[BT][2];
#pragma unroll
            for (int u = 0; u < BT; ++u) {
                const int q = 4 * (i0 + u) + ((tid >> 3) & 3);
                v[u] = make_uint4(0, 0, 0, 0);
                if (q < QN && srow < M) v[u] = __ldg(reinterpret_cast<const uint4*>(A + (size_t)srow * K) + q);
                if (q < QN && plus) {
                    const float4* at = reinterpret_cast<const float4*>(add + (size_t)srow * K + 8 * q);
                    a[u][0] = at[0];
                    a[u][1] = at[1];
                }
            }
#pragma unroll
            for (int u = 0; u < BT; ++u) {
                const int q = 4 * (i0 + u) + ((tid >> 3) & 3);
                if (q >= QN) continue;
                if (plus) {
                    const uint4 h = v[u];
                    const float4 a0 = a[u][0], a1 = a[u][1];
                    v[u] = make_uint4(pack2(bf((uint16_t)h.x) + a0.x, bf((uint16_t)(h.x >> 16)) + a0.y),
                                      pack2(bf((uint16_t)h.y) + a0.z, bf((uint16_t)(h.y >> 16)) + a0.w),
                                      pack2(bf((uint16_t)h.z) + a1.x, bf((uint16_t)(h.z >> 16)) + a1.y),
                                      pack2(bf((uint16_t)h.w) + a1.z, bf((uint16_t)(h.w >> 16)) + a1.w));
                    if (clear) {
                        float4* at = reinterpret_cast<float4*>(add + (size_t)srow * K + 8 * q);
                        at[0] = at[1] = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
                *reinterpret_cast<uint4*>(sA + tile_off(st, 8 * q, K)) = v[u];
                if (a_out && srow < M) reinterpret_cast<uint4*>(a_out + (size_t)srow * K)[q] = v[u];
            }
        }
        operands_ready();
        if (tid == 0) {
            umma::fence_after();
            umma::mma_tile(tmem, sA, sB, K, idesc, false);
            umma::commit(&bars[0]);
        }
        pending = true;
        if (!mma_done(bars, phase, mine)) {
            failed = true;
            break;
        }
        pending = false;
        // columns of this thread: [hh NH, hh NH + NH), or all 16 (thread rt) when N = 16
        constexpr int W = N < 32 ? 16 : 32, NH = N < 32 ? N : N / kRT;
        static_assert(N < 32 || NH % 32 == 0, "k_rows column split");
#pragma unroll
        for (int c0 = hh * NH; c0 < hh * NH + NH && c0 < N; c0 += W) {
            float v[32];
            if (N < 32)
                umma::tmem_ld16(umma::taddr(tmem, 32 * (warp & 3), c0), v);
            else
                umma::tmem_ld32(umma::taddr(tmem, 32 * (warp & 3), c0), v);
            if (row < M) {
                if (EPI == EPI_F32) {
                    float4* o = reinterpret_cast<float4*>(out_f32 + (size_t)row * N + c0);
#pragma unroll
                    for (int i = 0; i < W; ++i) v[i] += sbias[c0 + i];
#pragma unroll
                    for (int i = 0; i < W / 4; ++i) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    if (z_out) {
                        float4* o2 = reinterpret_cast<float4*>(z_out + (size_t)row * N + c0);
#pragma unroll
                        for (int i = 0; i < W / 4; ++i)
                            o2[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < W; ++i) v[i] += sbias[c0 + i];
                    if (z_out) {
                        float4* o = reinterpret_cast<float4*>(z_out + (size_t)row * N + c0);
#pragma unroll
                        for (int i = 0; i < W / 4; ++i) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    }
                    uint4* o = reinterpret_cast<uint4*>(out_bf + (size_t)row * N + c0);
#pragma unroll
                    for (int i = 0; i < W / 8; ++i)
                        o[i] = make_uint4(pack2(silu(v[8 * i]), silu(v[8 * i + 1])),
                                          pack2(silu(v[8 * i + 2]), silu(v[8 * i + 3])),
                                          pack2(silu(v[8 * i + 4]), silu(v[8 * i + 5])),
                                          pack2(silu(v[8 * i + 6]), silu(v[8 * i + 7])));
                }
            }
        }
        umma::fence_before();
        __syncthreads();
    }
    cta_end(bars, phase, pending && !mine, tmem, kCols, status, failed);
}

// ---------------------------------------------------------------------------
// fused edge pass
// ---------------------------------------------------------------------------
struct EdgeArgs {
    const float4* pos;
    const float4* vel;
    const int* offset;
    const int* sender;
    const int* receiver;
    int n_recv, cap;
    float inv_r, inv_vs, inv_norm;
    const uint16_t* img_e1;
    const uint16_t* img_e2;
    const float* b2;
    // forward: agg[r] += s * sum f (.) h[j]
    const uint16_t* h;
    float* agg;
    // backward (second round): dh[j] += s * f (.) g[r]
    const float* g;
    float* dh;
    // backward (first round + edge MLP)
    const float* g1;       // [n_recv,128]
    const float* g2;       // [n_recv,128]
    const uint16_t* h0;    // [n,128]
    const uint16_t* h2;    // [n,128]
    float* dh0;            // [n,128]
    float* partial;        // [grid][kBwdStride]
    int32_t* status;
    int early;             // inference: the weight images are copied before the previous kernel is done
};

constexpr uint32_t kImg16 = 128 * 16 * 2;   // 4 KB
constexpr uint32_t kImg128 = 128 * 128 * 2;  // 32 KB
// k_edges shared memory: the weight images once, then per pipeline an edge
// feature tile, the hidden-activation tile, receiver/sender ids and an mbarrier.
// The forward pass also stages the senders' latent rows (128 x 256 B); their
// copies are issued with layer 1 and land during it and its epilogue.
constexpr uint32_t EF_IMG1 = 0, EF_IMG2 = EF_IMG1 + kImg16, EF_B1 = EF_IMG2 + kImg128, EF_B2 = EF_B1 + 512,
                   EF_BARS = EF_B2 + 512, EF_SLOT = EF_BARS + 48, EF_PIPE = (EF_SLOT + 16 + 1023) / 1024 * 1024,
                   EF_P_XS = 0, EF_P_ZR = EF_P_XS + kImg16, EF_P_SR = EF_P_ZR + kImg128, EF_P_SJ = EF_P_SR + 512,
                   EF_P_END = EF_P_SJ + 512, EF_P_H = EF_P_END + 16;
template <int MODE>
struct EdgeSmem {
    static constexpr uint32_t pipe = EF_P_H + (MODE == MODE_AGG ? kImg128 : 0u), bytes = EF_PIPE + 2 * pipe;
    static constexpr int ctas = MODE == MODE_AGG ? 1 : 2;  // per SM
};
static_assert(EF_PIPE % 1024 == 0 && EF_P_H % 16 == 0, "k_edges shared memory alignment");
static_assert(EdgeSmem<MODE_AGG>::bytes <= 227 * 1024 && 2 * (EdgeSmem<MODE_SCATTER>::bytes + 1024) <= 228 * 1024,
              "k_edges shared memory");

struct EdgeLoad {
    int r, j;
    float4 pr, pj, vr, vj;
};

// Edge ids of edge e (-1 past the end); positions and velocities follow in
// edge_load_state, so the two dependent loads can be issued at different points.
__device__ __forceinline__ void edge_load_ids(const EdgeArgs& a, int e, int E, EdgeLoad& L) {
    L.r = -1;
    L.j = -1;
    if ((unsigned)e < (unsigned)E) {
        L.r = __ldg(a.receiver + e);
        L.j = __ldg(a.sender + e);
    }
}

__device__ __forceinline__ void edge_load_state(const EdgeArgs& a, EdgeLoad& L) {
    if (L.r >= 0) {
        L.pr = __ldg(a.pos + L.r);
        L.pj = __ldg(a.pos + L.j);
        L.vr = __ldg(a.vel + L.r);
        L.vj = __ldg(a.vel + L.j);
    }
}

// Edge features: ((x_j-x_i)/R, |x_j-x_i|/R, (v_j-v_i)/v_s, 1) as 8 BF16 values
// (zeros past the end); the other 8 input columns are zero.
__device__ __forceinline__ uint4 edge_pack(const EdgeArgs& a, const EdgeLoad& L) {
    if (L.r < 0) return make_uint4(0, 0, 0, 0);
    const float dx = L.pj.x - L.pr.x, dy = L.pj.y - L.pr.y, dz = L.pj.z - L.pr.z;
    const float dist = sqrtf(fmaf(dz, dz, fmaf(dx, dx, __fmul_rn(dy, dy))));  // the same bits in every kernel
    return make_uint4(pack2(dx * a.inv_r, dy * a.inv_r), pack2(dz * a.inv_r, dist * a.inv_r),
                      pack2((L.vj.x - L.vr.x) * a.inv_vs, (L.vj.y - L.vr.y) * a.inv_vs),
                      pack2((L.vj.z - L.vr.z) * a.inv_vs, 1.0f));
}

// Two independent pipelines of 8 warps per CTA (warps 0-7, 8-15), each owning
// TMEM columns [128 p, 128 p + 128): layer 1 lands there (lane = edge), is
// consumed by its epilogue, and layer 2 (lane = feature) overwrites it.  In
// both epilogues warps w and w + 4 of a pipeline read the same 32 TMEM lanes
// and split the 128 columns.  The next tile's edge features are built while
// layer 1 runs and written once it has read the current ones.  Aggregation
// copies the senders' latent rows into shared memory as soon as a tile's
// edges are known, which leaves room for one CTA per SM; it is bound by the
// waits between its MMAs and epilogues (509k edges: 62 us with 16-byte
// asynchronous copies by all threads, 64 us with a 256-byte bulk copy per
// edge and a barrier to wait on).  The scatter needs no rows, runs two
// CTAs per SM and is bound by its 4-byte atomic adds (one per edge and
// feature): 509k edges in 74 us, against 189 us with one CTA, the epilogue's
// columns indexed at run time (in local memory) and a load of the receiver's g
// waited for at each new receiver.  Aggregation without staged rows, two CTAs
// per SM: no faster.
constexpr int kPT = 256;  // threads per pipeline

// Barrier of one 256-thread pipeline (named barrier 1 or 2, immediate ids).
__device__ __forceinline__ void pipe_sync256(int id) {
    if (id == 1)
        asm volatile("bar.sync 1, 256;" ::: "memory");
    else
        asm volatile("bar.sync 2, 256;" ::: "memory");
}
__device__ __forceinline__ bool pipe_or256(bool v, int id) {
    uint32_t r;
    if (id == 1)
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "bar.red.or.pred q, 1, 256, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(r)
            : "r"((uint32_t)v)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "bar.red.or.pred q, 2, 256, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(r)
            : "r"((uint32_t)v)
            : "memory");
    return r != 0;
}

template <int MODE>
__global__ void __launch_bounds__(2 * kPT, EdgeSmem<MODE>::ctas) k_edges(EdgeArgs a) {
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t* img1 = sm + EF_IMG1;
    uint8_t* img2 = sm + EF_IMG2;
    float* b2 = reinterpret_cast<float*>(sm + EF_B2);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + EF_BARS);  // [0],[1] MMAs, [2] weights
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + EF_SLOT);
    const int tid = threadIdx.x, warp = tid >> 5, p = warp >> 3, plt = tid & (kPT - 1);
    const int wq = warp & 7, lanes = 32 * (wq & 3), half = wq >> 2;
    const int lt = plt & (kT - 1);  // TMEM lane of this thread
    const bool loader = plt < kT;
    uint8_t* pb = sm + EF_PIPE + p * EdgeSmem<MODE>::pipe;
    uint8_t* xs = pb + EF_P_XS;
    uint8_t* zr = pb + EF_P_ZR;
    int* sr = reinterpret_cast<int*>(pb + EF_P_SR);
    int* sj = reinterpret_cast<int*>(pb + EF_P_SJ);
    uint8_t* hs = pb + EF_P_H;  // [128 edges][128] BF16 sender rows
    uint64_t* bar = &bars[p];
    const int bid = 1 + p;
    if (tid == 0) {
        for (int b = 0; b < 3; ++b) mbar_init(&bars[b], 1);
        fence_mbar_init();
        if (a.early) {  // the weight images are fixed: copy them while the previous kernel drains
            mbar_arrive_expect_tx(&bars[2], kImg16 + kImg128);
            tma_load_1d(img1, a.img_e1, kImg16, &bars[2]);
            tma_load_1d(img2, a.img_e2, kImg128, &bars[2]);
        }
    }
    pdl_wait();
    pdl_launch();
    const int E = min(__ldg(a.offset + a.n_recv), a.cap);
    if (warp == 0) umma::tmem_alloc(slot, 256);
    if (tid < 128) b2[tid] = a.b2[tid];
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = *slot + 128u * p;
    if (tid == 0 && !a.early) {
        mbar_arrive_expect_tx(&bars[2], kImg16 + kImg128);
        tma_load_1d(img1, a.img_e1, kImg16, &bars[2]);
        tma_load_1d(img2, a.img_e2, kImg128, &bars[2]);
    }
    bool failed = __syncthreads_or(!mbar_wait(&bars[2], 0, kPolls));
    bool mine = true, pending = false;
    uint32_t phase = 0;
    constexpr uint32_t idesc = umma::idesc_bf16(128, 128);
    const int stride = 2 * gridDim.x;
    int tile = 2 * blockIdx.x + p;
    EdgeLoad nxt;  // ids of the next tile; its particle state until it is packed
    int r0 = -1, j0 = -1;
    nxt.r = nxt.j = -1;
    if (loader) {
        edge_load_ids(a, tile * kT + lt, E, nxt);
        edge_load_state(a, nxt);
        r0 = nxt.r;
        j0 = nxt.j;
        *reinterpret_cast<uint4*>(xs + tile_off(lt, 0, 16)) = edge_pack(a, nxt);
        *reinterpret_cast<uint4*>(xs + tile_off(lt, 8, 16)) = make_uint4(0, 0, 0, 0);
        edge_load_ids(a, (tile + stride) * kT + lt, E, nxt);
    }
    for (; !failed && tile * kT < E; tile += stride) {
        if (loader) {
            sr[lt] = r0;
            sj[lt] = j0;
        }
        fence_proxy_async_smem();
        umma::fence_before();
        pipe_sync256(bid);
        if (plt == 0) {
            umma::fence_after();
            umma::mma_tile(tmem, xs, img1, 16, idesc, false);  // D[e][k], layer-1 bias included
            umma::commit(bar);
        }
        if (loader) {
            if (MODE == MODE_AGG) {
                // edges after which the running sum is flushed: the last edge of a
                // receiver's run, and the last valid edge of each half-tile
                const int r = sr[lt];
                const bool flush = r >= 0 && (lt == kT - 1 || lt == kT / 2 - 1 || sr[lt + 1] != r);
                const unsigned m = __ballot_sync(0xffffffffu, flush);
                if ((lt & 31) == 0) reinterpret_cast<uint32_t*>(pb + EF_P_END)[lt >> 5] = m;
            } else {
                // first edges of the receivers' runs, and of each half-tile
                const int r = sr[lt];
                const bool start = r >= 0 && (lt == 0 || lt == kT / 2 || sr[lt - 1] != r);
                const unsigned m = __ballot_sync(0xffffffffu, start);
                if ((lt & 31) == 0) reinterpret_cast<uint32_t*>(pb + EF_P_END)[lt >> 5] = m;
            }
            edge_load_state(a, nxt);  // the next tile's particle state
        }
        if (MODE == MODE_AGG) {  // the senders' latent rows, 16 bytes a thread
            const int l = plt & 15;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = 16 * i + (plt >> 4), j = sj[e];
                if (j >= 0)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                     smem_u32(hs + e * 256 + 16 * l)),
                                 "l"(a.h + (size_t)j * kH + 8 * l)
                                 : "memory");
            }
        }
        pending = true;
        // A wait that gives up is reported at the pipeline's next barrier,
        // which then reduces the outcome (what is read meanwhile is discarded).
        mine = mbar_wait(bar, phase, kPolls);
        if (mine) {
            phase ^= 1u;
            pending = false;
        }
        umma::fence_after();
        if (loader && mine) {  // layer 1 has read its tile: the next one's edge features
            *reinterpret_cast<uint4*>(xs + tile_off(lt, 0, 16)) = edge_pack(a, nxt);
            r0 = nxt.r;
            j0 = nxt.j;
            edge_load_ids(a, (tile + 2 * stride) * kT + lt, E, nxt);
        }
        // layer-1 epilogue: lane = edge, this half's 64 hidden units
#pragma unroll
        for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 32) {
            float v[32];
            umma::tmem_ld32(umma::taddr(tmem, lanes, c0), v);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = c0 + 8 * q;
                uint4 w;
                w.x = pack2_relu(v[8 * q], v[8 * q + 1]);
                w.y = pack2_relu(v[8 * q + 2], v[8 * q + 3]);
                w.z = pack2_relu(v[8 * q + 4], v[8 * q + 5]);
                w.w = pack2_relu(v[8 * q + 6], v[8 * q + 7]);
                *reinterpret_cast<uint4*>(zr + tile_off(lt, k, 128)) = w;
            }
        }
        if (MODE == MODE_AGG) asm volatile("cp.async.wait_all;" ::: "memory");
        fence_proxy_async_smem();
        umma::fence_before();
        if (pipe_or256(!mine, bid)) { failed = true; break; }
        if (plt == 0) {
            umma::fence_after();
            umma::mma_tile(tmem, img2, zr, 128, idesc, false);  // D[c][e], over layer 1's columns
            umma::commit(bar);
        }
        float gnext = 0.0f;
        if (MODE == MODE_SCATTER && sr[64 * half] >= 0) gnext = __ldg(a.g + (size_t)sr[64 * half] * kH + lt);
        pending = true;
        mine = mbar_wait(bar, phase, kPolls);
        if (mine) {
            phase ^= 1u;
            pending = false;
        }
        umma::fence_after();
        // layer-2 epilogue: lane = feature c, this half's 64 edges of the tile
        const int c = lt;
        const float bc = b2[c];
        float gval = 0.0f;
        if (MODE == MODE_AGG) {
            const uint16_t* h16 = reinterpret_cast<const uint16_t*>(hs) + c;
            const uint32_t* ends = reinterpret_cast<const uint32_t*>(pb + EF_P_END);
            // Segmented sums over the receiver-sorted edges; a group of 8
            // edges that ends no run (most of them: ~30 edges per receiver)
            // runs without the per-edge flush tests.
            float acc = 0.0f;
#pragma unroll 1
            for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 32) {
                float v[32];
                umma::tmem_ld32(umma::taddr(tmem, lanes, c0), v);
                const uint32_t em = ends[c0 >> 5];  // warp-uniform: the same edges end a run for every feature
#pragma unroll
                for (int g = 0; g < 32; g += 8) {
                    if (((em >> g) & 0xffu) == 0u) {
#pragma unroll
                        for (int i = g; i < g + 8; ++i) acc = fmaf(v[i] + bc, bf(h16[(c0 + i) * kH]), acc);
                    } else {
#pragma unroll
                        for (int i = g; i < g + 8; ++i) {
                            const float t = fmaf(v[i] + bc, bf(h16[(c0 + i) * kH]), acc);
                            if (em & (1u << i)) {
                                atomicAdd(a.agg + (size_t)sr[c0 + i] * kH + c, t * a.inv_norm);
                                acc = 0.0f;
                            } else {
                                acc = t;
                            }
                        }
                    }
                }
            }
        } else {
            // Edges of one receiver follow each other: its g is read once, one
            // run ahead of its use.
            const uint32_t* first = reinterpret_cast<const uint32_t*>(pb + EF_P_END) + 2 * half;
            const unsigned long long starts = first[0] | (unsigned long long)first[1] << 32;
            const int valid = E - tile * kT - 64 * half;  // edges of this half-tile
            float* dhc = a.dh + c;
#pragma unroll 1
            for (int w = 0; w < 64 && w < valid; w += 8) {
                const int c0 = 64 * half + w;
                int j[8];
                *reinterpret_cast<int4*>(j) = *reinterpret_cast<const int4*>(sj + c0);
                *reinterpret_cast<int4*>(j + 4) = *reinterpret_cast<const int4*>(sj + c0 + 4);
                float v[8];
                umma::tmem_ld8(umma::taddr(tmem, lanes, c0), v);
                const uint32_t runs = (uint32_t)(starts >> w) & 0xffu;
                if (runs == 0u && w + 8 <= valid) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) atomicAdd(dhc + (size_t)j[i] * kH, (v[i] + bc) * gval);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (runs & (1u << i)) {
                            gval = gnext * a.inv_norm;
                            const unsigned long long later = starts >> (w + i) >> 1;
                            if (later) gnext = __ldg(a.g + (size_t)sr[c0 + i + __ffsll(later)] * kH + c);
                        }
                        if (j[i] >= 0) atomicAdd(dhc + (size_t)j[i] * kH, (v[i] + bc) * gval);
                    }
                }
            }
        }
        umma::fence_before();
        if (pipe_or256(!mine, bid)) { failed = true; break; }
    }
    if (failed && plt == 0) raise_flag(a.status, SPHDEM_FLAG_TIMEOUT);
    if (pending && !mine) mbar_wait(bar, phase, kPolls);
    umma::fence_before();
    __syncthreads();
    if (warp == 0) {
        umma::fence_after();
        umma::tmem_dealloc(*slot, 256);
    }
}

// k_edges_bwd shared memory.  Every operand is stored once, by the rows its
// epilogue owns, and enters its second product MN-major (umma.cuh): the hidden
// tile Z by edges, dF by features, dP by hidden units (over Z's space), the
// edge inputs by edges, W2 as the forward image.
constexpr uint32_t EB_IMG1 = 0, EB_IMG2 = EB_IMG1 + kImg16, EB_XS = EB_IMG2 + kImg128, EB_ZR = EB_XS + kImg16,
                   EB_DFT = EB_ZR + kImg128, EB_B2 = EB_DFT + kImg128, EB_SR = EB_B2 + 512, EB_SJ = EB_SR + 512,
                   EB_MASK = EB_SJ + 512, EB_START = EB_MASK + 2048, EB_BARS = EB_START + 16,
                   EB_SLOT = EB_BARS + 16, EB_BYTES = EB_SLOT + 16;
static_assert(2 * (EB_BYTES + 1024) <= 228 * 1024, "k_edges_bwd: two CTAs per SM");
constexpr int kBT = 512;  // threads: warps w, w + 4, w + 8, w + 12 share 32 TMEM lanes and split the 128 columns

// Backward of the first message round and of the edge MLP, per 128-edge tile:
// layer 1 and layer 2 again, dF = g1 h0 + g2 h2, the scatter of dh0, dW2 +=
// dF^T Z, dZ = W2^T dF^T, dP = dZ relu', dW1 += dP^T X.  What bounds it is the
// work between the MMAs (per edge and feature: the products, a 4-byte atomic
// add, two roundings), so it takes 4 threads per TMEM lane and two CTAs per SM
// that fill each other's waits, and reads eight senders' rows at a time and a
// receiver's g one run of edges ahead.  One thread per lane, one CTA per SM
// and transposed copies of Z, dF and X written element by element took 1,108
// us for 509k edges, an edge at a time 254 us; this form takes 188 us.
// TMEM columns: [0,128) layer 1, layer 2, dZ, then dW1 of the tile; [128,256) dW2.
__global__ void __launch_bounds__(kBT, 2) k_edges_bwd(EdgeArgs a) {
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t* img1 = sm + EB_IMG1;
    uint8_t* img2 = sm + EB_IMG2;
    uint8_t* xs = sm + EB_XS;
    uint8_t* zr = sm + EB_ZR;  // Z rows, then dP rows
    uint8_t* dft = sm + EB_DFT;
    float* b2 = reinterpret_cast<float*>(sm + EB_B2);
    int* sr = reinterpret_cast<int*>(sm + EB_SR);
    int* sj = reinterpret_cast<int*>(sm + EB_SJ);
    uint32_t* mask = reinterpret_cast<uint32_t*>(sm + EB_MASK);  // [hidden unit / 32][edge]: z > 0
    uint32_t* start = reinterpret_cast<uint32_t*>(sm + EB_START);  // bit per edge: the first of its receiver's
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + EB_BARS);
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + EB_SLOT);
    const int tid = threadIdx.x, warp = tid >> 5, lanes = 32 * (warp & 3), c0 = 32 * (warp >> 2);
    const int row = lanes + (tid & 31);  // TMEM lane: edge, feature or hidden unit
    const int E = min(__ldg(a.offset + a.n_recv), a.cap);

    const uint32_t tmem = cta_begin(bars, slot, 256);
    if (tid < 128) b2[tid] = a.b2[tid];
    if (tid == 0) {
        mbar_arrive_expect_tx(&bars[1], kImg16 + kImg128);
        tma_load_1d(img1, a.img_e1, kImg16, &bars[1]);
        tma_load_1d(img2, a.img_e2, kImg128, &bars[1]);
    }
    bool failed = __syncthreads_or(!mbar_wait(&bars[1], 0, kPolls));
    bool mine = true, pending = false, first = true;
    uint32_t phase = 0;
    constexpr uint32_t id128 = umma::idesc_bf16(128, 128), id16 = umma::idesc_bf16(128, 16);
    float db1 = 0.0f, db2 = 0.0f, w1[4] = {0.f, 0.f, 0.f, 0.f};
    EdgeLoad nxt;
    uint4 xin = make_uint4(0, 0, 0, 0);  // the next tile's edge features
    nxt.r = nxt.j = -1;
    if (tid < kT) {
        edge_load_ids(a, blockIdx.x * kT + tid, E, nxt);
        edge_load_state(a, nxt);
        xin = edge_pack(a, nxt);
    }
    for (int tile = blockIdx.x; !failed && tile * kT < E; tile += gridDim.x) {
        if (tid < kT) {
            sr[tid] = nxt.r;
            sj[tid] = nxt.j;
            *reinterpret_cast<uint4*>(xs + tile_off(tid, 0, 16)) = xin;
            *reinterpret_cast<uint4*>(xs + tile_off(tid, 8, 16)) = make_uint4(0, 0, 0, 0);
        }
        operands_ready();
        if (tid == 0) {
            umma::fence_after();
            umma::mma_tile(tmem, xs, img1, 16, id128, false);  // P[e][k]
            umma::commit(&bars[0]);
        }
        if (tid < kT) {
            // first edges of the receivers' runs, and of each 32 edges
            const int r = sr[tid];
            const unsigned m = __ballot_sync(0xffffffffu, r >= 0 && ((tid & 31) == 0 || sr[tid - 1] != r));
            if ((tid & 31) == 0) start[tid >> 5] = m;
            edge_load_ids(a, (tile + gridDim.x) * kT + tid, E, nxt);
        }
        pending = true;
        if (!mma_done(bars, phase, mine)) { failed = true; break; }
        pending = false;
        {  // lane = edge: Z row, z > 0
            float v[32];
            umma::tmem_ld32(umma::taddr(tmem, lanes, c0), v);
            uint32_t on = 0u;
#pragma unroll
            for (int i = 0; i < 32; ++i) on |= v[i] > 0.0f ? 1u << i : 0u;
            mask[(c0 >> 5) * kT + row] = on;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<uint4*>(zr + tile_off(row, c0 + 8 * q, 128)) =
                    make_uint4(pack2_relu(v[8 * q], v[8 * q + 1]), pack2_relu(v[8 * q + 2], v[8 * q + 3]),
                               pack2_relu(v[8 * q + 4], v[8 * q + 5]), pack2_relu(v[8 * q + 6], v[8 * q + 7]));
        }
        operands_ready();
        if (tid == 0) {
            umma::fence_after();
            umma::mma_tile(tmem, img2, zr, 128, id128, false);  // F[c][e]
            umma::commit(&bars[0]);
        }
        if (tid < kT) edge_load_state(a, nxt);
        float g1n = 0.0f, g2n = 0.0f;
        if (sr[c0] >= 0) {
            g1n = __ldg(a.g1 + (size_t)sr[c0] * kH + row);
            g2n = __ldg(a.g2 + (size_t)sr[c0] * kH + row);
        }
        pending = true;
        if (!mma_done(bars, phase, mine)) { failed = true; break; }
        pending = false;
        if (tid < kT) xin = edge_pack(a, nxt);
        {  // lane = feature: dF row, scatter of dh0, db2
            // Edges of one receiver follow each other: its g1, g2 are read
            // once, one run ahead of their use.
            const float bc = b2[row];
            const uint32_t sw = start[c0 >> 5];
            const int valid = E - tile * kT - c0;
            float g1v = 0.0f, g2v = 0.0f;
#pragma unroll 2
            for (int g = 0; g < 32; g += 8) {
                int jj[8];
                *reinterpret_cast<int4*>(jj) = *reinterpret_cast<const int4*>(sj + c0 + g);
                *reinterpret_cast<int4*>(jj + 4) = *reinterpret_cast<const int4*>(sj + c0 + g + 4);
                uint16_t h0v[8], h2v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const size_t at = (size_t)max(jj[i], 0) * kH + row;
                    h0v[i] = __ldg(a.h0 + at);
                    h2v[i] = __ldg(a.h2 + at);
                }
                float v[8];
                umma::tmem_ld8(umma::taddr(tmem, lanes, c0 + g), v);
                const uint32_t runs = (sw >> g) & 0xffu;
                if (runs == 0u && g + 8 <= valid) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        atomicAdd(a.dh0 + (size_t)jj[i] * kH + row, (v[i] + bc) * g1v);
                        v[i] = g1v * bf(h0v[i]) + g2v * bf(h2v[i]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (runs & (1u << i)) {
                            g1v = g1n * a.inv_norm;
                            g2v = g2n * a.inv_norm;
                            const uint32_t later = sw >> (g + i) >> 1;
                            if (later) {
                                const size_t at = (size_t)sr[c0 + g + i + __ffs(later)] * kH + row;
                                g1n = __ldg(a.g1 + at);
                                g2n = __ldg(a.g2 + at);
                            }
                        }
                        const bool on = g + i < valid;
                        if (on) atomicAdd(a.dh0 + (size_t)jj[i] * kH + row, (v[i] + bc) * g1v);
                        v[i] = on ? g1v * bf(h0v[i]) + g2v * bf(h2v[i]) : 0.0f;
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) db2 += v[i];
                *reinterpret_cast<uint4*>(dft + tile_off(row, c0 + g, 128)) =
                    make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
            }
        }
        operands_ready();
        if (tid == 0) {
            umma::fence_after();
            umma::mma_tile_mn(tmem + 128, dft, 0, zr, 128, 128, id128 | umma::kBMn, !first);  // dW2[c][k] += dF^T Z
            umma::mma_tile_mn(tmem, img2, 128, dft, 128, 128, id128 | umma::kAMn | umma::kBMn, false);  // dZ[k][e]
            umma::commit(&bars[0]);
        }
        pending = true;
        if (!mma_done(bars, phase, mine)) { failed = true; break; }
        pending = false;
        {  // lane = hidden unit: dP row, db1
            float v[32];
            umma::tmem_ld32(umma::taddr(tmem, lanes, c0), v);
            const uint4* on = reinterpret_cast<const uint4*>(mask + (warp & 3) * kT + c0);
            const uint32_t bit = 1u << (tid & 31);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint4 m = on[q];
                if (!(m.x & bit)) v[4 * q] = 0.0f;
                if (!(m.y & bit)) v[4 * q + 1] = 0.0f;
                if (!(m.z & bit)) v[4 * q + 2] = 0.0f;
                if (!(m.w & bit)) v[4 * q + 3] = 0.0f;
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) db1 += v[i];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<uint4*>(zr + tile_off(row, c0 + 8 * q, 128)) =
                    make_uint4(pack2(v[8 * q], v[8 * q + 1]), pack2(v[8 * q + 2], v[8 * q + 3]),
                               pack2(v[8 * q + 4], v[8 * q + 5]), pack2(v[8 * q + 6], v[8 * q + 7]));
        }
        operands_ready();
        if (tid == 0) {
            umma::fence_after();
            umma::mma_tile_mn(tmem, zr, 0, xs, 16, 128, id16 | umma::kBMn, false);  // dW1[k][in] of this tile
            umma::commit(&bars[0]);
        }
        pending = true;
        if (!mma_done(bars, phase, mine)) { failed = true; break; }
        pending = false;
        {
            float v[4];
            umma::tmem_ld4(umma::taddr(tmem, lanes, c0 >> 3), v);  // this thread's 4 of the 16 inputs
#pragma unroll
            for (int i = 0; i < 4; ++i) w1[i] += v[i];
        }
        first = false;
    }
    float* part = a.partial + (size_t)blockIdx.x * kBwdStride;
    __syncthreads();
    if (!failed) {
        float v[32];
        umma::tmem_ld32(umma::taddr(tmem + 128, lanes, c0), v);
#pragma unroll
        for (int i = 0; i < 32; ++i) part[row * 128 + c0 + i] = first ? 0.0f : v[i];
        const int in = c0 >> 3;
#pragma unroll
        for (int i = 0; i < 4; ++i) part[128 * 128 + row * 16 + in + i] = in + i < kBiasCol ? w1[i] : 0.0f;
        float* red = reinterpret_cast<float*>(dft);  // the four threads of a lane, in order
        red[tid] = db1;
        red[kBT + tid] = db2;
        __syncthreads();
        if (warp < 4) {
            part[128 * 128 + 128 * 16 + tid] = ((red[tid] + red[tid + 128]) + red[tid + 256]) + red[tid + 384];
            const float* r2 = red + kBT;
            part[128 * 128 + 128 * 16 + 128 + tid] = ((r2[tid] + r2[tid + 128]) + r2[tid + 256]) + r2[tid + 384];
        }
    }
    cta_end(bars, phase, pending && !mine, tmem, 256, a.status, failed);
}

// ---------------------------------------------------------------------------
// weight gradients of the node layers: C[128][N] = sum_r P[r][:]^T Q[r][:]
// ---------------------------------------------------------------------------
// Both operands are staged by rows (16-byte stores, 8 rows x 64 bytes per
// warp) and enter the product MN-major; 512 threads stage and read out.  With
// list, the rows are 0 .. n_direct - 1 and the list[0] rows list[1 ..], as in
// k_rows; n_rows bounds both.  80k rows: 53 us with one thread per row and
// transposed 2-byte stores; 27 us for the 29k rows that take part.
template <int N>
__global__ void __launch_bounds__(kRT * kT) k_wgrad(const uint16_t* __restrict__ P, const uint16_t* __restrict__ Q,
                                                    int n_rows, const int* __restrict__ list, int n_direct,
                                                    float* __restrict__ partial, int32_t* status) {
    constexpr uint32_t kA = 128 * 128 * 2, kB = N * 128 * 2;
    constexpr uint32_t kCols = N < 32 ? 32 : N;
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t* sA = sm;
    uint8_t* sB = sm + kA;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + kB);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lanes = 32 * (warp & 3), grp = warp >> 2;
    const uint32_t tmem = cta_begin(bars, slot, kCols);
    bool mine = true, failed = false, pending = false, first = true;
    uint32_t phase = 0;
    constexpr uint32_t idesc = umma::idesc_bf16(128, N) | umma::kAMn | umma::kBMn;
    const int rows = list ? min(n_rows, n_direct + __ldg(list)) : n_rows;
    auto stage = [&](uint8_t* to, const uint16_t* from, int chunk, int cols) {
        // (rows / 8) x (cols / 32) warp pieces of 8 rows x 4 16-byte words
        const int per = max(cols / 32, 1), words = cols / 8;
        for (int w = warp; w < 16 * per; w += kRT * 4) {
            const int r = 8 * (w / per) + (lane & 7), q = 4 * (w % per) + (lane >> 3);
            if (q >= words) continue;
            int row = chunk * kT + r;
            if (list && row >= n_direct) row = row < rows ? __ldg(list + 1 + (row - n_direct)) : n_rows;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (row < n_rows && chunk * kT + r < rows)
                v = __ldg(reinterpret_cast<const uint4*>(from + (size_t)row * cols) + q);
            *reinterpret_cast<uint4*>(to + tile_off(r, 8 * q, cols)) = v;
        }
    };
    for (int chunk = blockIdx.x; chunk * kT < rows; chunk += gridDim.x) {
        stage(sA, P, chunk, 128);
        stage(sB, Q, chunk, N);
        operands_ready();
        if (tid == 0) {
            umma::fence_after();
            umma::mma_tile_mn(tmem, sA, 128, sB, N, 128, idesc, !first);
            umma::commit(&bars[0]);
        }
        pending = true;
        if (!mma_done(bars, phase, mine)) { failed = true; break; }
        pending = false;
        first = false;
    }
    if (!failed) {
        float* part = partial + (size_t)blockIdx.x * 128 * N + (lanes + lane) * N;
        if (N < 32) {
            float v[4];
            umma::tmem_ld4(umma::taddr(tmem, lanes, 4 * grp), v);
#pragma unroll
            for (int i = 0; i < 4; ++i) part[4 * grp + i] = first ? 0.0f : v[i];
        } else {
            float v[32];
            umma::tmem_ld32(umma::taddr(tmem, lanes, 32 * grp), v);
#pragma unroll
            for (int i = 0; i < 32; ++i) part[32 * grp + i] = first ? 0.0f : v[i];
        }
    }
    cta_end(bars, phase, pending && !mine, tmem, kCols, status, failed);
}

// Sums of per-CTA partials, in a fixed order: segment s is `count` sums over n
// partials of `stride` floats at src, written to dst (transposed from
// [rows_t][cols_t] when rows_t > 0).  A CTA takes 32 sums; its 8 warps each add
// every eighth partial (a thread that adds all of them waits for one load
// after another: 15 us per segment; all ten segments take 12 us now).
struct Segment {
    const float* src;
    float* dst;
    int n, stride, count, rows_t, cols_t;
};
constexpr int kSegments = 10;
struct Segments {
    Segment s[kSegments];
    int n;
};
__global__ void __launch_bounds__(256) k_reduce(Segments g) {
    __shared__ float red[8][32];
    int b = blockIdx.x, k = 0;
    while (k < g.n && b >= (g.s[k].count + 31) / 32) b -= (g.s[k++].count + 31) / 32;
    if (k >= g.n) return;
    const Segment s = g.s[k];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = 32 * b + lane;
    float t = 0.0f;
    if (i < s.count) {
#pragma unroll 8
        for (int p = w; p < s.n; p += 8) t += s.src[(size_t)p * s.stride + i];
    }
    red[w][lane] = t;
    __syncthreads();
    if (w != 0 || i >= s.count) return;
#pragma unroll
    for (int p = 1; p < 8; ++p) t += red[p][lane];
    s.dst[s.rows_t > 0 ? (i % s.cols_t) * s.rows_t + i / s.cols_t : i] = t;
}

// ---------------------------------------------------------------------------
// elementwise pieces
// ---------------------------------------------------------------------------
// Row of index i in the node order of k_rows: 0 .. n_direct - 1, then the list.
__device__ __forceinline__ int node_row(int i, int n_direct, const int* __restrict__ list) {
    return list && i >= n_direct ? __ldg(list + 1 + (i - n_direct)) : i;
}

// Sum over the 8 row groups of a CTA of 256 threads (32 threads x 4 columns
// each), written to part[blockIdx.x * cols ..].
__device__ __forceinline__ void store_colsum(float4 s, int cols, float* __restrict__ part) {
    __shared__ float4 red[8][32];
    const int t = threadIdx.x & 31, g = threadIdx.x >> 5;
    red[g][t] = s;
    __syncthreads();
    if (g != 0 || 4 * t >= cols) return;
#pragma unroll
    for (int k = 1; k < 8; ++k) {
        const float4 o = red[k][t];
        s = make_float4(s.x + o.x, s.y + o.y, s.z + o.z, s.w + o.w);
    }
    float* to = part + (size_t)blockIdx.x * cols + 4 * t;  // the caller's scratch: any alignment
    to[0] = s.x;
    to[1] = s.y;
    to[2] = s.z;
    to[3] = s.w;
}

// out = d * silu'(z) as BF16 and its column sums (one partial row per CTA), for
// the node rows of the layer.
__global__ void __launch_bounds__(256) k_act_grad(const float* __restrict__ d, const float* __restrict__ z, int n_rows,
                                                  const int* __restrict__ list, int n_direct,
                                                  uint16_t* __restrict__ out, float* __restrict__ part) {
    const int rows = list ? min(n_rows, n_direct + __ldg(list)) : n_rows;
    const int t = threadIdx.x & 31;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < rows; i += gridDim.x * 8) {
        const size_t at = (size_t)node_row(i, n_direct, list) * kH / 4 + t;
        const float4 dv = reinterpret_cast<const float4*>(d)[at], zv = reinterpret_cast<const float4*>(z)[at];
        const float4 v = make_float4(dv.x * silu_grad(zv.x), dv.y * silu_grad(zv.y), dv.z * silu_grad(zv.z),
                                     dv.w * silu_grad(zv.w));
        reinterpret_cast<uint2*>(out)[at] = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
        s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
    }
    store_colsum(s, kH, part);
}

// The output gradient [n][16]: BF16 copy and column sums; zeroes the gradient
// rows dh of the nodes that only send (the scatter adds to them).
__global__ void __launch_bounds__(256) k_out_grad(const float* __restrict__ d, int n, uint16_t* __restrict__ out,
                                                  float* __restrict__ part, float* __restrict__ dh, int n_nodes,
                                                  const int* __restrict__ list) {
    const int t = threadIdx.x & 31, g = threadIdx.x >> 5;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < 4)
        for (int i = blockIdx.x * 8 + g; i < n; i += gridDim.x * 8) {
            const float* q = d + (size_t)i * 16 + 4 * t;  // the caller's: any alignment
            const float4 v = make_float4(q[0], q[1], q[2], q[3]);
            reinterpret_cast<uint2*>(out)[(size_t)i * 4 + t] = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
            s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
        }
    const int rows = list ? min(n_nodes, n + __ldg(list)) : n_nodes;
    for (int i = n + blockIdx.x * 8 + g; i < rows; i += gridDim.x * 8)
        reinterpret_cast<float4*>(dh)[(size_t)node_row(i, n, list) * kH / 4 + t] = make_float4(0.f, 0.f, 0.f, 0.f);
    store_colsum(s, 16, part);
}

// Loss and its gradient: one cluster of 8 CTAs (16,759 rows: 9.6 us; one CTA
// took 122), whose sums meet in the first CTA's shared memory in a fixed order.
constexpr int kLossCtas = 8;
__global__ void __cluster_dims__(kLossCtas, 1, 1) __launch_bounds__(1024)
    k_loss(const float* __restrict__ out, const float* __restrict__ target, int n, float* __restrict__ loss,
           float* __restrict__ d_out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    cluster_started();
    __shared__ float red[32];
    __shared__ float sums[kLossCtas];
    const float inv = n > 0 ? 1.0f / (6.0f * (float)n) : 0.0f;
    float s = 0.0f;
    for (long i = blockIdx.x * 1024L + threadIdx.x; i < (long)n * 16; i += kLossCtas * 1024L) {
        float g = 0.0f;
        if ((i & 15) < 6) {
            const float d = out[i] - target[i];
            s += d * d;
            g = 2.0f * d * inv;
        }
        d_out[i] = g;
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    cluster_wait_started();  // the first CTA's shared memory is written next
    if (threadIdx.x < 32) {
        const float t = warp_sum(red[threadIdx.x]);
        if (threadIdx.x == 0) cluster.map_shared_rank(sums, 0)[cluster.block_rank()] = t;
    }
    cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x == 0) {
        float t = 0.0f;
        for (int k = 0; k < kLossCtas; ++k) t += sums[k];
        *loss = t * inv;
    }
}

// Edge term of the loss: lambda / E * sum over edges (i <- j) of
// |dx_i - dx_j|^2, dx = out[:, 0:3] - target[:, 0:3] (senders that are not
// receivers do not move: dx_j = 0).  Adds its gradient to d_out and its value
// to *loss (atomics: the order of the FP32 additions is not fixed).
__global__ void k_edge_loss(const int* __restrict__ offset, const int* __restrict__ sender,
                            const int* __restrict__ receiver, int n_recv, int cap, const float* __restrict__ out,
                            const float* __restrict__ target, float lambda, float* __restrict__ d_out,
                            float* __restrict__ loss) {
    const int E = min(offset[n_recv], cap);
    const float w = E > 0 ? lambda / (float)E : 0.0f;
    float part = 0.0f;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += gridDim.x * blockDim.x) {
        const int i = receiver[e], j = sender[e];
        const bool jr = j < n_recv;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float di = out[16 * i + d] - target[16 * i + d];
            const float dj = jr ? out[16 * j + d] - target[16 * j + d] : 0.0f;
            const float g = di - dj;
            part += g * g;
            atomicAdd(d_out + 16 * i + d, 2.0f * w * g);
            if (jr) atomicAdd(d_out + 16 * j + d, -2.0f * w * g);
        }
    }
    part = warp_sum(part * w);
    if ((threadIdx.x & 31) == 0 && part != 0.0f) atomicAdd(loss, part);
}

__global__ void k_adam(float* __restrict__ th, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    th[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
}

struct ApplyArgs {
    float* pos[2];
    float* vel[2];
    const float* acc[2];
    int n[2];
    const float* out;
    int m;
    float dt;
    float sx[2], sv[2];
    const float* x_t;
    const float* v_t;
    float* target;
};

__global__ void k_apply(ApplyArgs a) {
    pdl_wait();
    pdl_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n[0] + a.n[1]) return;
    const int s = i < a.n[0] ? 0 : 1;
    const int k = s ? i - a.n[0] : i;
    const float m = (float)a.m, dt = a.dt;
    const float cx = 0.5f * dt * dt * m * (m + 1.0f), cv = m * dt;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float x = a.pos[s][3 * k + d], v = a.vel[s][3 * k + d], acc = a.acc[s][3 * k + d];
        const float px = x + cv * v + cx * acc;  // prior: m substeps at constant acceleration
        const float pv = v + cv * acc;
        if (a.target) {
            a.target[16 * i + d] = (a.x_t[3 * i + d] - px) / a.sx[s];
            a.target[16 * i + 3 + d] = (a.v_t[3 * i + d] - pv) / a.sv[s];
        } else {
            a.pos[s][3 * k + d] = px + a.sx[s] * a.out[16 * i + d];
            a.vel[s][3 * k + d] = pv + a.sv[s] * a.out[16 * i + 3 + d];
        }
    }
    if (a.target) {
#pragma unroll
        for (int d = 6; d < 16; ++d) a.target[16 * i + d] = 0.0f;
    }
}

__global__ void k_maxdev(const float* __restrict__ a, const float* __restrict__ b, float ref, int n, float inv,
                         float* __restrict__ out) {
    pdl_wait();
    pdl_launch();
    float m = 0.0f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        m = fmaxf(m, fabsf(a[i] - (b ? b[i] : ref)) * inv);
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(reinterpret_cast<int*>(out), __float_as_int(m));
}

// ---------------------------------------------------------------------------
// node inputs and the radius graph
// ---------------------------------------------------------------------------
__global__ void k_nodes(sphdem_mpnn_nodes_t a) {
    pdl_wait();
    pdl_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nf = a.n_fluid, nd = a.n_dem, nb = a.n_wall, nw = a.n_dem_wall;
    if (i >= nf + nd + nb + nw) return;
    float p[3], v[3] = {0, 0, 0}, ac[3] = {0, 0, 0};
    float rho = 0.0f, por = 0.0f, rad = 0.0f;
    int type;
    if (i < nf) {
        type = 0;
        for (int d = 0; d < 3; ++d) {
            p[d] = a.f_pos[3 * i + d];
            v[d] = a.f_vel[3 * i + d];
            ac[d] = a.f_acc[3 * i + d];
        }
        rho = (a.f_rho[i] / a.rho0 - 1.0f) * 100.0f;
        por = a.f_por[i] - 1.0f;
    } else if (i < nf + nd) {
        type = 1;
        const int k = i - nf;
        for (int d = 0; d < 3; ++d) {
            p[d] = a.d_pos[3 * k + d];
            v[d] = a.d_vel[3 * k + d];
            ac[d] = a.d_acc[3 * k + d];
        }
        rad = a.d_rad[k] * a.inv_radius;
    } else if (i < nf + nd + nb) {
        type = 2;
        const int k = i - nf - nd;
        for (int d = 0; d < 3; ++d) p[d] = a.b_pos[3 * k + d];
        rho = (a.b_rho[k] / a.rho0 - 1.0f) * 100.0f;
    } else {
        type = 3;
        const int k = i - nf - nd - nb;
        for (int d = 0; d < 3; ++d) p[d] = a.w_pos[3 * k + d];
        rad = a.w_rad[k] * a.inv_radius;
    }
    for (int d = 0; d < 3; ++d) a.node_pos3[3 * i + d] = p[d];
    reinterpret_cast<float4*>(a.node_pos4)[i] = make_float4(p[0], p[1], p[2], 0.0f);
    reinterpret_cast<float4*>(a.node_vel4)[i] = make_float4(v[0], v[1], v[2], 0.0f);
    float f[16] = {v[0] * a.inv_vscale, v[1] * a.inv_vscale, v[2] * a.inv_vscale, ac[0] * a.inv_ascale,
                   ac[1] * a.inv_ascale, ac[2] * a.inv_ascale, rho, por, 0, 0, 0, 0, rad, 0, 0, 0};
    f[8 + type] = 1.0f;
    uint4* o = reinterpret_cast<uint4*>(a.x + (size_t)i * 16);
    o[0] = make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
    o[1] = make_uint4(pack2(f[8], f[9]), pack2(f[10], f[11]), pack2(f[12], f[13]), pack2(f[14], f[15]));
}

// One warp per receiver: the lanes test 32 candidate slots at a time (ranges
// of the ball-trimmed cell columns, in column order); accepted senders are
// compacted in slot order by ballot, so the list is deterministic.
template <bool FILL>
__global__ void k_graph(Geo g, const float4* __restrict__ pos, int n_recv, float r2, float rq, int* __restrict__ offset,
                        int* __restrict__ sender, int* __restrict__ receiver, int cap, sphdem_ctl_t* ctl) {
    pdl_wait();
    pdl_launch();
    const int i = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= n_recv) return;  // warp-uniform
    const float4 p = __ldg(pos + i);
    const int inst = inst_of(g, i);
    const int base = FILL ? offset[i] : 0;
    const unsigned below = (1u << lane) - 1u;
    int cnt = 0;
    warp_ranges_ball(g, p.x, p.y, p.z, rq, inst, [&](int s, int e) {
        for (int k0 = s; k0 < e; k0 += 32) {
            const int k = k0 + lane;
            bool in = false;
            int j = -1;
            if (k < e) {
                j = __ldg(g.order + k);
                if (j != i) {
                    const float4 q = __ldg(pos + j);
                    in = d2_exact(p.x, p.y, p.z, q.x, q.y, q.z).d2 < r2;
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (FILL && in) {
                const int slot = base + cnt + __popc(m & below);
                if (slot < cap) {
                    sender[slot] = j;
                    receiver[slot] = i;
                }
            }
            cnt += __popc(m);
        }
    });
    if (lane == 0) {
        if (!FILL) offset[i] = cnt;
        else if (i == n_recv - 1 && base + cnt > cap) flag(ctl, SPHDEM_FLAG_ROW_OVERFLOW);
    }
}

// ---------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------
int sm_count() {
    static int n[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (n[dev] == 0) {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        n[dev] = v > 0 ? v : 1;
    }
    return n[dev];
}

// Opt a kernel into `bytes` of dynamic shared memory (once per kernel and device).
template <class Kern>
int smem_opt_in(Kern k, uint32_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, uint32_t> done;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_pair(reinterpret_cast<const void*>(k), dev);
    std::lock_guard<std::mutex> lock(mu);
    auto it = done.find(key);
    if (it != done.end() && it->second >= bytes) return SPHDEM_OK;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) {
        set_error("mpnn: shared memory opt-in", e);
        return SPHDEM_ERR_CUDA;
    }
    done[key] = bytes;
    return SPHDEM_OK;
}

template <int K, int N, int EPI, bool IMG>
int rows(const uint16_t* A, int M, const uint16_t* B, const float* bias, float* out_f32, uint16_t* out_bf,
         float* z_out, int32_t* status, cudaStream_t st, float* add = nullptr, int n_add = 0, bool clear = false,
         const int* list = nullptr, int n_direct = 0, int early = 0, uint16_t* a_out = nullptr) {
    if (M <= 0) return SPHDEM_OK;
    constexpr uint32_t bytes = N * K * 2 + kT * K * 2 + 4 * (N < 2 ? 2 : N) + 16 + 16;
    int rc = smem_opt_in(k_rows<K, N, EPI, IMG>, bytes);
    if (rc) return rc;
    const int tiles = (M + kT - 1) / kT;
    const int grid = tiles < 2 * sm_count() ? tiles : 2 * sm_count();
    launch_pdl(k_rows<K, N, EPI, IMG>, grid, kRT * kT, bytes, st, A, M, add, n_add, clear, B, bias, out_f32, out_bf, z_out, status,
               list, n_direct, early, a_out);
    return launch_status("mpnn rows");
}

template <int N>
int wgrad(const uint16_t* P, const uint16_t* Q, int n_rows, float* partial, int& ncta, int32_t* status,
          cudaStream_t st, const int* list = nullptr, int n_direct = 0) {
    constexpr uint32_t bytes = 128 * 128 * 2 + N * 128 * 2 + 16 + 16;
    int rc = smem_opt_in(k_wgrad<N>, bytes);
    if (rc) return rc;
    const int chunks = (n_rows + kT - 1) / kT;
    ncta = chunks < 1 ? 1 : chunks;
    if (ncta > sm_count()) ncta = sm_count();
    if (ncta > kMaxCtas) ncta = kMaxCtas;
    k_wgrad<N><<<ncta, kRT * kT, bytes, st>>>(P, Q, n_rows, list, n_direct, partial, status);
    return launch_status("mpnn wgrad");
}

void add_segment(Segments& g, const float* src, int n, int stride, int count, float* dst, int rows_t = 0,
                 int cols_t = 0) {
    g.s[g.n++] = {src, dst, n, stride, count, rows_t, cols_t};
}

int reduce(const Segments& g, cudaStream_t st) {
    int blocks = 0;
    for (int k = 0; k < g.n; ++k) blocks += (g.s[k].count + 31) / 32;
    if (blocks > 0) k_reduce<<<blocks, 256, 0, st>>>(g);
    return launch_status("mpnn reduce");
}

EdgeArgs edge_args(const sphdem_mpnn_net_t* n) {
    EdgeArgs a;
    memset(&a, 0, sizeof(a));
    a.pos = reinterpret_cast<const float4*>(n->node_pos4);
    a.vel = reinterpret_cast<const float4*>(n->node_vel4);
    a.offset = n->offset;
    a.sender = n->sender;
    a.receiver = n->receiver;
    a.n_recv = n->n_recv;
    a.cap = n->edge_capacity;
    a.inv_r = n->inv_radius;
    a.inv_vs = n->inv_vscale;
    a.inv_norm = n->inv_norm;
    a.img_e1 = n->packed + P_E1;
    a.img_e2 = n->packed + P_E2;
    a.b2 = n->theta + SPHDEM_MPNN_E2_B;
    a.status = n->status;
    return a;
}

int edge_grid(const sphdem_mpnn_net_t* n, int per_sm) {
    const long tiles = ((long)n->edge_capacity + kT - 1) / kT;
    long g = (long)per_sm * sm_count();
    if (g > tiles) g = tiles;
    if (g > kMaxCtas) g = kMaxCtas;
    return g < 1 ? 1 : (int)g;
}

template <int MODE>
int edges(const EdgeArgs& a, int grid, cudaStream_t st) {
    int rc = smem_opt_in(k_edges<MODE>, EdgeSmem<MODE>::bytes);
    if (rc) return rc;
    launch_pdl(k_edges<MODE>, grid, 2 * kPT, EdgeSmem<MODE>::bytes, st, a);
    return launch_status("mpnn edges");
}

// The rows of these buffers are moved 16 bytes at a time.
bool aligned16(std::initializer_list<const void*> buffers) {
    uintptr_t bits = 0;
    for (const void* p : buffers) bits |= (uintptr_t)p;
    if (bits & 15u) set_error_msg("mpnn: row buffers must be 16-byte aligned");
    return (bits & 15u) == 0;
}

bool net_ok(const sphdem_mpnn_net_t* n) {
    return n && n->n_nodes >= n->n_recv && n->n_recv >= 0 && n->edge_capacity > 0 && n->node_pos4 &&
           n->node_vel4 && n->x && n->offset && n->sender && n->receiver && n->theta && n->packed && n->h0 &&
           n->agg && n->h1 && n->h2 && n->h3 && n->out;
}

}  // namespace
}  // namespace sd

using namespace sd;

extern "C" int64_t sphdem_mpnn_partial_floats(void) { return (int64_t)kMaxCtas * kBwdStride; }

extern "C" int sphdem_mpnn_pack(const float* theta, uint16_t* packed, sphdem_stream_t stream) {
    if (!theta || !packed) {
        set_error_msg("mpnn_pack: NULL pointer");
        return SPHDEM_ERR_INVALID;
    }
    k_pack<<<dim3(128, 8), 128, 0, as_stream(stream)>>>(theta, packed);
    return launch_status("mpnn_pack");
}

extern "C" int sphdem_mpnn_nodes(const sphdem_mpnn_nodes_t* in, sphdem_stream_t stream) {
    if (!in || !in->node_pos3 || !in->node_pos4 || !in->node_vel4 || !in->x) {
        set_error_msg("mpnn_nodes: NULL pointer");
        return SPHDEM_ERR_INVALID;
    }
    const long n = (long)in->n_fluid + in->n_dem + in->n_wall + in->n_dem_wall;
    if (n <= 0) return SPHDEM_OK;
    launch_pdl(k_nodes, blocks_for(n, 256), 256, 0, as_stream(stream), *in);
    return launch_status("mpnn_nodes");
}

extern "C" int sphdem_mpnn_graph(sphdem_grid_t* grid, const float* node_pos3, const float* node_pos4, int32_t n_recv,
                                 float radius, int32_t* offset, int32_t* sender, int32_t* receiver,
                                 int32_t edge_capacity, int32_t* scan_scratch, sphdem_ctl_t* ctl,
                                 sphdem_stream_t stream) {
    if (!grid || !node_pos3 || !node_pos4 || !offset || !sender || !receiver || !scan_scratch || n_recv < 0 ||
        n_recv > grid->n || !(radius > 0.0f) || edge_capacity <= 0 || grid->cell < radius) {
        set_error_msg("mpnn_graph: invalid arguments (cell must be >= radius, n_recv <= nodes)");
        return SPHDEM_ERR_INVALID;
    }
    cudaStream_t st = as_stream(stream);
    int rc = build_grid(grid, node_pos3, ctl, st);
    if (rc) return rc;
    if (n_recv == 0) {
        cudaError_t e = cudaMemsetAsync(offset, 0, sizeof(int32_t), st);
        if (e != cudaSuccess) {
            set_error("mpnn_graph", e);
            return SPHDEM_ERR_CUDA;
        }
        return SPHDEM_OK;
    }
    const Geo g = make_geo(*grid);
    const float r2 = radius * radius;
    const float rq = pad_radius(radius);
    const float4* p4 = reinterpret_cast<const float4*>(node_pos4);
    const int nb = blocks_for((long)n_recv * 32, 256);
    launch_pdl(k_graph<false>, nb, 256, 0, st, g, p4, n_recv, r2, rq, offset, sender, receiver, edge_capacity, ctl);
    rc = scan_counts(offset, n_recv, scan_scratch, st);
    if (rc) return rc;
    launch_pdl(k_graph<true>, nb, 256, 0, st, g, p4, n_recv, r2, rq, offset, sender, receiver, edge_capacity, ctl);
    return launch_status("mpnn_graph");
}

namespace sd {
namespace {
// Before a forward pass: sender flags, the length of their list (if there is
// one) and the aggregation sums of the first round.
__global__ void k_clear(int* __restrict__ active, int n_nodes, int* __restrict__ list, float4* __restrict__ agg,
                        long n_agg) {
    pdl_wait();
    pdl_launch();
    const long i0 = blockIdx.x * (long)blockDim.x + threadIdx.x, stride = (long)gridDim.x * blockDim.x;
    if (list && i0 == 0) list[0] = 0;
    for (long i = i0; i < n_nodes; i += stride) active[i] = 0;
    for (long i = i0; i < n_agg; i += stride) agg[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}
// Non-receiver senders of the current graph, each listed once: list[0] is
// their count, list[1 ..] the nodes (order immaterial: node rows are
// independent).  Edge count from the CSR offsets, bounded by the edge buffer
// (an overflowing graph keeps its full count there but only `cap` edges).
__global__ void k_mark_senders(const int* __restrict__ offset, const int* __restrict__ sender, int n_recv,
                               int n_nodes, int cap, int* __restrict__ active, int* __restrict__ list) {
    pdl_wait();
    pdl_launch();
    const int E = min(__ldg(offset + n_recv), cap);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += gridDim.x * blockDim.x) {
        const int s = __ldg(sender + e);
        if (s >= n_recv && s < n_nodes && atomicExch(active + s, 1) == 0) list[1 + atomicAdd(list, 1)] = s;
    }
}
}  // namespace
}  // namespace sd

extern "C" int sphdem_mpnn_forward(const sphdem_mpnn_net_t* n, int store_pre, sphdem_stream_t stream) {
    if (!net_ok(n) || (store_pre && (!n->z0 || !n->z2))) {
        set_error_msg("mpnn_forward: invalid network state");
        return SPHDEM_ERR_INVALID;
    }
    if (!aligned16({n->x, n->h0, n->agg, n->h1, n->h2, n->h3, n->out}) || (store_pre && !aligned16({n->z0, n->z2})))
        return SPHDEM_ERR_INVALID;
    cudaStream_t st = as_stream(stream);
    const int nn = n->n_nodes, nr = n->n_recv;
    // node layers on the receivers and the other nodes that send (no other
    // node's rows are read, and none has a gradient)
    const int* list = nullptr;
    const bool listed = n->active && n->active_list && nn > nr;
    launch_pdl(k_clear, 4 * sm_count(), 256, 0, st, n->active, listed ? nn : 0, listed ? n->active_list : nullptr,
               reinterpret_cast<float4*>(n->agg), (long)nr * (kH / 4));
    if (listed) {
        launch_pdl(k_mark_senders, 2 * sm_count(), 256, 0, st, n->offset, n->sender, nr, nn, n->edge_capacity,
                   n->active, n->active_list);
        list = n->active_list;
    }
    int rc = rows<16, 128, EPI_SILU, true>(n->x, nn, n->packed + P_N1, n->theta + SPHDEM_MPNN_N1_B, nullptr, n->h0,
                                           store_pre ? n->z0 : nullptr, n->status, st, nullptr, 0, false, list, nr,
                                           list != nullptr && !store_pre);
    if (rc) return rc;
    // Inference copies the weight images early: every kernel of the chain
    // runs behind kernels that do not write them (the first node layer only
    // behind the sender marking, which itself waits on whatever packed them).
    EdgeArgs a = edge_args(n);
    a.early = !store_pre;
    const int eg = edge_grid(n, 1);
    for (int round = 0; round < 2; ++round) {
        a.h = round == 0 ? n->h0 : n->h2;
        a.agg = n->agg;
        if (nr > 0 && (rc = edges<MODE_AGG>(a, eg, st))) return rc;
        if (round == 0)  // h1 = h0 + agg formed while staging (the backward pass reads it)
            if ((rc = rows<128, 128, EPI_SILU, true>(n->h0, nn, n->packed + P_N2, n->theta + SPHDEM_MPNN_N2_B, nullptr,
                                                     n->h2, store_pre ? n->z2 : nullptr, n->status, st, n->agg, nr,
                                                     true, list, nr, !store_pre, store_pre ? n->h1 : nullptr)))
                return rc;
    }
    rc = rows<128, 16, EPI_F32, true>(n->h2, nr, n->packed + P_N3, n->theta + SPHDEM_MPNN_N3_B, n->out, nullptr, nullptr,
                                      n->status, st, n->agg, nr, false, nullptr, 0, !store_pre, store_pre ? n->h3 : nullptr);
    if (rc) return rc;
    return launch_status("mpnn_forward");
}

extern "C" int sphdem_mpnn_backward(const sphdem_mpnn_net_t* n, const sphdem_mpnn_grad_t* g,
                                    sphdem_stream_t stream) {
    if (!net_ok(n) || !n->z0 || !n->z2 || !g || !g->d_out || !g->g2 || !g->d_h2 || !g->d_h1 || !g->d_h0 ||
        !g->bf_a || !g->bf_b || !g->partial || !g->grad) {
        set_error_msg("mpnn_backward: invalid arguments");
        return SPHDEM_ERR_INVALID;
    }
    if (!aligned16({n->x, n->h0, n->h1, n->h2, n->h3, n->z0, n->z2, g->g2, g->d_h2, g->d_h1, g->d_h0, g->bf_a, g->bf_b}))
        return SPHDEM_ERR_INVALID;
    cudaStream_t st = as_stream(stream);
    const int nn = n->n_nodes, nr = n->n_recv;
    // the node rows of the forward pass
    const int* list = n->active && n->active_list && nn > nr ? n->active_list : nullptr;
    float* grad = g->grad;
    int ncta = 0, rc;
    // every kernel below leaves per-CTA partials at a place of its own; one
    // launch at the end sums them all
    Segments sums;
    sums.n = 0;
    float* part = g->partial;
    const float* const end = part + (size_t)kMaxCtas * kBwdStride;
    const int bg = edge_grid(n, 2), cg = min(2 * sm_count(), kMaxCtas);
    if (part + (size_t)bg * kBwdStride + (size_t)sm_count() * 128 * (16 + 128 + 16) + (size_t)cg * (16 + 128 + 128) > end) {
        set_error_msg("mpnn_backward: partials larger than their buffer");
        return SPHDEM_ERR_INVALID;
    }
    auto take = [&](int n_part, int stride) {
        float* p = part;
        part += (size_t)n_part * stride;
        return p;
    };
    // output layer
    float* p = take(cg, 16);
    k_out_grad<<<cg, 256, 0, st>>>(g->d_out, nr, g->bf_b, p, g->d_h2, nn, list);
    add_segment(sums, p, cg, 16, 16, grad + SPHDEM_MPNN_N3_B);
    if ((rc = wgrad<16>(n->h3, g->bf_b, nr, part, ncta, n->status, st))) return rc;
    add_segment(sums, take(ncta, 128 * 16), ncta, 128 * 16, 128 * 16, grad + SPHDEM_MPNN_N3_W, 128, 16);
    // second message round: d_h2 = g2 on the receivers, + the scatter
    if ((rc = rows<16, 128, EPI_F32, true>(g->bf_b, nr, n->packed + P_N3T, nullptr, g->g2, nullptr, g->d_h2,
                                           n->status, st)))
        return rc;
    EdgeArgs a = edge_args(n);
    a.g = g->g2;
    a.dh = g->d_h2;
    if (nr > 0 && (rc = edges<MODE_SCATTER>(a, edge_grid(n, EdgeSmem<MODE_SCATTER>::ctas), st))) return rc;
    // second node layer
    p = take(cg, 128);
    k_act_grad<<<cg, 256, 0, st>>>(g->d_h2, n->z2, nn, list, nr, g->bf_a, p);
    add_segment(sums, p, cg, 128, 128, grad + SPHDEM_MPNN_N2_B);
    if ((rc = wgrad<128>(g->bf_a, n->h1, nn, part, ncta, n->status, st, list, nr))) return rc;
    add_segment(sums, take(ncta, 128 * 128), ncta, 128 * 128, 128 * 128, grad + SPHDEM_MPNN_N2_W);
    // first message round and the edge MLP: d_h0 = d_h1, + the scatter
    if ((rc = rows<128, 128, EPI_F32, true>(g->bf_a, nn, n->packed + P_N2T, nullptr, g->d_h1, nullptr, g->d_h0,
                                            n->status, st, nullptr, 0, false, list, nr)))
        return rc;
    a.g1 = g->d_h1;
    a.g2 = g->g2;
    a.h0 = n->h0;
    a.h2 = n->h2;
    a.dh0 = g->d_h0;
    if ((rc = smem_opt_in(k_edges_bwd, EB_BYTES))) return rc;
    if (nr > 0) {
        a.partial = take(bg, kBwdStride);
        k_edges_bwd<<<bg, kBT, EB_BYTES, st>>>(a);
        if ((rc = launch_status("mpnn edges_bwd"))) return rc;
        add_segment(sums, a.partial, bg, kBwdStride, 128 * 128, grad + SPHDEM_MPNN_E2_W);
        add_segment(sums, a.partial + 128 * 128, bg, kBwdStride, 128 * 16, grad + SPHDEM_MPNN_E1_W);
        add_segment(sums, a.partial + 128 * 128 + 128 * 16, bg, kBwdStride, 128, grad + SPHDEM_MPNN_E1_B);
        add_segment(sums, a.partial + 128 * 128 + 128 * 16 + 128, bg, kBwdStride, 128, grad + SPHDEM_MPNN_E2_B);
    } else {
        const cudaError_t e = cudaMemsetAsync(grad, 0, sizeof(float) * SPHDEM_MPNN_N1_W, st);
        if (e != cudaSuccess) {
            set_error("mpnn_backward", e);
            return SPHDEM_ERR_CUDA;
        }
    }
    // first node layer
    p = take(cg, 128);
    k_act_grad<<<cg, 256, 0, st>>>(g->d_h0, n->z0, nn, list, nr, g->bf_a, p);
    add_segment(sums, p, cg, 128, 128, grad + SPHDEM_MPNN_N1_B);
    if ((rc = wgrad<16>(g->bf_a, n->x, nn, part, ncta, n->status, st, list, nr))) return rc;
    add_segment(sums, take(ncta, 128 * 16), ncta, 128 * 16, 128 * 16, grad + SPHDEM_MPNN_N1_W);
    if ((rc = reduce(sums, st))) return rc;
    return launch_status("mpnn_backward");
}

extern "C" int sphdem_mpnn_loss(const float* out, const float* target, int32_t n, float* loss, float* d_out,
                                sphdem_stream_t stream) {
    if (!out || !target || !loss || !d_out || n < 0) {
        set_error_msg("mpnn_loss: invalid arguments");
        return SPHDEM_ERR_INVALID;
    }
    k_loss<<<kLossCtas, 1024, 0, as_stream(stream)>>>(out, target, n, loss, d_out);
    return launch_status("mpnn_loss");
}

extern "C" int sphdem_mpnn_edge_loss(const int32_t* offset, const int32_t* sender, const int32_t* receiver,
                                     int32_t n_recv, int32_t edge_capacity, const float* out, const float* target,
                                     float lambda, float* loss, float* d_out, sphdem_stream_t stream) {
    if (!offset || !sender || !receiver || !out || !target || !loss || !d_out || n_recv < 0 || edge_capacity < 0) {
        set_error_msg("mpnn_edge_loss: invalid arguments");
        return SPHDEM_ERR_INVALID;
    }
    if (n_recv == 0 || edge_capacity == 0) return SPHDEM_OK;
    int grid = blocks_for(edge_capacity, 256);
    if (grid > 8 * sm_count()) grid = 8 * sm_count();
    k_edge_loss<<<grid, 256, 0, as_stream(stream)>>>(offset, sender, receiver, n_recv, edge_capacity, out, target,
                                                    lambda, d_out, loss);
    return launch_status("mpnn_edge_loss");
}

extern "C" int sphdem_mpnn_adam(float* theta, const float* grad, float* m, float* v, int32_t n, float lr, float beta1,
                                float beta2, float eps, int32_t step, sphdem_stream_t stream) {
    if (!theta || !grad || !m || !v || n < 0 || step < 1) {
        set_error_msg("mpnn_adam: invalid arguments");
        return SPHDEM_ERR_INVALID;
    }
    const float c1 = (float)(1.0 / (1.0 - pow((double)beta1, step)));
    const float c2 = (float)(1.0 / (1.0 - pow((double)beta2, step)));
    k_adam<<<blocks_for(n > 0 ? n : 1, 256), 256, 0, as_stream(stream)>>>(theta, grad, m, v, n, lr, beta1, beta2, eps,
                                                                          c1, c2);
    return launch_status("mpnn_adam");
}

extern "C" int sphdem_mpnn_apply(float* f_pos, float* f_vel, const float* f_acc, int32_t n_fluid, float* d_pos,
                                 float* d_vel, const float* d_acc, int32_t n_dem, const float* out, int32_t m,
                                 float dt, const float* scale4, const float* x_t, const float* v_t, float* target,
                                 sphdem_stream_t stream) {
    if (!scale4 || n_fluid < 0 || n_dem < 0 || (n_fluid > 0 && (!f_pos || !f_vel || !f_acc)) ||
        (n_dem > 0 && (!d_pos || !d_vel || !d_acc)) || (!target && !out) || (target && (!x_t || !v_t))) {
        set_error_msg("mpnn_apply: invalid arguments");
        return SPHDEM_ERR_INVALID;
    }
    ApplyArgs a;
    a.pos[0] = f_pos;
    a.pos[1] = d_pos;
    a.vel[0] = f_vel;
    a.vel[1] = d_vel;
    a.acc[0] = f_acc;
    a.acc[1] = d_acc;
    a.n[0] = n_fluid;
    a.n[1] = n_dem;
    a.out = out;
    a.m = m;
    a.dt = dt;
    a.sx[0] = scale4[0];
    a.sv[0] = scale4[1];
    a.sx[1] = scale4[2];
    a.sv[1] = scale4[3];
    a.x_t = x_t;
    a.v_t = v_t;
    a.target = target;
    const int n = n_fluid + n_dem;
    if (n == 0) return SPHDEM_OK;
    launch_pdl(k_apply, blocks_for(n, 256), 256, 0, as_stream(stream), a);
    return launch_status("mpnn_apply");
}

namespace sd {

// Largest correction displacement of a jump: max over the receivers (fluid
// rows first, then DEM) of |s_x out[0:3]| + mdt |s_v out[3:6]| into *dst
// (float bits, atomicMax; values >= 0; *dst starts at 0).
__global__ void k_corrmax(const float* __restrict__ out, int nf, int nd, float4 sc, float mdt, float* dst) {
    pdl_wait();
    pdl_launch();
    float m = 0.0f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf + nd; i += gridDim.x * blockDim.x) {
        const float sx = i < nf ? sc.x : sc.z, sv = i < nf ? sc.y : sc.w;
        const float* o = out + 16 * (size_t)i;
        const float dx = sx * sqrtf(o[0] * o[0] + o[1] * o[1] + o[2] * o[2]);
        const float dv = sv * sqrtf(o[3] * o[3] + o[4] * o[4] + o[5] * o[5]);
        m = fmaxf(m, dx + mdt * dv);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(reinterpret_cast<int*>(dst), __float_as_int(m));
}

int run_corrmax(const float* out, int nf, int nd, const float* scale4, float mdt, float* dst, cudaStream_t st) {
    if (nf + nd <= 0) return SPHDEM_OK;
    int grid = blocks_for(nf + nd, 256);
    if (grid > 4 * sm_count()) grid = 4 * sm_count();
    launch_pdl(k_corrmax, grid, 256, 0, st, out, nf, nd, make_float4(scale4[0], scale4[1], scale4[2], scale4[3]),
               mdt, dst);
    return launch_status("jump correction");
}

}  // namespace sd

extern "C" int sphdem_mpnn_maxdev(const float* a, const float* b, float ref, int32_t n, float inv, float* out,
                                  sphdem_stream_t stream) {
    if (!a || !out || n < 0) {
        set_error_msg("mpnn_maxdev: invalid arguments");
        return SPHDEM_ERR_INVALID;
    }
    if (n == 0) return SPHDEM_OK;
    int grid = blocks_for(n, 256);
    if (grid > 4 * sm_count()) grid = 4 * sm_count();
    launch_pdl(k_maxdev, grid, 256, 0, as_stream(stream), a, b, ref, n, inv, out);
    return launch_status("mpnn_maxdev");
}

extern "C" int sphdem_mpnn_gemm(const uint16_t* a, const uint16_t* b, float* c, int32_t m, int32_t n, int32_t k,
                                int32_t* status, sphdem_stream_t stream) {
    if (!a || !b || !c || m < 0 || (n != 16 && n != 128) || (k != 16 && k != 128)) {
        set_error_msg("mpnn_gemm: N and K must be 16 or 128");
        return SPHDEM_ERR_INVALID;
    }
    cudaStream_t st = as_stream(stream);
    if (k == 16 && n == 16) return rows<16, 16, EPI_F32, false>(a, m, b, nullptr, c, nullptr, nullptr, status, st);
    if (k == 16 && n == 128) return rows<16, 128, EPI_F32, false>(a, m, b, nullptr, c, nullptr, nullptr, status, st);
    if (k == 128 && n == 16) return rows<128, 16, EPI_F32, false>(a, m, b, nullptr, c, nullptr, nullptr, status, st);
    return rows<128, 128, EPI_F32, false>(a, m, b, nullptr, c, nullptr, nullptr, status, st);
}

extern "C" int sphdem_mpnn_wgrad(const uint16_t* p, const uint16_t* q, float* c, int32_t n_rows, int32_t n,
                                 float* partial, int32_t* status, sphdem_stream_t stream) {
    if (!p || !q || !c || !partial || n_rows < 0 || (n != 16 && n != 128)) {
        set_error_msg("mpnn_wgrad: N must be 16 or 128");
        return SPHDEM_ERR_INVALID;
    }
    cudaStream_t st = as_stream(stream);
    int ncta = 0, rc;
    if (n == 16)
        rc = wgrad<16>(p, q, n_rows, partial, ncta, status, st);
    else
        rc = wgrad<128>(p, q, n_rows, partial, ncta, status, st);
    if (rc) return rc;
    Segments sums;
    sums.n = 0;
    add_segment(sums, partial, ncta, 128 * n, 128 * n, c);
    return reduce(sums, st);
}
