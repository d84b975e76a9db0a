// sph.cu -- WCSPH neighbour loops on the sorted fluid / wall copies.
//
// One thread per subject (LANES = 1) or, for systems that leave the GPU idle
// then, 4 or 8 lanes per subject whose sums run in the order of the one thread
// and give the same bits (walk.cuh); or one warp per subject with a sum order
// of its own (LANES = 32: the launch option lanes_sph = 32).  Subjects are
// taken in cell order (grid order), so the lanes of a warp query the same few
// cell columns and their float4 neighbour loads hit the same L1 lines.
// Neighbour membership uses the exact FP32 predicates of the reference; the
// physics sums use contracted FP32.
//
//   k_density        Kernel_shepard_sph + Kernel_density_sph + Kernel_pres_sph
//                    (kernel/KERNEL_rho.py:6-82, kernel/KERNEL_pres.py:6-23) in
//                    one pass: the Shepard sum, when due, shares the loop.
//   k_density_wall   Kernel_density_bnd + Kernel_pres_bnd (KERNEL_rho.py:87-126,
//                    KERNEL_pres.py:26-45) with the constant wall-wall part cached.
//   k_force          Kernel_force_sph (kernel/KERNEL_force.py:7-71) and the
//                    pressure-gradient half of Kernel_prep_sphdem
//                    (kernel/KERNEL_SPHDEM_interaction.py:97-112): same
//                    neighbours, same support, one loop.
//   k_step_sph       Kernel_step_sph (kernel/KERNEL_step.py:6-22).
//
// Neighbour records (one thread per subject): the density pass already
// decides every fluid-fluid and fluid-wall membership of the step (same
// support, same exact predicate as the force pass), so it records them and the
// force pass loops over exactly those members instead of testing every
// candidate.  A thread walking cells evaluates the force body for ~1 in 5
// candidates, and the warp pays for the body on every candidate some lane
// accepts; from the record every iteration is a member.  Same members, same
// order, same arithmetic: the forces are bit-identical.  Two forms
// (params.nbr_format): int32 member slots (SPHDEM_NBR_SLOTS, 4 bytes per
// member), or walk masks (SPHDEM_NBR_MASKS, one bit per walked slot, ~5 per
// member: a sixth of the bytes, but the force pass re-trims the ranges and
// decodes the bits).
#include "common.cuh"
#include "walk.cuh"

namespace sd {

namespace {

extern __shared__ __align__(16) unsigned char sph_smem[];

// kern_w(k, fast_sqrt(d2)) of a finite d2, same bits: the guard of the root at
// 0 and the end of the support are a maximum each.  Not for a warp per subject:
// with it and Near2 that loop takes 40 registers instead of 31 and an SM holds
// fewer warps (density of 33k particles 51 us against 43, of 387k walls 171
// against 144).
template <int LANES>
__device__ __forceinline__ float member_w(const Kern& k, float d2) {
    if (LANES == 32) return kern_w(k, fast_sqrt(d2));
    const float q = (d2 * rsqrtf(fmaxf(d2, 1.0e-37f))) * k.inv_h;
    const float u = fmaxf(1.0f - 0.5f * q, 0.0f);
    const float u2 = u * u;
    return k.cw * u2 * u2 * (1.0f + 2.0f * q);
}

// Squared distance to a candidate with d2_exact's rounding, x and y as an FP32
// pair (a packed product is an FMA onto 0: the same rounding).
struct Near2 {
    unsigned long long nxy;
    float z;
    __device__ __forceinline__ explicit Near2(const float4& p) : z(p.z) {
        asm("mov.b64 %0, {%1, %2};" : "=l"(nxy) : "f"(-p.x), "f"(-p.y));
    }
    __device__ __forceinline__ float d2(const float4& q) const {
        float sx, sy;
        asm("{\n\t.reg .b64 d;\n\tmov.b64 d, {%2, %3};\n\tadd.rn.ftz.f32x2 d, d, %4;\n\t"
            "fma.rn.ftz.f32x2 d, d, d, %5;\n\tmov.b64 {%0, %1}, d;\n\t}"
            : "=f"(sx), "=f"(sy)
            : "f"(q.x), "f"(q.y), "l"(nxy), "l"(0ull));
        const float dz = __fsub_rn(z, q.z);
        return __fadd_rn(__fadd_rn(sx, sy), __fmul_rn(dz, dz));
    }
};

// Subject of this thread and its lane among the subject's LANES.
template <int LANES>
__device__ __forceinline__ int subject_index(int& lane) {
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    lane = (int)(threadIdx.x % LANES);
    return (int)(t / LANES);
}

// body(ok, j, q, d2) over the members (exact d2 < s2) of this lane's subject: a
// thread that walks every slot of the ball-trimmed ranges (LANES = 1), a warp
// whose lanes stride through each range together (LANES = 32; its sums are
// reduced across lanes at the end, a different, equally valid FP32 summation
// order), or walk.cuh's walk.
//
// One thread per subject waits for its candidates more than it computes, so it
// loads BATCH of them before it looks at the first.  Fluid density, 752k
// particles: 585 us one at a time, 528 with 4, 510-520 with 6, 525 with 8; 100k,
// nothing recorded: 97, 84, 80, 79.  The walls, most of which have no candidate
// at all, take one at a time (178 us for 3.1M; 197 with 6).
template <int LANES, int BATCH = 1, class F>
__device__ __forceinline__ void visit_members(const Geo& g, const float4* __restrict__ posm, bool mine,
                                              const float4& p, float rq, float s2, int inst, int lane, F&& body) {
    const Near2 near(p);
    auto one = [&](int j) {
        const float4 q = posm[j];
        const float d2 = near.d2(q);
        if (d2 < s2) body(true, j, q, d2);
    };
    if constexpr (LANES == 1 && BATCH == 1) {
        for_each_range_ball(g, p.x, p.y, p.z, rq, inst, [&](int s, int e) {
            for (int j = s; j < e; ++j) one(j);
        });
    } else if constexpr (LANES == 1) {
        for_each_range_ball(g, p.x, p.y, p.z, rq, inst, [&](int s, int e) {
            for (int j = s; j < e; j += BATCH) {
                float4 q[BATCH];
#pragma unroll
                for (int u = 0; u < BATCH; ++u)
                    if (u == 0 || j + u < e) q[u] = posm[j + u];
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const float d2 = near.d2(q[u]);
                    if ((u == 0 || j + u < e) && d2 < s2) body(true, j + u, q[u], d2);
                }
            }
        });
    } else if constexpr (LANES == 32) {
        warp_ranges_ball(g, p.x, p.y, p.z, rq, inst, [&](int s, int e) {
            for (int j = s + lane; j < e; j += 32) {
                const float4 q = posm[j];
                const D2 r = d2_exact(p.x, p.y, p.z, q.x, q.y, q.z);
                if (r.d2 < s2) body(true, j, q, r.d2);
            }
        });
    } else {
        WarpWalk<LANES>* walks = reinterpret_cast<WarpWalk<LANES>*>(sph_smem);
        warp_walk<LANES>(g, posm, mine, p.x, p.y, p.z, rq, s2, inst, walks[threadIdx.x >> 5],
                         [&](bool ok, int j, const float4& q, const D2& r) { body(ok, j, q, r.d2); });
    }
}

template <int LANES>
__device__ __forceinline__ float lanes_sum(float v) {
    return LANES == 32 ? warp_sum(v) : v;
}

// Thread-per-subject walk of the ball-trimmed ranges that records the walk mask
// in rows: body(j, q, d2) for the members; each range is taken in segments that
// end where a 32-bit mask word ends, the segment's member bits gathered in a
// register and stored with the word.  Returns the slots walked.
template <class Body>
__device__ __forceinline__ int walk_record(const Geo& g, const float4* __restrict__ posm, const float4& p, float rq,
                                           int inst, float s2, int32_t* __restrict__ rows, size_t n, int k, int cap,
                                           Body&& body) {
    int pos = 0;
    uint32_t word = 0u;
    for_each_range_ball(g, p.x, p.y, p.z, rq, inst, [&](int s, int e) {
        for (int j0 = s; j0 < e;) {
            const int b = pos + (j0 - s);
            const int sh = b & 31;
            const int j1 = min(j0 + 32 - sh, e);
            uint32_t m = 0u, bit = 1u << sh;
            for (int j = j0; j < j1; ++j, bit <<= 1) {
                const float4 q = posm[j];
                const D2 r = d2_exact(p.x, p.y, p.z, q.x, q.y, q.z);
                if (r.d2 < s2) {
                    body(j, q, r.d2);
                    m |= bit;
                }
            }
            word |= m;
            if (sh + (j1 - j0) == 32) {
                if ((b >> 5) < cap) rows[(size_t)(b >> 5) * n + k] = (int32_t)word;
                word = 0u;
            }
            j0 = j1;
        }
        pos += e - s;
    });
    if ((pos & 31) && (pos >> 5) < cap) rows[(size_t)(pos >> 5) * n + k] = (int32_t)word;
    return pos;
}

constexpr int kBatch = 6;       // candidates a thread of the density pass loads at a time
constexpr int kNoRecord = -1;  // beside SPHDEM_NBR_SLOTS and SPHDEM_NBR_MASKS: no neighbour record kept

struct DensArgs {
    Geo gs, gb;
    const float4* __restrict__ f_posm;
    const float* __restrict__ f_vprev;  // m/rho before this pass (Shepard input)
    const float4* __restrict__ b_posm;
    const float* __restrict__ b_vprev;
    float* flt;
    float* rho;
    float* pres;
    float4* f_rp;    // out: rho, pres, pres/rho^2, 1/rho  (sorted)
    float4* f_posv;  // out: x, y, z, m/rho                 (sorted)
    int* nbr;        // out: neighbour records (sphdem_work_t.nbr), or null
    int cap;         // per subject and kind: slots or mask words
    int fmt;         // SPHDEM_NBR_SLOTS or SPHDEM_NBR_MASKS
    int n;
    float s2, rq;
    Kern kern;
    float rho0, B, gamma;
};

template <int LANES, bool FLT, bool RHO, bool PRES, int REC>
__global__ void __launch_bounds__(256) k_density(DensArgs a) {
    pdl_wait();
    pdl_launch();
    int lane;
    const int k = subject_index<LANES>(lane);
    const bool mine = k < a.n;
    const size_t n = (size_t)a.n;
    const int o = mine ? a.gs.order[k] : 0;
    const float4 p = mine ? a.f_posm[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int inst = mine ? inst_of(a.gs, o) : 0;
    float rho_sum = 0.0f, flt_sum = 0.0f;
    if ((LANES == 1 || LANES == 32) && !mine) return;
    if constexpr (LANES == 1 && REC == SPHDEM_NBR_MASKS) {
        int32_t* rows = a.nbr;
        const int wf = walk_record(a.gs, a.f_posm, p, a.rq, inst, a.s2, rows, n, k, a.cap,
                                   [&](int j, const float4& q, float d2) {
                                       const float w = member_w<LANES>(a.kern, d2);
                                       if (RHO) rho_sum += q.w * w;
                                       if (FLT) flt_sum += a.f_vprev[j] * w;
                                   });
        int wb = 0;
        if (a.gb.ncl > 0)
            wb = walk_record(a.gb, a.b_posm, p, a.rq, inst, a.s2, rows + (size_t)a.cap * n, n, k, a.cap,
                             [&](int j, const float4& q, float d2) {
                                 const float w = member_w<LANES>(a.kern, d2);
                                 if (RHO) rho_sum += q.w * w;
                                 if (FLT) flt_sum += a.b_vprev[j] * w;
                             });
        rows[(size_t)(2 * a.cap) * n + k] = wf;
        rows[(size_t)(2 * a.cap + 1) * n + k] = wb;
    } else {
        constexpr bool list = LANES != 32 && REC == SPHDEM_NBR_SLOTS;
        const int shift = (threadIdx.x & 31) - lane;  // first lane of this subject
        // one kind's members: sums, and their slots into rows, up to the capacity
        auto kind = [&](const Geo& g, const float4* __restrict__ posm, const float* __restrict__ vprev, int first_row,
                        int count_row) {
            int found = 0;
            visit_members<LANES, kBatch>(g, posm, mine, p, a.rq, a.s2, inst, lane, [&](bool ok, int j,
                                                                                      const float4& q, float d2) {
                if constexpr (LANES == 1 || LANES == 32) {
                    const float w = member_w<LANES>(a.kern, d2);
                    if (RHO) rho_sum += q.w * w;
                    if (FLT) flt_sum += vprev[j] * w;
                    if (list) {
                        if (found < a.cap) a.nbr[(size_t)(first_row + found) * n + k] = j;
                        ++found;
                    }
                } else {
                    const float w = ok ? member_w<LANES>(a.kern, d2) : 0.0f;
                    if (list) {
                        const unsigned of = (__ballot_sync(0xffffffffu, ok) >> shift) & ((1u << (LANES & 31)) - 1u);
                        const int row = found + __popc(of & ((1u << lane) - 1u));
                        if (ok && row < a.cap) a.nbr[(size_t)(first_row + row) * n + k] = j;
                        found += __popc(of);
                    }
                    if (RHO) rho_sum = ordered_fma<LANES>(rho_sum, ok ? q.w : 0.0f, w);
                    if (FLT) flt_sum = ordered_fma<LANES>(flt_sum, ok ? vprev[j] : 0.0f, w);
                }
            });
            if (list && mine && lane == 0) a.nbr[(size_t)count_row * n + k] = found;
        };
        kind(a.gs, a.f_posm, a.f_vprev, 0, 2 * a.cap);
        if (a.gb.ncl > 0)
            kind(a.gb, a.b_posm, a.b_vprev, a.cap, 2 * a.cap + 1);
        else if (list && mine && lane == 0)
            a.nbr[(size_t)(2 * a.cap + 1) * n + k] = 0;
    }
    if (RHO) rho_sum = lanes_sum<LANES>(rho_sum);
    if (FLT) flt_sum = lanes_sum<LANES>(flt_sum);
    if (lane != 0 || !mine) return;
    if (FLT) a.flt[o] = flt_sum;
    if (RHO) {
        const float flt = FLT ? flt_sum : a.flt[o];
        const float rho = rho_sum / flt;
        a.rho[o] = rho;
        if (PRES) {
            const float pr = tait(rho, a.rho0, a.B, a.gamma);
            a.pres[o] = pr;
            const float irho = 1.0f / rho;
            a.f_rp[k] = make_float4(rho, pr, pr * irho * irho, irho);
            a.f_posv[k] = make_float4(p.x, p.y, p.z, p.w * irho);
        }
    }
}

struct WallArgs {
    Geo gs, gb;
    const float4* __restrict__ f_posm;
    const float4* __restrict__ b_posm;
    const float* __restrict__ b_self;
    float* rho;
    float* pres;
    float4* b_rp;
    int n;
    float s2, rq;
    Kern kern;
    float rho0, B, gamma;
};

template <int LANES, bool PRES>
__global__ void __launch_bounds__(256) k_density_wall(WallArgs a) {
    pdl_wait();
    pdl_launch();
    int lane;
    const int k = subject_index<LANES>(lane);
    const bool mine = k < a.n;
    if ((LANES == 1 || LANES == 32) && !mine) return;
    const int o = mine ? a.gb.order[k] : 0;
    const float4 p = mine ? a.b_posm[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int inst = mine ? inst_of(a.gb, o) : 0;
    float rho_sum = 0.0f;
    // One thread a particle: most walls stand where there is no fluid, and a slab
    // of whole columns (all y and z of the window at one x) without particles
    // shows it in two loads.  3.1M walls of 64 dam breaks: 181 -> 149 us, 2.2M of
    // one: 85 -> 52 (4 lanes a particle, which trim 32 columns at once: no gain).
    bool wet = a.gs.ncl > 0;
    if (LANES == 1 && wet) {
        const Win w = window(a.gs, p.x, p.y, p.z, a.rq);
        wet = false;
        for (int cx = w.x0; cx <= w.x1; ++cx) {
            const int* at = a.gs.start + inst * a.gs.ncl + (size_t)(cx * a.gs.dim[1]) * a.gs.dim[2];
            wet |= __ldg(at + w.y0 * a.gs.dim[2]) != __ldg(at + (w.y1 + 1) * a.gs.dim[2]);
        }
    }
    if (wet)
        visit_members<LANES>(a.gs, a.f_posm, mine, p, a.rq, a.s2, inst, lane,
                             [&](bool ok, int j, const float4& q, float d2) {
                                 if constexpr (LANES == 1 || LANES == 32)
                                     rho_sum += q.w * member_w<LANES>(a.kern, d2);
                                 else
                                     rho_sum = ordered_fma<LANES>(rho_sum, ok ? q.w : 0.0f,
                                                                  ok ? member_w<LANES>(a.kern, d2) : 0.0f);
                             });
    rho_sum = lanes_sum<LANES>(rho_sum);
    if (lane != 0 || !mine) return;
    const float rho = rho_sum + a.b_self[k];
    a.rho[o] = rho;
    if (PRES) {
        const float pr = tait(rho, a.rho0, a.B, a.gamma);
        a.pres[o] = pr;
        const float irho = 1.0f / rho;
        a.b_rp[k] = make_float4(rho, pr, pr * irho * irho, irho);
    }
}

struct ForceArgs {
    Geo gs, gb;
    const float4* __restrict__ f_posm;
    const float4* __restrict__ f_vel;
    const float4* __restrict__ f_rp;
    const float4* __restrict__ b_posm;
    const float4* __restrict__ b_vel;
    const float4* __restrict__ b_rp;
    float* acc;
    float* pgf;
    float4* f_pgf;     // out (sorted): pgf x, y, z, rho
    const int* nbr;    // neighbour records of this step's density pass, or null
    int cap;           // per subject and kind: slots or mask words
    int fmt;           // SPHDEM_NBR_SLOTS or SPHDEM_NBR_MASKS
    int n;
    float s2, rq;
    Kern kern;
    float two_mu, eps_h2, g;
};

// Pair terms of the fluid and wall loops.  MODE bit 1: acceleration (fx, fy,
// fz to be added), bit 2: negative pressure gradient (c, and grad_i W in gx,
// gy, gz: the sum takes -c grad W).
struct Pair {
    float fx, fy, fz, c, gx, gy, gz;
};
template <int MODE>
__device__ __forceinline__ Pair force_pair(const ForceArgs& a, const D2& r, const float4& vi, float pr_i, float p_i,
                                           float irho_i, const float4& q, const float4& rpj, const float4& vj) {
    Pair f;
    const float rinv = rsqrtf(r.d2);
    const float dist = r.d2 * rinv;
    const float dwr = kern_dw(a.kern, dist) * rinv;  // (dW/dr) / r
    f.gx = dwr * r.dx;
    f.gy = dwr * r.dy;
    f.gz = dwr * r.dz;
    if (MODE & 1) {
        const float sc = q.w * (pr_i + rpj.z);
        const float visc =
            __fdividef(a.two_mu * (r.dx * f.gx + r.dy * f.gy + r.dz * f.gz) * irho_i * rpj.w, r.d2 + a.eps_h2);
        const float mv = q.w * visc;
        f.fx = mv * (vi.x - vj.x) - sc * f.gx;
        f.fy = mv * (vi.y - vj.y) - sc * f.gy;
        f.fz = mv * (vi.z - vj.z) - sc * f.gz;
    }
    if (MODE & 2) f.c = q.w * rpj.w * (rpj.y - p_i);
    return f;
}

// Adds this lane's pair (nothing if !ok) to the subject's sums.
template <int LANES, int MODE>
__device__ __forceinline__ void force_sum(bool ok, const Pair& f, float3& acc, float3& pgf) {
    if constexpr (LANES == 1 || LANES == 32) {
        if (!ok) return;
        if (MODE & 1) acc = make_float3(acc.x + f.fx, acc.y + f.fy, acc.z + f.fz);
        if (MODE & 2) pgf = make_float3(fmaf(-f.c, f.gx, pgf.x), fmaf(-f.c, f.gy, pgf.y), fmaf(-f.c, f.gz, pgf.z));
    } else {
#pragma unroll
        for (int s = 0; s < LANES; ++s) {
            auto of = [&](float v) { return __shfl_sync(0xffffffffu, ok ? v : 0.0f, s, LANES); };
            if (MODE & 1) acc = make_float3(acc.x + of(f.fx), acc.y + of(f.fy), acc.z + of(f.fz));
            if (MODE & 2) {
                const float c = of(f.c);
                pgf = make_float3(fmaf(-c, of(f.gx), pgf.x), fmaf(-c, of(f.gy), pgf.y), fmaf(-c, of(f.gz), pgf.z));
            }
        }
    }
}

// The c member slots rows[t * n + k] recorded for subject k, in walk order,
// kUnroll per lane and round: their slots, then their fields, are loaded
// together so the gathers overlap (the loop is latency bound).  With LANES > 1
// all lanes of the warp call it; the rounds are the warp's.
template <int LANES, int MODE>
__device__ __forceinline__ void force_slots(const ForceArgs& a, const float4* __restrict__ posm,
                                            const float4* __restrict__ rp, const float4* __restrict__ vel,
                                            const int32_t* __restrict__ rows, int c, const float4& p,
                                            const float4& vi, const float4& rpi, int k, int lane, float3& acc,
                                            float3& pgf) {
    constexpr int kUnroll = LANES == 1 ? 4 : 2;
    const size_t n = (size_t)a.n;
    const int trips = LANES == 1 ? c : __reduce_max_sync(0xffffffffu, c);
    for (int t = 0; t < trips; t += kUnroll * LANES) {
        int js[kUnroll];
        float4 qs[kUnroll], rs[kUnroll], vs[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const int i = t + u * LANES + lane;
            js[u] = i < c ? rows[(size_t)i * n + k] : 0;
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) qs[u] = posm[js[u]];
        if (LANES > 1) {
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                rs[u] = rp[js[u]];
                vs[u] = vel[js[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const D2 r = d2_exact(p.x, p.y, p.z, qs[u].x, qs[u].y, qs[u].z);
            const bool ok = t + u * LANES + lane < c && r.d2 > kR2Min;
            if (LANES == 1) {
                if (ok)
                    force_sum<1, MODE>(true, force_pair<MODE>(a, r, vi, rpi.z, rpi.y, rpi.w, qs[u], rp[js[u]], vel[js[u]]),
                                       acc, pgf);
            } else {
                force_sum<LANES, MODE>(ok, force_pair<MODE>(a, r, vi, rpi.z, rpi.y, rpi.w, qs[u], rs[u], vs[u]), acc,
                                       pgf);
            }
        }
    }
}

// Ball-trimmed ranges a subject's walk-mask decode keeps in shared memory.
constexpr int kForceRanges = 16;

// The members a walk mask records for subject k over geometry g, in walk
// order, summed four per round (their slots, then their positions, are loaded
// together so the gathers overlap: the loop is latency bound).  The subject's
// non-empty ball-trimmed ranges are trimmed once into a table in shared memory
// -- per range, slot - walk position and the walk position where it ends -- so
// a member costs a find-first-set on its mask word and one table step.
// Returns false, having summed nothing, when the walk it re-trims is not the
// one recorded (more ranges than the table holds, or another length): the
// caller then walks the cells.
template <int MODE>
__device__ __forceinline__ bool force_members(const ForceArgs& a, const Geo& g, const float4* __restrict__ posm,
                                              const float4* __restrict__ rp, const float4* __restrict__ vel,
                                              const int32_t* __restrict__ rows, int walked, const float4& p,
                                              const float4& vi, const float4& rpi, int inst, int k, int32_t* tab,
                                              int ts, float3& acc, float3& pgf) {
    int nr = 0, pos = 0;
    for_each_range_ball(g, p.x, p.y, p.z, a.rq, inst, [&](int s, int e) {
        if (nr < kForceRanges) {
            tab[(2 * nr) * ts] = s - pos;  // slot of walk position q in this range: q + (s - pos)
            tab[(2 * nr + 1) * ts] = pos + (e - s);
        }
        ++nr;
        pos += e - s;
    });
    if (nr > kForceRanges || pos != walked) return false;
    const size_t n = (size_t)a.n;
    const int nwords = (pos + 31) >> 5;
    int wi = 0, base = 0, ri = 0;
    uint32_t word = nwords > 0 ? (uint32_t)__ldg(rows + k) : 0u;
    int off = nr > 0 ? tab[0] : 0, end = nr > 0 ? tab[ts] : 0;
    for (bool more = nwords > 0; more;) {
        int js[4] = {-1, -1, -1, -1};
#pragma unroll 1
        for (int u = 0; u < 4;) {
            if (word == 0u) {
                if (++wi >= nwords) {
                    more = false;
                    break;
                }
                word = (uint32_t)__ldg(rows + (size_t)wi * n + k);
                base = wi << 5;
                continue;
            }
            const int q = base + __ffs(word) - 1;
            word &= word - 1u;
            while (q >= end) {
                ++ri;
                off = tab[(2 * ri) * ts];
                end = tab[(2 * ri + 1) * ts];
            }
            js[0] = js[1];
            js[1] = js[2];
            js[2] = js[3];
            js[3] = q + off;
            ++u;
        }
        if (js[3] < 0) break;
        float4 qv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) qv[u] = posm[js[u] < 0 ? js[3] : js[u]];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const D2 r = d2_exact(p.x, p.y, p.z, qv[u].x, qv[u].y, qv[u].z);
            if (js[u] >= 0 && r.d2 > kR2Min)
                force_sum<1, MODE>(true, force_pair<MODE>(a, r, vi, rpi.z, rpi.y, rpi.w, qv[u], rp[js[u]], vel[js[u]]),
                                   acc, pgf);
        }
    }
    return true;
}

template <int LANES, int MODE>
__global__ void __launch_bounds__(256, 4) k_force(ForceArgs a) {
    pdl_wait();
    pdl_launch();
    int lane;
    const int k = subject_index<LANES>(lane);
    const bool mine = k < a.n;
    if ((LANES == 1 || LANES == 32) && !mine) return;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int o = mine ? a.gs.order[k] : 0;
    const float4 p = mine ? a.f_posm[k] : zero;
    const float4 vi = mine ? a.f_vel[k] : zero;
    const float4 rpi = mine ? a.f_rp[k] : zero;
    const int inst = mine ? inst_of(a.gs, o) : 0;
    const size_t n = (size_t)a.n;
    float3 acc = make_float3(0.f, 0.f, 0.f), pgf = make_float3(0.f, 0.f, 0.f);
    bool walk = mine;
    if (LANES == 1 && a.nbr != nullptr && a.fmt == SPHDEM_NBR_MASKS) {
        // the members recorded by the density pass (all with d2 < s2), in walk order
        int32_t* force_tab = reinterpret_cast<int32_t*>(sph_smem);
        const int wf = a.nbr[(size_t)(2 * a.cap) * n + k], wb = a.nbr[(size_t)(2 * a.cap + 1) * n + k];
        if (wf <= 32 * a.cap && wb <= 32 * a.cap) {
            float3 af = acc, pf = pgf;
            bool ok = force_members<MODE>(a, a.gs, a.f_posm, a.f_rp, a.f_vel, a.nbr, wf, p, vi, rpi, inst, k,
                                          force_tab + threadIdx.x, blockDim.x, af, pf);
            if (ok && a.gb.ncl > 0 && wb > 0)
                ok = force_members<MODE>(a, a.gb, a.b_posm, a.b_rp, a.b_vel, a.nbr + (size_t)a.cap * n, wb, p, vi,
                                         rpi, inst, k, force_tab + threadIdx.x, blockDim.x, af, pf);
            if (ok) {
                walk = false;
                acc = af;
                pgf = pf;
            }
        }
    } else if (LANES != 32 && a.nbr != nullptr) {
        // the member slots recorded by the density pass (all with d2 < s2), in walk order
        const int cf = mine ? a.nbr[(size_t)(2 * a.cap) * n + k] : 0;
        const int cb = mine ? a.nbr[(size_t)(2 * a.cap + 1) * n + k] : 0;
        const bool listed = cf <= a.cap && cb <= a.cap;
        if (listed) walk = false;
        if (LANES != 1 || listed) {
            constexpr int G = LANES == 32 ? 1 : LANES;
            force_slots<G, MODE>(a, a.f_posm, a.f_rp, a.f_vel, a.nbr, listed ? cf : 0, p, vi, rpi, k, lane, acc, pgf);
            force_slots<G, MODE>(a, a.b_posm, a.b_rp, a.b_vel, a.nbr + (size_t)a.cap * n, listed ? cb : 0, p, vi, rpi,
                                 k, lane, acc, pgf);
        }
    }
    // subjects without a record (none kept, or one that overflowed): the walk
    auto visit = [&](const Geo& g, const float4* __restrict__ posm, const float4* __restrict__ rp,
                     const float4* __restrict__ vel) {
        auto member = [&](bool ok, int j, const float4& q) {
            const D2 r = d2_exact(p.x, p.y, p.z, q.x, q.y, q.z);
            ok = ok && r.d2 > kR2Min && r.d2 < a.s2;
            Pair f = {};
            if (ok) f = force_pair<MODE>(a, r, vi, rpi.z, rpi.y, rpi.w, q, rp[j], vel[j]);
            force_sum<LANES, MODE>(ok, f, acc, pgf);
        };
        // one test per candidate, on the differences that the pair term needs
        // (262k particles 291 us, 309 with a test of its own before it)
        if constexpr (LANES == 1)
            for_each_range_ball(g, p.x, p.y, p.z, a.rq, inst, [&](int s, int e) {
                for (int j = s; j < e; ++j) member(true, j, posm[j]);
            });
        else
            visit_members<LANES>(g, posm, walk, p, a.rq, a.s2, inst, lane,
                                 [&](bool ok, int j, const float4& q, float) { member(ok, j, q); });
    };
    if (LANES == 1 || LANES == 32 ? walk : __any_sync(0xffffffffu, walk)) {
        visit(a.gs, a.f_posm, a.f_rp, a.f_vel);
        if (a.gb.ncl > 0) visit(a.gb, a.b_posm, a.b_rp, a.b_vel);
    }
    if (MODE & 1) {
        acc.x = lanes_sum<LANES>(acc.x);
        acc.y = lanes_sum<LANES>(acc.y);
        acc.z = lanes_sum<LANES>(acc.z);
    }
    if (MODE & 2) {
        pgf.x = lanes_sum<LANES>(pgf.x);
        pgf.y = lanes_sum<LANES>(pgf.y);
        pgf.z = lanes_sum<LANES>(pgf.z);
    }
    if (lane != 0 || !mine) return;
    if (MODE & 1) st3(a.acc, o, make_float3(acc.x, acc.y, acc.z - a.g));
    if (MODE & 2) {
        if (a.pgf) st3(a.pgf, o, pgf);
        a.f_pgf[k] = make_float4(pgf.x, pgf.y, pgf.z, rpi.x);
    }
}

__global__ void k_pres(const float* __restrict__ rho, float* __restrict__ pres, int n, float rho0, float B,
                       float gamma) {
    pdl_wait();
    pdl_launch();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pres[i] = tait(rho[i], rho0, B, gamma);
}

}  // namespace

namespace {
__global__ void k_step_sph(float* pos, float* vel, const float* __restrict__ acc, int n, float dt) {
    pdl_wait();
    pdl_launch();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) euler_store(pos, vel, i, ld3(acc, i), dt);
}
}  // namespace

static float tait_B(float rho0, float c0, float gamma) { return rho0 * c0 * c0 / gamma; }

// Threads per block of the neighbour loops: 64, 128 or 256 (default 128).
static int launch_block(int b) { return (b == 64 || b == 256) ? b : 128; }

// Largest systems that take several lanes per subject; beyond them one thread
// per subject fills the GPU and executes fewer instructions.  The loops of a step
// share the GPU with one another (the walls' with the density's, the porosity pass
// with the force), and the shared memory of the several-lane walks is taken from
// the others' L1, so the lines are drawn by whole steps, not by a loop's own time.
// Step (us) with density, walls, force by one thread 000 ... by several lanes 111,
// the form taken here marked *; SPH only, then coupled with spheres above the water:
//   fluid  walls        000   001   010   011   111        000   001   010   011   111
//    25k    118k        170   152   171   133   100*       164   137   188   149   113*
//    49k    118k        181   172   197   156   145*       174   160   206   179   158*
//    64k    180k        190   185   204   167   172*       175   171   212   193   191*
//    96k    180k        245   238   261   217*  223        232   213   283   234*  246
//   125k    278k        262   261*  283   245   278        246   245*  314   270   302
//   150k    278k        267*  277   292   265   321        269*  279   323   295   351
//   262k    450k        416*  439   485   432   536        409*  431   521   475   566
// Ensembles: 55k / 242k 193 193 242 201 190*, 98k / 387k 235 245* 321 288 292,
// 143k / 580k 293* 326 379 372 414.  Alone, 55k density 79 | 79 (lanes | one
// thread), 435k walls 51 | 51, force from records 64k 55 | 54, 98k 79 | 62; by
// walks (no records) 80k 125 | 151, 98k 164 | 166, 123k 202 | 179.
constexpr int kDensityLanesMax = 64 * 1024;
constexpr int kWallLanesMax = 256 * 1024;
constexpr int kForceLanesMax = 128 * 1024, kForceWalkLanesMax = 100 * 1024;

// Blocks and shared memory of a loop with LANES lanes per subject (the walks
// need 6-8 KB per warp: at most 128 threads, 48 KB without an opt-in).
template <int LANES>
static void loop_shape(int n, int& block, int& blocks, size_t& smem) {
    if (LANES != 1 && LANES != 32 && block > 128) block = 128;
    blocks = blocks_for((long)n * LANES, block);
    smem = LANES == 1 || LANES == 32 ? 0 : (size_t)(block / 32) * sizeof(WarpWalk<LANES == 32 ? 1 : LANES>);
}

// The steps' density, with the pressure and with or without records, and the
// single kernels: the Shepard filter alone, the density alone.
template <int LANES, int REC>
static void launch_density(const DensArgs& a, bool flt, bool pres, int bs, cudaStream_t st) {
    int nb;
    size_t smem;
    loop_shape<LANES>(a.n, bs, nb, smem);
    if (flt && pres)
        launch_pdl(k_density<LANES, true, true, true, REC>, nb, bs, smem, st, a);
    else if (pres)
        launch_pdl(k_density<LANES, false, true, true, REC>, nb, bs, smem, st, a);
    else if constexpr (REC == kNoRecord) {
        if (flt)
            launch_pdl(k_density<LANES, true, false, false, REC>, nb, bs, smem, st, a);
        else
            launch_pdl(k_density<LANES, false, true, false, REC>, nb, bs, smem, st, a);
    }
}

template <int LANES>
static void launch_wall(const WallArgs& a, bool pres, int bs, cudaStream_t st) {
    int nb;
    size_t smem;
    loop_shape<LANES>(a.n, bs, nb, smem);
    if (pres)
        launch_pdl(k_density_wall<LANES, true>, nb, bs, smem, st, a);
    else
        launch_pdl(k_density_wall<LANES, false>, nb, bs, smem, st, a);
}

template <int LANES>
static void launch_force(const ForceArgs& a, int mode, int bs, cudaStream_t st) {
    int nb;
    size_t smem;
    loop_shape<LANES>(a.n, bs, nb, smem);
    if (LANES == 1 && a.nbr && a.fmt == SPHDEM_NBR_MASKS)  // the range tables (32 KB at 256 threads)
        smem = (size_t)2 * kForceRanges * bs * sizeof(int32_t);
    if (mode == 3)
        launch_pdl(k_force<LANES, 3>, nb, bs, smem, st, a);
    else if (mode == 2)
        launch_pdl(k_force<LANES, 2>, nb, bs, smem, st, a);
    else
        launch_pdl(k_force<LANES, 1>, nb, bs, smem, st, a);
}

// flt with pres: the Shepard filter and the density; without: the filter alone.
int run_density(const sphdem_ctx_t* c, float support, float h, bool flt, bool pres, float rho0, float c0, float gamma,
                cudaStream_t st, int block, int lanes, int nbr_cap, int nbr_format) {
    const int n = c->sph.n;
    if (n <= 0) return SPHDEM_OK;
    DensArgs a;
    a.gs = make_geo(c->grid_sph);
    a.gb = make_geo(c->grid_bnd);
    if (c->bnd.n <= 0) a.gb.ncl = 0;
    a.f_posm = (const float4*)c->work.f_posm;
    a.f_vprev = c->work.f_vprev;
    a.b_posm = (const float4*)c->work.b_posm;
    a.b_vprev = c->work.b_vprev;
    a.flt = c->sph.flt;
    a.rho = c->sph.rho;
    a.pres = c->sph.pres;
    a.f_rp = (float4*)c->work.f_rp;
    a.f_posv = (float4*)c->work.f_posv;
    a.nbr = (nbr_cap > 0 && lanes != 32) ? c->work.nbr : nullptr;
    a.cap = nbr_cap;
    a.fmt = nbr_format;
    a.n = n;
    a.s2 = support * support;
    a.rq = pad_radius(support);
    a.kern = make_kern(h);
    a.rho0 = rho0;
    a.B = tait_B(rho0, c0, gamma);
    a.gamma = gamma;
    const int bs = launch_block(block);
    if (lanes == 32)
        launch_density<32, kNoRecord>(a, flt, pres, bs, st);
    else if (a.nbr && a.fmt == SPHDEM_NBR_MASKS)
        launch_density<1, SPHDEM_NBR_MASKS>(a, flt, pres, bs, st);
    else if (a.nbr && n > kDensityLanesMax)
        launch_density<1, SPHDEM_NBR_SLOTS>(a, flt, pres, bs, st);
    else if (a.nbr)
        launch_density<8, SPHDEM_NBR_SLOTS>(a, flt, pres, bs, st);
    else if (n > kDensityLanesMax)
        launch_density<1, kNoRecord>(a, flt, pres, bs, st);
    else
        launch_density<8, kNoRecord>(a, flt, pres, bs, st);
    return launch_status("density");
}

int run_density_wall(const sphdem_ctx_t* c, float support, float h, bool pres, float rho0, float c0, float gamma,
                     cudaStream_t st, int block, int lanes) {
    const int n = c->bnd.n;
    if (n <= 0) return SPHDEM_OK;
    WallArgs a;
    a.gs = make_geo(c->grid_sph);
    if (c->sph.n <= 0) a.gs.ncl = 0;
    a.gb = make_geo(c->grid_bnd);
    a.f_posm = (const float4*)c->work.f_posm;
    a.b_posm = (const float4*)c->work.b_posm;
    a.b_self = c->work.b_self;
    a.rho = c->bnd.rho;
    a.pres = c->bnd.pres;
    a.b_rp = (float4*)c->work.b_rp;
    a.n = n;
    a.s2 = support * support;
    a.rq = pad_radius(support);
    a.kern = make_kern(h);
    a.rho0 = rho0;
    a.B = tait_B(rho0, c0, gamma);
    a.gamma = gamma;
    const int bs = launch_block(block);
    if (lanes == 32)
        launch_wall<32>(a, pres, bs, st);
    else if (n > kWallLanesMax)
        launch_wall<1>(a, pres, bs, st);
    else
        launch_wall<4>(a, pres, bs, st);
    return launch_status("density_wall");
}

int run_force(const sphdem_ctx_t* c, float support, float h, float mu, float g, int mode, cudaStream_t st, int block,
              int lanes, int nbr_cap, int nbr_format) {
    const int n = c->sph.n;
    if (n <= 0) return SPHDEM_OK;
    ForceArgs a;
    a.gs = make_geo(c->grid_sph);
    a.gb = make_geo(c->grid_bnd);
    if (c->bnd.n <= 0) a.gb.ncl = 0;
    a.f_posm = (const float4*)c->work.f_posm;
    a.f_vel = (const float4*)c->work.f_vel;
    a.f_rp = (const float4*)c->work.f_rp;
    a.b_posm = (const float4*)c->work.b_posm;
    a.b_vel = (const float4*)c->work.b_vel;
    a.b_rp = (const float4*)c->work.b_rp;
    a.acc = c->sph.acc;
    a.pgf = c->sph.pgf;
    a.f_pgf = (float4*)c->work.f_pgf;
    a.nbr = (nbr_cap > 0 && lanes != 32) ? c->work.nbr : nullptr;
    a.cap = nbr_cap;
    a.fmt = nbr_format;
    a.n = n;
    a.s2 = support * support;
    a.rq = pad_radius(support);
    a.kern = make_kern(h);
    a.two_mu = 2.0f * mu;
    a.eps_h2 = 0.01f * h * h;
    a.g = g;
    const int bs = launch_block(block);
    if (lanes == 32)
        launch_force<32>(a, mode, bs, st);
    else if ((a.nbr && a.fmt == SPHDEM_NBR_MASKS) || n > (a.nbr ? kForceLanesMax : kForceWalkLanesMax))
        launch_force<1>(a, mode, bs, st);
    else
        launch_force<4>(a, mode, bs, st);
    return launch_status("force");
}

int run_pres(const float* rho, float* pres, int n, float rho0, float c0, float gamma, cudaStream_t st) {
    if (n <= 0) return SPHDEM_OK;
    launch_pdl(k_pres, blocks_for(n, 256), 256, 0, st, rho, pres, n, rho0, tait_B(rho0, c0, gamma), gamma);
    return launch_status("pres");
}

int run_step_sph(const sphdem_ctx_t* c, float dt, cudaStream_t st) {
    const int n = c->sph.n;
    if (n <= 0) return SPHDEM_OK;
    launch_pdl(k_step_sph, blocks_for(n, 256), 256, 0, st, c->sph.pos, c->sph.vel, c->sph.acc, n, dt);
    return launch_status("step_sph");
}

}  // namespace sd
