// One token through all layers of a small model in ONE cooperative launch: a single user's drafted or decoded token.  (The logits are
// left to gemv.cu, whose loop streams the one large matrix faster: with them as a last phase here a step of one layer took 91 us instead of
// 75 at width 896, 157 instead of 120 at 1536.)
//
// As a chain of kernels (gemv.cu and the attention kernel, five a layer) such a step takes 4.9 us a kernel whatever its matrix weighs:
// hand-over of the grid, the activations' round trips through L2, reductions.  The weights of a layer (30 MB at width 896) are worth
// 4.6 us of HBM time.  Here a CTA per SM stays for the whole step:
//   * One warp streams the CTA's rows of every matrix, in the order of the phases, through a ring of panels of 16 rows in shared memory
//     (bulk copies; about 100 KB on their way).  Weights depend on nothing, so the stream runs across all hand-overs.
//   * Sixteen warps multiply: a warp has its part of k for all rows of a panel (mma.sync m16n8k16, the token is one of the eight columns),
//     the warps' sums meet in shared memory, one thread a row adds them in order and runs the epilogue.
//   * A hand-over is one trip through L2: every 64-bit word of an activation carries its phase's number beside the value, the reader
//     polls the words it needs, and no fence, flag or grid-wide barrier stands between them.  A word is written again only by a CTA that
//     has seen results of all its readers, so every CTA must have results of its own (one_step_sizes).
//   * A row of the residual belongs to the same thread in both of its projections and stays in a register.
//   * Attention runs on a CTA per query head and share of the keys, cache rows requested before the query is there, one worker of eight
//     (sixteen) lanes a key; shares meet at the head's first CTA.
// 24 layers of width 896 at 65 positions 594 -> 437 us, at 2048 879 -> 577; 28 of 1536 1051 -> 990; four of 1024 107 -> 91.  What bounds it
// now: 16 us a layer, of which the weights are worth 4.6: four hand-overs of a microsecond and as many input reads of half a one, 1 us a
// phase of its own code (each piece runs once a phase), shared memory that takes the stream in and gives it out again in the long ones.
// Same rounding points as gemv.cu: bf16 operands, fp32 sums, the fused RMSNorm's rstd and sums of squares; softmax weights stay fp32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "asd_internal.h"
#include "gemm.h"
#include "grid_turn.h"
#include "mma_sync.cuh"
#include "one_step.h"
#include "ptx.cuh"

namespace asd {

namespace {

constexpr int kOsWarps = 16, kOsThreads = (kOsWarps + 1) * 32;        // warps that multiply, and one that streams
constexpr int kOsMaxPiece = 1024;                                    // k elements of a panel
constexpr int kOsArrivals = 240;                                     // of a panel's readers together: 1, 2, 3, 4, 5, 8 or 16 warps
constexpr int kOsWords = 5;                                          // words a thread asks for at once
constexpr int kOsLine = 16;                                          // words of a line: what all CTAs poll stands alone in one
constexpr int kOsKeys = 512;                                         // cache rows of a share whose places are kept
constexpr int kOsAhead = 2;                                          // cache rows a worker has on their way

struct OsArgs {
    OneStep s;
    int grid, piece, slots, slot_bytes, x_bytes, splits, group;
    unsigned long long *w_qkv, *w_attn, *w_part, *w_x, *w_act, *w_sign;       // exchanged words; w_sign: [phase][grid] lines
};

struct OsShared {
    uint64_t full[16], empty[16];
    unsigned base;
    int failed, pos, slot;
    int first[4], count[4];                                           // this CTA's rows of every phase
    // How a phase's units (pieces of its panels) are shared out; divisions cost 0.1 us each here.  Units of a batch, warps of a unit, pieces
    // of a panel, what a warp arrives with; a warp's unit of a batch, its piece in the first batch, and its k steps of a whole piece and
    // of the last one; a panel's batch and first unit there
    int at_once[4], share[4], pieces[4], arrive[4], last_steps[4];
    struct {
        short unit, piece, lo, n, last_lo, last_n;
    } warp_plan[4][kOsWarps];
    int step_plan[4];                                                 // pieces that a warp's unit moves on by from batch to batch
    short2 panel_plan[4][kOsMaxPanels];
    float sumsq[kOsWarps], rstd;
    float head_m[kOsWarps], head_l[kOsWarps];
    float qkv[3][128];                                                // query, new key and value of the CTA's head
    int rows[kOsKeys];                                                // cache rows of the CTA's keys, in head rows
    float red[2][kOsMaxPanels][kOsWarps][kOsPanel];                   // of this phase and the one before: by batch of panels and warp
    float head_o[kOsWarps][128];
};

__device__ __forceinline__ unsigned long long os_load(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void os_store(unsigned long long* p, uint32_t value, unsigned epoch) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)epoch << 32 | value) : "memory");
}
// the word at p once it is of this phase; bounded (ptx.cuh): afterwards anything, and every later wait of the CTA ends at once
__device__ __forceinline__ uint32_t os_wait(const unsigned long long* p, unsigned long long v, unsigned epoch, volatile int* failed, int* err) {
    if ((unsigned)(v >> 32) != epoch) {
        const uint32_t t0 = clock_steps();
        do {
            v = os_load(p);
            if (*failed) break;
            if (clock_steps() - t0 > 4) wait_report(failed, err, WAIT_ONE_STEP << 8 | 1);
        } while ((unsigned)(v >> 32) != epoch);
    }
    return (uint32_t)v;
}
__device__ __forceinline__ uint32_t os_bits(float x) {
    const __nv_bfloat16 b = __float2bfloat16(x);
    return *reinterpret_cast<const unsigned short*>(&b);
}
__device__ __forceinline__ unsigned short os_raw(const __nv_bfloat16* p) {
    unsigned short v;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float os_low(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float os_high(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float os_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void os_arrive(uint64_t* bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
__device__ __forceinline__ void os_sync() { asm volatile("barrier.cta.sync.aligned 1, 512;" ::: "memory"); }

// place of element k of the input among xs: lane t of a product takes elements 2 t, 2 t + 1, 2 t + 8, 2 t + 9 of 16; those of two products
// lie side by side, 16 bytes a lane
__device__ __forceinline__ int os_place(int k) {
    return (k & ~31) | (k & 6) << 2 | (k >> 2 & 4) | (k >> 2 & 2) | (k & 1);
}
// this CTA's units of n: [first, first + count)
struct OsShare {
    int first, count;
};
__device__ __forceinline__ OsShare os_share(int n, int cta, int grid) {
    const int a = (int)((long long)n * cta / grid), b = (int)((long long)n * (cta + 1) / grid);
    return {a, b - a};
}

// Phases of a layer.  Row i of a CTA's share of a phase's matrix, in the order of its panels:
enum OsPhase { OS_QKV, OS_O, OS_GU, OS_DOWN };
template <int HD>
__device__ __forceinline__ int os_row(int phase, int first, int i) {
    constexpr int kHalf = HD / 2;
    const int u = first + (i >> 1);
    if (phase == OS_QKV) return u / kHalf * HD + u % kHalf + (i & 1) * kHalf;      // pairs (j, j + half) of a head
    if (phase == OS_GU) return (u >> 6) * 128 + (u & 63) + (i & 1) * 64;           // gate and up rows: 64 of each, alternately
    return first + i;
}

template <int HD>
__global__ void __launch_bounds__(kOsThreads, 1) one_step_kernel(const __grid_constant__ OsArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    const OneStep& s = a.s;
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(smem + (size_t)a.slots * a.slot_bytes);         // the phase's input
    OsShared* S = reinterpret_cast<OsShared*>(smem + (size_t)a.slots * a.slot_bytes + a.x_bytes);
    volatile int* failed = &S->failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x;
    const WaitGuard guard{failed, s.err, WAIT_ONE_STEP << 8};

    constexpr int kHalf = HD / 2;
    if (tid < 4) {
        // units: pairs of rows, rows, pairs of pairs (neighbours share a word of the result), rows
        const OsShare u = os_share(tid == OS_QKV ? s.nqkv / 2 : tid == OS_GU ? s.ffn / 2 : s.h, cta, a.grid);
        S->first[tid] = tid == OS_GU ? 2 * u.first : u.first;
        S->count[tid] = tid == OS_QKV ? 2 * u.count : tid == OS_GU ? 4 * u.count : u.count;
    }
    if (tid < 4 * kOsWarps) {
        const int e = tid / kOsWarps, w = tid % kOsWarps, K = e == OS_O ? s.qdim : e == OS_DOWN ? s.ffn : s.h;
        const OsShare r = os_share(e == OS_QKV ? s.nqkv / 2 : e == OS_GU ? s.ffn / 2 : s.h, cta, a.grid);
        const int rows = e == OS_QKV ? 2 * r.count : e == OS_GU ? 4 * r.count : r.count;
        const int panels = max(1, (rows + kOsPanel - 1) / kOsPanel), pieces = (K + a.piece - 1) / a.piece;
        const int at_once = min(min(a.slots, kOsWarps), panels * pieces), share = kOsWarps / at_once, u = w / share, sub = w - u * share;
        const int whole = a.piece >> 4, last = (K - (pieces - 1) * a.piece) >> 4;
        auto cut = [&](int steps, short& lo, short& n) {
            const int per = ((steps + share - 1) / share + 1) & ~1;           // (two steps' input is one load)
            lo = (short)min(sub * per, steps), n = (short)min(per, steps - lo);
        };
        auto& plan = S->warp_plan[e][w];
        plan.unit = (short)u, plan.piece = (short)(u % pieces);
        cut(whole, plan.lo, plan.n);
        cut(last, plan.last_lo, plan.last_n);
        if (w == 0) {
            S->at_once[e] = at_once, S->share[e] = share, S->pieces[e] = pieces, S->arrive[e] = kOsArrivals / share, S->last_steps[e] = last;
            S->step_plan[e] = at_once % pieces;
        }
        if (w < kOsMaxPanels) S->panel_plan[e][w] = make_short2((short)(w * pieces / at_once), (short)(w * pieces % at_once));
    }
    if (tid == 0) {
        for (int i = 0; i < a.slots; ++i) {
            mbar_init(&S->full[i], 1);
            mbar_init(&S->empty[i], kOsArrivals);
        }
        S->failed = 0;
        S->base = s.sync[0];
        S->pos = s.positions[0];
        S->slot = s.token_slot[0];
        fence_mbar_init();
    }
    __syncthreads();

    const int its = 4 * s.n_layers;            // four phases a layer
    auto k_of = [&](int phase) { return phase == OS_O ? s.qdim : phase == OS_DOWN ? s.ffn : s.h; };

    if (warp == kOsWarps) {
        // ------------------------------------------------------------------ weights: a lane per row of a panel
        int slot = 0, round = 0;
        bool ok = true;
        for (int it = 0; it < its && ok; ++it) {
            const int phase = it & 3, K = k_of(phase), first = S->first[phase], count = S->count[phase];
            const OneLayer& L = s.layers[it >> 2];
            const __nv_bfloat16* w = phase == OS_QKV ? L.wqkv : phase == OS_O ? L.wo : phase == OS_GU ? L.wgu : L.wdown;
            for (int p = 0; p < count && ok; p += kOsPanel) {
                const int n = min(kOsPanel, count - p);
                const __nv_bfloat16* src = w + (size_t)os_row<HD>(phase, first, p + min(lane, n - 1)) * K;
                for (int k = 0; k < K; k += a.piece) {
                    const int bytes = min(a.piece, K - k) * 2;
                    if (round > 0 && !(ok = __all_sync(0xffffffffu, mbar_wait(&S->empty[slot], (round - 1) & 1, guard)) != 0)) break;
                    if (lane == 0) mbar_expect_tx(&S->full[slot], n * bytes);
                    __syncwarp();
                    if (lane < n) bulk_g2s(smem + (size_t)slot * a.slot_bytes + lane * (bytes + 16), src + k, bytes, &S->full[slot]);
                    if (++slot == a.slots) slot = 0, ++round;
                }
            }
        }
    } else {
        // One loop over all phases, so that their common code is there once: a layer passes through it in a few microseconds, and what
        // does not fit the instruction caches is fetched again every time (158 KB of code unrolled by phase: 18.5 us a layer).
        const int pos = S->pos;
        unsigned epoch = S->base;              // of the words that the phase reads
        int slot = 0, buf = 0;                 // (a warp writes sums while others may still read those of the phase before)
        uint32_t parity = 0;
        float resid = 0.0f;                    // of row tid of this CTA's share of the hidden size

        // what stays the same in all layers: angles of this thread's pair, the cache rows of this CTA's share of the keys
        const int u_qkv = S->first[OS_QKV] + (tid >> 1), head = u_qkv / kHalf, jj = u_qkv % kHalf;
        const bool pair = tid < S->count[OS_QKV], rotates = head < s.nh + s.nkv;
        float cs = 1.0f, sn = 0.0f;
        if (pair && rotates) sincosf((float)pos * s.inv_freq[jj], &sn, &cs);
        const int* pt = s.page_table + (size_t)S->slot * s.max_pages;
        const int hq = cta / a.splits, sp = cta - hq * a.splits, kvh = hq / a.group;
        const bool attends = cta < s.nh * a.splits;
        const int keys = pos + 1, per_share = (keys + a.splits - 1) / a.splits, key0 = sp * per_share, key1 = min(keys, key0 + per_share);
        auto cache_row = [&](int key) {
            const int p = key / s.page_size;
            return (pt[p] * s.nkv + kvh) * s.page_size + (key - p * s.page_size);
        };
        if (attends)
            for (int i = tid; i < kOsKeys && key0 + i < key1; i += kOsWarps * 32) S->rows[i] = cache_row(key0 + i);
        long long kv_off = 0;                  // where this thread's new key or value pair goes
        if (pair && head >= s.nh)
            kv_off = ((long long)(pt[pos / s.page_size] * s.nkv + (rotates ? head - s.nh : head - s.nh - s.nkv)) * s.page_size + pos % s.page_size) * HD + jj;
        const int sum_warps = (a.grid + 31) >> 5;              // warps that add up the CTAs' sums of squares
        // attention: a worker of eight (sixteen) lanes a key, the cache rows that it has on their way
        constexpr int kLanes = HD / 8, kWorkers = 32 / kLanes, kStride = kOsWarps * kWorkers;
        const int d0 = (lane % kLanes) * 8;
        uint4 kr[kOsAhead], vr[kOsAhead];
        int kv_layer = 0;
        auto fetch = [&](int k) {
#pragma unroll
            for (int i = 0; i < kOsAhead; ++i) {
                const int key = k + i * kStride;
                kr[i] = vr[i] = make_uint4(0, 0, 0, 0);
                if (key < key1 && key < pos) {
                    const OneLayer& L = s.layers[kv_layer];
                    const size_t at = (size_t)(key - key0 < kOsKeys ? S->rows[key - key0] : cache_row(key)) * HD + d0;
                    kr[i] = __ldcg(reinterpret_cast<const uint4*>(L.k_cache + at));
                    vr[i] = __ldcg(reinterpret_cast<const uint4*>(L.v_cache + at));
                }
            }
        };
        // the embedding, by every CTA for itself
        {
            const __nv_bfloat16 *e = s.embed + (size_t)s.tokens[0] * s.h, *ln = s.layers[0].ln1;
            if (tid < S->count[OS_O]) resid = __bfloat162float(e[S->first[OS_O] + tid]);
            float t = 0.0f;
            if (warp < sum_warps)
                for (int i = tid; i < s.h; i += sum_warps * 32) {
                    const float x = __bfloat162float(e[i]);
                    xs[os_place(i)] = __float2bfloat16(x * __bfloat162float(ln[i]));
                    t += x * x;
                }
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
            if (lane == 0) S->sumsq[warp] = t;
            os_sync();
        }

#pragma unroll 1
        for (int it = 0; it < its; ++it) {
            const int phase = it & 3, K = k_of(phase), l = it >> 2, count = S->count[phase], first = S->first[phase];
            const bool normed = phase == OS_QKV || phase == OS_GU;
            const OneLayer& L = s.layers[l];
            // what the epilogue needs besides, as it lies in memory: nothing waits for it before
            unsigned short extra = 0;
            if (phase == OS_QKV) {
                if (pair) extra = os_raw(L.bqkv + head * HD + jj + (tid & 1) * kHalf);
            } else if (!normed && tid < count) {
                extra = os_raw((phase == OS_O ? L.ln2 : l + 1 < s.n_layers ? s.layers[l + 1].ln1 : s.final_norm) + first + tid);
            }
            // the weights of the first batch: nothing of the other CTAs' is needed for them
            const int panels = (count + kOsPanel - 1) / kOsPanel, at_once = S->at_once[phase], pieces = S->pieces[phase], share = S->share[phase];
            const auto plan = S->warp_plan[phase][warp];
            const int step = S->step_plan[phase], last_steps = S->last_steps[phase], arrive = S->arrive[phase];
            auto await = [&](int units) {
                if (plan.unit >= units) return;
                const int ring = slot + plan.unit;
                mbar_wait_timed(&S->full[ring >= a.slots ? ring - a.slots : ring], parity ^ (ring >= a.slots), guard, 2);
            };
            await(min(at_once, panels * pieces));
            if (phase == OS_QKV && attends) kv_layer = l, fetch(key0 + warp * kWorkers + lane / kLanes);       // (rows of earlier steps)
            // ---- input: words of one element (O, down: of two), and the CTAs' sums of squares
            if (it > 0) {
                const int n = normed ? s.h : K >> 1;
                constexpr int kStride = kOsWarps * 32;
                const unsigned long long* words = normed ? a.w_x : phase == OS_O ? a.w_attn : a.w_act;
                // A word of every CTA (head) first, which stands alone in its line: all words again and again, from all CTAs, are more
                // than L2 delivers, and words that are polled queue behind the polls of their line (3.6 us instead of 0.6)
                {
                    float x = 0.0f;
                    if (tid < (phase == OS_O ? s.nh : a.grid)) {
                        const unsigned long long* p = a.w_sign + ((size_t)(phase + 3 & 3) * a.grid + tid) * kOsLine;
                        x = __uint_as_float(os_wait(p, os_load(p), epoch, failed, s.err));
                    }
                    if (normed && warp < sum_warps) {
#pragma unroll
                        for (int d = 16; d >= 1; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
                        if (lane == 0) S->sumsq[warp] = x;
                    }
                    os_sync();
                }
#pragma unroll 1
                for (int i = tid; i < n; i += kOsWords * kStride) {
                    unsigned long long v[kOsWords];
#pragma unroll
                    for (int e = 0; e < kOsWords; ++e) v[e] = i + e * kStride < n ? os_load(words + i + e * kStride) : 0;
#pragma unroll
                    for (int e = 0; e < kOsWords; ++e)
                        if (i + e * kStride < n) {
                            const uint32_t w = os_wait(words + i + e * kStride, v[e], epoch, failed, s.err);
                            if (normed)
                                reinterpret_cast<unsigned short*>(xs)[os_place(i + e * kStride)] = (unsigned short)w;
                            else
                                reinterpret_cast<uint32_t*>(xs)[os_place(2 * (i + e * kStride)) >> 1] = w;
                        }
                }
                os_sync();
            }
            // the norm's factor, by a warp that has the least to multiply
            if (warp == kOsWarps - 1 && normed) {
                float t = lane < sum_warps ? S->sumsq[lane] : 0.0f;
#pragma unroll
                for (int d = 4; d >= 1; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
                if (lane == 0) S->rstd = rsqrtf(t / (float)s.h + s.eps);
            }
            // ---- products: the ring's panels a batch at a time, a panel's piece by as many warps as there are for each
            int piece = plan.piece, batch = 0;
#pragma unroll 1
            for (int u = 0; u < panels * pieces; u += at_once, ++batch) {
                const int units = min(at_once, panels * pieces - u);
                if (batch > 0) {               // (a slot's barrier is looked at only when its piece before has been read)
                    os_sync();
                    await(units);
                }
                if (plan.unit < units) {
                    int ring = slot + plan.unit;
                    if (ring >= a.slots) ring -= a.slots;
                    const bool last = piece == pieces - 1;
                    const int lo = last ? plan.last_lo : plan.lo, n = last ? plan.last_n : plan.n;
                    const int stride = (last ? last_steps : a.piece >> 4) * 32 + 16;
                    float c[2][4] = {};
                    uint32_t wa = smem_u32(smem + ring * a.slot_bytes) + (uint32_t)((lane & 15) * stride + (lane >> 4) * 16 + lo * 32);
                    const uint4* xp = reinterpret_cast<const uint4*>(xs + piece * a.piece + lo * 16) + (lane & 3);
#pragma unroll 2
                    for (int i = 0; i < n; i += 2, wa += 64, xp += 4) {
                        uint32_t w0[4], w1[4];
                        const uint4 x = lane < 4 ? *xp : make_uint4(0, 0, 0, 0);
                        ldsm_x4(wa, w0);
                        mma_bf16(c[0], w0, x.x, x.y);
                        if (i + 1 < n) {
                            ldsm_x4(wa + 32, w1);
                            mma_bf16(c[1], w1, x.z, x.w);
                        }
                    }
                    __syncwarp();
                    if (lane == 0) os_arrive(&S->empty[ring], arrive);
                    if ((lane & 3) == 0) {
                        S->red[buf][batch][warp][lane >> 2] = c[0][0] + c[1][0];
                        S->red[buf][batch][warp][(lane >> 2) + 8] = c[0][2] + c[1][2];
                    }
                }
                piece += step;
                if (piece >= pieces) piece -= pieces;
                slot += units;
                if (slot >= a.slots) slot -= a.slots, parity ^= 1;
            }
            os_sync();
            if (warp * 32 >= panels * kOsPanel) {              // (warps without rows)
                buf ^= 1;
                epoch += phase == OS_QKV ? 2 : 1;
            } else {
                float v = 0.0f, rstd = 1.0f;
                {                              // this row's panel: a run of units, from batch to batch
                    const short2 in = S->panel_plan[phase][tid >> 4];
                    const float* r = &S->red[buf][in.x][in.y * share][tid & 15];
                    const int n = pieces * share;
                    if (in.y + pieces <= at_once) {
                        float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                        for (int w = 0; w < kOsWarps; ++w) t[w & 3] += w < n ? r[w * kOsPanel] : 0.0f;
                        v = (t[0] + t[1]) + (t[2] + t[3]);
                    } else {
                        int bt = in.x, u = in.y;
                        for (int i = 0; i < pieces; ++i) {
                            r = &S->red[buf][bt][u * share][tid & 15];
                            for (int w = 0; w < share; ++w) v += r[w * kOsPanel];
                            if (++u == at_once) u = 0, ++bt;
                        }
                    }
                }
                buf ^= 1;
                if (normed) rstd = S->rstd;
                v *= rstd;
                ++epoch;
                if (phase == OS_QKV) {
                    v += os_low(extra);
                    const float o = __shfl_xor_sync(0xffffffffu, v, 1);
                    if (pair && (tid & 1) == 0) {
                        const uint32_t lo = os_bits(v * cs - o * sn), hi = os_bits(o * cs + v * sn);
                        os_store(a.w_qkv + u_qkv, lo | hi << 16, epoch);
                        if (head >= s.nh) {
                            __nv_bfloat16* dst = (rotates ? L.k_cache : L.v_cache) + kv_off;
                            *reinterpret_cast<unsigned short*>(dst) = (unsigned short)lo;
                            *reinterpret_cast<unsigned short*>(dst + kHalf) = (unsigned short)hi;
                        }
                    }
                    ++epoch;                   // of the attention's result
                } else if (phase == OS_GU) {
                    const float u = __shfl_xor_sync(0xffffffffu, v, 1);
                    const uint32_t b = os_bits(__fdividef(v, 1.0f + __expf(-v)) * u), n = __shfl_down_sync(0xffffffffu, b, 2);
                    if (tid < count && (tid & 3) == 0) os_store(a.w_act + (first + (tid >> 1)) / 2, b | n << 16, epoch);
                    if (tid == 0) os_store(a.w_sign + ((size_t)OS_GU * a.grid + cta) * kOsLine, 0, epoch);
                } else if (warp == 0) {        // residual += result; the next norm's input and this CTA's sum of squares
                    float y = 0.0f;
                    if (lane < count) {
                        y = resid + v;
                        resid = y;
                        const uint32_t x = os_bits(y * os_low(extra));
                        os_store(a.w_x + first + lane, x, epoch);
                        if (it == its - 1) reinterpret_cast<unsigned short*>(s.x_out)[first + lane] = (unsigned short)x;
                    }
                    float t = y * y;
#pragma unroll
                    for (int d = 16; d >= 1; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
                    if (lane == 0) {
                        os_store(a.w_sign + ((size_t)phase * a.grid + cta) * kOsLine, __float_as_uint(t), epoch);
                        if (it == its - 1) s.sums_out[cta] = t;
                    }
                }
            }
            if (phase != OS_QKV || !attends) continue;

            // ---- attention of query head hq over keys [key0, key1)
            int key = key0 + warp * kWorkers + lane / kLanes;
            if (tid < 3 * kHalf) {             // query, and the new token's key and value, which the cache does not hold yet
                const int which = tid / kHalf, j = tid % kHalf;
                const unsigned long long* p = a.w_qkv + (which == 0 ? hq : which == 1 ? s.nh + kvh : s.nh + s.nkv + kvh) * kHalf + j;
                const uint32_t w = os_wait(p, os_load(p), epoch - 1, failed, s.err);
                const float scale = which == 0 ? 1.4426950408889634f / sqrtf((float)HD) : 1.0f;
                S->qkv[which][j] = os_low(w) * scale;
                S->qkv[which][j + kHalf] = os_high(w) * scale;
            }
            os_sync();
            float q[8], o[8], m = -INFINITY, sum = 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) q[e] = S->qkv[0][d0 + e], o[e] = 0.0f;
            // (every lane walks as often as the first worker of the warp, so that the shuffles meet)
#pragma unroll 1
            for (int k1 = key0 + warp * kWorkers; k1 < key1; k1 += kOsAhead * kStride) {
                float sc[kOsAhead], vx[kOsAhead][8], mn = m;
#pragma unroll
                for (int i = 0; i < kOsAhead; ++i) {
                    const int kk = key + i * kStride;
                    const uint32_t kw[4] = {kr[i].x, kr[i].y, kr[i].z, kr[i].w}, vw[4] = {vr[i].x, vr[i].y, vr[i].z, vr[i].w};
                    float t = 0.0f;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        t = fmaf(q[2 * e], os_low(kw[e]), t);
                        t = fmaf(q[2 * e + 1], os_high(kw[e]), t);
                        vx[i][2 * e] = os_low(vw[e]), vx[i][2 * e + 1] = os_high(vw[e]);
                    }
                    if (kk == pos && kk < key1) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) t = fmaf(q[e], S->qkv[1][d0 + e], t), vx[i][e] = S->qkv[2][d0 + e];
                    }
                    sc[i] = t;
                }
#pragma unroll
                for (int i = 0; i < kOsAhead; ++i) {
#pragma unroll
                    for (int d = kLanes / 2; d >= 1; d >>= 1) sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], d);
                    if (key + i * kStride >= key1) sc[i] = -INFINITY;
                    mn = fmaxf(mn, sc[i]);
                }
                key += kOsAhead * kStride;
                if (k1 + kOsAhead * kStride < key1) fetch(key);
                if (mn > -INFINITY) {
                    const float corr = os_ex2(m - mn);
                    sum *= corr;
#pragma unroll
                    for (int e = 0; e < 8; ++e) o[e] *= corr;
#pragma unroll
                    for (int i = 0; i < kOsAhead; ++i) {
                        const float p = os_ex2(sc[i] - mn);
                        sum += p;
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[e] = fmaf(p, vx[i][e], o[e]);
                    }
                    m = mn;
                }
            }
            // the warp's workers, then the warps
            auto merge = [&](float om, float& f, float& g) {
                const float mn = fmaxf(m, om);
                f = m > -INFINITY ? os_ex2(m - mn) : 0.0f, g = om > -INFINITY ? os_ex2(om - mn) : 0.0f;
                m = mn;
            };
#pragma unroll
            for (int d = kLanes; d < 32; d <<= 1) {
                float f, g;
                merge(__shfl_xor_sync(0xffffffffu, m, d), f, g);
                sum = sum * f + __shfl_xor_sync(0xffffffffu, sum, d) * g;
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = o[e] * f + __shfl_xor_sync(0xffffffffu, o[e], d) * g;
            }
            if (lane < kLanes)
#pragma unroll
                for (int e = 0; e < 8; ++e) S->head_o[warp][d0 + e] = o[e];
            if (lane == 0) S->head_m[warp] = m, S->head_l[warp] = sum;
            os_sync();
            if (tid < HD) {
                float al = 0.0f, ao = 0.0f;
                const int busy = min(kOsWarps, (key1 - key0 + kWorkers - 1) / kWorkers);        // warps that had a key
                float hm[kOsWarps];
                m = -INFINITY;
#pragma unroll
                for (int w = 0; w < kOsWarps; ++w) hm[w] = w < busy ? S->head_m[w] : -INFINITY, m = fmaxf(m, hm[w]);
#pragma unroll
                for (int w = 0; w < kOsWarps; ++w) {
                    const float f = w < busy ? os_ex2(hm[w] - m) : 0.0f;
                    al += w < busy ? S->head_l[w] * f : 0.0f;
                    ao += w < busy ? S->head_o[w][tid] * f : 0.0f;
                }
                unsigned long long* part = a.w_part + (size_t)hq * (a.splits - 1) * (HD + 2);
                if (sp > 0) {
                    part += (size_t)(sp - 1) * (HD + 2);
                    os_store(part + tid, __float_as_uint(ao), epoch);
                    if (tid == 0) os_store(part + HD, __float_as_uint(m), epoch), os_store(part + HD + 1, __float_as_uint(al), epoch);
                } else {
#pragma unroll 1
                    for (int i = 1; i < a.splits; ++i, part += HD + 2) {
                        const unsigned long long vm = os_load(part + HD), vl = os_load(part + HD + 1), vo = os_load(part + tid);
                        float f, g;
                        merge(__uint_as_float(os_wait(part + HD, vm, epoch, failed, s.err)), f, g);
                        al = al * f + __uint_as_float(os_wait(part + HD + 1, vl, epoch, failed, s.err)) * g;
                        ao = ao * f + __uint_as_float(os_wait(part + tid, vo, epoch, failed, s.err)) * g;
                    }
                    const uint32_t b = os_bits(ao / al), n = __shfl_down_sync(0xffffffffu, b, 1);
                    if ((tid & 1) == 0) os_store(a.w_attn + (hq * HD + tid) / 2, b | n << 16, epoch);
                    if (tid == 0) os_store(a.w_sign + hq * kOsLine, 0, epoch);        // (phase OS_QKV's place)
                }
            }
        }
    }
    __syncthreads();
    wait_settle(guard);
    if (tid == 0 && atomicAdd(&s.sync[1], 1u) == (unsigned)a.grid - 1) {       // the last CTA out: numbers for the next step
        s.sync[1] = 0;
        s.sync[0] = S->base + 5u * s.n_layers;
    }
}

size_t os_words(int h, int nqkv, int qdim, int ffn, int grid) {
    return (size_t)nqkv / 2 + qdim / 2 + (size_t)grid * 130 + h + ffn / 2 + 4 * grid * kOsLine + 3 * kOsLine;
}

}  // namespace

int one_step_sums() { return sm_count(); }

size_t one_step_bytes(int h, int nqkv, int qdim, int ffn) { return 64 + 8 * os_words(h, nqkv, qdim, ffn, sm_count()); }

bool one_step_takes(const OneStep& s) {
    DeviceLimits dev;
    if (device_limits(&dev)) return false;
    return one_step_sizes(s, dev.sms) && one_step_bytes(s.h, s.nqkv, s.qdim, s.ffn) > 0 && s.work;
}

int one_step_launch(const OneStep& s, int max_kv_len, cudaStream_t stream) {
    DeviceLimits dev;
    if (device_limits(&dev)) return -1;
    OsArgs a = {};
    a.s = s;
    a.grid = dev.sms, a.group = s.nh / s.nkv;
    a.s.sync = static_cast<unsigned*>(s.work);
    unsigned long long* w = reinterpret_cast<unsigned long long*>(static_cast<char*>(s.work) + 64);
    a.w_qkv = w, w += s.nqkv / 2;
    a.w_attn = w, w += s.qdim / 2;
    a.w_part = w, w += (size_t)a.grid * 130;
    a.w_x = w, w += s.h;
    a.w_act = w, w += s.ffn / 2;
    a.w_sign = reinterpret_cast<unsigned long long*>((reinterpret_cast<uintptr_t>(w) + 127) & ~uintptr_t(127));
    // a share of the keys is what its workers have on their way at once, if there are SMs for as many
    const int at_once = kOsAhead * kOsWarps * (256 / s.hd);
    a.splits = std::max(1, std::min(a.grid / s.nh, (max_kv_len + at_once - 1) / at_once));
    // panels as long as the rows of the hidden size, at most 1024, in whole swaths of 64 (rows 16 bytes longer than a multiple of 128 lie
    // on different banks)
    a.piece = s.h <= kOsMaxPiece ? (s.h + 63) / 64 * 64 : kOsMaxPiece;
    a.slot_bytes = kOsPanel * (a.piece * 2 + 16);
    a.x_bytes = (std::max(std::max(s.h, s.qdim), s.ffn) * 2 + 127) / 128 * 128;
    a.slots = std::min(16, (dev.smem_optin - a.x_bytes - (int)sizeof(OsShared) - 128) / a.slot_bytes);
    if (a.slots < 3) return 1;
    // batches of units that the ring holds: at most as many as there is room for their sums
    const int once = std::min(a.slots, kOsWarps);
    auto batches = [&](int rows, int K) { return ((rows + kOsPanel - 1) / kOsPanel * ((K + a.piece - 1) / a.piece) + once - 1) / once; };
    auto most = [&](int n) { return (n + a.grid - 1) / a.grid; };
    if (std::max(std::max(batches(2 * most(s.nqkv / 2), s.h), batches(most(s.h), s.qdim)),
                 std::max(batches(4 * most(s.ffn / 2), s.h), batches(most(s.h), s.ffn))) > kOsMaxPanels)
        return 1;
    const int smem = a.slots * a.slot_bytes + a.x_bytes + (int)sizeof(OsShared);
    auto fn = s.hd == 64 ? one_step_kernel<64> : one_step_kernel<128>;
    if (preload_one_step()) return -1;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;       // all CTAs resident, or an error
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3(a.grid);
    cfg.blockDim = dim3(kOsThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (const int rc = grid_in_turn(stream, [&] { return cudaLaunchKernelEx(&cfg, fn, a); })) return rc;
    count_kernel(KERNEL_ONE_STEP);
    return 0;
}

int preload_one_step() {
    static PerDeviceOnce once;
    ASD_ONCE(once, {
        DeviceLimits dev;
        if (device_limits(&dev)) return -1;
        ASD_CUDA(cudaFuncSetAttribute(one_step_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.smem_optin));
        ASD_CUDA(cudaFuncSetAttribute(one_step_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.smem_optin));
    });
    return 0;
}

}  // namespace asd
