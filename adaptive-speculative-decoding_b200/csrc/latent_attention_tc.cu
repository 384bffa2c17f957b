// Latent key/value attention in latent space on tcgen05 / TMEM for bf16 cache rows: the kernel of every call that brings
// enough query rows (prompts, verifications, single tokens of many heads).  Same contract as latent_attention.cu.
//
// What bounds it: the fp32 query enters as three bf16 terms (24 bits) and the fp32 weights as two, so a (query row, key)
// pair costs 3 (R + dr) + 2 R multiply-adds; on mma.sync (latent_attn_mma) that ran at a fifth of the legacy rate.
//   * CTA = 128 query rows (consecutive tokens x all heads of one sequence: they share their keys) x half of the latent
//     columns of the result x one share of the keys.  128 lanes x 256 result columns and two 128-key score tiles fill the
//     512 columns of TMEM, so a latent of 512 takes two CTAs that both form the scores; one CTA would have to spill.
//   * Keys come by TMA straight from the paged pool, 64 row elements x one page a box, in the K-major 128-byte swizzle.  The
//     chunks that hold this CTA's result columns wait in a ring of six 16 KB slots, because the same bytes are the value
//     operand (MN-major: keys are the contraction dimension); the others pass through two slots of their own.
//   * The query's terms do not fit beside the keys (442 KB): the three planes that the projection wrote stream from L2
//     through two 48 KB slots, one 3-D box (64 columns of all three) a chunk, once per 128 keys.
//   * The order inside a tile hides the softmax and the value product: scores of tile j + 1 over the chunks that are only
//     keys, then the value product of tile j, which frees its slots, then the chunks that are values too.  Four warps
//     (thread = query row = TMEM lane) meanwhile take the running maximum of tile j and write its weights back over the
//     scores as two bf16 terms, the A operand of the value product.  The result accumulates in TMEM; it is rescaled only
//     when a row's maximum has grown by more than 8 (in log2) over the one its weights refer to, which keeps every weight
//     below 2^8 and the sums exact in fp32.
//   * A thread needs ~200 clocks to wait for a barrier and issue one box or four products, so boxes are as large as the
//     layout allows, a query slot feeds twelve products, three warps load, and the issuing warp walks its loops whole (a
//     first form with 16 KB slots, one loader and one issuing thread took 666 us where the next took 366).
// Four prompts of 1024 tokens, 16 heads, latent 512 + 64: 1350 us on mma.sync, 354 here (185 GFLOP: 0.52 PFLOP/s).
// Every wait is bounded: on expiry the kernel raises the caller's error flag, lets its copies land, frees its TMEM and ends.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "asd_internal.h"
#include "blocks.h"
#include "gemm.h"
#include "ptx.cuh"

namespace asd {

namespace {

constexpr int kLtThreads = 256;            // warps 0-3 softmax (thread = query row), 4 query loader, 5 MMA, 6-7 key loaders
constexpr int kLtKeys = 128;               // keys per tile
constexpr int kLtSlot = 128 * 128;         // bytes of 128 rows x 64 bf16
constexpr int kLtVSlots = 6;               // ring of key chunks that are values too
constexpr int kLtKSlots = 2;               // ring of the other key chunks
constexpr int kLtQSlots = 2;               // ring of query chunks, three terms each
constexpr int kLtMaxV = 4;                 // chunks of 64 result columns per CTA
constexpr float kLtSlack = 8.0f;           // log2 growth of a row maximum that the weights tolerate before a rescale
constexpr uint32_t kLtSpin = 1u << 20;
// Query rows of a tile from which this kernel is the better one.  A tile costs what 128 rows cost, however many are real:
// 64 single tokens of 32 heads at 1024 positions: 146 us on mma.sync, 96 us here; 16 of 16 heads at 1500: 58 us there, 72 here
// when the line was drawn (4096 prompt tokens of 16 heads, 128 rows a tile: 1350 and 354).
constexpr int kLtMinRows = 32;

struct LtArgs {
    const int* positions;
    const int* cu_q;
    const int* seq_slot;
    const int* page_table;
    int max_pages, page_shift;
    int heads, HG, TQ, R, rw, parts, hgs, nsplit, window, box_rows;
    float scale2;                          // score scale x log2(e)
    float* out_lat;                        // [M][heads][R]
    float *ws_o, *ws_ml;
    int* err;
};

struct LtBars {
    uint64_t q_full[kLtQSlots], q_empty[kLtQSlots], k_full[kLtKSlots], k_empty[kLtKSlots], v_full[kLtVSlots], s_full[2],
        pv_done[2], p_full;
    uint32_t tmem;
    int failed;
};

__device__ __forceinline__ void lt_report(LtBars* B, int* err) {
    *reinterpret_cast<volatile int*>(&B->failed) = 1;
    if (err) {
        *const_cast<volatile int*>(err) = WAIT_LATENT << 8 | 1;
        __threadfence_system();
    }
}
__device__ __forceinline__ bool lt_wait(uint64_t* bar, uint32_t parity, LtBars* B, int* err) {
    for (uint32_t i = 0; i < kLtSpin; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*reinterpret_cast<volatile int*>(&B->failed)) return false;
    }
    lt_report(B, err);
    return false;
}
// the same by a whole warp, one answer for all lanes: what follows stays uniform
__device__ __forceinline__ bool lt_wait_warp(uint64_t* bar, uint32_t parity, LtBars* B, int* err) {
    for (uint32_t i = 0; i < kLtSpin; ++i) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        if (__any_sync(0xffffffffu, *reinterpret_cast<volatile int*>(&B->failed))) return false;
    }
    lt_report(B, err);
    return false;
}
// a place in a ring of barriers and the parity of its current round
struct LtRing {
    int slot = 0;
    uint32_t round = 0;
    __device__ __forceinline__ void step(int n) {
        if (++slot == n) slot = 0, round ^= 1;
    }
};
__device__ __forceinline__ void lt_settle(uint64_t* bar, uint32_t parity) {     // after a failure: let a copy land, bounded
    for (uint32_t i = 0; i < kLtSpin && !mbar_try_wait(bar, parity); ++i) {
    }
}
// MN-major SW128 operand (keys along rows of 128 B = 64 columns, 8-key atoms 1024 B apart, the next 64 columns a slot further)
__device__ __forceinline__ uint64_t lt_desc_mn(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(kLtSlot >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// {columns, rows, planes} box into shared memory
__device__ __forceinline__ void lt_load_3d(void* dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ float lt_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// weights of 32 scores -> 16 packed pairs of their high terms and 16 of what is left (a score of -inf: weight 0)
__device__ __forceinline__ void lt_weights(const uint32_t (&v)[32], float scale, float nref, uint32_t (&ph)[16], uint32_t (&pl)[16],
                                           float (&sum)[4]) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const float p0 = lt_ex2(fmaf(__uint_as_float(v[i]), scale, nref));
        const float p1 = lt_ex2(fmaf(__uint_as_float(v[i + 1]), scale, nref));
        sum[(i >> 1) & 3] += p0 + p1;
        const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
        const float2 f = __bfloat1622float2(h);
        const __nv_bfloat162 r = __floats2bfloat162_rn(p0 - f.x, p1 - f.y);
        ph[i >> 1] = *reinterpret_cast<const uint32_t*>(&h);
        pl[i >> 1] = *reinterpret_cast<const uint32_t*>(&r);
    }
}
// bits i of 32 elements with lo <= i <= hi
__device__ __forceinline__ uint32_t lt_bits(int lo, int hi) {
    const uint32_t upto = hi < 0 ? 0u : (hi >= 31 ? 0xffffffffu : (2u << hi) - 1u);
    const uint32_t from = lo <= 0 ? 0xffffffffu : (lo > 31 ? 0u : 0xffffffffu << lo);
    return upto & from;
}

__global__ void __launch_bounds__(kLtThreads, 1)
    latent_attn_tc(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv, const LtArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sV = smem;                                        // [kLtVSlots]
    uint8_t* sK = sV + kLtVSlots * kLtSlot;                    // [kLtKSlots]
    uint8_t* sQ = sK + kLtKSlots * kLtSlot;                    // [kLtQSlots][3 terms]
    LtBars* B = reinterpret_cast<LtBars*>(sQ + kLtQSlots * 3 * kLtSlot);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int seq = blockIdx.y / a.nsplit, split = blockIdx.y % a.nsplit;
    // the CTAs that share a query tile are neighbours (its terms then meet in L2); the last tiles see the most keys and start first
    const int shared = a.hgs * a.parts, tile_x = (int)(gridDim.x / shared) - 1 - (int)blockIdx.x / shared;
    const int part = blockIdx.x % a.parts, h0 = (int)(blockIdx.x % shared) / a.parts * a.HG;
    const int t0 = a.cu_q[seq] + tile_x * a.TQ;
    const int t_end = a.cu_q[seq + 1];
    const int* pt = a.page_table + (long long)a.seq_slot[seq] * a.max_pages;
    if (t0 >= t_end) return;
    const int n_tok = min(a.TQ, t_end - t0);
    const int p_first = a.positions[t0], p_last = a.positions[t0 + n_tok - 1];
    const int j_lo = max(p_first - a.window + 1, 0);
    const int base = j_lo & ~(kLtKeys - 1);                    // tiles start at multiples of 128 positions: whole pages
    const int tiles = (p_last - base) / kLtKeys + 1, per = (tiles + a.nsplit - 1) / a.nsplit;
    const int ts = split * per, nt = min(tiles, ts + per) - ts;
    const int vcols = a.R / a.parts, vch = vcols >> 6, v0 = part * vch, nch = a.rw >> 6;

    // query row of this thread (warps 0-3): row r = (token r / HG, head h0 + r % HG)
    const int tq = tid / a.HG, hd = h0 + tid % a.HG;
    const bool real = tid < a.TQ * a.HG && tq < n_tok && hd < a.heads;
    const long long row = (long long)(t0 + (real ? tq : 0)) * a.heads + (real ? hd : 0);
    if (nt <= 0) {                                             // an empty share of a short sequence
        if (real && warp < 4) {
            float* dst = a.ws_o + (row * a.nsplit + split) * a.R + part * vcols;
            for (int c = 0; c < vcols; ++c) dst[c] = 0.0f;
            if (part == 0) a.ws_ml[(row * a.nsplit + split) * 2] = -INFINITY, a.ws_ml[(row * a.nsplit + split) * 2 + 1] = 0.0f;
        }
        return;
    }
    const int psh = a.page_shift, pages = kLtKeys >> psh, last_page = p_last >> psh;
    const int my = (warp - 6) * ((pages + 1) / 2) + lane;
    const bool mine = warp >= 6 && lane < (pages + 1) / 2 && my < pages;
    const int first_page = mine ? pt[min((base + ts * kLtKeys >> psh) + my, last_page)] : 0;
    if (tid == 0) {
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_kv);
        for (int i = 0; i < kLtQSlots; ++i) {
            mbar_init(&B->q_full[i], 1);
            mbar_init(&B->q_empty[i], 1);
        }
        for (int i = 0; i < kLtKSlots; ++i) {
            mbar_init(&B->k_full[i], 2);       // two loading warps
            mbar_init(&B->k_empty[i], 1);
        }
        for (int i = 0; i < kLtVSlots; ++i) mbar_init(&B->v_full[i], 2);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->s_full[i], 1);
            mbar_init(&B->pv_done[i], 1);
        }
        mbar_init(&B->p_full, 4);
        B->failed = 0;
        fence_mbar_init();
    }
    if (warp == 5) {
        tmem_alloc(&B->tmem, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = B->tmem;                             // columns 0-255: scores / weights of two tiles, 256-: result

    // chunk i of a tile, in the order of its products: first the chunks that are only keys, then this CTA's values
    // (its ring: two tiles' worth, of four chunks one and a half; a slot's earlier user is then at most two tiles back, so that
    // the parity of pv_done names it)
    const int kch = nch - vch, nv = min(kLtVSlots, 2 * vch);
    auto chunk_at = [&](int i) { return i >= kch ? v0 + i - kch : (i < v0 ? i : i + vch); };

    if (warp == 4) {
        // ------------------------------------------------------------------ query loader
        if (lane == 0) {
            const int q_row = t0 * a.heads + h0, bytes = 3 * a.box_rows * 128, total = nt * nch;
            LtRing rq;
            int it = 0, i = 0;
            for (bool ok = true; it < total && ok; ++it) {
                if (it >= kLtQSlots) ok = lt_wait(&B->q_empty[rq.slot], rq.round ^ 1, B, a.err);
                if (!ok) break;
                mbar_expect_tx(&B->q_full[rq.slot], bytes);
                lt_load_3d(sQ + rq.slot * 3 * kLtSlot, &map_q, chunk_at(i) * 64, q_row, 0, &B->q_full[rq.slot]);
                rq.step(kLtQSlots);
                if (++i == nch) i = 0;
            }
            if (it < total)                                    // given up: what is in flight lands before the memory goes
                for (int s = 0; s < kLtQSlots && s < it; ++s) lt_settle(&B->q_full[s], ((it - 1 - s) / kLtQSlots) & 1);
        }
        __syncwarp();
    } else if (warp >= 6) {
        // ------------------------------------------------------------------ key loaders: a lane per page, half of them each
        const int n_mine = __popc(__ballot_sync(0xffffffffu, mine));
        LtRing rk, rv;
        int kn = 0, vn = 0;                                    // chunks begun
        bool ok = true;
        // pages past the end repeat the sequence's last one: their keys are masked, their values zeroed
        int next = first_page;
        for (int j = 0; j < nt && ok; ++j) {
            const int page = next;
            if (j + 1 < nt && mine) next = pt[min((base + (ts + j + 1) * kLtKeys >> psh) + my, last_page)];
            for (int i = 0; i < nch; ++i) {
                uint64_t* bar;
                uint8_t* dst;
                if (i < kch) {
                    if (kn >= kLtKSlots) ok = lt_wait_warp(&B->k_empty[rk.slot], rk.round ^ 1, B, a.err);
                    bar = &B->k_full[rk.slot];
                    dst = sK + rk.slot * kLtSlot;
                } else {
                    if (vn >= nv) {                            // the tile that used the slot before has been multiplied
                        const int jp = i - kch + vch >= nv ? j - 1 : j - 2;
                        ok = lt_wait_warp(&B->pv_done[jp & 1], (jp >> 1) & 1, B, a.err);
                    }
                    bar = &B->v_full[rv.slot];
                    dst = sV + rv.slot * kLtSlot;
                }
                if (!ok) break;
                if (i < kch)
                    ++kn, rk.step(kLtKSlots);
                else
                    ++vn, rv.step(nv);
                if (lane == 0) mbar_expect_tx(bar, n_mine << (psh + 7));
                __syncwarp();
                if (mine) tma_load_2d(dst + ((size_t)my << (psh + 7)), &map_kv, chunk_at(i) * 64, page << psh, bar);
                __syncwarp();
            }
        }
        if (!ok) {
            for (int s = 0; s < kLtKSlots && s < kn; ++s) lt_settle(&B->k_full[s], ((kn - 1 - s) / kLtKSlots) & 1);
            for (int s = 0; s < nv && s < vn; ++s) lt_settle(&B->v_full[s], ((vn - 1 - s) / nv) & 1);
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------------ MMA issuer
        // The whole warp walks the loops, so that addresses and descriptors stay in uniform registers, and one lane issues.
        const bool lead = elect_one();
        const uint32_t id_s = umma_idesc_bf16(128, 128);
        const uint32_t uV = smem_u32(sV), uK = smem_u32(sK), uQ = smem_u32(sQ);
        const uint32_t term = (uint32_t)a.box_rows * 128u >> 4;        // between a slot's terms, in descriptor units
        LtRing rq, rk, rv;
        int pv_slot = 0;
        bool ok = true;
        auto scores = [&](int j, int i0, int i1) {
            const uint32_t d = tmem + (uint32_t)((j & 1) * 128);
            for (int i = i0; i < i1 && ok; ++i) {
                uint64_t *bar, *free_k = nullptr;
                uint32_t k_addr;
                if (i < kch) {
                    ok = lt_wait_warp(&B->k_full[rk.slot], rk.round, B, a.err);
                    k_addr = uK + (uint32_t)(rk.slot * kLtSlot);
                    free_k = &B->k_empty[rk.slot];
                    rk.step(kLtKSlots);
                } else {
                    ok = lt_wait_warp(&B->v_full[rv.slot], rv.round, B, a.err);
                    k_addr = uV + (uint32_t)(rv.slot * kLtSlot);
                    rv.step(nv);
                }
                ok = ok && lt_wait_warp(&B->q_full[rq.slot], rq.round, B, a.err);
                if (!ok) break;
                tc_fence_after();
                const uint64_t kd = umma_desc_sw128(k_addr), qd = umma_desc_sw128(uQ + (uint32_t)(rq.slot * 3 * kLtSlot));
                bar = &B->q_empty[rq.slot];
                rq.step(kLtQSlots);
                if (lead) {
#pragma unroll
                    for (int u = 2; u >= 0; --u)               // the low term first
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16(d, qd + u * term + 2 * k, kd + 2 * k, id_s, u != 2 || k != 0 || i != 0);
                    umma_commit(bar);
                    if (free_k) umma_commit(free_k);
                }
                __syncwarp();
            }
        };
        auto values = [&](int j) {
            ok = ok && lt_wait_warp(&B->p_full, j & 1, B, a.err);
            if (!ok) return;
            tc_fence_after();
            const uint32_t p = tmem + (uint32_t)((j & 1) * 128);
            // a tile's chunks lie in consecutive slots of the ring, or in two runs of them
            for (int c = 0; c < vch;) {
                const int n = min(vch - c, nv - pv_slot);
                const uint32_t id_v = umma_idesc_bf16(128, (uint32_t)n * 64) | (1u << 16);     // B is MN-major
                const uint64_t vd = lt_desc_mn(uV + (uint32_t)(pv_slot * kLtSlot));
                const uint32_t d = tmem + 256u + (uint32_t)c * 64u;
                if (lead) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {              // 16 keys; their high and low terms lie 32 columns apart
                        const uint32_t pc = p + (uint32_t)((k >> 2) * 64 + (k & 3) * 8);
                        umma_f16_ts(d, pc + 32, vd + k * (2048 >> 4), id_v, (j | k) != 0);
                        umma_f16_ts(d, pc, vd + k * (2048 >> 4), id_v, 1);
                    }
                }
                __syncwarp();
                c += n;
                pv_slot += n;
                if (pv_slot == nv) pv_slot = 0;
            }
            if (lead) umma_commit(&B->pv_done[j & 1]);
            __syncwarp();
        };
        for (int j = 0; j < nt && ok; ++j) {
            // the scores of tile j take the buffer of tile j - 2, whose value product was issued before them
            if (j >= 2) ok = lt_wait_warp(&B->pv_done[j & 1], ((j >> 1) - 1) & 1, B, a.err);
            scores(j, 0, kch);
            if (j > 0) values(j - 1);
            scores(j, kch, nch);
            if (lead) umma_commit(&B->s_full[j & 1]);
            __syncwarp();
        }
        values(nt - 1);
    } else {
        // ------------------------------------------------------------------ softmax (thread = query row)
        const int pos = real ? a.positions[t0 + tq] : -1;
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
        float ref = -INFINITY, l = 0.0f;                       // the maximum the weights refer to (log2), and their sum
        bool ok = true;
        // A row's 128 scores are read once and stay in registers.  Cut tiles turn what a row may not see into -inf beforehand, by
        // bits (as comparisons the compiler branched on every element: 10000 to 14000 clocks a cut tile).  4 prompts of 1024 tokens, 16
        // heads: 370 -> 354 us, 64 single tokens of 32 heads at 1024 positions 104 -> 96; the products wait for their operands, from
        // L2, most of what is left.
        auto tile = [&](int j, bool whole) {
            const int key0 = base + (ts + j) * kLtKeys;
            const uint32_t tS = lanes + (uint32_t)((j & 1) * 128);
            uint32_t x[4][32];
#pragma unroll
            for (int q = 0; q < 4; ++q) tmem_ld_32x32(tS + (uint32_t)(q * 32), x[q]);
            tmem_ld_wait();
            if (!whole) {
                const int hi = pos - key0, lo = pos - a.window + 1 - key0;      // element i is visible iff lo <= i <= hi
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t bits = lt_bits(lo - q * 32, hi - q * 32);
#pragma unroll
                    for (int i = 0; i < 32; ++i) x[q][i] = bits & (1u << i) ? x[q][i] : 0xff800000u;
                }
            }
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(x[q][i]));
            // rn products with a positive scale keep the order; a negative or zero one is refused by the host
            const float top = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale2;
            const bool grow = real && (top > ref + kLtSlack || (ref == -INFINITY && top > -INFINITY));
            if (__any_sync(0xffffffffu, grow)) {
                const float corr = grow ? lt_ex2(ref - top) : 1.0f;        // ref = -inf: 0, of a row that is 0 so far
                if (j > 0) {
                    if (!lt_wait_warp(&B->pv_done[(j - 1) & 1], ((j - 1) >> 1) & 1, B, a.err)) {
                        ok = false;
                        return;
                    }
                    tc_fence_after();
                    for (int c = 0; c < vcols; c += 32) {
                        uint32_t v[32], w[16];
                        tmem_ld_32x32(lanes + 256u + (uint32_t)c, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * corr);
#pragma unroll
                        for (int i = 0; i < 16; ++i) w[i] = v[i];
                        tmem_st_32x16(lanes + 256u + (uint32_t)c, w);
#pragma unroll
                        for (int i = 0; i < 16; ++i) w[i] = v[16 + i];
                        tmem_st_32x16(lanes + 256u + (uint32_t)c + 16u, w);
                    }
                }
                l *= corr;
                if (grow) ref = top;
            }
            const float nref = ref == -INFINITY ? 0.0f : -ref;
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int q = 0; q < 4; ++q) {      // two quarters' high terms lie side by side, then their low terms
                uint32_t ph[16], pl[16];
                lt_weights(x[q], a.scale2, nref, ph, pl, sum);
                const uint32_t at = tS + (uint32_t)((q >> 1) * 64 + (q & 1) * 16);
                tmem_st_32x16(at, ph);
                tmem_st_32x16(at + 32u, pl);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        };
        for (int j = 0; j < nt && ok; ++j) {
            const int key0 = base + (ts + j) * kLtKeys;
            if (!lt_wait_warp(&B->s_full[j & 1], (j >> 1) & 1, B, a.err)) break;
            tc_fence_after();
            const bool whole = key0 + kLtKeys <= p_first + 1 && key0 >= p_last - a.window + 1;     // every row sees every key
            tile(j, whole);
            if (!ok) break;
            if (key0 + kLtKeys > p_last + 1 || key0 < j_lo) {
                // keys that no row of the tile may see: whatever the pool holds there must not meet the zero weights
                const int kp = key0 + tid;
                if (kp > p_last || kp < j_lo)
                    for (int c = 0, sl = j * vch % nv; c < vch; ++c, sl = sl + 1 == nv ? 0 : sl + 1) {
                        uint4* dst = reinterpret_cast<uint4*>(sV + sl * kLtSlot + tid * 128);
#pragma unroll
                        for (int i = 0; i < 8; ++i) dst[i] = make_uint4(0, 0, 0, 0);
                    }
                fence_proxy_async_smem();
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->p_full);
        }
        ok = ok && lt_wait_warp(&B->pv_done[(nt - 1) & 1], ((nt - 1) >> 1) & 1, B, a.err);
        tc_fence_after();
        if (ok) {
            const bool direct = a.nsplit == 1;
            const float mul = direct ? 1.0f / l : 1.0f;
            // rows through shared memory (every load and product has ended): a warp then writes whole rows, 16 bytes a lane side
            // by side, where a thread per row wrote 16 bytes here and there (14000 clocks of the tile's end)
            const int ld = vcols / 4 + 1;                      // float4s; odd: the lanes' rows spread over the banks
            float4* own = reinterpret_cast<float4*>(smem) + (size_t)warp * 32 * ld;
            for (int c = 0; c < vcols; c += 32) {
                uint32_t v[32];
                tmem_ld_32x32(lanes + 256u + (uint32_t)c, v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; i += 4)
                    own[lane * ld + (c + i) / 4] = make_float4(__uint_as_float(v[i]) * mul, __uint_as_float(v[i + 1]) * mul,
                                                               __uint_as_float(v[i + 2]) * mul, __uint_as_float(v[i + 3]) * mul);
            }
            __syncwarp();
            const unsigned live = __ballot_sync(0xffffffffu, real);
            float* const to = direct ? a.out_lat : a.ws_o;
            const long long at = (direct ? row : row * a.nsplit + split) * a.R + part * vcols;
            const int q4 = vcols / 4;                          // at most 64
#pragma unroll 8
            for (int r = 0; r < 32; ++r) {
                float4* dst = reinterpret_cast<float4*>(to + __shfl_sync(0xffffffffu, at, r));
                const bool put = live >> r & 1;
                if (put && lane < q4) dst[lane] = own[r * ld + lane];
                if (put && lane + 32 < q4) dst[lane + 32] = own[r * ld + lane + 32];
            }
            if (real && !direct && part == 0) {
                a.ws_ml[(row * a.nsplit + split) * 2] = ref * 0.69314718055994531f;    // natural units, as the merge expects
                a.ws_ml[(row * a.nsplit + split) * 2 + 1] = l;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace

// How launch_latent_attention_tc cuts a call: rows per tile and the number of (tile, head group, part) CTAs per share.
struct LtPlan {
    int HG, TQ, hgs, parts, rows, q_tiles;
};
static LtPlan lt_plan(const LatentDims& d, int max_qlen) {
    LtPlan p;
    p.HG = d.heads < 128 ? d.heads : 128;
    p.TQ = std::min(128 / p.HG, max_qlen);
    p.hgs = (d.heads + p.HG - 1) / p.HG;
    p.parts = d.R > 256 ? 2 : 1;
    p.rows = p.TQ * p.HG;
    p.q_tiles = (max_qlen + p.TQ - 1) / p.TQ;
    return p;
}

bool latent_attention_tc_takes(const LatentDims& d, const PagedRows& cache, int max_qlen, int tiled) {
    const int parts = d.R > 256 ? 2 : 1, rw = d.R + d.dr;
    if (tiled < 2 || cache.f32 || cache.rows <= 0 || cache.rows >= (1ll << 31) || max_qlen <= 0 || !(d.scale > 0.f)) return false;
    if (d.R <= 0 || d.R > 512 || d.R % (64 * parts) || rw % 64 || d.window <= 0) return false;
    if (cache.page_size < 8 || cache.page_size > kLtKeys || (cache.page_size & (cache.page_size - 1))) return false;
    if (reinterpret_cast<uintptr_t>(cache.pool) & 15) return false;
    return lt_plan(d, max_qlen).rows >= kLtMinRows;
}

int launch_latent_attention_tc(const SeqIndex& ix, const int* cu_q, const int* seq_slot, int nseq, int max_qlen,
                               int max_kv_len, const __nv_bfloat16* q_terms, const LatentDims& d, const PagedRows& cache,
                               float* out_lat, const AttnSplit& ws, int* err, cudaStream_t stream) {
    if (ix.M <= 0 || nseq <= 0) return 0;
    const LtPlan p = lt_plan(d, max_qlen);
    const int rw = d.R + d.dr;
    const long long rows = (long long)ix.M * d.heads;
    if (3 * rows >= (1ll << 31)) return set_error("latent attention: too many query rows");
    LtArgs a;
    a.positions = ix.positions, a.cu_q = cu_q, a.seq_slot = seq_slot;
    a.page_table = cache.page_table, a.max_pages = cache.max_pages;
    a.page_shift = 0;
    while ((1 << a.page_shift) < cache.page_size) ++a.page_shift;
    a.heads = d.heads, a.HG = p.HG, a.TQ = p.TQ, a.R = d.R, a.rw = rw, a.parts = p.parts, a.hgs = p.hgs, a.window = d.window;
    a.box_rows = std::min(128, (p.rows + 7) & ~7);
    a.scale2 = d.scale * 1.4426950408889634f;
    a.out_lat = out_lat, a.ws_o = ws.o, a.ws_ml = ws.ml, a.err = err;
    // few query tiles: the keys are cut into shares until every SM has a CTA, of at least two tiles each
    a.nsplit = 1;
    const long long ctas = (long long)p.q_tiles * p.hgs * p.parts * nseq;
    const int sms = sm_count();
    if (ws.o && ws.ml && ctas < sms) {
        const long long keys = std::min<long long>(d.window, max_kv_len) + p.TQ + kLtKeys;
        long long n = std::min<long long>(sms / ctas, keys / (2 * kLtKeys));
        n = std::min(n, std::min(ws.rows / rows, ws.o_elems / (rows * d.R)));
        a.nsplit = (int)std::max<long long>(1, std::min<long long>(n, 64));
    }
    if ((long long)nseq * a.nsplit > 65535) return set_error("latent attention: too many sequences");
    CUtensorMap mq, mk;
    if (make_tmap_bf16_planes(&mq, q_terms, rows, rw, 3, a.box_rows)) return -1;
    if (make_tmap_bf16(&mk, cache.pool, cache.rows, rw, rw, cache.page_size)) return -1;
    const int smem = 1024 + (kLtVSlots + kLtKSlots + 3 * kLtQSlots) * kLtSlot + (int)sizeof(LtBars);
    static PerDeviceOnce once;
    ASD_ONCE(once, ASD_CUDA(cudaFuncSetAttribute(latent_attn_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)));
    const dim3 grid(p.q_tiles * p.hgs * p.parts, nseq * a.nsplit);
    latent_attn_tc<<<grid, kLtThreads, smem, stream>>>(mq, mk, a);
    count_kernel(KERNEL_LATENT_TC);
    ASD_CUDA(cudaGetLastError());
    if (a.nsplit > 1) return launch_latent_combine(ws.o, ws.ml, a.nsplit, d.R, out_lat, rows, stream);
    return 0;
}

}  // namespace asd
