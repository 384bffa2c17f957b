// Latent key/value attention of prompts in HEAD space on tcgen05 / TMEM: the same result as latent_attention_tc.cu, which scores every
// (query row, key) pair in the latent space, over 3 (R + dr) + 2 R products of which two CTAs form the first part twice: 4480
// multiply-adds a pair at 512 + 64.  That serves few tokens over many cached positions.  A prompt brings about as many tokens as it
// sees positions, and carrying the POSITIONS through the up-projections once, instead of every query through the key's and every
// result through the value's, leaves 960 a pair and neither head product:
//   * latent_rows_kernel copies the visible cache rows of every sequence out of their pages, padded with zeros to whole tiles of 128;
//   * gemm_tc.cu multiplies them with the stacked key / value up-projection of all heads and writes two bf16 terms (16 bits) of each
//     fp32 result, a plane each;
//   * latent_prompt_kernel: CTA = 128 consecutive query tokens of one head.  Scores: (q1 q0)(k1 k0) without the product of the two
//     low terms, over dn, and the rotated part as three query terms against the cached key.  Values: likewise, weights in two terms.
// No operand has fewer bits than in latent space: there the head products round queries and results to one bf16 term (2^-9), here
// both sides keep two (2^-17) and the result is rounded once, to the output's type.
// Mezilix prompt, 4 x 1024 tokens, 16 heads of 128 + 64: head products and attention 86 + 354 + 58 us before, 12 + 33 + 87
// here; 3 prompts of up to 777 tokens 47 + 160 + 30 and 11 + 24 + 54.
//
// Inside the attention kernel (the frame of window_attention_tc.cu): two warps load, two issue the products, four take the softmax
// (thread = query row = TMEM lane).  A head's keys are its own, so every tile of 128 brings nine 16 KB boxes from L2 for 60 products of
// about 60 clocks; a tile takes 2.7 us (tensor pipes active 38 % of the kernel).  The query's two terms stand in TMEM (the A operand of the scores), the three of its rotated part in shared memory; what is
// left of that holds rings of two and three 32 KB units for the terms of keys and values (both chunks of a term together, so that a value
// product has all of its 128 columns), and one box for the rotated key part.  The scores' columns are free as soon as the softmax has its
// row in registers, since the weights have columns of their own: scores of tile j + 1 and values of tile j run side by side.
// Shared memory (226 KB) and TMEM (512 columns) allow one CTA per SM.  Launched plainly, never triggers (ptx.cuh).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "asd_internal.h"
#include "blocks.h"
#include "gemm.h"
#include "ptx.cuh"
#include "softmax_tile.cuh"

namespace asd {

namespace {

constexpr int kLpThreads = 256;            // warps 0-3 softmax (thread = query row), 4 and 7 loads, 5 and 6 products
constexpr int kLpKeys = 128;               // keys per tile
constexpr int kLpDn = 128, kLpDr = 64, kLpDv = 128;
constexpr int kLpKUnits = 2, kLpVUnits = 3;     // rings of keys and values: units of two boxes
constexpr int kLpMinTokens = 9;            // of a sequence, below which neither form was compared
constexpr float kLpSlack = 8.0f;           // log2 growth of a row maximum that the weights tolerate before a rescale

// first position a sequence's rows start at, and how many positions of it this call sees
struct LpSpan {
    int base, n;
};
__device__ __forceinline__ LpSpan lp_span(const int* positions, int t0, int t_end, int window) {
    const int p0 = positions[t0], base = max(p0 - window + 1, 0) & ~(kLpKeys - 1);
    return {base, p0 + (t_end - t0) - base};
}

// rows [seq * cap + i] = cache row of position base + i; zeros up to the end of the last tile
__global__ void __launch_bounds__(256) latent_rows_kernel(const int* positions, const int* cu_q, const int* seq_slot, PagedRows cache,
                                                          int rw, int window, int cap, uint4* rows) {
    pdl_enter();
    const int seq = blockIdx.y, t0 = cu_q[seq], t_end = cu_q[seq + 1];
    if (t0 >= t_end) return;
    const LpSpan sp = lp_span(positions, t0, t_end, window);
    const int i0 = blockIdx.x * 32, end = min((sp.n + kLpKeys - 1) & ~(kLpKeys - 1), cap), per = rw >> 3;
    const int* pt = cache.page_table + (long long)seq_slot[seq] * cache.max_pages;
    const uint4* pool = static_cast<const uint4*>(cache.pool);
    for (int t = threadIdx.x; t < 32 * per; t += 256) {
        const int r = t / per, c = t - r * per, i = i0 + r;
        if (i >= end) break;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (i < sp.n) {
            const int p = sp.base + i;
            v = pool[((long long)pt[p / cache.page_size] * cache.page_size + p % cache.page_size) * per + c];
        }
        rows[((long long)seq * cap + i) * per + c] = v;
    }
}

struct LpArgs {
    const int* positions;
    const int* cu_q;
    const float* q;                        // [M][ldq], head h at h * (dn + dr): dn unrotated, dr rotated
    long long ldq;
    int heads, window, cap, plane_rows, R;
    float scale2;                          // score scale x log2(e)
    __nv_bfloat16* out;                    // [M][heads * dv]
    int* err;
};

struct LpBars {
    uint64_t q_full, r_full, r_empty, k_full[kLpKUnits], k_empty[kLpKUnits], v_full[kLpVUnits], v_empty[kLpVUnits], s_full, s_read, p_full, pv_done, cut_full[2];
    uint32_t tmem;
    int failed;
};

__global__ void __launch_bounds__(kLpThreads, 1)
    latent_prompt_kernel(const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_rot, const LpArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sT = smem;                                        // [3 terms] of the query's rotated part
    uint8_t* sK = sT + 3 * kStSlot;                            // [kLpKUnits][2 chunks]
    uint8_t* sV = sK + 2 * kLpKUnits * kStSlot;                // [kLpVUnits][2 chunks]
    uint8_t* sR = sV + 2 * kLpVUnits * kStSlot;                // rotated key part
    LpBars* B = reinterpret_cast<LpBars*>(sR + kStSlot);
    const WaitGuard guard{reinterpret_cast<volatile int*>(&B->failed), a.err, WAIT_LATENT_PROMPT << 8};

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // neighbours are the heads of a sequence's same tile (they read the same rotated keys); the last tiles see the most keys and start first
    const int seq = blockIdx.x / a.heads, h = blockIdx.x - seq * a.heads, tile_x = (int)gridDim.y - 1 - (int)blockIdx.y;
    const int first = a.cu_q[seq], t_end = a.cu_q[seq + 1], t0 = first + tile_x * 128;
    if (t0 >= t_end) return;
    const LpSpan sp = lp_span(a.positions, first, t_end, a.window);
    const int n_tok = min(128, t_end - t0);
    // positions and keys from here on count from the sequence's first row
    const int p_first = a.positions[first] + (t0 - first) - sp.base, p_last = p_first + n_tok - 1;
    const int j_lo = max(p_first - a.window + 1, 0), key_base = j_lo & ~(kLpKeys - 1);
    const int nt = (p_last - key_base) / kLpKeys + 1;
    const int row0 = seq * a.cap + key_base;                   // of the first tile
    auto cut = [&](int j) { const int key0 = key_base + j * kLpKeys; return key0 + kLpKeys > p_last + 1 || key0 < j_lo; };

    if (tid == 0) {
        tma_prefetch_desc(&map_kv);
        tma_prefetch_desc(&map_rot);
        mbar_init(&B->q_full, 4);
        mbar_init(&B->r_full, 1);
        mbar_init(&B->r_empty, 1);
        for (int i = 0; i < kLpKUnits; ++i) {
            mbar_init(&B->k_full[i], 1);
            mbar_init(&B->k_empty[i], 1);
        }
        for (int i = 0; i < kLpVUnits; ++i) {
            mbar_init(&B->v_full[i], 1);
            mbar_init(&B->v_empty[i], 1);
        }
        mbar_init(&B->s_full, 1);
        mbar_init(&B->s_read, 4);
        mbar_init(&B->p_full, 4);
        mbar_init(&B->pv_done, 1);
        mbar_init(&B->cut_full[0], 1);
        mbar_init(&B->cut_full[1], 1);
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
    const uint32_t tmem = B->tmem;                             // columns 0-127: scores, 128-: weights, 256-: result, 384-: the query's two terms

    // the query's terms, a row a thread (rows that are not there: zeros).  A warp reads 32 floats of four rows an instruction and turns
    // them in its own rows of sT; the next ones' loads are on their way
    if (warp < 4) {
        auto terms = [&](float u, float v, uint32_t (&t)[3]) {
            const __nv_bfloat162 t0 = __floats2bfloat162_rn(u, v);
            const float2 f0 = __bfloat1622float2(t0);
            const __nv_bfloat162 t1 = __floats2bfloat162_rn(u - f0.x, v - f0.y);
            const float2 f1 = __bfloat1622float2(t1);
            const __nv_bfloat162 t2 = __floats2bfloat162_rn(u - f0.x - f1.x, v - f0.y - f1.y);
            t[0] = *reinterpret_cast<const uint32_t*>(&t0);
            t[1] = *reinterpret_cast<const uint32_t*>(&t1);
            t[2] = *reinterpret_cast<const uint32_t*>(&t2);
        };
        const int piece = lane & 7, first_row = lane >> 3;
        const float* src = a.q + (long long)(t0 + warp * 32) * a.ldq + h * (kLpDn + kLpDr) + piece * 4;
        float4 x[8];
        auto fetch = [&](int c) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = first_row + 4 * i;
                x[i] = warp * 32 + r < n_tok ? *reinterpret_cast<const float4*>(src + (long long)r * a.ldq + c * 32) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        };
        uint8_t* turned = sT + warp * 32 * 128;
        auto put = [&](int slot) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = first_row + 4 * i;
                *reinterpret_cast<float4*>(turned + slot * kStSlot + r * 128 + ((piece ^ (r & 7)) << 4)) = x[i];
            }
        };
        auto own = [&](int slot, int i) {
            return *reinterpret_cast<const float4*>(turned + slot * kStSlot + lane * 128 + ((i ^ (lane & 7)) << 4));
        };
        const uint32_t to = tmem + ((uint32_t)(warp * 32) << 16) + 384u;
        fetch(0);
#pragma unroll 1
        for (int c = 0; c < kLpDn / 32; ++c) {
            put(c & 1);                                        // (read by the other lanes two rounds ago)
            fetch(c + 1);
            __syncwarp();
            uint32_t hi[16], lo[16], t[3];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 v = own(c & 1, i);
                terms(v.x, v.y, t);
                hi[2 * i] = t[0], lo[2 * i] = t[1];
                terms(v.z, v.w, t);
                hi[2 * i + 1] = t[0], lo[2 * i + 1] = t[1];
            }
            tmem_st_32x16(to + (uint32_t)(c * 16), hi);
            tmem_st_32x16(to + 64u + (uint32_t)(c * 16), lo);
        }
        put(0);
        fetch(kLpDn / 32 + 1);
        __syncwarp();                                          // (slot 1: read a round ago)
        put(1);
        __syncwarp();
        float4 v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = own(i >> 3, i & 7);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint32_t t[4][3];
            terms(v[2 * i].x, v[2 * i].y, t[0]);
            terms(v[2 * i].z, v[2 * i].w, t[1]);
            terms(v[2 * i + 1].x, v[2 * i + 1].y, t[2]);
            terms(v[2 * i + 1].z, v[2 * i + 1].w, t[3]);
            uint8_t* dst = turned + lane * 128 + ((i ^ (lane & 7)) << 4);
#pragma unroll
            for (int u = 0; u < 3; ++u) *reinterpret_cast<uint4*>(dst + u * kStSlot) = make_uint4(t[0][u], t[1][u], t[2][u], t[3][u]);
        }
        tmem_st_wait();
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&B->q_full);
    }

    if (warp == 4 || warp == 7) {
        // ------------------------------------------------------------------ loads of keys and of values: the low term of each first
        const bool vals = warp == 7;
        auto load = [&]() {
            const int col = vals ? a.heads * kLpDn + h * kLpDv : h * kLpDn, units = vals ? kLpVUnits : kLpKUnits;
            uint64_t *full = vals ? B->v_full : B->k_full, *empty = vals ? B->v_empty : B->k_empty;
            uint8_t* ring = vals ? sV : sK;
            int slot = 0, round = 0;
            auto unit = [&](int row) {
                if (round > 0 && !mbar_wait(&empty[slot], (round - 1) & 1, guard)) return false;
                mbar_expect_tx(&full[slot], 2 * kStSlot);
                tma_load_2d(ring + 2 * slot * kStSlot, &map_kv, col, row, &full[slot]);
                tma_load_2d(ring + (2 * slot + 1) * kStSlot, &map_kv, col + 64, row, &full[slot]);
                if (++slot == units) slot = 0, ++round;
                return true;
            };
            for (int j = 0; j < nt; ++j) {
                const int row = row0 + j * kLpKeys;
                if (!vals) {
                    if (j > 0 && !mbar_wait(&B->r_empty, (j - 1) & 1, guard)) return;
                    mbar_expect_tx(&B->r_full, kStSlot);
                    tma_load_2d(sR, &map_rot, a.R, row, &B->r_full);
                }
                if (!unit(row + a.plane_rows) || !unit(row)) return;
            }
        };
        if (lane == 0) load();
        __syncwarp();
    } else if (warp == 5 || warp == 6) {
        // ------------------------------------------------------------------ products: scores and values by a warp each
        // A product of either leaves every 60 clocks and few wait behind it, while a look at a barrier takes 130: one warp for both
        // left the tensor cores idle for a third of a tile.
        // The whole warp walks the loop, so that addresses and descriptors stay in uniform registers, and one lane issues.
        const bool lead = elect_one();
        auto ready = [&](uint64_t* bar, int phase) { return __all_sync(0xffffffffu, mbar_wait(bar, phase & 1, guard)) != 0; };
        bool ok = true;
        if (warp == 5) {
            const uint32_t id_s = umma_idesc_bf16(128, kLpKeys), uT = smem_u32(sT), uK = smem_u32(sK), uR = smem_u32(sR);
            // scores += term `u` of the queries times the unit's keys
            auto keys = [&](int slot, int u) {
                if (lead) {
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const uint64_t kd = umma_desc_sw128(uK + (uint32_t)((2 * slot + c) * kStSlot));
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16_ts(tmem, tmem + 384u + (uint32_t)(u * 64 + c * 32 + k * 8), kd + 2 * k, id_s, 1);
                    }
                }
                __syncwarp();
            };
            int slot = 0, round = 0;
            auto freed = [&]() {
                if (lead) umma_commit(&B->k_empty[slot]);
                __syncwarp();
                if (++slot == kLpKUnits) slot = 0, ++round;
            };
            ok = ready(&B->q_full, 0);
            for (int j = 0; j < nt && ok; ++j) {
                ok = ready(&B->r_full, j);
                if (j > 0) ok = ok && ready(&B->s_read, j - 1);        // the softmax's warps hold the tile before
                if (!ok) break;
                tc_fence_after();
                if (lead) {
                    const uint64_t kd = umma_desc_sw128(uR);
#pragma unroll
                    for (int u = 2; u >= 0; --u)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16(tmem, umma_desc_sw128(uT + (uint32_t)(u * kStSlot)) + 2 * k, kd + 2 * k, id_s, u != 2 || k != 0);
                    umma_commit(&B->r_empty);
                }
                __syncwarp();
                if (!(ok = ready(&B->k_full[slot], round))) break;
                tc_fence_after();
                keys(slot, 0);                                 // low keys
                freed();
                if (!(ok = ready(&B->k_full[slot], round))) break;
                tc_fence_after();
                keys(slot, 1);
                keys(slot, 0);
                freed();
                if (lead) umma_commit(&B->s_full);
                __syncwarp();
            }
        } else {
            const uint32_t id_v = umma_idesc_bf16(128, kLpDv) | (1u << 16), uV = smem_u32(sV);      // values are MN-major
            // result += term `u` of the weights (high 0, low 1: 32 columns apart) times the unit's values
            auto weigh = [&](int unit, int u, bool fresh) {
                const uint32_t p = tmem + 128u + (uint32_t)(u * 32);
                const uint64_t vd = st_desc_mn(uV + (uint32_t)(2 * unit * kStSlot));
                if (lead) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        umma_f16_ts(tmem + 256u, p + (uint32_t)((k >> 2) * 64 + (k & 3) * 8), vd + k * (2048 >> 4), id_v, !fresh || k != 0);
                }
                __syncwarp();
            };
            for (int j = 0; j < nt && ok; ++j) {
                const int u0 = 2 * j % kLpVUnits, u1 = (2 * j + 1) % kLpVUnits;
                ok = ready(&B->v_full[u0], 2 * j / kLpVUnits) && ready(&B->v_full[u1], (2 * j + 1) / kLpVUnits);
                if (ok && cut(j)) {                            // the softmax's warps zero some of its values (first or last tile)
                    if (lead) mbar_arrive(&B->cut_full[j == nt - 1]);
                    __syncwarp();
                }
                ok = ok && ready(&B->p_full, j);
                if (!ok) break;
                tc_fence_after();
                weigh(u0, 0, j == 0);                          // high weights, low values
                if (lead) umma_commit(&B->v_empty[u0]);
                __syncwarp();
                weigh(u1, 1, false);
                weigh(u1, 0, false);
                if (lead) {
                    umma_commit(&B->v_empty[u1]);
                    umma_commit(&B->pv_done);
                }
                __syncwarp();
            }
        }
    } else if (warp < 4) {
        // ------------------------------------------------------------------ softmax (thread = query row)
        const bool real = tid < n_tok;
        const int pos = real ? p_first + tid : -1;
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
        float ref = -INFINITY, l = 0.0f;                       // the maximum the weights refer to (log2), and their sum
        // a wait that gave up is reported; the walk goes on to the end, so that every barrier of these warps is met
        // A row's 128 scores are read once and stay in registers; cut tiles turn what a row may not see into -inf, by bits.
        auto tile = [&](int j, bool whole) {
            const int key0 = key_base + j * kLpKeys;
            uint32_t x[4][32];
#pragma unroll
            for (int q = 0; q < 4; ++q) tmem_ld_32x32(lanes + (uint32_t)(q * 32), x[q]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->s_read);            // the next tile's scores may come
            if (!whole) {
                const StSeen seen{pos - a.window + 1 - key0, pos - key0, 0};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t bits = seen.bits(q * 32);
#pragma unroll
                    for (int i = 0; i < 32; ++i) x[q][i] = bits & (1u << i) ? x[q][i] : 0xff800000u;
                }
            }
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(x[q][i]));
            // rn products with a positive scale keep the order; a negative or zero one is not taken
            const float top = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale2;
            const bool grow = real && (top > ref + kLpSlack || (ref == -INFINITY && top > -INFINITY));
            if (__any_sync(0xffffffffu, grow)) {
                const float corr = grow ? st_ex2(ref - top) : 1.0f;        // ref = -inf: 0, of a row that is 0 so far
                if (j > 0) {
                    mbar_wait_timed(&B->pv_done, (j - 1) & 1, guard, 2);
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < kLpDv; c += 16) {
                        uint32_t v[16];
                        tmem_ld_32x16(lanes + 256u + (uint32_t)c, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * corr);
                        tmem_st_32x16(lanes + 256u + (uint32_t)c, v);
                    }
                }
                l *= corr;
                if (grow) ref = top;
            }
            const float nref = ref == -INFINITY ? 0.0f : -ref;
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            uint32_t ph[4][16], pl[4][16];
#pragma unroll
            for (int q = 0; q < 4; ++q) st_weights<false>(x[q], 0u, a.scale2, nref, ph[q], pl[q], sum);
            if (j > 0) {                                       // the last tile's are multiplied
                mbar_wait_timed(&B->pv_done, (j - 1) & 1, guard, 5);
                tc_fence_after();
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {      // a half's terms: 32 columns of high ones, 32 of low ones
                tmem_st_32x16(lanes + 128u + (uint32_t)((q >> 1) * 64 + (q & 1) * 16), ph[q]);
                tmem_st_32x16(lanes + 128u + (uint32_t)((q >> 1) * 64 + (q & 1) * 16 + 32), pl[q]);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        };
        for (int j = 0; j < nt; ++j) {
            const int key0 = key_base + j * kLpKeys;
            mbar_wait_timed(&B->s_full, j & 1, guard, 1);
            tc_fence_after();
            tile(j, key0 + kLpKeys <= p_first + 1 && key0 >= p_last - a.window + 1);
            if (cut(j)) {
                // keys that no row of the tile may see: whatever was computed for them must not meet the zero weights
                const int kp = key0 + tid;
                mbar_wait_timed(&B->cut_full[j == nt - 1], 0, guard, 3);
                if (kp > p_last || kp < j_lo)
                    for (int c = 0; c < 4; ++c) {
                        uint4* dst = reinterpret_cast<uint4*>(sV + (2 * ((2 * j + (c >> 1)) % kLpVUnits) + (c & 1)) * kStSlot + tid * 128);
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
        mbar_wait_timed(&B->pv_done, (nt - 1) & 1, guard, 4);
        tc_fence_after();
        // every load and product has ended: shared memory is free.  Rows through it, so that a warp writes whole rows
        const float inv = 1.0f / l;
        constexpr int kLd = kLpDv * 2 + 16;                    // bytes; 16 of padding spread the lanes' rows over the banks
        uint8_t* own = sK + (size_t)warp * 32 * kLd;
#pragma unroll 1
        for (int c = 0; c < kLpDv; c += 16) {
            uint32_t v[16], b[8];
            tmem_ld_32x16(lanes + 256u + (uint32_t)c, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const __nv_bfloat162 y = __floats2bfloat162_rn(__uint_as_float(v[2 * i]) * inv, __uint_as_float(v[2 * i + 1]) * inv);
                b[i] = *reinterpret_cast<const uint32_t*>(&y);
            }
            *reinterpret_cast<uint4*>(own + lane * kLd + c * 2) = make_uint4(b[0], b[1], b[2], b[3]);
            *reinterpret_cast<uint4*>(own + lane * kLd + c * 2 + 16) = make_uint4(b[4], b[5], b[6], b[7]);
        }
        __syncwarp();
        const int c = lane & 15;                               // 16 lanes write a row's 16-byte pieces
        __nv_bfloat16* out0 = a.out + ((long long)t0 * a.heads + h) * kLpDv + c * 8;
#pragma unroll 4
        for (int r = lane >> 4; r < 32; r += 2) {
            const uint4 x = *reinterpret_cast<const uint4*>(own + r * kLd + c * 16);
            if (warp * 32 + r < n_tok) *reinterpret_cast<uint4*>(out0 + (long long)(warp * 32 + r) * a.heads * kLpDv) = x;
        }
    }
    wait_settle(guard);
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace

// rows that a call's positions take, a sequence's apart
static long long lp_cap(int max_kv_len) { return ((long long)max_kv_len + kLpKeys - 1) & ~(long long)(kLpKeys - 1); }

bool latent_prompt_takes(const LatentDims& d, const PagedRows& cache, int M, int nseq, int max_qlen, int max_kv_len, const float* q,
                         long long ldq, const LatentPromptWs& ws, int tiled) {
    if (tiled < 2 || ws.mode <= 0 || cache.f32 || !ws.w || !ws.rows || !ws.planes || max_qlen <= 0 || max_kv_len <= 0 || nseq <= 0 || !(d.scale > 0.f))
        return false;
    if (d.dn != kLpDn || d.dr != kLpDr || d.dv != kLpDv || d.R <= 0 || d.R % 8 || d.window <= 0) return false;
    const uintptr_t at = reinterpret_cast<uintptr_t>(cache.pool) | reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(ws.w) |
                         reinterpret_cast<uintptr_t>(ws.rows) | reinterpret_cast<uintptr_t>(ws.planes);
    if ((at & 15) || ldq % 4 || cache.page_size <= 0) return false;
    const long long rows = lp_cap(max_kv_len) * nseq, cols = (long long)d.heads * (kLpDn + kLpDv);
    if (2 * rows >= (1ll << 31) || cols >= (1ll << 31) || nseq > 65535 || (long long)nseq * d.heads >= (1ll << 31)) return false;
    if (rows * (d.R + kLpDr) > ws.row_elems || 2 * rows * cols > ws.plane_elems) return false;
    if (ws.mode > 1) return true;
    if (max_qlen < kLpMinTokens) return false;
    return latent_prompt_gain(d.heads, d.R, sm_count(), M, nseq, max_qlen, max_kv_len) > 0.0;
}

int launch_latent_prompt(const SeqIndex& ix, const int* cu_q, const int* seq_slot, int nseq, int max_qlen, int max_kv_len,
                         const float* q, long long ldq, const LatentDims& d, const PagedRows& cache, const LatentPromptWs& ws,
                         void* out, int* err, cudaStream_t stream) {
    if (ix.M <= 0 || nseq <= 0) return 0;
    const int cap = (int)lp_cap(max_kv_len), rows = cap * nseq, cols = d.heads * (kLpDn + kLpDv), rw = d.R + kLpDr;
    ASD_CUDA(launch_pdl(latent_rows_kernel, dim3(cap / 32, nseq), 256, 0, stream, ix.positions, cu_q, seq_slot, cache, rw, d.window, cap,
                        static_cast<uint4*>(ws.rows)));
    count_launch(1);
    if (launch_gemm_tc_terms(ws.rows, rw, ws.w, rows, cols, d.R, ws.planes, stream)) return -1;
    LpArgs a;
    a.positions = ix.positions, a.cu_q = cu_q, a.q = q, a.ldq = ldq;
    a.heads = d.heads, a.window = std::min(d.window, 1 << 30), a.cap = cap, a.plane_rows = rows, a.R = d.R;
    a.scale2 = d.scale * 1.4426950408889634f;
    a.out = static_cast<__nv_bfloat16*>(out), a.err = err;
    CUtensorMap mk, mr;
    if (make_tmap_bf16(&mk, ws.planes, 2ull * rows, cols, cols, kLpKeys)) return -1;
    if (make_tmap_bf16(&mr, ws.rows, rows, rw, rw, kLpKeys)) return -1;
    const int smem = 1024 + (4 + 2 * (kLpKUnits + kLpVUnits)) * kStSlot + (int)sizeof(LpBars);
    static PerDeviceOnce once;
    ASD_ONCE(once, ASD_CUDA(cudaFuncSetAttribute(latent_prompt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)));
    const dim3 grid(nseq * d.heads, (max_qlen + 127) / 128);
    if (grid.y > 65535) return set_error("latent attention: too many tokens");
    latent_prompt_kernel<<<grid, kLpThreads, smem, stream>>>(mk, mr, a);
    ASD_CUDA(cudaGetLastError());
    count_kernel(KERNEL_LATENT_PROMPT);
    return 0;
}

}  // namespace asd
