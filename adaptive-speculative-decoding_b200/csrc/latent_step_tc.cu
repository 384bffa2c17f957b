// Latent key/value attention of few query rows (single tokens of many heads, small verifications) on tcgen05 / TMEM: the contract of
// latent_attention_tc.cu, whose tile costs what 128 query rows cost and brings the query's three planes from L2 again for every tile
// of keys (590 KB; 64 tokens of 32 heads at 1024 positions 95 us, the cache rows' bytes are worth 12).  Here up to 32 rows (that call 31 us;
// 16 tokens of 16 heads at 1500, 42 on mma.sync, 18):
//   * The three bf16 terms of a row (24 bits of its fp32 query) are stacked along the lanes: lane 32 t + r holds term t of row r, all
//     of R + dr, 288 columns of TMEM that stay for the CTA's life as the A operand of the scores.  One product of 16 elements then
//     serves all terms, shared memory is left to the keys alone, and a key is read once.
//   * Keys come by TMA from the paged pool in tiles of 64 positions, pairs of 64-column chunks in a ring of ten 16 KB units (two and a
//     half tiles on their way) and the rotated part in a ring of its own.
//   * The terms' scores meet in shared memory, where four threads a row take the softmax of a tile and write its weights as two bf16
//     terms: the B operand of the value product, which is transposed - 128 latent columns on the lanes, the rows as columns - so that
//     512 latent columns of 32 rows take 128 columns of TMEM and nothing is scored twice.
//   * The sums are rescaled only when a row's maximum has grown by 2^8.
// What bounds it: a tile is 36 + 32 products of 50 clocks, 1.6 us of the 2 a tile takes; the queries' way into TMEM is 4 us a CTA.
// Launched plainly, never triggers (ptx.cuh); one CTA per SM.
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
#include "softmax_tile.cuh"

namespace asd {

namespace {

constexpr int kLsThreads = 224;            // warps 0-3 softmax and results, 4 loads, 5 and 6 products
constexpr int kLsKeys = 64;                // keys per tile
constexpr int kLsRows = 32;                // query rows of a CTA
constexpr int kLsUnit = 2 * kLsKeys * 128; // bytes of two chunks of 64 columns
constexpr int kLsUnits = 10;
constexpr int kLsRots = 3;                 // ring of rotated parts
constexpr int kLsLd = kLsKeys + 4;         // floats of a row of a term's scores in shared memory
// Row tiles of a sequence up to which this form is taken (its keys are read once for each), unless fewer than 32 rows see a single tile of
// keys, which latent_attn_mma does in 2 % less of a step.  One layer of the Mezilix family, us a step with latent_attention_tc.cu or
// latent_attn_mma and here: 64 tokens of 32 heads at 1024 positions 269, 216; 16 tokens of 16 heads at 2500 159, 130; 1 of 32 163, 146;
// 64 x 3 of 8 heads at 256 190, 163; two row tiles: 64 x 2 of 32 heads at 1024 296, 251; 16 tokens of 16 heads at 33 106, 108.
constexpr int kLatentStepTiles = 2;
constexpr float kLsSlack = 8.0f;           // log2 growth of a row maximum that the weights tolerate before a rescale

struct LsArgs {
    const int* positions;
    const int* cu_q;
    const int* seq_slot;
    const int* page_table;
    int max_pages, page_shift;
    const __nv_bfloat16* q;                // [3][M][heads][rw]
    long long plane;
    int heads, HG, TQ, R, rw, hgs, nsplit, window, box_rows, n_cols;
    float scale2;                          // score scale x log2(e)
    float* out_lat;                        // [M][heads][R]
    float *ws_o, *ws_ml;
    int* err;
};

struct LsShared {
    uint64_t q_full, u_full[kLsUnits], u_empty[kLsUnits], r_full[kLsRots], r_empty[kLsRots], s_full, s_read, p_full, pv_done;
    uint32_t tmem;
    int failed;
    float corr[kLsRows], inv[kLsRows];
    __align__(16) float scores[3][kLsRows * kLsLd];
};

__device__ __forceinline__ bool ls_any(bool x) {              // over the four softmax warps; a barrier of theirs
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred.aligned q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)x)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void ls_sync() { asm volatile("barrier.cta.sync.aligned 1, 128;" ::: "memory"); }

// A operand of the value product: MN-major SW128 (keys along rows of 128 B = 64 columns, the next 64 columns half a unit further)
__device__ __forceinline__ uint64_t ls_desc_mn(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)((kLsUnit / 2) >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

__global__ void __launch_bounds__(kLsThreads, 1) latent_step_kernel(const __grid_constant__ CUtensorMap map_kv, const LsArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sU = smem;                                        // [kLsUnits]
    uint8_t* sR = sU + kLsUnits * kLsUnit;                     // [kLsRots]
    uint8_t* sP = sR + kLsRots * (kLsUnit / 2);                // [2 terms][32 rows][64 keys]
    LsShared* B = reinterpret_cast<LsShared*>(sP + 2 * kLsRows * kLsKeys * 2);
    const WaitGuard guard{reinterpret_cast<volatile int*>(&B->failed), a.err, WAIT_LATENT_STEP << 8};

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int seq = blockIdx.y / a.nsplit, split = blockIdx.y - seq * a.nsplit;
    const int h0 = (int)(blockIdx.x % a.hgs) * a.HG, t0 = a.cu_q[seq] + (int)(blockIdx.x / a.hgs) * a.TQ, t_end = a.cu_q[seq + 1];
    if (t0 >= t_end) return;
    const int n_tok = min(a.TQ, t_end - t0), n_head = min(a.HG, a.heads - h0);
    const int p_first = a.positions[t0], p_last = p_first + n_tok - 1;
    const int j_lo = max(p_first - a.window + 1, 0), base = j_lo & ~(kLsKeys - 1);
    const int tiles = (p_last - base) / kLsKeys + 1, per = (tiles + a.nsplit - 1) / a.nsplit;
    const int ts = split * per, nt = min(tiles, ts + per) - ts;
    const int nb = a.R >> 7;                                   // blocks of 128 latent columns: units a tile
    // row r = (token r / HG, head h0 + r % HG): with several head groups there is one token, so that rows are neighbours in either case
    const int n_rows = a.hgs == 1 ? n_tok * a.HG : n_head;
    const long long row0 = (long long)t0 * a.heads + h0;
    if (nt <= 0) {                                             // an empty share of a short sequence
        for (int r = 0; r < n_rows; ++r) {
            const long long at = (row0 + r) * a.nsplit + split;
            for (int c = tid; c < a.R; c += kLsThreads) a.ws_o[at * a.R + c] = 0.0f;
            if (tid == 0) a.ws_ml[at * 2] = -INFINITY, a.ws_ml[at * 2 + 1] = 0.0f;
        }
        return;
    }
    if (tid == 0) {
        tma_prefetch_desc(&map_kv);
        mbar_init(&B->q_full, 3);
        for (int i = 0; i < kLsUnits; ++i) {
            mbar_init(&B->u_full[i], 1);
            mbar_init(&B->u_empty[i], 1);
        }
        for (int i = 0; i < kLsRots; ++i) {
            mbar_init(&B->r_full[i], 1);
            mbar_init(&B->r_empty[i], 1);
        }
        mbar_init(&B->s_full, 1);
        mbar_init(&B->s_read, 4);                              // every warp that waits for s_full: none of them may be lapped
        mbar_init(&B->p_full, 4);
        mbar_init(&B->pv_done, 1);
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
    const uint32_t tmem = B->tmem;                             // columns 0-287: queries, 288-351: scores, 352-: sums of the blocks
    constexpr uint32_t kScores = 288, kSums = 352;

    if (warp == 4) {
        // ------------------------------------------------------------------ loads: a lane per box of positions
        const int boxes = kLsKeys / a.box_rows, box = lane * a.box_rows, last_page = p_last >> a.page_shift;
        const int* pt = a.page_table + (long long)a.seq_slot[seq] * a.max_pages;
        // boxes past the end repeat the sequence's last page: their keys are masked, their values zeroed
        auto row_of = [&](int j) {
            const int kp = base + (ts + j) * kLsKeys + box, page = min(kp >> a.page_shift, last_page);
            return lane < boxes ? (pt[page] << a.page_shift) + (kp & ((1 << a.page_shift) - 1)) : 0;
        };
        int next = row_of(0), us = 0, ur = 0, rs = 0, rr = 0;  // slots and rounds of both rings
        bool ok = true;
        for (int j = 0; j < nt && ok; ++j) {
            const int row = next;
            if (j + 1 < nt) next = row_of(j + 1);
            if (rr > 0) ok = __all_sync(0xffffffffu, mbar_wait(&B->r_empty[rs], (rr - 1) & 1, guard)) != 0;
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(&B->r_full[rs], kLsUnit / 2);
            __syncwarp();
            if (lane < boxes) tma_load_2d(sR + rs * (kLsUnit / 2) + box * 128, &map_kv, a.R, row, &B->r_full[rs]);
            if (++rs == kLsRots) rs = 0, ++rr;
            for (int b = 0; b < nb && ok; ++b) {
                if (ur > 0) ok = __all_sync(0xffffffffu, mbar_wait(&B->u_empty[us], (ur - 1) & 1, guard)) != 0;
                if (!ok) break;
                if (lane == 0) mbar_expect_tx(&B->u_full[us], kLsUnit);
                __syncwarp();
                if (lane < boxes) {
                    uint8_t* dst = sU + us * kLsUnit + box * 128;
                    tma_load_2d(dst, &map_kv, b * 128, row, &B->u_full[us]);
                    tma_load_2d(dst + kLsUnit / 2, &map_kv, b * 128 + 64, row, &B->u_full[us]);
                }
                if (++us == kLsUnits) us = 0, ++ur;
            }
        }
        __syncwarp();
    } else if (warp >= 5) {
        // ------------------------------------------------------------------ products: scores and values by a warp each (a look at a
        // barrier takes as long as two of them, and few wait behind the one that runs)
        const bool lead = elect_one();
        auto ready = [&](uint64_t* bar, int phase) { return __all_sync(0xffffffffu, mbar_wait(bar, phase & 1, guard)) != 0; };
        const uint32_t uU = smem_u32(sU), uR = smem_u32(sR), uP = smem_u32(sP);
        bool ok = true;
        int us = 0;
        if (warp == 5) {
            const uint32_t id_s = umma_idesc_bf16(128, kLsKeys);
            int ur = 0, rs = 0, rr = 0;
            ok = ready(&B->q_full, 0);
            for (int j = 0; j < nt && ok; ++j) {
                ok = ready(&B->r_full[rs], rr);
                if (j > 0) ok = ok && ready(&B->s_read, j - 1);        // the softmax's warps hold the tile before
                if (!ok) break;
                tc_fence_after();
                if (lead) {
                    const uint64_t kd = umma_desc_sw128(uR + (uint32_t)(rs * (kLsUnit / 2)));
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_f16_ts(tmem + kScores, tmem + (uint32_t)(nb * 64 + k * 8), kd + 2 * k, id_s, k != 0);
                    umma_commit(&B->r_empty[rs]);
                }
                __syncwarp();
                if (++rs == kLsRots) rs = 0, ++rr;
                for (int b = 0; b < nb && ok; ++b) {
                    ok = ready(&B->u_full[us], ur);
                    if (!ok) break;
                    tc_fence_after();
                    if (lead) {
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const uint64_t kd = umma_desc_sw128(uU + (uint32_t)(us * kLsUnit + c * (kLsUnit / 2)));
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                umma_f16_ts(tmem + kScores, tmem + (uint32_t)(b * 64 + c * 32 + k * 8), kd + 2 * k, id_s, 1);
                        }
                    }
                    __syncwarp();
                    if (++us == kLsUnits) us = 0, ++ur;
                }
                if (!ok) break;
                if (lead) umma_commit(&B->s_full);
                __syncwarp();
            }
        } else {
            const uint32_t id_v = umma_idesc_bf16(128, (uint32_t)a.n_cols) | (1u << 15);       // A: MN-major
            for (int j = 0; j < nt && ok; ++j) {
                ok = ready(&B->p_full, j);
                if (!ok) break;
                tc_fence_after();
                for (int b = 0; b < nb; ++b) {
                    const uint64_t vd = ls_desc_mn(uU + (uint32_t)(us * kLsUnit)), pd = umma_desc_sw128(uP);
                    const uint32_t d = tmem + kSums + (uint32_t)(b * kLsRows);
                    if (lead) {
#pragma unroll
                        for (int k = 0; k < kLsKeys / 16; ++k)
#pragma unroll
                            for (int u = 1; u >= 0; --u)       // the low term first
                                umma_f16(d, vd + k * (2048 >> 4), pd + u * ((kLsRows * kLsKeys * 2) >> 4) + 2 * k, id_v, (j | k) != 0 || u == 0);
                        umma_commit(&B->u_empty[us]);
                    }
                    __syncwarp();
                    if (++us == kLsUnits) us = 0;
                }
                if (lead) umma_commit(&B->pv_done);
                __syncwarp();
            }
        }
    } else {
        // ------------------------------------------------------------------ queries, softmax, results
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
        if (warp < 3) {                                        // term `warp` of row `lane`
            // 64 elements of four rows an instruction, three such chunks on their way, turned in shared memory
            constexpr int kLd = 144;                           // bytes of a row there
            uint8_t* own = reinterpret_cast<uint8_t*>(B->scores[warp]);
            const int piece = lane & 7, first = lane >> 3, chunks = a.rw >> 6;
            const uint4* src = reinterpret_cast<const uint4*>(a.q + warp * a.plane + (row0 + first) * a.rw) + piece;
#pragma unroll 1
            for (int c0 = 0; c0 < chunks; c0 += 3) {
                uint4 x[3][8];
#pragma unroll
                for (int u = 0; u < 3; ++u)
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        x[u][i] = first + 4 * i < n_rows && c0 + u < chunks ? src[(i * a.rw >> 1) + (c0 + u) * 8] : make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    if (c0 + u >= chunks) break;
#pragma unroll
                    for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(own + (first + 4 * i) * kLd + piece * 16) = x[u][i];
                    __syncwarp();
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        uint32_t w[16];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint4 v = *reinterpret_cast<const uint4*>(own + lane * kLd + g * 64 + i * 16);
                            w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
                        }
                        tmem_st_32x16(lanes + (uint32_t)((c0 + u) * 32 + g * 16), w);
                    }
                    __syncwarp();
                }
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->q_full);
        }
        // four threads a row, thread c of them keys 16 i + 4 c .. + 3
        const int r = tid >> 2, c4 = (tid & 3) * 4;
        const bool real = r < n_rows;
        const int pos = real ? p_first + r / a.HG : -1;
        float ref = -INFINITY, l = 0.0f;                       // the maximum the weights refer to (log2), and this thread's part of their sum
        // a wait that gave up is reported; the walk goes on to the end, so that every barrier of these warps is met
        for (int j = 0; j < nt; ++j) {
            const int key0 = base + (ts + j) * kLsKeys;
            mbar_wait_timed(&B->s_full, j & 1, guard, 1);
            tc_fence_after();
            if (warp < 3) {
                uint32_t x[2][32];
                tmem_ld_32x32(lanes + kScores, x[0]);
                tmem_ld_32x32(lanes + kScores + 32u, x[1]);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&B->s_read);        // the next tile's scores may come
                float4* dst = reinterpret_cast<float4*>(B->scores[warp] + lane * kLsLd);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const uint32_t* v = &x[i >> 3][(i & 7) * 4];
                    dst[i] = make_float4(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), __uint_as_float(v[3]));
                }
            } else {                                           // has no scores to read; every lane has seen that they are there
                __syncwarp();
                if (lane == 0) mbar_arrive(&B->s_read);
            }
            if (key0 + kLsKeys > p_last + 1 || key0 < j_lo) {
                // keys that no row may see: whatever the pool holds there must not meet the zero weights (the scores have read them)
                const int kp = key0 + (tid & 63);
                if (kp > p_last || kp < j_lo)
                    for (int b = tid >> 6; b < 2 * nb; b += 2) {
                        const int u = (j * nb + (b >> 1)) % kLsUnits;
                        uint4* dst = reinterpret_cast<uint4*>(sU + u * kLsUnit + (b & 1) * (kLsUnit / 2) + (tid & 63) * 128);
#pragma unroll
                        for (int i = 0; i < 8; ++i) dst[i] = make_uint4(0, 0, 0, 0);
                    }
            }
            __syncwarp();
            ls_sync();
            float s[16];
            const int hi = pos - key0, lo = pos - a.window + 1 - key0;     // key i is visible iff lo <= i <= hi
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int at = r * kLsLd + i * 16 + c4;
                const float4 s0 = *reinterpret_cast<const float4*>(B->scores[0] + at), s1 = *reinterpret_cast<const float4*>(B->scores[1] + at),
                             s2 = *reinterpret_cast<const float4*>(B->scores[2] + at);
                s[4 * i] = s0.x + (s1.x + s2.x), s[4 * i + 1] = s0.y + (s1.y + s2.y);
                s[4 * i + 2] = s0.z + (s1.z + s2.z), s[4 * i + 3] = s0.w + (s1.w + s2.w);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int k = i * 16 + c4 + e;
                    if (k > hi || k < lo) s[4 * i + e] = -INFINITY;
                }
            }
            float m = -INFINITY;
#pragma unroll
            for (int i = 0; i < 16; ++i) m = fmaxf(m, s[i]);
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            // rn products with a positive scale keep the order; a negative or zero one is not taken
            const float top = m * a.scale2;
            const bool grow = real && (top > ref + kLsSlack || (ref == -INFINITY && top > -INFINITY));
            const float corr = grow ? st_ex2(ref - top) : 1.0f;            // ref = -inf: 0, of a row that is 0 so far
            if (c4 == 0) B->corr[r] = corr;
            l *= corr;
            if (grow) ref = top;
            const bool any = ls_any(grow);
            const float nref = ref == -INFINITY ? 0.0f : -ref;
            uint32_t ph[8], pl[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float p0 = st_ex2(fmaf(s[2 * i], a.scale2, nref)), p1 = st_ex2(fmaf(s[2 * i + 1], a.scale2, nref));
                l += p0 + p1;
                const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
                const float2 f = __bfloat1622float2(h);
                const __nv_bfloat162 d = __floats2bfloat162_rn(p0 - f.x, p1 - f.y);
                ph[i] = *reinterpret_cast<const uint32_t*>(&h);
                pl[i] = *reinterpret_cast<const uint32_t*>(&d);
            }
            if (j > 0) {                                       // the last tile's weights are multiplied
                mbar_wait_timed(&B->pv_done, (j - 1) & 1, guard, 2);
                tc_fence_after();
                if (any)
                    for (int b = 0; b < nb; ++b) {
                        uint32_t v[32], w[16];
                        tmem_ld_32x32(lanes + kSums + (uint32_t)(b * kLsRows), v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * B->corr[i]);
#pragma unroll
                        for (int i = 0; i < 16; ++i) w[i] = v[i];
                        tmem_st_32x16(lanes + kSums + (uint32_t)(b * kLsRows), w);
#pragma unroll
                        for (int i = 0; i < 16; ++i) w[i] = v[16 + i];
                        tmem_st_32x16(lanes + kSums + (uint32_t)(b * kLsRows + 16), w);
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint8_t* dst = sP + r * 128 + (((2 * i + (c4 >> 3)) ^ (r & 7)) << 4) + (c4 & 4) * 2;
                *reinterpret_cast<uint2*>(dst) = make_uint2(ph[2 * i], ph[2 * i + 1]);
                *reinterpret_cast<uint2*>(dst + kLsRows * kLsKeys * 2) = make_uint2(pl[2 * i], pl[2 * i + 1]);
            }
            fence_proxy_async_smem();
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->p_full);
        }
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        const bool direct = a.nsplit == 1;
        if (c4 == 0) {
            B->inv[r] = direct ? 1.0f / l : 1.0f;
            if (real && !direct) {
                const long long at = (row0 + r) * a.nsplit + split;
                a.ws_ml[at * 2] = ref * 0.69314718055994531f;  // natural units, as the merge expects
                a.ws_ml[at * 2 + 1] = l;
            }
        }
        mbar_wait_timed(&B->pv_done, (nt - 1) & 1, guard, 3);
        tc_fence_after();
        ls_sync();
        float* const to = direct ? a.out_lat + row0 * a.R + tid : a.ws_o + (row0 * a.nsplit + split) * a.R + tid;
        const int step = a.nsplit * a.R;
        for (int b = 0; b < nb; ++b) {                         // thread = latent column
            uint32_t v[32];
            tmem_ld_32x32(lanes + kSums + (uint32_t)(b * kLsRows), v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (i < n_rows) to[i * step + b * 128] = __uint_as_float(v[i]) * B->inv[i];
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

// rows per CTA
struct LsPlan {
    int HG, TQ, hgs, q_tiles;
};
LsPlan ls_plan(const LatentDims& d, int max_qlen) {
    LsPlan p;
    p.HG = std::min(d.heads, kLsRows);
    p.TQ = std::min(kLsRows / p.HG, max_qlen);
    p.hgs = (d.heads + p.HG - 1) / p.HG;
    p.q_tiles = (max_qlen + p.TQ - 1) / p.TQ;
    return p;
}

}  // namespace

bool latent_step_takes(const LatentDims& d, const PagedRows& cache, int max_qlen, int max_kv_len, int tiled) {
    if (tiled < 2 || cache.f32 || cache.rows <= 0 || cache.rows >= (1ll << 31) || max_qlen <= 0 || !(d.scale > 0.f)) return false;
    if (d.R <= 0 || d.R > 512 || d.R % 128 || d.dr != 64 || d.window <= 0) return false;
    if (cache.page_size < 8 || (cache.page_size & (cache.page_size - 1))) return false;
    if (reinterpret_cast<uintptr_t>(cache.pool) & 15) return false;
    const LsPlan p = ls_plan(d, max_qlen);
    if (p.HG * p.TQ < 32 && std::min(max_kv_len, d.window) <= kLsKeys) return false;
    return (long long)p.q_tiles * p.hgs <= kLatentStepTiles;
}

int launch_latent_step(const SeqIndex& ix, const int* cu_q, const int* seq_slot, int nseq, int max_qlen, int max_kv_len,
                       const __nv_bfloat16* q_terms, const LatentDims& d, const PagedRows& cache, float* out_lat, const AttnSplit& ws,
                       int* err, cudaStream_t stream) {
    if (ix.M <= 0 || nseq <= 0) return 0;
    const LsPlan p = ls_plan(d, max_qlen);
    const long long rows = (long long)ix.M * d.heads;
    LsArgs a;
    a.positions = ix.positions, a.cu_q = cu_q, a.seq_slot = seq_slot;
    a.page_table = cache.page_table, a.max_pages = cache.max_pages;
    a.page_shift = 0;
    while ((1 << a.page_shift) < cache.page_size) ++a.page_shift;
    a.q = q_terms, a.rw = d.R + d.dr, a.plane = rows * a.rw;
    a.heads = d.heads, a.HG = p.HG, a.TQ = p.TQ, a.R = d.R, a.hgs = p.hgs, a.window = std::min(d.window, 1 << 30);
    a.box_rows = std::min(cache.page_size, kLsKeys);
    a.n_cols = p.HG * p.TQ <= 16 ? 16 : 32;
    a.scale2 = d.scale * 1.4426950408889634f;
    a.out_lat = out_lat, a.ws_o = ws.o, a.ws_ml = ws.ml, a.err = err;
    // few sequences: the keys are cut into shares until every SM has a CTA, of at least two tiles each
    a.nsplit = 1;
    const long long ctas = (long long)p.q_tiles * p.hgs * nseq;
    const int sms = sm_count();
    if (ws.o && ws.ml && ctas < sms) {
        const long long keys = std::min<long long>(d.window, max_kv_len) + p.TQ + kLsKeys;
        long long n = std::min<long long>(sms / ctas, keys / (2 * kLsKeys));
        n = std::min(n, std::min(ws.rows / rows, ws.o_elems / (rows * d.R)));
        a.nsplit = (int)std::max<long long>(1, std::min<long long>(n, 64));
    }
    if ((long long)nseq * a.nsplit > 65535) return set_error("latent attention: too many sequences");
    CUtensorMap mk;
    if (make_tmap_bf16(&mk, cache.pool, cache.rows, a.rw, a.rw, a.box_rows)) return -1;
    const int smem = 1024 + kLsUnits * kLsUnit + kLsRots * (kLsUnit / 2) + 2 * kLsRows * kLsKeys * 2 + (int)sizeof(LsShared);
    static PerDeviceOnce once;
    ASD_ONCE(once, ASD_CUDA(cudaFuncSetAttribute(latent_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)));
    latent_step_kernel<<<dim3(p.q_tiles * p.hgs, nseq * a.nsplit), kLsThreads, smem, stream>>>(mk, a);
    ASD_CUDA(cudaGetLastError());
    count_kernel(KERNEL_LATENT_STEP);
    if (a.nsplit > 1) return launch_latent_combine(ws.o, ws.ml, a.nsplit, d.R, out_lat, rows, stream);
    return 0;
}

}  // namespace asd
