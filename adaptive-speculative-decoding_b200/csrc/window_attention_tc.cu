// Windowed grouped-query attention (window_attention.cu's contract) on tcgen05 / TMEM for bf16 cache rows and calls that bring
// enough query rows: prompts, and verifications of models with many query heads per key/value head.
//
// What bounded the mma.sync form (window_attn_mma): 256 legacy instructions per 16 rows x 64 keys, because the fp32 queries and
// weights enter as two bf16 terms each, and a sincosf per result coordinate at the end: 189 us for 3 prompts of up to 777 tokens,
// 16 heads on 4 of 128.  Here a term's product of 128 rows x 128 keys is 8 instructions: 40 us (a CTA of seven tiles 16 us:
// 2.5 to bring the queries, 1.5 to the first scores, 1.5 a tile, 3 behind the last).
//   * CTA = 128 query rows (consecutive tokens x the query heads of one key/value head, which share their keys); the last tiles see
//     the most keys and start first.
//   * Both terms of the queries stand in shared memory (K-major 128-byte swizzle) for the CTA's life; key and value tiles of 128
//     positions come by TMA straight from the paged pool, 64 columns x one page a box, two tiles of each on their way.
//   * One warp issues the products: scores of tile j + 1, then the values of tile j, so that the tensor cores work while four
//     warps (thread = query row = TMEM lane) take the maxima of tile j + 1 and write its weights back over the scores as two bf16
//     terms, the A operand of the value product (keys are the contraction dimension: V is MN-major as it lies in the pool).
//   * The result accumulates in TMEM and is rescaled only when a row's maximum has grown by 2^8.  The sink joins the sum at the end;
//     the angles of the turn back by the query's position come from window_post_kernel.
// Shared memory (192 KB at 128 / 128) and TMEM (512 columns) allow one CTA per SM.  Launched plainly, never triggers (ptx.cuh).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "asd_internal.h"
#include "blocks.h"
#include "elem.cuh"
#include "gemm.h"
#include "ptx.cuh"
#include "softmax_tile.cuh"

namespace asd {

namespace {

constexpr int kWtThreads = 256;            // warps 0-3 softmax (thread = query row), 4 keys, 5 products, 6 values
constexpr int kWtKeys = 128;               // keys per tile
constexpr float kWtSlack = 8.0f;           // log2 growth of a row maximum that the weights tolerate before a rescale
// Query rows of a tile from which this kernel is the better one: all that the single-token form of the mma.sync kernel (up to 16
// rows) does not take.  20 rows: 16 sequences at 900 positions 86 us there, 29 here; 64 at 200 41 and 33; one at 64 25 and 15.
constexpr int kWtMinRows = 17;

struct WtArgs {
    const int* positions;
    const int* cu_q;
    const int* seq_slot;
    const int* page_table;
    int max_pages, page_shift;
    const float* q;
    long long ldq;
    WindowDims d;
    int group, TQ, inv_group;              // inv_group: r / group == r * inv_group >> 16 for every row r of a tile
    float scale2;                          // score scale x log2(e)
    const float* sink;
    const float2* turns;                   // [M][dv / 2] cos, sin of a token's value angles
    __nv_bfloat16* out;
    int* err;
};

struct WtBars {
    uint64_t q_full, k_full[2], k_empty[2], v_full[2], s_full[2], p_full[2], pv_done[2];
    uint32_t tmem;
    int failed;
};

__global__ void __launch_bounds__(kWtThreads, 1) window_attn_tc(const __grid_constant__ CUtensorMap map_kv, const WtArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const WindowDims& d = a.d;
    const int kc = d.dk >> 6, vc = d.dv >> 6;                  // chunks of 64 columns
    uint8_t* sQ = smem;                                        // [2 terms][kc]
    uint8_t* sK = sQ + 2 * kc * kStSlot;                       // [2 tiles][kc]
    uint8_t* sV = sK + 2 * kc * kStSlot;                       // [2 tiles][vc]
    WtBars* B = reinterpret_cast<WtBars*>(sV + 2 * vc * kStSlot);
    const WaitGuard guard{reinterpret_cast<volatile int*>(&B->failed), a.err, WAIT_WINDOW << 8};

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int seq = blockIdx.x / d.kv_heads, g = blockIdx.x - seq * d.kv_heads, tile_x = (int)gridDim.y - 1 - (int)blockIdx.y;
    const int t0 = a.cu_q[seq] + tile_x * a.TQ, t_end = a.cu_q[seq + 1];
    if (t0 >= t_end) return;
    const int n_tok = min(a.TQ, t_end - t0);
    const int p_first = a.positions[t0], p_last = p_first + n_tok - 1;
    // tiles start at multiples of 128 positions: those of the kept first positions, then those from the window's start on
    const int j_lo = max(p_first - d.window + 1, 0), base = j_lo & ~(kWtKeys - 1);
    const int nA = min((min(d.keep_first, j_lo) + kWtKeys - 1) / kWtKeys, base / kWtKeys);
    const int nt = nA + (p_last - base) / kWtKeys + 1;
    auto first_key = [&](int j) { return j < nA ? j * kWtKeys : base + (j - nA) * kWtKeys; };

    if (tid == 0) {
        tma_prefetch_desc(&map_kv);
        mbar_init(&B->q_full, 6);              // the warps that stage the queries
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->k_full[i], 1);
            mbar_init(&B->k_empty[i], 1);
            mbar_init(&B->v_full[i], 1);
            mbar_init(&B->s_full[i], 1);
            mbar_init(&B->p_full[i], 4);
            mbar_init(&B->pv_done[i], 1);
        }
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

    // both terms of the queries, by the warps that do not load (rows that are not there: zeros): eight elements a step, six steps'
    // loads on their way together
    if (warp != 4 && warp != 6) {
        const int ksh = kc == 2 ? 4 : 3;
        constexpr int kStagers = kWtThreads - 64, kAhead = 6;
        const int first = (warp < 4 ? warp : (warp == 5 ? 4 : 5)) * 32 + lane, total = 128 * kc * 8;
        for (int i0 = first; i0 < total; i0 += kAhead * kStagers) {
            float4 x[kAhead][2];
#pragma unroll
            for (int n = 0; n < kAhead; ++n) {
                const int i = i0 + n * kStagers, r = i >> ksh, c = i - (r << ksh), tq = r * a.inv_group >> 16;
                x[n][0] = x[n][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (i < total && tq < n_tok && r < a.TQ * a.group) {
                    const float4* src = reinterpret_cast<const float4*>(a.q + (long long)(t0 + tq) * a.ldq +
                                                                        (long long)(g * a.group + r - tq * a.group) * d.dk + c * 8);
                    x[n][0] = src[0];
                    x[n][1] = src[1];
                }
            }
#pragma unroll
            for (int n = 0; n < kAhead; ++n) {
                const int i = i0 + n * kStagers, r = i >> ksh, c = i - (r << ksh);
                if (i >= total) break;
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float u = e & 1 ? x[n][e >> 1].z : x[n][e >> 1].x, v = e & 1 ? x[n][e >> 1].w : x[n][e >> 1].y;
                    const __nv_bfloat162 h = __floats2bfloat162_rn(u, v);
                    const float2 f = __bfloat1622float2(h);
                    const __nv_bfloat162 l = __floats2bfloat162_rn(u - f.x, v - f.y);
                    hi[e] = *reinterpret_cast<const uint32_t*>(&h);
                    lo[e] = *reinterpret_cast<const uint32_t*>(&l);
                }
                uint8_t* dst = sQ + (c >> 3) * kStSlot + r * 128 + (((c & 7) ^ (r & 7)) << 4);
                *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(dst + kc * kStSlot) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&B->q_full);
    }

    if (warp == 4 || warp == 6) {
        // ------------------------------------------------------------------ key and value loaders: a lane per page
        const bool keys = warp == 4;
        const int psh = a.page_shift, pages = kWtKeys >> psh, last_page = p_last >> psh, nc = keys ? kc : vc;
        const int col = keys ? g * d.dk : d.kv_heads * d.dk + g * d.dv;
        const int* pt = a.page_table + (long long)a.seq_slot[seq] * a.max_pages;
        uint8_t* ring = keys ? sK : sV;
        uint64_t *full = keys ? B->k_full : B->v_full, *freed = keys ? B->k_empty : B->pv_done;
        // pages past the end repeat the sequence's last one: their keys are masked, their values zeroed
        auto page_of = [&](int j) { return lane < pages ? pt[min((first_key(j) >> psh) + lane, last_page)] : 0; };
        int next = page_of(0);
        for (int j = 0; j < nt; ++j) {
            const int page = next, s = j & 1;
            if (j + 1 < nt) next = page_of(j + 1);
            if (j >= 2 && !__all_sync(0xffffffffu, mbar_wait(&freed[s], ((j >> 1) - 1) & 1, guard))) break;
            if (lane == 0) mbar_expect_tx(&full[s], (uint32_t)(nc * kStSlot));
            __syncwarp();
            if (lane < pages)
                for (int c = 0; c < nc; ++c)
                    tma_load_2d(ring + (s * nc + c) * kStSlot + ((size_t)lane << (psh + 7)), &map_kv, col + c * 64, page << psh,
                                &full[s]);
            __syncwarp();
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------------ products
        // The whole warp walks the loops, so that addresses and descriptors stay in uniform registers, and one lane issues.
        const bool lead = elect_one();
        const uint32_t id_s = umma_idesc_bf16(128, 128), id_v = umma_idesc_bf16(128, (uint32_t)d.dv) | (1u << 16);   // V: MN-major
        const uint32_t uQ = smem_u32(sQ), uK = smem_u32(sK), uV = smem_u32(sV);
        auto ready = [&](uint64_t* bar, int phase) { return __all_sync(0xffffffffu, mbar_wait(bar, phase & 1, guard)) != 0; };
        bool ok = ready(&B->q_full, 0);
        auto values = [&](int j) {
            const int s = j & 1;
            ok = ok && ready(&B->v_full[s], j >> 1) && ready(&B->p_full[s], j >> 1);
            if (!ok) return;
            tc_fence_after();
            const uint32_t p = tmem + (uint32_t)(s * 128);
            const uint64_t vd = st_desc_mn(uV + (uint32_t)(s * vc * kStSlot));
            if (lead) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {                  // 16 keys; their high and low terms lie 32 columns apart
                    const uint32_t pc = p + (uint32_t)((k >> 2) * 64 + (k & 3) * 8);
                    umma_f16_ts(tmem + 256u, pc + 32, vd + k * (2048 >> 4), id_v, (j | k) != 0);
                    umma_f16_ts(tmem + 256u, pc, vd + k * (2048 >> 4), id_v, 1);
                }
                umma_commit(&B->pv_done[s]);
            }
            __syncwarp();
        };
        for (int j = 0; j < nt && ok; ++j) {
            const int s = j & 1;
            // the scores of tile j take the buffer of tile j - 2's weights
            if (j >= 2) ok = ready(&B->pv_done[s], (j >> 1) - 1);
            ok = ok && ready(&B->k_full[s], j >> 1);
            if (!ok) break;
            tc_fence_after();
            if (lead) {
                for (int u = 1; u >= 0; --u)                   // the low term first
                    for (int c = 0; c < kc; ++c) {
                        const uint64_t qd = umma_desc_sw128(uQ + (uint32_t)((u * kc + c) * kStSlot));
                        const uint64_t kd = umma_desc_sw128(uK + (uint32_t)((s * kc + c) * kStSlot));
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16(tmem + (uint32_t)(s * 128), qd + 2 * k, kd + 2 * k, id_s, u != 1 || c != 0 || k != 0);
                    }
                umma_commit(&B->k_empty[s]);
                umma_commit(&B->s_full[s]);
            }
            __syncwarp();
            if (j > 0) values(j - 1);
        }
        values(nt - 1);
    } else if (warp < 4) {
        // ------------------------------------------------------------------ softmax (thread = query row)
        const int tq = tid * a.inv_group >> 16;
        const bool real = tid < a.TQ * a.group && tq < n_tok;
        const int head = g * a.group + tid - tq * a.group;
        const int pos = real ? p_first + tq : -1;
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
        float ref = -INFINITY, l = 0.0f;                       // the maximum the weights refer to (log2), and their sum
        // a wait that gave up is reported; the walk goes on to the end, so that every barrier of these warps is met
        // (rolled loops: most tiles are the first or second of their kind on their SM)
        auto tile = [&](int j, auto masked_tag) {
            constexpr bool MASKED = decltype(masked_tag)::value;
            const int key0 = first_key(j);
            const StSeen seen{pos - d.window + 1 - key0, pos - key0, d.keep_first - key0};
            const uint32_t tS = lanes + (uint32_t)((j & 1) * 128);
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {
                uint32_t v[32];
                const uint32_t bits = MASKED ? seen.bits(q * 32) : 0u;
                tmem_ld_32x32(tS + (uint32_t)(q * 32), v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    float x = __uint_as_float(v[i]);
                    if (MASKED) x = bits & (1u << i) ? x : -INFINITY;
                    m4[i & 3] = fmaxf(m4[i & 3], x);
                }
            }
            // rn products with a positive scale keep the order; a negative or zero one is refused by the host
            const float top = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * a.scale2;
            const bool grow = real && (top > ref + kWtSlack || (ref == -INFINITY && top > -INFINITY));
            if (__any_sync(0xffffffffu, grow)) {
                const float corr = grow ? st_ex2(ref - top) : 1.0f;        // ref = -inf: 0, of a row that is 0 so far
                if (j > 0) {
                    mbar_wait_timed(&B->pv_done[(j - 1) & 1], ((j - 1) >> 1) & 1, guard, 2);
                    tc_fence_after();
                    for (int c = 0; c < d.dv; c += 32) {
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
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {      // both quarters of a half are read before its weights overwrite them
                uint32_t x0[32], x1[32], ph[16], pl[16];
                tmem_ld_32x32(tS + (uint32_t)(h * 64), x0);
                tmem_ld_32x32(tS + (uint32_t)(h * 64 + 32), x1);
                tmem_ld_wait();
                st_weights<MASKED>(x0, MASKED ? seen.bits(h * 64) : 0u, a.scale2, nref, ph, pl, sum);
                tmem_st_32x16(tS + (uint32_t)(h * 64), ph);
                tmem_st_32x16(tS + (uint32_t)(h * 64 + 32), pl);
                st_weights<MASKED>(x1, MASKED ? seen.bits(h * 64 + 32) : 0u, a.scale2, nref, ph, pl, sum);
                tmem_st_32x16(tS + (uint32_t)(h * 64 + 16), ph);
                tmem_st_32x16(tS + (uint32_t)(h * 64 + 48), pl);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        };
        for (int j = 0; j < nt; ++j) {
            const int key0 = first_key(j), s = j & 1;
            mbar_wait_timed(&B->s_full[s], (j >> 1) & 1, guard, 1);
            tc_fence_after();
            // every row sees every key
            const bool whole = key0 + kWtKeys <= p_first + 1 && (key0 >= p_last - d.window + 1 || key0 + kWtKeys <= d.keep_first);
            if (whole)
                tile(j, std::false_type{});
            else
                tile(j, std::true_type{});
            if (key0 + kWtKeys > p_last + 1 || (key0 < j_lo && key0 + kWtKeys > d.keep_first)) {
                // keys that no row of the tile may see: whatever the pool holds there must not meet the zero weights
                const int kp = key0 + tid;
                mbar_wait_timed(&B->v_full[s], (j >> 1) & 1, guard, 3);
                if (kp > p_last || (kp < j_lo && kp >= d.keep_first))
                    for (int c = 0; c < vc; ++c) {
                        uint4* dst = reinterpret_cast<uint4*>(sV + (s * vc + c) * kStSlot + tid * 128);
#pragma unroll
                        for (int i = 0; i < 8; ++i) dst[i] = make_uint4(0, 0, 0, 0);
                    }
                fence_proxy_async_smem();
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->p_full[s]);
        }
        mbar_wait_timed(&B->pv_done[(nt - 1) & 1], ((nt - 1) >> 1) & 1, guard, 4);
        tc_fence_after();
        // every load and product has ended: shared memory is free
        float inv = 1.0f / l;
        if (a.sink && real) {                                  // one more term of the denominator, without a value
            const float sk = a.sink[head] * 1.4426950408889634f, mf = fmaxf(ref, sk), so = exp2f(ref - mf);
            inv = so / (l * so + exp2f(sk - mf));
        }
        // rows through shared memory, so that a warp writes whole rows
        const int ld = d.dv * 2 + 16;                          // bytes; 16 of padding spread the lanes' rows over the banks
        uint8_t* own = sK + (size_t)warp * 32 * ld;
        const int half = d.dv >> 1;
        const float2* tr = a.turns + (long long)(t0 + (real ? tq : 0)) * half;
        for (int c = 0; c < (d.interleaved ? d.dv : half); c += 32) {
            uint32_t v[32], w[32];
            tmem_ld_32x32(lanes + 256u + (uint32_t)c, v);
            if (!d.interleaved) tmem_ld_32x32(lanes + 256u + (uint32_t)(c + half), w);
            tmem_ld_wait();
            // turned back: (u, v) of a pair becomes (u cos + v sin, v cos - u sin)
            if (d.interleaved) {
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float2 t = tr[(c + i) >> 1];
                    const float x = __uint_as_float(v[i]) * inv, y = __uint_as_float(v[i + 1]) * inv;
                    v[i] = __float_as_uint(x * t.x + y * t.y);
                    v[i + 1] = __float_as_uint(y * t.x - x * t.y);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float2 t = tr[c + i];
                    const float x = __uint_as_float(v[i]) * inv, y = __uint_as_float(w[i]) * inv;
                    v[i] = __float_as_uint(x * t.x + y * t.y);
                    w[i] = __float_as_uint(y * t.x - x * t.y);
                }
            }
            auto put = [&](int at, const uint32_t (&r)[32]) {
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    uint32_t b[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[i + 2 * e]), __uint_as_float(r[i + 2 * e + 1]));
                        b[e] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                    *reinterpret_cast<uint4*>(own + lane * ld + (at + i) * 2) = make_uint4(b[0], b[1], b[2], b[3]);
                }
            };
            put(c, v);
            if (!d.interleaved) put(c + half, w);
        }
        __syncwarp();
        const int lanes_row = d.dv >> 3, rows_step = 32 / lanes_row;       // 8 or 16 lanes write a row's 16-byte pieces
        const int c = lane & (lanes_row - 1);
        __nv_bfloat16* out0 = a.out + ((long long)t0 * d.heads + g * a.group) * d.dv + c * 8;
#pragma unroll 4
        for (int r = lane >> (d.dv == 128 ? 4 : 3); r < 32; r += rows_step) {
            const int rr = warp * 32 + r, t = rr * a.inv_group >> 16;
            const uint4 x = *reinterpret_cast<const uint4*>(own + r * ld + c * 16);
            if (rr < a.TQ * a.group && t < n_tok) {
                const int row = rr + t * (d.heads - a.group);
                *reinterpret_cast<uint4*>(out0 + (long long)row * d.dv) = x;
            }
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

bool window_attention_tc_takes(const WindowDims& d, const PagedRows& cache, int max_qlen, const float* q, long long ldq,
                               const void* out, int of32) {
    const int group = d.heads / d.kv_heads;
    if (cache.f32 || of32 || cache.rows <= 0 || cache.rows >= (1ll << 31) || max_qlen <= 0 || !(d.scale > 0.f)) return false;
    if ((d.dk != 64 && d.dk != 128) || (d.dv != 64 && d.dv != d.dk) || group > 128) return false;
    if (cache.page_size < 8 || cache.page_size > kWtKeys || (cache.page_size & (cache.page_size - 1))) return false;
    if (((reinterpret_cast<uintptr_t>(cache.pool) | reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) || ldq % 4)
        return false;
    return std::min(128 / group, max_qlen) * group >= kWtMinRows;
}

int launch_window_attention_tc(const SeqIndex& ix, const int* cu_q, const int* seq_slot, int nseq, int max_qlen, const float* q,
                               long long ldq, const WindowDims& d, const float* sink, const float2* turns,
                               const PagedRows& cache, void* out, cudaStream_t stream) {
    const int rowlen = d.kv_heads * (d.dk + d.dv), kc = d.dk / 64, vc = d.dv / 64;
    WtArgs a;
    a.positions = ix.positions, a.cu_q = cu_q, a.seq_slot = seq_slot;
    a.page_table = cache.page_table, a.max_pages = cache.max_pages;
    a.page_shift = 0;
    while ((1 << a.page_shift) < cache.page_size) ++a.page_shift;
    a.q = q, a.ldq = ldq, a.d = d;
    a.d.window = std::min(d.window, 1 << 30);
    a.group = d.heads / d.kv_heads;
    a.TQ = 128 / a.group, a.inv_group = (65536 + a.group - 1) / a.group;
    a.scale2 = d.scale * 1.4426950408889634f;
    a.sink = sink, a.turns = turns, a.out = static_cast<__nv_bfloat16*>(out), a.err = wait_word();
    const dim3 grid(nseq * d.kv_heads, (max_qlen + a.TQ - 1) / a.TQ);
    if (grid.y > 65535 || (long long)nseq * d.kv_heads >= (1ll << 31)) return set_error("windowed attention: too many tokens, sequences or heads");
    CUtensorMap mk;
    if (make_tmap_bf16(&mk, cache.pool, cache.rows, rowlen, rowlen, cache.page_size)) return -1;
    const int smem = 1024 + (4 * kc + 2 * vc) * kStSlot + (int)sizeof(WtBars);
    static PerDeviceOnce once;
    ASD_ONCE(once, ASD_CUDA(cudaFuncSetAttribute(window_attn_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024)));
    window_attn_tc<<<grid, kWtThreads, smem, stream>>>(mk, a);
    ASD_CUDA(cudaGetLastError());
    count_kernel(KERNEL_WINDOW_TC);
    return 0;
}

}  // namespace asd
