// Paged-KV attention of few query rows (head_dim 128, pages of 16 positions): a drafted token's group of query heads, a
// verification's few positions.
//
// attention_tc.cu walks a sequence's keys tile by tile on the tensor cores, 128 lanes for what may be 7 rows: 1.2 us a tile of
// 128 keys, one after the other.  Here no key waits for another:
//   * the pages of a CTA's share are requested at once (24 of them, 8 KB each; the rest as slots empty), those that hold no new
//     position before griddepcontrol.wait;
//   * eight warps for every 16 query rows take the pages in turn: scores, running softmax and value product of 16 keys by mma.sync
//     m16n8k16, operands by ldmatrix from the 128-byte swizzle that TMA wrote, weights straight from the score fragments.  Bound by the
//     latency of the first pages and of the final sums while a share is short, by HBM beyond;
//   * the warps' results meet in shared memory, a sequence's shares by the last CTA of them.
// Rounding as in attention_tc.cu: bf16 queries, keys, values and weights, fp32 sums, the weights' sum takes them unrounded.
//
// A layer of a step with it and with attention_tc.cu: 16 sequences of 512 keys, 4 key/value heads of 7 rows 38 and 43 us, of 2048 keys 50
// and 54; 4 such sequences of 2048 keys 39 and 49; 64 sequences of 512 keys 61 and 67; 8 heads of 2 rows, 128 sequences of 512 keys 103
// and 123; 8 heads of 30 rows, 16 sequences of 512 keys 56.6 and 58.1, of 2048 keys 75 and 81, one of 2048 keys 45 and 55.5.  (32 rows in
// eight warps, a warp both tiles: 58.1 and 78.6.)  A drafted token through four 7B layers (16 sequences, 512 keys): 588 -> 567 us.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "asd_internal.h"
#include "layers.h"
#include "mma_sync.cuh"
#include "ptx.cuh"

namespace asd {

namespace {

constexpr int kAfWarps = 8;                        // that take pages in turn, for every tile of 16 query rows
constexpr int kAfPage = 16;                        // positions of a page
constexpr int kAfHalf = kAfPage * 128;             // bytes of a page's first or last 64 dimensions
constexpr int kAfSlot = 4 * kAfHalf;               // keys and values of a page
constexpr int kAfSlots = 24;                       // a multiple of the warps: a slot's pages are one warp's (one of each tile's)
constexpr int kAfQLd = 272;                        // bytes of a query row in shared memory
constexpr int kAfOLd = 132;                        // floats of a result row there

struct AfArgs {
    const __nv_bfloat16* q;        // [M, nh, 128]
    const int *positions, *cu_q, *seq_slot, *page_table;
    int max_pages, nh, nkv, split_keys, nsplit_max;
    long long k_row0, v_row0;      // first pool row (position-major rows of 128 dims) of this layer's K / V
    float scale_log2;
    float *o_part, *ml_part;
    int* tickets;
    __nv_bfloat16* out;
    int* err;
};

__device__ __forceinline__ float af_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <int RT>      // tiles of 16 query rows, eight warps each
__global__ void __launch_bounds__(256 * RT, 1) attn_few_kernel(const __grid_constant__ CUtensorMap kv_map, const AfArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full[kAfSlots];
    __shared__ __align__(16) uint8_t sQ[RT * 16 * kAfQLd];
    __shared__ float sM[kAfWarps][RT * 16], sL[kAfWarps][RT * 16];
    __shared__ int s_failed, s_last;
    const WaitGuard guard{&s_failed, a.err, WAIT_ATTENTION << 8};
    constexpr int kThreads = 256 * RT;
    const int tid = threadIdx.x, warp = (tid >> 5) & 7, tile = tid >> 8, lane = tid & 31, gr = lane >> 2, t4 = lane & 3;
    const int seq = blockIdx.x, g = blockIdx.y, sp = blockIdx.z, G = a.nh / a.nkv;
    const int q0 = a.cu_q[seq], qlen = a.cu_q[seq + 1] - q0;
    if (qlen <= 0) return;
    const int R = qlen * G, kv_len = a.positions[q0] + qlen;
    const int kbeg = sp * a.split_keys;
    if (kbeg >= kv_len) return;
    const int kend = min(kv_len, kbeg + a.split_keys), pages = (kend - kbeg + kAfPage - 1) / kAfPage;
    const int nsplit_seq = (kv_len + a.split_keys - 1) / a.split_keys, ready = kv_len - qlen;      // keys that earlier forwards wrote
    const int* pt = a.page_table + (size_t)a.seq_slot[seq] * a.max_pages + kbeg / kAfPage;
    if (tid == 0) {
        tma_prefetch_desc(&kv_map);
        for (int i = 0; i < kAfSlots; ++i) mbar_init(&full[i], 1);
        s_failed = 0;
        fence_mbar_init();
    }
    __syncthreads();
    auto request = [&](int p) {        // a lane's job
        const int slot = p % kAfSlots;
        const long long row = ((long long)pt[p] * a.nkv + g) * kAfPage;
        uint8_t* dst = ring + slot * kAfSlot;
        mbar_expect_tx(&full[slot], kAfSlot);
        tma_load_2d(dst, &kv_map, 0, (int)(a.k_row0 + row), &full[slot]);
        tma_load_2d(dst + kAfHalf, &kv_map, 64, (int)(a.k_row0 + row), &full[slot]);
        tma_load_2d(dst + 2 * kAfHalf, &kv_map, 0, (int)(a.v_row0 + row), &full[slot]);
        tma_load_2d(dst + 3 * kAfHalf, &kv_map, 64, (int)(a.v_row0 + row), &full[slot]);
    };
    // the warp's own first pages (slots warp, warp + 8, ...), a lane each
    const int mine = warp + lane * kAfWarps;
    const bool asks = tile == 0 && lane < kAfSlots / kAfWarps && mine < pages, old = kbeg + (mine + 1) * kAfPage <= ready;
    if (asks && old) request(mine);
    grid_dep_wait();
    grid_dep_launch();
    if (asks && !old) request(mine);
    for (int i = tid; i < RT * 16 * 16; i += kThreads) {
        const int r = i >> 4, c = i & 15, t = r / G;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r < R) v = *reinterpret_cast<const uint4*>(a.q + ((size_t)(q0 + t) * a.nh + g * G + (r - t * G)) * 128 + c * 8);
        *reinterpret_cast<uint4*>(sQ + r * kAfQLd + c * 16) = v;
    }
    __syncthreads();

    float o[16][4], m[2], l[2];
    int last[2];                       // a row's last visible key (rows that are not there: none)
#pragma unroll
    for (int n = 0; n < 16; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = tile * 16 + gr + 8 * h;
        m[h] = -INFINITY, l[h] = 0.0f, last[h] = r < R ? ready + r / G : -1;
    }
#pragma unroll 1
    for (int p = warp; p < pages; p += kAfWarps) {
        const int slot = p % kAfSlots, key0 = kbeg + p * kAfPage;
        uint8_t* pg = ring + slot * kAfSlot;
        mbar_wait_timed(&full[slot], (p / kAfSlots) & 1, guard, 16);
        if (key0 + kAfPage > kend) {   // places that nobody wrote must not meet the zero weights
            for (int i = lane; i < (key0 + kAfPage - kend) * 16; i += 32) {
                const int r = kend - key0 + (i >> 4), c = i & 15;
                *reinterpret_cast<uint4*>(pg + (2 + (c >> 3)) * kAfHalf + r * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
            }
            __syncwarp();
        }
        // scores of 16 keys: two tiles of eight, eight steps of 16 dimensions
        float sc[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.0f;
        const uint32_t kb = smem_u32(pg);
        const int kr = (lane & 7) + ((lane >> 4) << 3), kc = (lane >> 3) & 1;      // key row and 8-dimension half of this lane's address
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint32_t b[4], q[4];       // keys 0-7: dimensions 0-7, 8-15; keys 8-15 the same
            const int c = (k & 3) * 2 + kc;
            ldsm_x4(kb + (uint32_t)((k >> 2) * kAfHalf + kr * 128 + ((c ^ (kr & 7)) << 4)), b);
            ldsm_x4(smem_u32(sQ) + (uint32_t)((tile * 16 + (lane & 15)) * kAfQLd + k * 32 + (lane >> 4) * 16), q);
            mma_bf16(sc[0], q, b[0], b[1]);
            mma_bf16(sc[1], q, b[2], b[3]);
        }
        // running softmax: a thread has keys 2 t4, 2 t4 + 1 of either tile for rows gr and gr + 8
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int kp = key0 + (e >> 1) * 8 + t4 * 2 + (e & 1);
                x[e] = kp <= last[h] && kp < kend ? sc[e >> 1][2 * h + (e & 1)] * a.scale_log2 : -INFINITY;
            }
            float top = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float mn = fmaxf(m[h], top), ref = mn == -INFINITY ? 0.0f : mn, corr = af_ex2(m[h] - ref);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = af_ex2(x[e] - ref);
            l[h] = l[h] * corr + ((x[0] + x[1]) + (x[2] + x[3]));      // (of this thread's keys)
            m[h] = mn;
            w[h] = pack_bf16(x[0], x[1]), w[2 + h] = pack_bf16(x[2], x[3]);
#pragma unroll
            for (int n = 0; n < 16; ++n) o[n][2 * h] *= corr, o[n][2 * h + 1] *= corr;
        }
        // values: 16 dimensions a load
        const int vr = lane & 15, vc = lane >> 4;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            uint32_t b[4];
            const int c = (n & 3) * 2 + vc;
            ldsm_x4_t(kb + (uint32_t)((2 + (n >> 2)) * kAfHalf + vr * 128 + ((c ^ (vr & 7)) << 4)), b);
            mma_bf16(o[2 * n], w, b[0], b[1]);
            mma_bf16(o[2 * n + 1], w, b[2], b[3]);
        }
        if (p + kAfSlots < pages) {    // the slot is free when every tile's warp has read it
            if (RT > 1)
                asm volatile("bar.sync %0, %1;" ::"r"(1 + warp), "n"(32 * RT) : "memory");
            else
                __syncwarp();
            if (tile == 0) {
                fence_proxy_async_smem();
                if (lane == 0) request(p + kAfSlots);
            }
        }
    }
    __syncthreads();                   // every page has come and been read: the ring is free
    float* part = reinterpret_cast<float*>(ring) + (size_t)warp * RT * 16 * kAfOLd;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = tile * 16 + gr + 8 * h;
        float t = l[h];
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        if (t4 == 0) sM[warp][r] = m[h], sL[warp][r] = t;
#pragma unroll
        for (int n = 0; n < 16; ++n) *reinterpret_cast<float2*>(part + r * kAfOLd + n * 8 + t4 * 2) = make_float2(o[n][2 * h], o[n][2 * h + 1]);
    }
    __syncthreads();
    const int busy = min(kAfWarps, pages);
    for (int i = tid; i < R * 32; i += kThreads) {
        const int r = i >> 5, d4 = i & 31, t = r / G;
        const size_t th = (size_t)(q0 + t) * a.nh + g * G + (r - t * G);
        float mx = -INFINITY, sum = 0.0f;
        for (int w = 0; w < busy; ++w) mx = fmaxf(mx, sM[w][r]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int w = 0; w < busy; ++w) {
            const float f = sM[w][r] == -INFINITY ? 0.0f : af_ex2(sM[w][r] - mx);
            const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(ring) + (size_t)(w * RT * 16 + r) * kAfOLd + d4 * 4);
            sum += sL[w][r] * f;
            acc.x += v.x * f, acc.y += v.y * f, acc.z += v.z * f, acc.w += v.w * f;
        }
        if (nsplit_seq == 1) {
            const float inv = 1.0f / sum;
            __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(a.out + th * 128) + d4 * 2;
            op[0] = __floats2bfloat162_rn(acc.x * inv, acc.y * inv);
            op[1] = __floats2bfloat162_rn(acc.z * inv, acc.w * inv);
        } else {
            const size_t at = th * a.nsplit_max + sp;
            *(reinterpret_cast<float4*>(a.o_part + at * 128) + d4) = acc;
            if (d4 == 0) a.ml_part[at * 2] = mx, a.ml_part[at * 2 + 1] = sum;
        }
    }
    wait_settle(guard);
    if (nsplit_seq == 1) return;
    // the last CTA of this (sequence, kv head) merges the shares
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int tk = atomicAdd(&a.tickets[q0 * a.nkv + g], 1);
        s_last = tk == nsplit_seq - 1;
        if (s_last) a.tickets[q0 * a.nkv + g] = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int i = tid; i < R * 32; i += kThreads) {
        const int r = i >> 5, d4 = i & 31, t = r / G;
        const size_t th = (size_t)(q0 + t) * a.nh + g * G + (r - t * G), base = th * a.nsplit_max;
        const int ns = min(nsplit_seq, (ready + t) / a.split_keys + 1);        // shares that hold a visible key
        float mx = -INFINITY, sum = 0.0f;
        for (int s2 = 0; s2 < ns; ++s2) mx = fmaxf(mx, __ldcg(&a.ml_part[(base + s2) * 2]));
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s2 = 0; s2 < ns; ++s2) {
            const float f = af_ex2(__ldcg(&a.ml_part[(base + s2) * 2]) - mx);
            sum += __ldcg(&a.ml_part[(base + s2) * 2 + 1]) * f;
            const float4 v = __ldcg(reinterpret_cast<const float4*>(a.o_part + (base + s2) * 128) + d4);
            acc.x += v.x * f, acc.y += v.y * f, acc.z += v.z * f, acc.w += v.w * f;
        }
        const float inv = 1.0f / sum;
        __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(a.out + th * 128) + d4 * 2;
        op[0] = __floats2bfloat162_rn(acc.x * inv, acc.y * inv);
        op[1] = __floats2bfloat162_rn(acc.z * inv, acc.w * inv);
    }
}

constexpr int kAfSmem = 1024 + kAfSlots * kAfSlot;

}  // namespace

// Keys of a share, whole pages; 0: not taken.
// Up to 16 rows it was faster at every length (16 to 8192 keys) and number of sequences (1 to 128, up to 1024 CTAs): by 3 to 5 us a layer
// where the CTAs fit the SMs, by up to 28 beyond.  17 to 32 rows of up to 256 tokens: 2 to 11 us (27 where attention_tc.cu does not split
// 8192 keys), at worst equal (64 sequences of 4 heads, 28 rows, 384 keys: 104.2 and 104.4).  More tokens come from the CTA-pair GEMM, whose
// glue kernel leaves no time to request pages ahead: 0.3 to 12 us faster up to 256 keys, from 384 on between 2 faster and 4 slower.
// A split ends with one more pass through memory, 2.5 us: 768 keys in one share cost 38.0 to 40.5 us a layer, in two to four 38.9 to 42;
// 1024 the reverse, 39.4 and 40.  Beyond 16 shares their merge grows faster than the keys shrink (8192 keys of one sequence: 46.1 us in 37
// shares of 14 pages, 44 in 16).
int attention_few_split(int M, int nseq, int nkv, int hd, int page_size, int rows, int max_kv_len) {
    if (hd != 128 || page_size != kAfPage || rows > 32 || max_kv_len <= 0) return 0;
    if (rows > 16 && M > 256 && max_kv_len > 256) return 0;
    const int items = std::max(nseq * nkv, 1), sms = sm_count(), pages = (max_kv_len + kAfPage - 1) / kAfPage;
    const int shares = pages <= 48 ? 1 : std::max(1, std::min({sms / items, pages / 16, 16}));
    return (pages + shares - 1) / shares * kAfPage;
}

int launch_attention_few(const AttnLaunch& L, cudaStream_t stream) {
    if (preload_attention_few()) return -1;
    AfArgs a;
    a.q = L.q, a.positions = L.positions, a.cu_q = L.cu_q, a.seq_slot = L.seq_slot, a.page_table = L.page_table;
    a.max_pages = L.max_pages, a.nh = L.nh, a.nkv = L.nkv, a.split_keys = L.split_keys, a.nsplit_max = L.nsplit_max;
    a.k_row0 = L.k_row0, a.v_row0 = L.v_row0;
    a.scale_log2 = 1.4426950408889634f / sqrtf((float)L.hd);
    a.o_part = L.o_part, a.ml_part = L.ml_part, a.tickets = L.tickets, a.out = L.out, a.err = wait_word();
    const bool two = L.max_qlen * (L.nh / L.nkv) > 16;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(L.nseq, L.nkv, L.nsplit_max);
    cfg.blockDim = dim3(two ? 512 : 256);
    cfg.dynamicSmemBytes = kAfSmem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().glue_pdl ? 1 : 0;
    ASD_CUDA(cudaLaunchKernelEx(&cfg, two ? attn_few_kernel<2> : attn_few_kernel<1>, *L.kv_map, a));
    count_kernel(KERNEL_ATTENTION_FEW);
    return 0;
}

int preload_attention_few() {
    static PerDeviceOnce once;
    ASD_ONCE(once, {
        ASD_CUDA(cudaFuncSetAttribute(attn_few_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAfSmem));
        ASD_CUDA(cudaFuncSetAttribute(attn_few_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAfSmem));
        prefer_max_smem(attn_few_kernel<1>);
        prefer_max_smem(attn_few_kernel<2>);
    });
    return 0;
}

}  // namespace asd
