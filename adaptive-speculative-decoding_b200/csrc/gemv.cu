// Projections of ONE token on the CUDA cores: a single user's drafted or decoded token on a small model.
//
// Such a step is a chain of kernels that each read one weight matrix once, bound by each kernel's own latency: the
// weight-streaming tcgen05 kernel (gemm.cu) pays for tensor-map fetches, a barrier ring, TMEM and the cluster reduction of its
// K splits in every launch, 7 us in stream for matrices whose bytes take 0.3 to 3 us.  Here a warp owns pairs of weight rows
// and reads them 16 bytes a lane straight into registers; the first 4 KB of every warp are requested BEFORE
// griddepcontrol.wait, which for those matrices is most of what it will ever read.  The activations sit in shared memory as
// bf16.  Rows pair up as their epilogue needs them (rotary pair, gate and up row), so an epilogue is one lane's work after a
// butterfly, its operands requested before the products.  Where the rows are few and long, 2 to 8 warps share a pair and
// add their parts in order through shared memory.
// Same rounding points as gemm.cu: bf16 operands, fp32 sums, the fused RMSNorm's rstd and per-block sums of squares.
// A whole step of the 24-layer model of width 896 at 65 positions: 868 -> 594 us, 121 launches of 7.2 and 4.9 us.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "asd_internal.h"
#include "gemm.h"
#include "ptx.cuh"

namespace asd {

namespace {

constexpr int kGvThreads = 256, kGvWarps = kGvThreads / 32;
constexpr int kGvStep = 256;          // k elements of a row that a warp reads at once (16 bytes a lane)

struct GvArgs {
    const __nv_bfloat16* x;
    const __nv_bfloat16* w;
    int K, mode, units, ksplit, steps;      // steps: k steps of a row per warp
    int n_valid;
    void* out;
    QkvEpilogue qkv;
    NormFusion norm;
};

__device__ __forceinline__ float gv_silu_mul(float g, float u) { return __fdividef(g, 1.0f + __expf(-g)) * u; }
__device__ __forceinline__ void gv_unpack(const uint4& v, float (&f)[8]) {
    const uint32_t r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(r[i] << 16);
        f[2 * i + 1] = __uint_as_float(r[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ uint4 gv_load(const __nv_bfloat16* p) {        // a weight is read once: keep it out of L1
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// UN: row pairs a warp works on at once
template <int UN>
__global__ void __launch_bounds__(kGvThreads, 2) gemv_kernel(const GvArgs a) {
    constexpr int S = 4 / UN, R = 2 * UN;       // k steps of a row in flight, rows
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float rstd_s, part[kGvWarps][R], sq_s[kGvWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kpad = (a.K + kGvStep - 1) / kGvStep * kGvStep;
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(smem);                     // [kpad]
    const int groups = (a.units + UN - 1) / UN, at_once = kGvWarps / a.ksplit;      // groups of UN pairs; a block's at a time
    const int sub = warp % a.ksplit, k_first = sub * a.steps * kGvStep;
    const int half = a.mode == GEMM_OUT_QKV ? a.qkv.hd >> 1 : 0;

    // weight rows of a pair
    auto rows_of = [&](int u, int& r0, int& r1) {
        if (a.mode == GEMM_OUT_QKV) {
            r0 = u / half * a.qkv.hd + u % half;
            r1 = r0 + half;
        } else if (a.mode == GEMM_OUT_SWIGLU) {
            r0 = (u >> 6) * 128 + (u & 63);
            r1 = r0 + 64;
        } else {
            r0 = 2 * u;
            r1 = min(2 * u + 1, a.n_valid - 1);
        }
    };
    const __nv_bfloat16* wp[R];
    auto point = [&](int g) {
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            int r0, r1;
            rows_of(min(g * UN + i, a.units - 1), r0, r1);
            wp[2 * i] = a.w + (size_t)r0 * a.K;
            wp[2 * i + 1] = a.w + (size_t)r1 * a.K;
        }
    };
    uint4 buf[2][R][S];
    auto fetch = [&](uint4 (&b)[R][S], int step) {
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int k = k_first + (step + s) * kGvStep + lane * 8;
            const bool in = step + s < a.steps && k < a.K;
#pragma unroll
            for (int r = 0; r < R; ++r) b[r][s] = in ? gv_load(wp[r] + k) : make_uint4(0, 0, 0, 0);
        }
    };
    int g = blockIdx.x * at_once + warp / a.ksplit;
    if (g < groups) {
        point(g);
        fetch(buf[0], 0);
    }
    grid_dep_wait();                    // the weights never change; everything below reads what earlier kernels wrote
    for (int k = tid * 8; k < kpad; k += kGvThreads * 8)
        *reinterpret_cast<uint4*>(xs + k) = k < a.K ? *reinterpret_cast<const uint4*>(a.x + k) : make_uint4(0, 0, 0, 0);
    if (warp == kGvWarps - 1) {
        float ss = 0.0f;
        for (int t = lane; t < a.norm.parts; t += 32) ss += a.norm.sumsq_in[(size_t)t * a.norm.ld];
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
        if (lane == 0) rstd_s = a.norm.sumsq_in ? rsqrtf(ss / (float)a.norm.hidden + a.norm.eps) : 1.0f;
    }
    // what a pair's epilogue reads, one pair a lane: requested before the products
    const bool residual = a.norm.sumsq_out != nullptr;
    float e0 = 0.f, e1 = 0.f, l0 = 0.f, l1 = 0.f;      // old residual | biases; next norm's weights | cos, sin
    __nv_bfloat16* dst = nullptr;
    auto operands = [&](int g0) {
        const int u = g0 * UN + lane;
        if (lane >= UN || u >= a.units || sub != 0) return;
        if (residual) {
            const bool two = 2 * u + 1 < a.n_valid;
            const float* o = static_cast<const float*>(a.out) + 2 * u;
            e0 = o[0], e1 = two ? o[1] : 0.0f;
            l0 = __bfloat162float(a.norm.ln_w[2 * u]), l1 = two ? __bfloat162float(a.norm.ln_w[2 * u + 1]) : 0.0f;
        } else if (a.mode == GEMM_OUT_QKV) {
            const QkvEpilogue& e = a.qkv;
            const int head = u / half, j = u % half;
            const bool rot = head < e.nh + e.nkv;
            e0 = __bfloat162float(e.bias[head * e.hd + j]), e1 = __bfloat162float(e.bias[head * e.hd + j + half]);
            const float2 cs = rot ? e.cs[j] : make_float2(1.0f, 0.0f);
            l0 = cs.x, l1 = cs.y;
            if (head < e.nh) {
                dst = e.q_out + head * e.hd + j;
            } else {
                const int pos = e.positions[0];
                const int page = e.page_table[(size_t)e.token_slot[0] * e.max_pages + pos / e.page_size];
                const int kvh = rot ? head - e.nh : head - e.nh - e.nkv;
                dst = (rot ? e.k_cache : e.v_cache) + ((size_t)(page * e.nkv + kvh) * e.page_size + pos % e.page_size) * e.hd + j;
            }
        }
    };
    operands(g);
    __syncthreads();
    grid_dep_launch();                  // the next kernel may request its weights

    float sq = 0.0f;
    const int rounds = (groups + gridDim.x * at_once - 1) / (gridDim.x * at_once);
    for (int it = 0; it < rounds; ++it, g += gridDim.x * at_once) {
        const bool live = g < groups;
        if (it > 0) operands(g);
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = 0.0f;
        if (live) {
            auto use = [&](const uint4 (&b)[R][S], int step) {
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    if (step + s >= a.steps) break;
                    const int k = min(k_first + (step + s) * kGvStep, kpad - kGvStep) + lane * 8;      // (past the end: zero weights)
                    float x[8];
                    gv_unpack(*reinterpret_cast<const uint4*>(xs + k), x);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        float w[8];
                        gv_unpack(b[r][s], w);
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[r] = fmaf(w[i], x[i], acc[r]);
                    }
                }
            };
            for (int step = 0; step < a.steps; step += 2 * S) {        // the next steps' rows are on their way meanwhile
                if (step + S < a.steps) fetch(buf[1], step + S);
                use(buf[0], step);
                if (step + 2 * S < a.steps) fetch(buf[0], step + 2 * S);
                if (step + S < a.steps) use(buf[1], step + S);
            }
        }
        if (g + (int)gridDim.x * at_once < groups) {                   // the next group's first rows, before the epilogue
            point(g + gridDim.x * at_once);
            fetch(buf[0], 0);
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], d);
        if (a.ksplit > 1) {             // parts of a pair meet in shared memory, added in order
            if (lane == 0)
#pragma unroll
                for (int r = 0; r < R; ++r) part[warp][r] = acc[r];
            __syncthreads();
            if (sub == 0)
#pragma unroll
                for (int r = 0; r < R; ++r)
                    for (int s = 1; s < a.ksplit; ++s) acc[r] += part[warp + s][r];
            __syncthreads();
        }
        const int u = g * UN + lane;
        if (!live || sub != 0 || lane >= UN || u >= a.units) continue;
        const float v0 = UN == 2 && lane ? acc[R - 2] : acc[0], v1 = UN == 2 && lane ? acc[R - 1] : acc[1];
        if (a.mode == GEMM_OUT_QKV) {
            const float x1 = v0 * rstd_s + e0, x2 = v1 * rstd_s + e1;
            dst[0] = __float2bfloat16(x1 * l0 - x2 * l1);
            dst[half] = __float2bfloat16(x2 * l0 + x1 * l1);
        } else if (a.mode == GEMM_OUT_SWIGLU) {
            static_cast<__nv_bfloat16*>(a.out)[u] = __float2bfloat16(gv_silu_mul(v0 * rstd_s, v1 * rstd_s));
        } else {
            float* o = static_cast<float*>(a.out) + 2 * u;
            const bool two = 2 * u + 1 < a.n_valid;
            if (residual) {             // residual += result; the next norm's input and sum of squares
                const float y0 = e0 + v0, y1 = two ? e1 + v1 : 0.0f;
                __nv_bfloat16* b = a.norm.resid_bf + 2 * u;
                o[0] = y0;
                b[0] = __float2bfloat16(y0 * l0);
                if (two) o[1] = y1, b[1] = __float2bfloat16(y1 * l1);
                sq += y0 * y0 + y1 * y1;
            } else {
                o[0] = v0 * rstd_s;
                if (two) o[1] = v1 * rstd_s;
            }
        }
    }
    if (residual) {
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, d);
        if (lane == 0) sq_s[warp] = sq;
        __syncthreads();
        if (tid == 0) {
            float s = 0.0f;
            for (int w = 0; w < kGvWarps; ++w) s += sq_s[w];
            a.norm.sumsq_out[(size_t)blockIdx.x * a.norm.ld] = s;
        }
    }
}

template <int UN>
int gv_launch(const GvArgs& a, int blocks, size_t smem, cudaStream_t stream) {
    ASD_CUDA(launch_pdl(gemv_kernel<UN>, blocks, kGvThreads, smem, stream, a));
    count_kernel(KERNEL_GEMV);
    return 0;
}

}  // namespace

// One token, matrices of at most 128 MB (the largest of the layer's), activations within the default shared memory.  On a
// width-896 model (17 MB at most) a step of eight layers takes 235 us here and 329 with gemm.cu, on a width-1536 one (55 MB)
// 351 and 450; with 272 MB the streams weigh more than the latencies (four layers of width 3584: 572 in this kernel's first
// form, 553 in gemm.cu).  A form for two to four tokens gained little with two where one gains most (318 and 333) and lost
// elsewhere (471 and 445): the products are CUDA-core work per token.
bool gemv_takes(int M, int max_k, size_t max_bytes) { return M == 1 && max_k <= 16384 && max_bytes <= (size_t)128 << 20; }

// x bf16 [K], w bf16 [N][K] row major; max_parts bounds the blocks of a launch that writes sums of squares (one per block, norm.ld
// apart; gemv_max_blocks() never bounds it), *blocks_out their number.
int gemv_launch(int mode, const __nv_bfloat16* x, const __nv_bfloat16* w, int K, int n_valid, void* out, const QkvEpilogue* qkv,
                const NormFusion* norm, int max_parts, int* blocks_out, cudaStream_t stream) {
    if (K <= 0 || K > 16384 || (K & 7) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15))
        return set_error("gemv: shape or alignment outside the kernel's contract");
    GvArgs a = {};
    a.x = x, a.w = w, a.K = K, a.mode = mode, a.n_valid = n_valid, a.out = out;
    if (qkv) a.qkv = *qkv;
    if (norm) a.norm = *norm;
    a.units = mode == GEMM_OUT_QKV ? n_valid / 2 : (mode == GEMM_OUT_SWIGLU ? n_valid : (n_valid + 1) / 2);
    // Two blocks of eight warps per SM.  Enough pairs: each warp takes two at once (an activation read serves four rows);
    // too few for the chip: warps share a pair's k range, 512 elements or more each.
    const int at_a_time = 2 * sm_count(), want = at_a_time * kGvWarps;
    const int un = a.units >= 2 * want ? 2 : 1;
    const int steps = (K + kGvStep - 1) / kGvStep;
    a.ksplit = 1;
    while (un == 1 && a.ksplit < kGvWarps && 4 * a.units * a.ksplit < 3 * want && steps / (2 * a.ksplit) >= 2) a.ksplit *= 2;
    a.steps = (steps + a.ksplit - 1) / a.ksplit;
    const int groups = (a.units + un - 1) / un, at_once = kGvWarps / a.ksplit;
    int blocks = std::min((groups + at_once - 1) / at_once, at_a_time);
    if (a.norm.sumsq_out) blocks = std::max(1, std::min(blocks, max_parts));
    if (blocks_out) *blocks_out = blocks;
    const size_t smem = (size_t)steps * kGvStep * 2;
    return un == 2 ? gv_launch<2>(a, blocks, smem, stream) : gv_launch<1>(a, blocks, smem, stream);
}

int gemv_max_blocks() { return 2 * sm_count(); }

int preload_gemv() {
    cudaFuncAttributes fa;
    ASD_CUDA(cudaFuncGetAttributes(&fa, gemv_kernel<1>));
    ASD_CUDA(cudaFuncGetAttributes(&fa, gemv_kernel<2>));
    return 0;
}

}  // namespace asd
