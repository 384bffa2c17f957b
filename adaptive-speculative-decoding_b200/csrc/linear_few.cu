// Dense projections of a few tokens, y fp32 [M][ldc] = x bf16 [M][K] * w bf16 [N][K]^T with M <= 16: what a step of a few sequences
// asks of a layer's smaller matrices.
//
// Such a step is a chain of kernels that read a matrix of 4 to 60 MB once, 1 to 10 us at HBM speed, and what they cost beside that
// is their head and tail.  The weight-streaming tcgen05 kernel (gemm.cu) pays for barrier rings, TMEM and a cluster reduction of its
// K splits (5 us) in every launch.  Here a block owns groups of 16 weight rows and its eight warps share K:
//   * a warp reads its part of the rows 16 bytes a lane straight into registers, eight 32-element pieces of both row tiles on their
//     way (8 KB a warp, 128 KB an SM), the first of them requested BEFORE griddepcontrol.wait;
//   * a lane's 16 bytes are eight consecutive k of one weight row, and of two tokens from shared memory: the operands of two
//     mma.sync m16n8k16 whose k indexes are permuted alike on both sides, so that neither needs a transpose or ldmatrix;
//   * the warps' sums meet in shared memory, added in warp order, one barrier per group.
// The sums of a token depend on neither M nor the other tokens.
// 16 tokens, cold matrices, us (gemm.cu before): 2048 x 2048 10.3 -> 5.6, 6144 x 2048 12.4 -> 9.4, 8224 x 2048 13.1 -> 9.8,
// 3072 x 1024 8.3 -> 5.4, 4096 x 4096 14.2 -> 10.2, 6720 x 4096 22.3 -> 13.4; 2048 x 6144 13.8 -> 12.1,
// 128 x 6144 10.3 -> 10.4.  In a step gemm.cu's launches overlap; dense.h says which matrices a step leaves to them.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "asd_internal.h"
#include "blocks.h"
#include "mma_sync.cuh"
#include "ptx.cuh"

namespace asd {

namespace {

constexpr int kLfThreads = 256, kLfWarps = 8;
constexpr int kLfTok = 16, kLfRows = 16; // tokens, weight rows a group
constexpr int kLfAhead = 8;              // pieces of 32 k on their way per warp

struct LfArgs {
    const __nv_bfloat16* x;
    const __nv_bfloat16* w;
    float* y;
    int M, N, K, ldc;
    int pieces;                          // of 32 k per warp
    int row_bytes;                       // of a warp's slice of a token in shared memory: an odd multiple of 64
};

__device__ __forceinline__ uint4 lf_load(const __nv_bfloat16* p) {        // a weight is read once: keep it out of L1
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 lf_shared(uint32_t addr) {      // in its place among the products: all at once they do not fit registers
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

__global__ void __launch_bounds__(kLfThreads, 2) linear_few_kernel(const LfArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float red[2][kLfWarps][kLfTok * kLfRows];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int groups = (a.N + kLfRows - 1) / kLfRows;
    const int k0 = warp * a.pieces * 32 + t * 8;                           // this lane's first k
    uint8_t* xs = smem + (size_t)warp * kLfTok * a.row_bytes;               // [tokens][row_bytes]

    // loads run one block of kLfAhead pieces before the products, over the borders of groups
    int lg = blockIdx.x, lc = 0, there = 0;      // group and first piece of the block that is loaded next; pieces of it that exist
    const __nv_bfloat16 *w0, *w1;                // at that piece
    auto point = [&]() {
        const int n = min(lg, groups - 1) * kLfRows + g;
        w0 = a.w + (size_t)min(n, a.N - 1) * a.K + k0 + lc * 32;
        w1 = a.w + (size_t)min(n + 8, a.N - 1) * a.K + k0 + lc * 32;
        there = lg < groups ? min(a.pieces - lc, (a.K - k0 - lc * 32 + 31) >> 5) : 0;
    };
    auto fetch = [&](int j, uint4 (&b)[2]) {
        b[0] = j < there ? lf_load(w0 + j * 32) : make_uint4(0, 0, 0, 0);
        b[1] = j < there ? lf_load(w1 + j * 32) : make_uint4(0, 0, 0, 0);
    };
    auto next = [&]() {
        lc += kLfAhead;
        if (lc >= a.pieces) lc = 0, lg += gridDim.x;
        point();
    };
    uint4 buf[kLfAhead][2];
    point();
#pragma unroll
    for (int j = 0; j < kLfAhead; ++j) fetch(j, buf[j]);
    next();
    grid_dep_wait();                     // the weights never change; everything below reads what earlier kernels wrote
    grid_dep_launch();
    {
        const int per = a.pieces * 4;    // 16-byte places of a token in the warp's slice
        for (int m = 0; m < kLfTok; ++m)
            for (int i = lane; i < per; i += 32) {
                const int k = warp * a.pieces * 32 + i * 8;
                const bool in = m < a.M && k < a.K;
                cp_async16(smem_u32(xs + m * a.row_bytes + i * 16), a.x + (in ? (size_t)m * a.K + k : 0), in);
            }
        cp_async_commit();
        cp_async_wait<0>();
        __syncwarp();
    }
    int b = 0;
    const uint32_t xl = smem_u32(xs) + g * a.row_bytes + t * 16;
#pragma unroll 1
    for (int cg = blockIdx.x; cg < groups; cg += gridDim.x) {
        float acc[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll 1
        for (int c = 0; c < a.pieces; c += kLfAhead) {
#pragma unroll
            for (int j = 0; j < kLfAhead; ++j) {
                const uint4 u0 = buf[j][0], u1 = buf[j][1];
                if (c + j < a.pieces) {              // (the same in every warp)
                    const uint4 p = lf_shared(xl + (c + j) * 64), q = lf_shared(xl + 8 * a.row_bytes + (c + j) * 64);
                    const uint32_t a0[4] = {p.x, q.x, p.y, q.y}, a1[4] = {p.z, q.z, p.w, q.w};
                    mma_bf16(acc[0], a0, u0.x, u0.y);
                    mma_bf16(acc[1], a0, u1.x, u1.y);
                    mma_bf16(acc[0], a1, u0.z, u0.w);
                    mma_bf16(acc[1], a1, u1.z, u1.w);
                }
                fetch(j, buf[j]);
            }
            next();
        }
        // the group's sums: element (token, row) of all warps, in order
        float* mine = red[b][warp];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            float* at = mine + g * kLfRows + n * 8 + t * 2;
            at[0] = acc[n][0], at[1] = acc[n][1];
            at[8 * kLfRows] = acc[n][2], at[8 * kLfRows + 1] = acc[n][3];
        }
        __syncthreads();
        float s = 0.f;                   // (as many threads as sums)
#pragma unroll
        for (int w = 0; w < kLfWarps; ++w) s += red[b][w][tid];
        const int m = tid / kLfRows, n = cg * kLfRows + tid % kLfRows;
        if (m < a.M && n < a.N) a.y[(size_t)m * a.ldc + n] = s;
        b ^= 1;                          // (written again two barriers from here)
    }
}

static_assert(kLfThreads == kLfTok * kLfRows, "one sum per thread");

int lf_pieces(int K) { return ((K + 31) / 32 + kLfWarps - 1) / kLfWarps; }
size_t lf_smem(int K) { return (size_t)kLfWarps * kLfTok * ((lf_pieces(K) | 1) * 64); }
constexpr int kLfSmemMax = 224 * 1024 - (int)sizeof(float) * 2 * kLfWarps * kLfTok * kLfRows;

}  // namespace

// Matrices up to 64 MB: beyond, gemm.cu's stream covers its head and tail (32768 x 2048: 26.1 us there, 27.1 here; steps of three
// Rivetar layers of width 4096, 100 to 134 MB matrices here too: 1 token 388 and 398 us, with this line 383 and 381).  With a second
// tile of tokens (17 to 32) this form was 20 us a step slower.
bool linear_few_takes(const void* x, const void* w, int M, int N, int K) {
    if (M <= 0 || M > kLfTok || N <= 0 || K <= 0 || K % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15))
        return false;
    return (size_t)N * K <= (32u << 20) && lf_smem(K) <= (size_t)kLfSmemMax;
}

int launch_linear_few(const void* x, const void* w, float* y, int M, int N, int K, int ldc, cudaStream_t stream) {
    LfArgs a;
    a.x = static_cast<const __nv_bfloat16*>(x), a.w = static_cast<const __nv_bfloat16*>(w), a.y = y;
    a.M = M, a.N = N, a.K = K, a.ldc = ldc;
    a.pieces = lf_pieces(K);
    a.row_bytes = (a.pieces | 1) * 64;
    const size_t smem = lf_smem(K);
    static PerDeviceOnce once;
    ASD_ONCE(once, ASD_CUDA(cudaFuncSetAttribute(linear_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLfSmemMax)));
    const int groups = (N + kLfRows - 1) / kLfRows, per_sm = smem <= 96 * 1024 ? 2 : 1;
    ASD_CUDA(launch_pdl(linear_few_kernel, std::min(groups, per_sm * sm_count()), kLfThreads, smem, stream, a));
    ASD_CUDA(cudaGetLastError());
    count_kernel(KERNEL_LINEAR_FEW);
    return 0;
}

}  // namespace asd

#include "../../include/asd_b200.h"
extern "C" int asd_linear_bf16_few(const void* x, const void* w, void* out, int M, int N, int K, void* stream) {
    using namespace asd;
    if (!out || !linear_few_takes(x, w, M, N, K)) return set_error("asd_linear_bf16_few: shape or alignment outside the kernel's contract");
    return launch_linear_few(x, w, static_cast<float*>(out), M, N, K, N, static_cast<cudaStream_t>(stream));
}
