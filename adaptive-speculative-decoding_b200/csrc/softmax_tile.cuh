// Pieces of the tcgen05 attention kernels whose thread = query row = TMEM lane takes a tile of 128 scores through the softmax:
// window_attention_tc.cu and latent_prompt_tc.cu.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace asd {

constexpr int kStSlot = 128 * 128;         // bytes of 128 rows x 64 bf16

// MN-major SW128 operand (keys along rows of 128 B = 64 columns, 8-key atoms 1024 B apart, the next 64 columns a slot further)
__device__ __forceinline__ uint64_t st_desc_mn(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(kStSlot >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ float st_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// element i of a tile is visible to a row iff i <= hi and (i >= lo or i < kept): as bits of 32 elements from i0 on, so that a test
// of one costs an instruction (as comparisons the compiler branched on every element: 14000 to 29000 clocks a tile)
struct StSeen {
    int lo, hi, kept;
    __device__ __forceinline__ static uint32_t below(int n) {          // bits 0 .. n - 1
        return n <= 0 ? 0u : (n >= 32 ? 0xffffffffu : (1u << n) - 1u);
    }
    __device__ __forceinline__ uint32_t bits(int i0) const { return below(hi + 1 - i0) & (~below(lo - i0) | below(kept - i0)); }
};
// weights of 32 scores -> 16 packed pairs of their high terms and 16 of what is left
template <bool MASKED>
__device__ __forceinline__ void st_weights(const uint32_t (&v)[32], uint32_t seen, float scale, float nref,
                                           uint32_t (&ph)[16], uint32_t (&pl)[16], float (&sum)[4]) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        float p0 = st_ex2(fmaf(__uint_as_float(v[i]), scale, nref));
        float p1 = st_ex2(fmaf(__uint_as_float(v[i + 1]), scale, nref));
        if (MASKED) {
            p0 = seen & (1u << i) ? p0 : 0.0f;
            p1 = seen & (2u << i) ? p1 : 0.0f;
        }
        sum[(i >> 1) & 3] += p0 + p1;
        const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
        const float2 f = __bfloat1622float2(h);
        const __nv_bfloat162 r = __floats2bfloat162_rn(p0 - f.x, p1 - f.y);
        ph[i >> 1] = *reinterpret_cast<const uint32_t*>(&h);
        pl[i >> 1] = *reinterpret_cast<const uint32_t*>(&r);
    }
}

}  // namespace asd
