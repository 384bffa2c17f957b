// Residual-stream kernels that are not contractions: embedding with a hashed token-pair table, scalar-gain RMS norm,
// token shift with carried state, the close of a parallel layer with depth-weighted averaging, row selection.
// One CTA per token row; the residual stream, the norms and the carried state are fp32 whatever the engine's type.
#include <cuda_bf16.h>

#include <initializer_list>

#include "asd_internal.h"
#include "blocks.h"
#include "elem.cuh"
#include "ptx.cuh"

namespace asd {

namespace {

// the row above is this sequence's previous position
__device__ __forceinline__ bool follows(const SeqIndex& ix, int m) {
    return m > 0 && ix.token_slot[m - 1] == ix.token_slot[m] && ix.positions[m - 1] == ix.positions[m] - 1;
}
// row m is one of the last `ring` rows of its run of consecutive positions: no later row of the batch lands on the
// same ring entry
__device__ __forceinline__ bool owns_ring_entry(const SeqIndex& ix, int m, int ring) {
    const int o = m + ring;
    return !(o < ix.M && ix.token_slot[o] == ix.token_slot[m] && ix.positions[o] == ix.positions[m] + ring);
}

__global__ void embed_pair_kernel(SeqIndex ix, const void* embed, const void* table, int wf32, int buckets, int mul_prev,
                                  int mul_cur, const int* tok_ring, int ring, float* x0, const void* g, float eps,
                                  float* hn, int D) {
    pdl_enter();
    __shared__ float red[33];
    const int m = blockIdx.x;
    const int tok = ix.tokens[m], pos = ix.positions[m], slot = ix.token_slot[m];
    long long row;
    if (pos == 0) {
        row = buckets;
    } else {
        const int prev = follows(ix, m) ? ix.tokens[m - 1] : tok_ring[(long long)slot * ring + (pos - 1) % ring];
        row = (long long)(((unsigned long long)prev * (unsigned long long)mul_prev +
                           (unsigned long long)tok * (unsigned long long)mul_cur) % (unsigned long long)buckets);
    }
    float ss = 0.f;
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
        const float v = ldx(embed, (long long)tok * D + d, wf32) + ldx(table, row * D + d, wf32);
        x0[(long long)m * D + d] = v;
        ss += v * v;
    }
    ss = block_sum(ss, red);
    const float r = ldx(g, 0, wf32) / sqrtf(ss / (float)D + eps);
    for (int d = threadIdx.x; d < D; d += blockDim.x) hn[(long long)m * D + d] = x0[(long long)m * D + d] * r;
}

// The row kernels below keep NV groups of four elements per thread in registers: a row's loads are on their way together and its
// sum costs one barrier.  The split depends on the width alone, so that a row's sums do not depend on the batch.
// 4096 rows of 2048, 100 MB: 33 -> 20 us.
template <int NV>
__global__ void __launch_bounds__(1024) embed_pair_regs_kernel(SeqIndex ix, const void* embed, const void* table, int wf32,
                                                               int buckets, int mul_prev, int mul_cur, const int* tok_ring,
                                                               int ring, float* x0, const void* g, float eps, float* hn, int D) {
    pdl_enter();
    __shared__ float red[32];
    const int m = blockIdx.x;
    const int tok = ix.tokens[m], pos = ix.positions[m], slot = ix.token_slot[m];
    float v[NV][4], ss[1] = {0.f};
    auto place = [&](int j) { return (j * (int)blockDim.x + (int)threadIdx.x) * 4; };
#pragma unroll
    for (int j = 0; j < NV; ++j)
        if (place(j) < D) ldx4(embed, (long long)tok * D + place(j), wf32, v[j]);
    long long row;
    if (pos == 0) {
        row = buckets;
    } else {
        const int prev = follows(ix, m) ? ix.tokens[m - 1] : tok_ring[(long long)slot * ring + (pos - 1) % ring];
        row = (long long)(((unsigned long long)prev * (unsigned long long)mul_prev +
                           (unsigned long long)tok * (unsigned long long)mul_cur) % (unsigned long long)buckets);
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        if (place(j) >= D) continue;
        float t[4];
        ldx4(table, row * D + place(j), wf32, t);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v[j][e] += t[e];
            ss[0] += v[j][e] * v[j][e];
        }
        stx4(x0, (long long)m * D + place(j), 1, v[j]);
    }
    const float gain = ldx(g, 0, wf32);
    block_sums<1>(ss, red);
    const float r = gain / sqrtf(ss[0] / (float)D + eps);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        if (place(j) >= D) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e) v[j][e] *= r;
        stx4(hn, (long long)m * D + place(j), 1, v[j]);
    }
}

__global__ void commit_tokens_kernel(SeqIndex ix, int* tok_ring, int ring) {
    pdl_enter();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= ix.M || !owns_ring_entry(ix, m, ring)) return;
    tok_ring[(long long)ix.token_slot[m] * ring + ix.positions[m] % ring] = ix.tokens[m];
}

__global__ void token_shift_kernel(SeqIndex ix, const float* hn, const float* state, int ring, const void* mu, int wf32,
                                   void* h, void* hs, int of32, int D) {
    pdl_enter();
    const int m = blockIdx.x;
    const int pos = ix.positions[m];
    const float* prev = nullptr;
    if (pos > 0)
        prev = follows(ix, m) ? hn + (long long)(m - 1) * D
                              : state + ((long long)ix.token_slot[m] * ring + (pos - 1) % ring) * D;
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
        const float v = hn[(long long)m * D + d];
        const float p = prev ? prev[d] : 0.f;
        stx(h, (long long)m * D + d, of32, v);
        stx(hs, (long long)m * D + d, of32, v + (p - v) * ldx(mu, d, wf32));
    }
}

// 4096 rows of 2048: 27 -> 19.5 us for 67 MB
__global__ void token_shift4_kernel(SeqIndex ix, const float* hn, const float* state, int ring, const void* mu, int wf32,
                                    void* h, void* hs, int of32, int D) {
    pdl_enter();
    const int m = blockIdx.y, d = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (d >= D) return;
    const long long at = (long long)m * D + d;
    float v[4], p[4] = {0.f, 0.f, 0.f, 0.f}, w[4];
    ldx4(hn, at, 1, v);
    ldx4(mu, d, wf32, w);
    const int pos = ix.positions[m];
    if (pos > 0) {
        if (follows(ix, m))
            ldx4(hn, at - D, 1, p);
        else
            ldx4(state, ((long long)ix.token_slot[m] * ring + (pos - 1) % ring) * D + d, 1, p);
    }
    stx4(h, at, of32, v);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = v[e] + (p[e] - v[e]) * w[e];
    stx4(hs, at, of32, v);
}

__global__ void commit_shift_kernel(SeqIndex ix, const float* hn, float* state, int ring, int D) {
    pdl_enter();
    const int m = blockIdx.x;
    if (!owns_ring_entry(ix, m, ring)) return;
    float* dst = state + ((long long)ix.token_slot[m] * ring + ix.positions[m] % ring) * D;
    for (int d = threadIdx.x; d < D; d += blockDim.x) dst[d] = hn[(long long)m * D + d];
}

__global__ void layer_close_kernel(LayerClose L, SeqIndex ix) {
    pdl_enter();
    __shared__ float red[33];
    const int m = blockIdx.x, D = L.D;
    const long long base = (long long)m * D;
    if (L.state_ring && owns_ring_entry(ix, m, L.ring)) {
        float* dst = L.state_ring + ((long long)ix.token_slot[m] * L.ring + ix.positions[m] % L.ring) * D;
        for (int d = threadIdx.x; d < D; d += blockDim.x) dst[d] = L.hn[base + d];
    }
    float* xnew = L.stack + (size_t)(L.layer + 1) * L.stack_stride + base;
    float ss = 0.f;
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
        float y = L.mix[base + d];
        if (L.top > 0) {
            float f = 0.f;
            for (int k = 0; k < L.top; ++k)
                f += L.gate[(long long)m * L.top + k] * L.expert_out[(long long)L.slot_of[(long long)m * L.top + k] * D + d];
            y += f;
        }
        const float xn = L.x_in[base + d] + y;
        xnew[d] = xn;
        float a = 0.f;
        for (int j = 0; j <= L.layer; ++j) a += ldx(L.coeff, j, L.wf32) * L.stack[(size_t)j * L.stack_stride + base + d];
        a += ldx(L.coeff, L.layer + 1, L.wf32) * xn;
        L.x_next[base + d] = a;
        ss += a * a;
    }
    ss = block_sum(ss, red);
    const float r = ldx(L.g_next, 0, L.wf32) / sqrtf(ss / (float)D + L.eps);
    for (int d = threadIdx.x; d < D; d += blockDim.x) L.hn[base + d] = L.x_next[base + d] * r;
}

// 4096 rows of 2048, two experts each, 300 MB: 85 -> 42 us (the step of 64 rows of 4096, all its
// row kernels together: 442 -> 405).  The bound of 1024 threads caps the registers at 64 and spills 48 bytes with four groups: bound to
// the 512 threads of rows up to 8192 it has 74 and fewer blocks an SM, 4096 rows of 4096 82 -> 100 us, of 8192 165 -> 255.
template <int NV>
__global__ void __launch_bounds__(1024) layer_close_regs_kernel(LayerClose L, SeqIndex ix) {
    pdl_enter();
    __shared__ float red[32];
    const int m = blockIdx.x, D = L.D;
    const long long base = (long long)m * D;
    auto place = [&](int j) { return (j * (int)blockDim.x + (int)threadIdx.x) * 4; };
    float y[NV][4], x[NV][4], t[NV][4];
    auto load = [&](const float* p, float (&r)[NV][4]) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            r[j][0] = r[j][1] = r[j][2] = r[j][3] = 0.f;
            if (place(j) < D) ldx4(p, place(j), 1, r[j]);
        }
    };
    auto store = [&](float* p, const float (&r)[NV][4]) {
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (place(j) < D) stx4(p, place(j), 1, r[j]);
    };
    load(L.mix + base, y);
    load(L.x_in + base, x);
    if (L.state_ring && owns_ring_entry(ix, m, L.ring)) {
        load(L.hn + base, t);
        store(L.state_ring + ((long long)ix.token_slot[m] * L.ring + ix.positions[m] % L.ring) * D, t);
    }
    if (L.top > 0) {
        float f[NV][4];
#pragma unroll
        for (int j = 0; j < NV; ++j) f[j][0] = f[j][1] = f[j][2] = f[j][3] = 0.f;
        for (int k = 0; k < L.top; ++k) {
            const float g = L.gate[(long long)m * L.top + k];
            load(L.expert_out + (long long)L.slot_of[(long long)m * L.top + k] * D, t);
#pragma unroll
            for (int j = 0; j < NV; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) f[j][e] += g * t[j][e];
        }
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) y[j][e] += f[j][e];
    }
    // y: the new residual, then its depth-weighted sum with the earlier ones
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[j][e] += x[j][e];
    store(L.stack + (size_t)(L.layer + 1) * L.stack_stride + base, y);
    float a[NV][4];
#pragma unroll
    for (int j = 0; j < NV; ++j) a[j][0] = a[j][1] = a[j][2] = a[j][3] = 0.f;
    for (int l = 0; l <= L.layer; ++l) {
        const float c = ldx(L.coeff, l, L.wf32);
        load(L.stack + (size_t)l * L.stack_stride + base, t);
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) a[j][e] += c * t[j][e];
    }
    const float c = ldx(L.coeff, L.layer + 1, L.wf32), gain = ldx(L.g_next, 0, L.wf32);
    float ss[1] = {0.f};
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            a[j][e] += c * y[j][e];
            ss[0] += a[j][e] * a[j][e];       // places beyond the row hold zeros
        }
    store(L.x_next + base, a);
    block_sums<1>(ss, red);
    const float r = gain / sqrtf(ss[0] / (float)D + L.eps);
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[j][e] *= r;
    store(L.hn + base, a);
}

__global__ void select_rows4_kernel(const float* src, const int* rows, void* dst, int of32, int D) {
    pdl_enter();
    const int r = blockIdx.y, d = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (d >= D) return;
    float v[4];
    ldx4(src, (long long)(rows ? rows[r] : r) * D + d, 1, v);
    stx4(dst, (long long)r * D + d, of32, v);
}

__global__ void select_rows_kernel(const float* src, const int* rows, void* dst, int of32, int D) {
    pdl_enter();
    const int r = blockIdx.x;
    const long long s = (long long)(rows ? rows[r] : r) * D;
    for (int d = threadIdx.x; d < D; d += blockDim.x) stx(dst, (long long)r * D + d, of32, src[s + d]);
}

inline bool in_regs(int D) { return D % 4 == 0 && D <= 16384; }
// about 256 threads a row
#define ASD_REG_LAUNCH(kernel, D, rows, ...)                                                       \
    {                                                                                              \
        const int nv = (D) <= 1024 ? 1 : ((D) <= 2048 ? 2 : 4);                                    \
        auto fn = nv == 1 ? kernel<1> : (nv == 2 ? kernel<2> : kernel<4>);                         \
        ASD_CUDA(launch_pdl(fn, rows, ((D) / 4 + nv * 32 - 1) / (nv * 32) * 32, 0, stream, __VA_ARGS__)); \
    }
inline bool aligned16(std::initializer_list<const void*> ps) {
    uintptr_t at = 0;
    for (const void* p : ps) at |= reinterpret_cast<uintptr_t>(p);
    return (at & 15) == 0;
}
inline int row_threads(int D) { return D >= 1024 ? 256 : (D >= 256 ? 128 : 64); }

}  // namespace

int launch_embed_pair(const SeqIndex& ix, const void* embed, const void* pair_table, int wf32, int buckets, int mul_prev,
                      int mul_cur, const int* tok_ring, int ring, float* x0, const void* g, float eps, float* hn, int D,
                      cudaStream_t stream) {
    if (ix.M <= 0) return 0;
    if (buckets <= 0 || ring <= 0) return set_error("embed_pair: buckets and ring must be positive");
    if (in_regs(D) && aligned16({embed, pair_table, x0, hn}))
        ASD_REG_LAUNCH(embed_pair_regs_kernel, D, ix.M, ix, embed, pair_table, wf32, buckets, mul_prev, mul_cur, tok_ring, ring, x0, g,
                       eps, hn, D)
    else
        ASD_CUDA(launch_pdl(embed_pair_kernel, ix.M, row_threads(D), 0, stream, ix, embed, pair_table, wf32, buckets,
                            mul_prev, mul_cur, tok_ring, ring, x0, g, eps, hn, D));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

int launch_commit_tokens(const SeqIndex& ix, int* tok_ring, int ring, cudaStream_t stream) {
    if (ix.M <= 0) return 0;
    ASD_CUDA(launch_pdl(commit_tokens_kernel, (ix.M + 127) / 128, 128, 0, stream, ix, tok_ring, ring));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

int launch_token_shift(const SeqIndex& ix, const float* hn, const float* state_ring, int ring, const void* mu, int wf32,
                       void* h, void* hs, int of32, int D, cudaStream_t stream) {
    if (ix.M <= 0) return 0;
    if (D % 4 == 0 && ix.M <= 65535 && aligned16({hn, state_ring, mu, h, hs}))
        ASD_CUDA(launch_pdl(token_shift4_kernel, dim3((D / 4 + 127) / 128, ix.M), 128, 0, stream, ix, hn, state_ring, ring, mu, wf32,
                            h, hs, of32, D));
    else
        ASD_CUDA(launch_pdl(token_shift_kernel, ix.M, row_threads(D), 0, stream, ix, hn, state_ring, ring, mu, wf32, h, hs,
                            of32, D));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

int launch_commit_shift_state(const SeqIndex& ix, const float* hn, float* state_ring, int ring, int D,
                              cudaStream_t stream) {
    if (ix.M <= 0) return 0;
    ASD_CUDA(launch_pdl(commit_shift_kernel, ix.M, row_threads(D), 0, stream, ix, hn, state_ring, ring, D));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

int launch_layer_close(const LayerClose& L, cudaStream_t stream) {
    if (L.M <= 0) return 0;
    if (L.state_ring && (!L.ix || L.ring <= 0)) return set_error("layer_close: the carried state needs the batch index and a ring");
    const SeqIndex ix = L.ix ? *L.ix : SeqIndex{nullptr, nullptr, nullptr, 0};
    if (in_regs(L.D) && L.stack_stride % 4 == 0 &&
        aligned16({L.mix, L.x_in, L.hn, L.state_ring, L.expert_out, L.stack, L.x_next}))
        ASD_REG_LAUNCH(layer_close_regs_kernel, L.D, L.M, L, ix)
    else
        ASD_CUDA(launch_pdl(layer_close_kernel, L.M, row_threads(L.D), 0, stream, L, ix));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

int launch_select_rows(const float* src, const int* rows, void* dst, int of32, int n, int D, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (D % 4 == 0 && n <= 65535 && aligned16({src, dst}))
        ASD_CUDA(launch_pdl(select_rows4_kernel, dim3((D / 4 + 127) / 128, n), 128, 0, stream, src, rows, dst, of32, D));
    else
        ASD_CUDA(launch_pdl(select_rows_kernel, n, row_threads(D), 0, stream, src, rows, dst, of32, D));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace asd
