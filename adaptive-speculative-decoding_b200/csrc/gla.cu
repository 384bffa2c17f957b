// Gated linear attention: a recurrence with a [dk][dv] state per head and a decay per key channel,
//   S_t = diag(alpha_t) S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t,   alpha_t = sigmoid(z_t)^(1 / tau).
// gla_decay_kernel:  alpha from the inner decay projection (a thread has 1 or 4 channels of 8 tokens, fp32).
// gla_recurrence_kernel: one CTA per (sequence, head, 32 value columns, or 16).  Columns of S never mix, so a CTA owns its
//   columns for the whole run of new positions: a thread keeps 8 key rows x 4 columns of the state in registers.  The
//   new positions are staged CH at a time in shared memory (q, k, decay rows and the CTA's value columns) by
//   cp.async, one chunk ahead; per position every thread updates its part and forms its rows' share of o, and after the
//   chunk the shares are added in index order.  The arithmetic per position is the same whatever the chunking or the
//   batch, so a sequence's outputs do not depend on how its tokens were cut into forwards.
//   The state lives in fp32 [slot][ring][head][dk][dv]; entry p % ring is the state after position p.
// gla_out_kernel: RMS norm of every head's o over dv (plain weight), times silu(gate).
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "asd_internal.h"
#include "blocks.h"
#include "elem.cuh"
#include "ptx.cuh"

namespace asd {

namespace {

constexpr int GLA_R = 8;     // key rows of the state per thread
constexpr int GLA_C = 4;     // and columns

__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid) {
    const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
    const int sz = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(addr), "l"(src), "r"(sz) : "memory");
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid) {
    const unsigned addr = (unsigned)__cvta_generic_to_shared(dst);
    const int sz = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(addr), "l"(src), "r"(sz) : "memory");
}

constexpr int GD_TOK = 32, GD_LANES = 64, GD_THREADS = 256;   // per CTA of the decay kernel: tokens, channel lanes, threads

// One CTA = 64 * CPT channels x 32 tokens: the channels' projection rows are staged transposed, [low][channels] with an odd
// row length (the stores of a warp, which go down a column, then meet 32 banks; with 256 floats a row they met one and the
// staging alone took a third of the kernel); a thread has CPT channels 64 apart and 8 tokens, so that a staged value feeds CPT
// or 8 products.  2151 tokens x 2048 channels, 32 inner: 53 -> 36 us (what is left is log1p, exp and expm1 of
// every element); 16 tokens: 18 -> 7 us (CPT 1: more CTAs).
template <int CPT>
__global__ void __launch_bounds__(GD_THREADS) gla_decay_kernel(const float* a, long long lda, const float* w_decay,
                                                          const float* b_decay, GlaDims d, float* alpha, int M) {
    pdl_enter();
    extern __shared__ float sm[];
    constexpr int CH = GD_LANES * CPT, ST = CH + 1, TT = GD_TOK / (GD_THREADS / GD_LANES);
    float* wT = sm;                      // [low][ST]
    float* av = sm + d.low * ST;         // [GD_TOK][low]
    const int n = d.heads * d.dk;
    const int c0 = blockIdx.x * CH, m0 = blockIdx.y * GD_TOK;
    const int nt = min(GD_TOK, M - m0);
    // eight loads on their way at a time; (outer, inner) of consecutive places GD_THREADS apart without a division each
    auto stage = [&](int total, auto load, auto store) {
        const int d_out = GD_THREADS / d.low, d_in = GD_THREADS - d_out * d.low;
        int out = threadIdx.x / d.low, in = threadIdx.x - out * d.low;
        for (int i = threadIdx.x; i < total; i += 8 * GD_THREADS) {
            float x[8];
            int o = out, r = in;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                x[j] = i + j * GD_THREADS < total ? load(o, r) : 0.f;
                o += d_out, r += d_in;
                if (r >= d.low) r -= d.low, ++o;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (i + j * GD_THREADS < total) store(out, in, x[j]);
                out += d_out, in += d_in;
                if (in >= d.low) in -= d.low, ++out;
            }
        }
    };
    stage(CH * d.low, [&](int c, int r) { return c0 + c < n ? w_decay[(long long)(c0 + c) * d.low + r] : 0.f; },
          [&](int c, int r, float x) { wT[r * ST + c] = x; });
    stage(GD_TOK * d.low, [&](int t, int r) { return t < nt ? a[(long long)(m0 + t) * lda + r] : 0.f; },
          [&](int t, int r, float x) { av[t * d.low + r] = x; });
    __syncthreads();
    const int lane = threadIdx.x & (GD_LANES - 1), first = threadIdx.x / GD_LANES * TT;
    float z[CPT][TT];
#pragma unroll
    for (int i = 0; i < CPT; ++i)
#pragma unroll
        for (int t = 0; t < TT; ++t) z[i][t] = 0.f;
    for (int r = 0; r < d.low; ++r) {
        float w[CPT];
#pragma unroll
        for (int i = 0; i < CPT; ++i) w[i] = wT[r * ST + i * GD_LANES + lane];
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            const float x = av[(first + t) * d.low + r];
#pragma unroll
            for (int i = 0; i < CPT; ++i) z[i][t] = fmaf(w[i], x, z[i][t]);
        }
    }
    const float inv_tau = 1.f / d.tau;
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
        const int c = c0 + i * GD_LANES + lane;
        const float bias = c < n ? b_decay[c] : 0.f;
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            if (c < n && first + t < nt) {
                const float zz = z[i][t] + bias;
                // log sigmoid(z) = min(z, 0) - log1p(exp(-|z|)).  A slow decay lies just below 1, where expf's two units in
                // the last place are a relative error of 1e-7 that hundreds of steps multiply; 1 + expm1 is rounded once
                const float ls = fminf(zz, 0.f) - log1pf(expf(-fabsf(zz)));
                alpha[(long long)(m0 + first + t) * n + c] = 1.f + expm1f(ls * inv_tau);
            }
        }
    }
}

struct Staged {                         // one position's values for a thread: its key rows in pairs, its columns
    float2 a[GLA_R / 2], k[GLA_R / 2], q[GLA_R / 2];
    float v[GLA_C];
};

// What bounds it: three fp32 operations per state element and position, and the staged values' way from shared memory into
// registers (128 bytes a clock and SM, broadcast or not).  With one column and 16 rows per thread (the form before) a position
// brought 12 bytes per element into registers, 780 clocks on an SM with two CTAs; with 8 rows x 4 columns it is 3.5, below the
// arithmetic, which runs on packed pairs of rows.  3 prompts of up to 777 positions, 16 heads of 128 x 128: 321 -> 174 us
// (436 clocks a position where an SM has two of the 192 CTAs, 245 where it has one; fp32 pipe 0.54 busy on the former).
// Rows beyond dk are staged as zeros and take no k v^T (an infinite v times zero would be NaN): they add nothing.  A thread that has
// nothing but such rows does what its warp does, and nobody reads its share: had it a loop of its own, a warp of key size 16 or 24
// would walk every position twice (2 sequences of 500, 4 heads of 24 x 40: 162 us so, now 101).  `vec`: sizes and addresses allow
// 16-byte copies.  MAXT: threads at most (COLS / 4 per 8 key rows); PIPE: loads a position ahead.
template <int MAXT, int MINB, bool PIPE, int COLS = 32>
__global__ void __launch_bounds__(MAXT, MINB) gla_recurrence_kernel(SeqIndex ix, const int* cu_q, const int* seq_slot, const float* q,
                                                              const float* k, const float* v, long long ld, const float* alpha,
                                                              GlaDims d, float* state, int ring, float* out, int CH, int vec) {
    pdl_enter();
    constexpr int CG = COLS / GLA_C;                    // column groups
    extern __shared__ __align__(16) float sm[];
    const int seq = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * COLS;
    const int t0 = cu_q[seq], t1 = cu_q[seq + 1];
    if (t0 >= t1) return;
    const int tid = threadIdx.x, nthr = blockDim.x, RG = nthr / CG;
    const int dkp = RG * GLA_R;                         // padded key size
    const int rg = tid / CG, r0 = rg * GLA_R, ca = tid % CG * GLA_C;   // the thread's rows and columns
    const int live = (d.dk + GLA_R - 1) / GLA_R;        // row groups that hold a row; what the others compute is used by nobody
    // no thread of the warp has rows on both sides of dk
    const bool whole = __all_sync(0xffffffffu, r0 + GLA_R <= d.dk || r0 >= d.dk);
    const int slot = seq_slot[seq];
    const int p0 = ix.positions[t0];
    // shared: two buffers of { q, k, decay [CH][dkp] each, v [CH][COLS] }, then the shares of o [RG][CH][COLS]
    const int buf_elems = 3 * CH * dkp + CH * COLS, share = CH * COLS;
    float* part = sm + 2 * buf_elems;
    const long long st_entry = (long long)d.heads * d.dk * d.dv;
    float* st_cta = state + (long long)slot * ring * st_entry + (long long)head * d.dk * d.dv + col0;
    float2 S[GLA_R / 2][GLA_C];                         // [pair of rows][column]
    auto copy_state = [&](float* entry, bool store) {
#pragma unroll
        for (int p = 0; p < GLA_R / 2; ++p)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + 2 * p + h;
                if (r >= d.dk) continue;
                float* at = entry + (long long)r * d.dv + ca;
                float x[GLA_C];
#pragma unroll
                for (int e = 0; e < GLA_C; ++e) x[e] = h ? S[p][e].y : S[p][e].x;
                if (vec) {
                    if (col0 + ca < d.dv) {
                        if (store)
                            *reinterpret_cast<float4*>(at) = make_float4(x[0], x[1], x[2], x[3]);
                        else
                            *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(at);
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < GLA_C; ++e)
                        if (col0 + ca + e < d.dv) {
                            if (store)
                                at[e] = x[e];
                            else
                                x[e] = at[e];
                        }
                }
                if (!store) {
#pragma unroll
                    for (int e = 0; e < GLA_C; ++e) {
                        if (h)
                            S[p][e].y = x[e];
                        else
                            S[p][e].x = x[e];
                    }
                }
            }
    };
#pragma unroll
    for (int p = 0; p < GLA_R / 2; ++p)
#pragma unroll
        for (int c = 0; c < GLA_C; ++c) S[p][c] = make_float2(0.f, 0.f);
    const int hq = head * d.dk, hv = head * d.dv;
    const int n_alpha = d.heads * d.dk;
    // W floats per copy, one chunk ahead of the arithmetic; a thread has the same places of every position
    auto fetch_w = [&](int buf, int c0, auto width) {
        constexpr int W = decltype(width)::value;
        const int nt = min(CH, t1 - c0), per = dkp / W;
        for (int i = tid; i < 3 * per + COLS / W; i += nthr) {
            const int arr = i >= 2 * per ? (i >= 3 * per ? 3 : 2) : (i >= per ? 1 : 0);
            const int c = (i - arr * per) * W;
            const bool ok = arr == 3 ? col0 + c < d.dv : c < d.dk;
            const long long step = arr == 2 ? n_alpha : ld;
            const float* src = arr == 0 ? q : (arr == 1 ? k : (arr == 2 ? alpha : v));
            if (ok) src += c0 * step + (arr == 3 ? hv + col0 + c : hq + c);
            const int width_s = arr == 3 ? COLS : dkp;
            float* dst = sm + buf * buf_elems + arr * CH * dkp + c;
            for (int t = 0; t < nt; ++t) {              // places beyond the chunk's positions are never read
                if constexpr (W == 4)
                    cp_async16(dst, src, ok);
                else
                    cp_async4(dst, src, ok);
                dst += width_s;
                if (ok) src += step;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto fetch = [&](int buf, int c0) {
        if (vec)
            fetch_w(buf, c0, std::integral_constant<int, 4>{});
        else
            fetch_w(buf, c0, std::integral_constant<int, 1>{});
    };
    fetch(0, t0);
    if (p0 > 0) copy_state(st_cta + (long long)((p0 - 1) % ring) * st_entry, false);
    int it = 0;
    for (int c0 = t0; c0 < t1; c0 += CH, ++it) {
        const int nt = min(CH, t1 - c0);
        if (c0 + CH < t1) {
            fetch((it + 1) & 1, c0 + CH);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();   // this chunk's rows have landed for every thread; the previous shares have been read
        const float* qs = sm + (it & 1) * buf_elems + r0;
        const float* vs = sm + (it & 1) * buf_elems + 3 * CH * dkp;
        float* ps = part + rg * share;
        auto load = [&](int t, Staged& x) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                *reinterpret_cast<float4*>(&x.a[2 * i]) = *reinterpret_cast<const float4*>(qs + 2 * CH * dkp + t * dkp + 4 * i);
                *reinterpret_cast<float4*>(&x.k[2 * i]) = *reinterpret_cast<const float4*>(qs + CH * dkp + t * dkp + 4 * i);
                *reinterpret_cast<float4*>(&x.q[2 * i]) = *reinterpret_cast<const float4*>(qs + t * dkp + 4 * i);
            }
            *reinterpret_cast<float4*>(x.v) = *reinterpret_cast<const float4*>(vs + t * COLS + ca);
        };
        auto position = [&](int t, const Staged& x, auto beyond) {
            float o[GLA_C];
#pragma unroll
            for (int c = 0; c < GLA_C; ++c) {
                const float2 vc = make_float2(x.v[c], x.v[c]);
                float2 s = make_float2(0.f, 0.f);
#pragma unroll
                for (int p = 0; p < GLA_R / 2; ++p) {
                    float2 kv = mul2(x.k[p], vc);
                    if constexpr (decltype(beyond)::value) {
                        if (r0 + 2 * p >= d.dk) kv.x = 0.f;
                        if (r0 + 2 * p + 1 >= d.dk) kv.y = 0.f;
                    }
                    S[p][c] = fma2(x.a[p], S[p][c], kv);
                    s = p ? fma2(S[p][c], x.q[p], s) : mul2(S[p][c], x.q[p]);
                }
                o[c] = s.x + s.y;
            }
            *reinterpret_cast<float4*>(ps + t * COLS + ca) = make_float4(o[0], o[1], o[2], o[3]);
        };
        // the last `ring` new positions leave their state behind
        const int quiet = min(nt, max(0, t1 - ring - c0));
        int t = 0;
        auto run = [&](auto beyond) {
            if constexpr (PIPE) {
                // the next position's values are on their way while this one's are used (one past the last reads what is there, in
                // bounds, for nothing); a share's store would otherwise hold its loads back
                if (quiet <= 0) return;
                Staged x0, x1;
                load(0, x0);
                for (; t + 1 < quiet; t += 2) {
                    load(t + 1, x1);
                    position(t, x0, beyond);
                    load(t + 2, x0);
                    position(t + 1, x1, beyond);
                }
                if (t < quiet) position(t++, x0, beyond);
            } else {
#pragma unroll 1
                for (; t < quiet; ++t) {
                    Staged x;
                    load(t, x);
                    position(t, x, beyond);
                }
            }
        };
        if (whole)
            run(std::false_type{});
        else
            run(std::true_type{});
#pragma unroll 1
        for (; t < nt; ++t) {
            Staged x;
            load(t, x);
            position(t, x, std::true_type{});
            if (t >= quiet) copy_state(st_cta + (long long)((p0 + (c0 + t - t0)) % ring) * st_entry, true);
        }
        __syncthreads();   // the chunk is consumed (its buffer may be refilled) and the shares are complete
        for (int i = tid; i < nt * CG; i += nthr) {
            const int tt = i / CG, c = i % CG * GLA_C;
            if (col0 + c >= d.dv) continue;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int w = 0; w < live; ++w) {
                const float4 x = *reinterpret_cast<const float4*>(part + w * share + tt * COLS + c);
                o.x += x.x, o.y += x.y, o.z += x.z, o.w += x.w;
            }
            o.x *= d.q_scale, o.y *= d.q_scale, o.z *= d.q_scale, o.w *= d.q_scale;
            float* dst = out + (long long)(c0 + tt) * d.heads * d.dv + hv + col0 + c;
            if (vec) {
                *reinterpret_cast<float4*>(dst) = o;
            } else {
                dst[0] = o.x;
                if (col0 + c + 1 < d.dv) dst[1] = o.y;
                if (col0 + c + 2 < d.dv) dst[2] = o.z;
                if (col0 + c + 3 < d.dv) dst[3] = o.w;
            }
        }
    }
}

// one warp per (token, head); a lane keeps its values between the sum and the result: VN groups of four (dv <= 128 * VN, sizes
// and addresses allow 16-byte accesses), or VN = 0: any size, read twice.  2151 tokens, 16 heads of 128: 22 -> 12.5 us.
template <int VN>
__global__ void gla_out_kernel(const float* o, const float* gate, long long ldg, const float* w, float eps, void* y,
                               int of32, long long pairs, int heads, int dv) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const long long i0 = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i0 >= pairs) return;
    const long long m = i0 / heads;
    const float* src = o + i0 * dv;
    const float* g = gate + m * ldg + (i0 - m * heads) * dv;
    float ss = 0.f;
    if constexpr (VN > 0) {
        float x[VN][4], gv[VN][4];
#pragma unroll
        for (int j = 0; j < VN; ++j) {
            const int i = (j * 32 + lane) * 4;
            if (i >= dv) break;
            ldx4(src, i, 1, x[j]);
            ldx4(g, i, 1, gv[j]);
#pragma unroll
            for (int e = 0; e < 4; ++e) ss += x[j][e] * x[j][e];
        }
        ss = warp_sum(ss);
        const float r = 1.f / sqrtf(ss / (float)dv + eps);
#pragma unroll
        for (int j = 0; j < VN; ++j) {
            const int i = (j * 32 + lane) * 4;
            if (i >= dv) break;
            float wv[4];
            ldx4(w, i, 1, wv);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[j][e] = x[j][e] * r * wv[e] * (gv[j][e] / (1.f + expf(-gv[j][e])));
            stx4(y, i0 * dv + i, of32, x[j]);
        }
    } else {
        for (int i = lane; i < dv; i += 32) ss += src[i] * src[i];
        ss = warp_sum(ss);
        const float r = 1.f / sqrtf(ss / (float)dv + eps);
        for (int i = lane; i < dv; i += 32) {
            const float gv = g[i];
            stx(y, i0 * dv + i, of32, src[i] * r * w[i] * (gv / (1.f + expf(-gv))));
        }
    }
}

}  // namespace

int launch_gla_decay(const float* a, long long lda, const float* w_decay, const float* b_decay, const GlaDims& d,
                     float* alpha, int M, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (d.low <= 0 || !(d.tau > 0.f)) return set_error("gla: decay projection of size %d, tau %f", d.low, d.tau);
    if ((size_t)d.low * (256 + GD_TOK) * sizeof(float) > 200 * 1024)
        return set_error("gla: decay projection of size %d does not fit shared memory", d.low);
    const int n = d.heads * d.dk, tiles = (M + GD_TOK - 1) / GD_TOK;
    if (tiles > 65535) return set_error("gla: too many tokens");
    // four channels a thread where that still gives every SM a CTA
    const int cpt = (n + 4 * GD_LANES - 1) / (4 * GD_LANES) * tiles >= sm_count() ? 4 : 1;
    const size_t smem = ((size_t)d.low * (GD_LANES * cpt + 1) + (size_t)d.low * GD_TOK) * sizeof(float);
    static PerDeviceOnce once;
    ASD_ONCE(once, {
        ASD_CUDA(cudaFuncSetAttribute(gla_decay_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
        ASD_CUDA(cudaFuncSetAttribute(gla_decay_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    });
    const dim3 grid((n + GD_LANES * cpt - 1) / (GD_LANES * cpt), tiles);
    ASD_CUDA(launch_pdl(cpt == 4 ? gla_decay_kernel<4> : gla_decay_kernel<1>, grid, GD_THREADS, smem, stream, a, lda, w_decay,
                        b_decay, d, alpha, M));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

int launch_gla_recurrence(const SeqIndex& ix, const int* cu_q, const int* seq_slot, int nseq, const float* q,
                          const float* k, const float* v, long long ld, const float* alpha, const GlaDims& d,
                          float* state, int ring, float* out, cudaStream_t stream) {
    if (ix.M <= 0 || nseq <= 0) return 0;
    if (d.dk <= 0 || d.dk > 1024) return set_error("gla: key size %d outside 1..1024", d.dk);
    if (ring <= 0 || !state) return set_error("gla: no state");
    const int groups = (d.dk + GLA_R - 1) / GLA_R, run = (ix.M + nseq - 1) / nseq;
    // 32 columns a CTA; steps of large heads 16, so that an SM holds several (64 single tokens, 4 heads of 512 x 512: one CTA of 512
    // threads per SM 252 us, two 150, four of 256 threads 136; 1 head of 1024 x 1024: one of 1024 threads 177, two of 512 152)
    int cols = groups > 32 && run <= 1 ? 16 : 32;
    // 48 columns where 32 leave some SMs with two CTAs, which are then the last, and these give every CTA an SM of its own: 436 clocks a
    // position there, 390 here (3 prompts of up to 777 positions, 16 heads of 128 x 128: 167 -> 158 us; four warps of 8 rows x 6 columns
    // a CTA instead of six of 8 x 4: 225).  Eleven head shapes, 38 to 148 pairs of sequence and head, a layer's step with and without: runs of
    // 2 to 64 positions within 2 us of each other or faster, of 128 and 256 up to 14 % faster (12 x 256, 8 heads of 32 x 48: 208 -> 179 us)
    const long long heads_all = (long long)nseq * d.heads, sms = sm_count();
    if (run > 1 && groups <= 16 && heads_all * ((d.dv + 31) / 32) > sms && heads_all * ((d.dv + 47) / 48) <= sms) cols = 48;
    const int cg = cols / GLA_C, whole = cols == 48 ? 96 : 32;         // threads: whole warps, and whole rows of column groups
    const int threads = (groups * cg + whole - 1) / whole * whole, RG = threads / cg, dkp = RG * GLA_R;
    // chunks as long as two (large heads: one) staged CTAs per SM allow, and no longer than the runs: a step's CTAs are then
    // small enough for an SM to hold all that its registers can
    int ch = dkp <= 128 ? 16 : (dkp <= 512 ? 8 : 4);
    ch = std::min(ch, run <= 1 ? 1 : std::max(4, run));
    const size_t smem = (size_t)(2 * (3 * ch * dkp + ch * cols) + RG * ch * cols) * sizeof(float);
    const dim3 grid(nseq, d.heads, (d.dv + cols - 1) / cols);
    if (grid.y > 65535 || grid.z > 65535) return set_error("gla: too many heads or value columns");
    const uintptr_t at = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                         reinterpret_cast<uintptr_t>(alpha) | reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(out);
    const int vec = (at & 15) == 0 && ld % 4 == 0 && d.dk % 4 == 0 && d.dv % 4 == 0;
    // steps and short runs of large heads wait for the state, not for their positions: no loads ahead, and the registers of as many
    // CTAs per SM as there can be (64 runs of 5, 4 heads of 512 x 512: one 295 us, two 191)
    const int form = cols == 16 ? (threads > 256 ? 0 : 1)
                : cols == 48 ? 7
                                : (threads > 512 ? 2 : (threads > 256 ? (2 * smem <= 220 * 1024 ? 3 : 4) : (ch == 1 ? 5 : 6)));
    const decltype(&gla_recurrence_kernel<256, 2, true>) forms[] = {
        gla_recurrence_kernel<512, 2, false, 16>, gla_recurrence_kernel<256, 4, false, 16>, gla_recurrence_kernel<1024, 1, false>,
        gla_recurrence_kernel<512, 2, false>,     gla_recurrence_kernel<512, 1, true>,      gla_recurrence_kernel<256, 4, false>,
        gla_recurrence_kernel<256, 2, true>,      gla_recurrence_kernel<192, 1, true, 48>};
    auto fn = forms[form];
    static PerDeviceOnce once[8];
    ASD_ONCE(once[form], ASD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024)));
    ASD_CUDA(launch_pdl(fn, grid, threads, smem, stream, ix, cu_q, seq_slot, q, k, v, ld, alpha, d, state, ring, out, ch, vec));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

int launch_gla_out(const float* o, const float* gate, long long ldg, const float* w, float eps, void* y, int of32, int M,
                   int heads, int dv, cudaStream_t stream) {
    if (M <= 0) return 0;
    const long long pairs = (long long)M * heads, blocks = (pairs + 7) / 8;
    if (blocks > 0x7fffffffLL) return set_error("gla: too many tokens");
    const uintptr_t at = reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(w) |
                         reinterpret_cast<uintptr_t>(y);
    const bool vec = (at & 15) == 0 && ldg % 4 == 0 && dv % 4 == 0 && dv <= 256;
    auto fn = !vec ? gla_out_kernel<0> : (dv <= 128 ? gla_out_kernel<1> : gla_out_kernel<2>);
    ASD_CUDA(launch_pdl(fn, (unsigned)blocks, 256, 0, stream, o, gate, ldg, w, eps, y, of32, pairs, heads, dv));
    count_launch(1);
    ASD_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace asd
