// Fused logits -> softmax -> rejection sampling -> residual resample -> stop-rule features, as a STREAMING pass:
// every logit of the verify step is read from HBM once, with no vocabulary-wide exchange in front of the exponentials.
//
//   sampler_stats_kernel   item = (row, chunk): 4096 consecutive logits of one row, the draft row's chunk next to the
//     target's; at most 3 CTAs of 256 threads per SM stay resident and walk the items.  Bound by HBM: a CTA keeps a ring
//     of two chunk pairs (four chunks when greedy) filled by 1-D bulk (TMA) copies, so an SM has 96 to 192 KB of loads in
//     flight all the time; a CTA per item, whose load, barriers, fence and ticket came one after the other, lived 7 us per
//     32 KB and held the kernel at 0.57 of the copy bandwidth.  Per chunk: maximum (warp reductions + one shared-memory
//     hop; the runner-up only where it can be: between the threads' maxima, and inside the one thread that owns the
//     maximum), exponentials relative to the CHUNK maximum (polynomial exp2 on the packed fp32x2 pipe), lane sums and
//     the canonical warp scan; one 32-byte record per (row, chunk), and nothing that waits for another CTA.
//   sampler_draw_kernel    grid = sequences x G (G CTAs share a sequence's chunks, enough to fill the SMs once), launched
//     programmatically behind it.  Every CTA merges the records of its sequence's rows, a warp per row (rescaling by
//     2^(m_c - M), lanes = chunks, sums chained in chunk order through shuffles), runs the min(1, p/q) accept test in
//     binary64 and finds the first-reject prefix: repeating this in the G CTAs is cheaper than tickets between them.  The
//     first of them writes the features and accepted tokens.  Then the ONE row that emits a new token: residual
//     max(0, p - q) chunk totals; the last CTA of the sequence walks the totals, re-reads the selected chunk (L2) and
//     finishes the inverse-CDF draw inside it.  Greedy verification needs the merge only (G = 1), and where
//     its items all fit the chip at once the first kernel's last CTA of a sequence does it: one launch.
// DRAM traffic = (1 + ~1/(k+1)) x the algorithmic bytes.
// Measured (V = 152064, all outputs the same bits), the CTA-per-item form -> this one: B = 64, k = 8: 195 -> 163 us (the
// first kernel 176 -> 132 us, 5.0 TB/s; what is left is its 10 cycles per issued instruction at 24 warps, six of them a
// scheduler's, and 31 us of the second kernel, of which 12 are the emitting rows' second read); B = 16, k = 5 greedy
// 37 -> 29 us; V = 151936, B = 1, k = 4: 22 -> 14 us, launches and the chain record -> merge -> residual -> draw.
//
// ARITHMETIC CONTRACT v2 (bit-exact with oracle/sampler_oracle.c - see that file's header): every contract
// operation below is an explicit round-to-nearest intrinsic so that nvcc can neither contract nor reorder it.
// Inside a chunk, local element u lives in lane (u / 4) mod 256 = thread, visited in increasing u.
//
// Replaces (reference): per-token softmax + log(probs[token]) with a host sync per token,
// src/training/generate_training_data.py:128-134, and the logprob feature
// reductions of docs/guides/RESEARCH_PROTOCOL.md:379-398.  The accept/resample rule itself has no
// reference implementation.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "asd_internal.h"
#include "ptx.cuh"

namespace asd {

constexpr int kChunk = 4096;             // logits per chunk
constexpr int kST = 256;                 // threads per CTA = lanes per chunk
constexpr int kSW = kST / 32;            // warps
constexpr int kSlots = kChunk / 4 / kST; // float4 per thread and row (4)
constexpr int kMaxChunks = 52;           // V <= 212992
constexpr int kMaxRows = 65;             // k <= 64
constexpr int kNFeat = ASD_NUM_FEATURES;

struct SamplerParams {
    const float* target;       // [B, k+1, V]
    const float* draft;        // [B, k, V] or null
    const int* draft_tokens;   // [B, k]
    const double* u_accept;    // [B, k]
    const double* u_resid;     // [B]
    int B, k, V, NC, greedy;
    int G;                     // CTAs of the draw kernel per sequence
    int fused;                 // greedy, an item per CTA: the sequence's last CTA merges in the first kernel
    float c1;
    // outputs
    uint8_t* accept_mask;
    int* accepted_len;
    int* out_tokens;
    float* out_logprobs;
    float* features;
    // workspace (ticket zero between launches)
    int* seq_ticket;    // [B]
    float4* rec_p;      // [rows][NC] {m, m2, Z, S} of the target chunk
    float4* rec_q;      // [rows][NC] {mq, Zq, e at the chunk arg-max, arg-max index (bits)}
    float* row_px;      // [rows] chunk-relative e_p of the draft token
    float* row_qx;      // [rows] chunk-relative e_q of the draft token
    float* seq_rc;      // [B][NC] residual chunk totals of the emitting row
    int* err;           // where a wait that ran out is reported
};

__device__ __forceinline__ float exp2p(float t) {
    const float tc = fmaxf(t, -125.0f);
    const float r = __fadd_rn(tc, 12582912.0f);
    const float nf = __fadd_rn(r, -12582912.0f);
    const float f = __fadd_rn(tc, -nf);
    float p = 0x1.5c08e6p-10f;
    p = __fmaf_rn(p, f, 0x1.3d0c52p-7f);
    p = __fmaf_rn(p, f, 0x1.c6b6e4p-5f);
    p = __fmaf_rn(p, f, 0x1.ebf918p-3f);
    p = __fmaf_rn(p, f, 0x1.62e428p-1f);
    p = __fmaf_rn(p, f, 0x1.000002p+0f);
    return __int_as_float(__float_as_int(p) + (__float_as_int(r) << 23));
}
// two lanes of the same polynomial on the packed fp32x2 pipe (FFMA2 / FADD2, sm_100): each component is an IEEE
// fma / add, so the results are bit-identical to the scalar contract
__device__ __forceinline__ float2 exp2p2(float2 t) {
    const float2 tc = make_float2(fmaxf(t.x, -125.0f), fmaxf(t.y, -125.0f));
    const float2 magic = make_float2(12582912.0f, 12582912.0f), nmagic = make_float2(-12582912.0f, -12582912.0f);
    const float2 r = __fadd2_rn(tc, magic);
    const float2 nf = __fadd2_rn(r, nmagic);
    const float2 f = __ffma2_rn(nf, make_float2(-1.0f, -1.0f), tc);   // tc - nf, exact
    float2 q = make_float2(0x1.5c08e6p-10f, 0x1.5c08e6p-10f);
    q = __ffma2_rn(q, f, make_float2(0x1.3d0c52p-7f, 0x1.3d0c52p-7f));
    q = __ffma2_rn(q, f, make_float2(0x1.c6b6e4p-5f, 0x1.c6b6e4p-5f));
    q = __ffma2_rn(q, f, make_float2(0x1.ebf918p-3f, 0x1.ebf918p-3f));
    q = __ffma2_rn(q, f, make_float2(0x1.62e428p-1f, 0x1.62e428p-1f));
    q = __ffma2_rn(q, f, make_float2(0x1.000002p+0f, 0x1.000002p+0f));
    return make_float2(__int_as_float(__float_as_int(q.x) + (__float_as_int(r.x) << 23)),
                       __int_as_float(__float_as_int(q.y) + (__float_as_int(r.y) << 23)));
}

// Hillis-Steele inclusive scan inside the warp (the contract's order)
__device__ __forceinline__ float warp_hs(float x, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x = __fadd_rn(x, up);
    }
    return x;
}

// warp_hs(x)'s last lane for three sums at once: the scan's last lane is the tree that pairs lanes 1, 2, 4, 8, 16 apart,
// so a butterfly gives its bits, and after the first two steps one exchange serves all three (16 instructions instead of
// 45).  Lanes with bit 1 set end up with q's total, the others with x's (bit 0 clear) or y's (bit 0 set).
__device__ __forceinline__ float warp_tree3(float x, float y, float q, int lane) {
    const unsigned all = 0xffffffffu;
    const bool odd = lane & 1, high = lane & 2;
    float a = __fadd_rn(odd ? y : x, __shfl_xor_sync(all, odd ? x : y, 1));
    q = __fadd_rn(q, __shfl_xor_sync(all, q, 1));
    a = __fadd_rn(high ? q : a, __shfl_xor_sync(all, high ? a : q, 2));
#pragma unroll
    for (int d = 4; d <= 16; d <<= 1) a = __fadd_rn(a, __shfl_xor_sync(all, a, d));
    return a;
}
// maximum over the warp in one instruction (NaN loses against a number, as in fmaxf)
__device__ __forceinline__ float warp_fmax(float x) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}

// e = exp2p(fma(z, c1, -m)) for the four logits of a float4, in place
__device__ __forceinline__ void exp4(float4& z, float2 c1v, float2 nmv, float2& t0, float2& t1) {
    t0 = __ffma2_rn(make_float2(z.x, z.y), c1v, nmv);
    t1 = __ffma2_rn(make_float2(z.z, z.w), c1v, nmv);
    const float2 e0 = exp2p2(t0), e1 = exp2p2(t1);
    z = make_float4(e0.x, e0.y, e1.x, e1.y);
}

// One row's statistics from its chunk records, by one warp (lanes = chunks lane and lane + 32; every sum is chained in
// chunk order): {M, Zp, Mq, Zq}, whether the draft token is accepted, and - `write` - the row's features.
struct RowMerge {
    float4 stat;
    int accept, amax;
    float lpx, lp_amax;
};
__device__ __forceinline__ RowMerge merge_row(const SamplerParams& p, int b, int i, int lane, bool write) {
    const unsigned all = 0xffffffffu;
    const int NC = p.NC, row = b * (p.k + 1) + i;
    const bool has_draft = i < p.k && !p.greedy;
    const float4 none = make_float4(-INFINITY, -INFINITY, 0.f, 0.f);
    float4 rp[2], rq[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const bool ok = lane + 32 * u < NC;
        rp[u] = ok ? __ldcg(&p.rec_p[(size_t)row * NC + lane + 32 * u]) : none;
        rq[u] = ok ? __ldcg(&p.rec_q[(size_t)row * NC + lane + 32 * u]) : none;
    }
    const int x = i < p.k ? p.draft_tokens[b * p.k + i] : -1;
    const bool x_ok = i < p.k && x >= 0 && x < p.V;
    const float px = x_ok ? __ldcg(&p.row_px[row]) : 0.0f, qx = x_ok && has_draft ? __ldcg(&p.row_qx[row]) : 0.0f;
    const double u_acc = has_draft ? p.u_accept[b * p.k + i] : 0.0;
    float M = fmaxf(rp[0].x, rp[1].x), M2 = fmaxf(fminf(rp[0].x, rp[1].x), fmaxf(rp[0].y, rp[1].y));
    float Mq = fmaxf(rq[0].x, rq[1].x);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const float o1 = __shfl_xor_sync(all, M, d), o2 = __shfl_xor_sync(all, M2, d);
        M2 = fmaxf(fminf(M, o1), fmaxf(M2, o2));
        M = fmaxf(M, o1);
        Mq = fmaxf(Mq, __shfl_xor_sync(all, Mq, d));
    }
    float sc[2], tz[2], ts[2], sq[2], tq[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const float d = __fadd_rn(rp[u].x, -M);
        sc[u] = exp2p(d);
        tz[u] = __fmul_rn(rp[u].z, sc[u]);
        ts[u] = __fmul_rn(__fmaf_rn(rp[u].z, d, rp[u].w), sc[u]);
        sq[u] = exp2p(__fadd_rn(rq[u].x, -Mq));
        tq[u] = __fmul_rn(rq[u].y, sq[u]);
    }
    float Zp = 0.0f, St = 0.0f, Zq = 0.0f;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll 8
        for (int c = 0; c < min(32, NC - 32 * u); ++c) {
            Zp = __fadd_rn(Zp, __shfl_sync(all, tz[u], c));
            St = __fadd_rn(St, __shfl_sync(all, ts[u], c));
            Zq = __fadd_rn(Zq, __shfl_sync(all, tq[u], c));
        }
    if (!has_draft) Zq = 0.0f;
    const int cx = x_ok ? x / kChunk : 0;
    const float s_x = __shfl_sync(all, cx < 32 ? sc[0] : sc[1], cx & 31);
    const float sq_x = __shfl_sync(all, cx < 32 ? sq[0] : sq[1], cx & 31);
    RowMerge r;
    r.stat = make_float4(M, Zp, Mq, Zq);
    const float Px = x_ok ? __fmul_rn(px, s_x) : 0.0f;
    r.amax = -1;
    float P_amax = 0.0f;
    if (p.greedy) {             // the first chunk that attains the row maximum holds its lowest index
        const unsigned h0 = __ballot_sync(all, rp[0].x == M && lane < NC), h1 = __ballot_sync(all, rp[1].x == M && lane + 32 < NC);
        if (h0 | h1) {
            const int src = h0 ? __ffs(h0) - 1 : __ffs(h1) - 1;
            r.amax = __shfl_sync(all, __float_as_int(h0 ? rq[0].w : rq[1].w), src);
            P_amax = __shfl_sync(all, h0 ? __fmul_rn(rq[0].z, sc[0]) : __fmul_rn(rq[1].z, sc[1]), src);
        }
    }
    r.accept = 0;
    if (p.greedy) {
        r.accept = x_ok && x == r.amax;
    } else if (has_draft && x_ok) {
        const float Qx = __fmul_rn(qx, sq_x);
        const double lhs = __dmul_rn(__dmul_rn(u_acc, (double)Qx), (double)Zp);
        const double rhs = __dmul_rn((double)Px, (double)Zq);
        r.accept = lhs <= rhs;
    }
    r.lpx = r.lp_amax = 0.0f;
    if (write) {
        const float logZ = logf(Zp), log2Z = log2f(Zp);
        r.lpx = x_ok ? logf(Px) - logZ : -INFINITY;
        if (p.greedy) r.lp_amax = logf(P_amax) - logZ;
        if (lane == 0) {
            float* f = p.features + (size_t)row * kNFeat;
            f[0] = __fmul_rn(__fadd_rn(M, log2Z), 0x1.62e43p-1f);
            f[1] = 1.0f / Zp;
            f[2] = f[1] - exp2p(__fadd_rn(M2, -M)) / Zp;
            f[3] = (log2Z - St / Zp) * 0x1.62e43p-1f;
            f[4] = r.lpx;
        }
    }
    return r;
}

// All rows of a sequence, a warp per row; returns the first-reject prefix.
struct SeqMerge {
    float4 stat[kMaxRows];
    int acc[kMaxRows], amax[kMaxRows];
    float lpx[kMaxRows], lpamax[kMaxRows];
};
__device__ __forceinline__ int merge_rows(const SamplerParams& p, int b, SeqMerge& s, bool write) {
    const int lane = threadIdx.x & 31, k1 = p.k + 1;
    for (int i = threadIdx.x >> 5; i < k1; i += kSW) {
        const RowMerge r = merge_row(p, b, i, lane, write);
        if (lane == 0) {
            s.stat[i] = r.stat;
            s.acc[i] = r.accept;
            s.amax[i] = r.amax;
            s.lpx[i] = r.lpx;
            s.lpamax[i] = r.lp_amax;
        }
    }
    __syncthreads();
    int n = 0;
    while (n < p.k && s.acc[n]) ++n;
    return n;
}
__device__ __forceinline__ void write_prefix(const SamplerParams& p, int b, int n, const SeqMerge& s) {
    const int tid = threadIdx.x, k1 = p.k + 1;
    if (tid < p.k) p.accept_mask[b * p.k + tid] = tid < n;
    if (tid == 0) p.accepted_len[b] = n;
    if (tid < k1 && (tid != n || p.greedy)) {       // position n of a sampled sequence: the draw
        int tok = -1;
        float lp = 0.0f;
        if (tid < n) {
            tok = p.draft_tokens[b * p.k + tid];
            lp = s.lpx[tid];
        } else if (tid == n) {
            tok = s.amax[n];
            lp = s.lpamax[n];
        }
        p.out_tokens[b * k1 + tid] = tok;
        p.out_logprobs[b * k1 + tid] = lp;
        p.features[(size_t)(b * k1 + tid) * kNFeat + 5] = lp;
    }
}

// ------------------------------------------------------------------------------------------------ kernel 1
__device__ __forceinline__ float max4(const float4& z) { return fmaxf(fmaxf(z.x, z.y), fmaxf(z.z, z.w)); }

template <bool GREEDY>
__global__ void __launch_bounds__(kST, 3) sampler_stats_kernel(const SamplerParams p) {
    constexpr int kStages = GREEDY ? 4 : 2, kPair = GREEDY ? kChunk / 4 : kChunk / 2;    // float4s per stage
    extern __shared__ __align__(128) float4 s_ring[];     // [kStages][target chunk | draft chunk]
    __shared__ __align__(8) uint64_t s_bar[kStages];
    __shared__ int4 s_item[kStages];                      // {row, chunk, float4s of the chunk | has_draft << 16, draft token in the chunk}
    __shared__ __align__(16) float2 s_red[2][kSW];        // (the record of an item is written while the next one's maxima arrive)
    __shared__ float s_own2[kSW], s_red2[kSW][3];
    __shared__ unsigned long long s_key[kSW];
    __shared__ int s_failed, s_last;
    __shared__ SeqMerge s_seq;
    const WaitGuard guard{&s_failed, p.err, WAIT_SAMPLER << 8};
    grid_dep_launch();      // the draw kernel may be scheduled; it waits for this grid before reading anything
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int total = p.B * (p.k + 1) * p.NC;
    const float c1 = p.c1;
    const float2 c1v = make_float2(c1, c1);
    // thread 0: bulk copies of one (row, chunk) item into a stage of the ring, and what the others need to know about it
    auto issue = [&](int item, int st) {
        const int V = p.V, row = item / p.NC, c = item - row * p.NC;
        const int b = row / (p.k + 1), i = row - b * (p.k + 1);
        const bool hd = !GREEDY && i < p.k;
        const int n4 = min(kChunk / 4, (V - c * kChunk) >> 2);
        const uint32_t bytes = (uint32_t)n4 * 16u;
        const int x = i < p.k ? p.draft_tokens[b * p.k + i] : -1;
        s_item[st] = make_int4(row, c, n4 | (hd ? 1 << 16 : 0), x >= 0 && x < V && x / kChunk == c ? x - c * kChunk : -1);
        float4* dst = s_ring + st * kPair;
        mbar_expect_tx(&s_bar[st], hd ? 2 * bytes : bytes);     // (its release covers s_item)
        bulk_g2s(dst, p.target + (size_t)row * V + (size_t)c * kChunk, bytes, &s_bar[st]);
        if (hd) bulk_g2s(dst + kChunk / 4, p.draft + ((size_t)b * p.k + i) * V + (size_t)c * kChunk, bytes, &s_bar[st]);
    };
    if (tid == 0) {
#pragma unroll
        for (int st = 0; st < kStages; ++st) mbar_init(&s_bar[st], 1);
        s_failed = 0;
        fence_mbar_init();
#pragma unroll
        for (int st = 0; st < kStages; ++st)
            if (blockIdx.x + (long long)st * gridDim.x < total) issue(blockIdx.x + st * gridDim.x, st);
    }
    __syncthreads();            // the barriers are initialised
    int it = 0;
    for (int item = blockIdx.x; item < total; item += gridDim.x, ++it) {
        const int st = it % kStages;
        const float4* zt = s_ring + st * kPair;
        const float4* zq = zt + kChunk / 4;
        mbar_wait_far(&s_bar[st], (it / kStages) & 1, guard, 1);
        const int4 what = s_item[st];
        const int n4 = what.z & 0xffff;
        const bool has_draft = !GREEDY && (what.z >> 16);
        // pass over the float4s this thread owns; a whole chunk needs no bounds
        auto each = [&](auto&& f) {
            if (n4 == kChunk / 4) {
#pragma unroll
                for (int s = 0; s < kSlots; ++s) f(s * kST + tid);
            } else {
#pragma unroll 1
                for (int v = tid; v < n4; v += kST) f(v);
            }
        };

        // ---- chunk maxima on the raw logits: rn multiplication by c1 > 0 is monotone, so the two largest a = z * c1 of
        // the multiset are the products of the two largest z (exact, order independent)
        float own = -INFINITY, mq = -INFINITY;
        each([&](int v) {
            own = fmaxf(own, max4(zt[v]));
            if (has_draft) mq = fmaxf(mq, max4(zq[v]));
        });
        const float wm = warp_fmax(own);
        mq = warp_fmax(mq);
        if (lane == 0) s_red[it & 1][warp] = make_float2(wm, mq);
        __syncthreads();
        float m1 = -INFINITY;
        mq = -INFINITY;
#pragma unroll
        for (int w = 0; w < kSW; w += 2) {
            const float4 o = *reinterpret_cast<const float4*>(&s_red[it & 1][w]);
            m1 = fmaxf(m1, fmaxf(o.x, o.z));
            mq = fmaxf(mq, fmaxf(o.y, o.w));
        }
        // runner-up of a warp that owns the maximum: between its other lanes and inside the owner (of several owners the
        // first leaves out its own maximum, and the others' stand in for the runner-up); of other warps: their maxima, below
        float second = -INFINITY;
        if (wm == m1) {
            const unsigned owners = __ballot_sync(0xffffffffu, own == m1);
            const bool first = lane == __ffs(owners) - 1;
            float a1 = -INFINITY, a2 = -INFINITY;
            if (first)
                for (int v = tid; v < n4; v += kST) {
                    const float4 z = zt[v];
                    const float a[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        a2 = fmaxf(a2, fminf(a1, a[e]));
                        a1 = fmaxf(a1, a[e]);
                    }
                }
            __syncwarp();
            second = warp_fmax(first ? a2 : own);
        }
        const float raw1 = m1;
        m1 = __fmul_rn(m1, c1);
        mq = __fmul_rn(mq, c1);

        // ---- exponentials relative to the chunk maximum; a lane keeps two running sums (elements with even / odd local
        // index, each left to right) on the packed fp32x2 pipe and adds them at the end
        float2 zs2 = make_float2(0.f, 0.f), ss2 = zs2, qs2 = zs2;
        const float2 nm1v = make_float2(-m1, -m1), nmqv = make_float2(-mq, -mq);
        each([&](int v) {
            float4 z = zt[v];
            float2 t0, t1;
            exp4(z, c1v, nm1v, t0, t1);
            zs2 = __fadd2_rn(__fadd2_rn(zs2, make_float2(z.x, z.y)), make_float2(z.z, z.w));
            ss2 = __fadd2_rn(__fadd2_rn(ss2, __fmul2_rn(make_float2(z.x, z.y), t0)), __fmul2_rn(make_float2(z.z, z.w), t1));
            if (has_draft) {
                float4 q = zq[v];
                exp4(q, c1v, nmqv, t0, t1);
                qs2 = __fadd2_rn(__fadd2_rn(qs2, make_float2(q.x, q.y)), make_float2(q.z, q.w));
            }
        });
        // ---- the draft token's exponentials (one thread recomputes them from the chunk in shared memory)
        if (tid == 32 && what.w >= 0) {
            p.row_px[what.x] = exp2p(__fmaf_rn(reinterpret_cast<const float*>(zt)[what.w], c1, -m1));
            if (has_draft) p.row_qx[what.x] = exp2p(__fmaf_rn(reinterpret_cast<const float*>(zq)[what.w], c1, -mq));
        }
        __syncwarp();
        // ---- canonical chunk totals: the warp's scan tree, sequential chain over the 8 warps
        const float sum = warp_tree3(__fadd_rn(zs2.x, zs2.y), __fadd_rn(ss2.x, ss2.y), __fadd_rn(qs2.x, qs2.y), lane);
        if (lane < 3) s_red2[warp][lane] = sum;         // lanes 0, 1, 2: Z, S, Zq
        if (lane == 3) s_own2[warp] = second;
        if (GREEDY) {               // (lowest index attaining the maximum, its e): only threads whose maximum attains it look
            unsigned long long key = ~0ull;
            if (__fmul_rn(own, c1) == m1)
                for (int v = tid; v < n4; v += kST) {
                    const float4 z = zt[v];
                    const float zz[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (key == ~0ull && __fmul_rn(zz[e], c1) == m1)
                            key = ((unsigned long long)(unsigned)(what.y * kChunk + v * 4 + e) << 32) |
                                  __float_as_uint(exp2p(__fmaf_rn(zz[e], c1, -m1)));
                }
            __syncwarp();
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) {
                const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, d);
                key = o < key ? o : key;
            }
            if (lane == 0) s_key[warp] = key;
        }
        __syncthreads();            // every thread is done with the stage
        if (tid == 0) {
            fence_proxy_async_smem();   // generic reads of the stage ordered before the async-proxy writes of the next copy
            if (item + (long long)kStages * gridDim.x < total && !*guard.failed) issue(item + kStages * gridDim.x, st);
            float Z = 0.0f, S = 0.0f, Zq = 0.0f, m2 = -INFINITY;
            unsigned long long kk = ~0ull;
            bool seen = false;          // the first warp that attains the maximum is the owner, the others are runners-up
#pragma unroll
            for (int w = 0; w < kSW; ++w) {
                Z = __fadd_rn(Z, s_red2[w][0]);
                S = __fadd_rn(S, s_red2[w][1]);
                Zq = __fadd_rn(Zq, s_red2[w][2]);
                const float wmax = s_red[it & 1][w].x;
                const bool owner = !seen && wmax == raw1;
                seen |= owner;
                m2 = fmaxf(m2, owner ? s_own2[w] : wmax);
                if (GREEDY) kk = s_key[w] < kk ? s_key[w] : kk;
            }
            const size_t at = (size_t)what.x * p.NC + what.y;
            p.rec_p[at] = make_float4(m1, __fmul_rn(m2, c1), Z, S);
            p.rec_q[at] = make_float4(mq, Zq, __uint_as_float((unsigned)(kk & 0xffffffffu)), __int_as_float((int)(kk >> 32)));
        }
    }
    wait_settle(guard);
    if (GREEDY && p.fused) {        // this CTA had one item
        const int b = blockIdx.x / (p.NC * (p.k + 1));
        if (tid == 0) {
            __threadfence();        // the record, and the draft token's term before the last barrier
            s_last = atomicAdd(&p.seq_ticket[b], 1) == p.NC * (p.k + 1) - 1;
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        if (tid == 0) p.seq_ticket[b] = 0;
        const int n = merge_rows(p, b, s_seq, true);
        write_prefix(p, b, n, s_seq);
    }
}

// ------------------------------------------------------------------------------------------------ kernel 2
// residual weights of this thread's elements of chunk c of the emitting row, whose logits lie at zt_s (draft: behind them):
// r -> zq[], P -> zt[]; returns the lane sum
__device__ __forceinline__ float residual_chunk(const SamplerParams& p, int row, int c, bool has_draft, const float4* zt_s,
                                                const float4& st, float4 (&zt)[kSlots], float4 (&zq)[kSlots],
                                                bool (&have)[kSlots]) {
    const int tid = threadIdx.x;
    const int n4 = min(kChunk / 4, (p.V - c * kChunk) >> 2);
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        have[s] = s * kST + tid < n4;
        zt[s] = have[s] ? zt_s[s * kST + tid] : make_float4(0.f, 0.f, 0.f, 0.f);
        zq[s] = (has_draft && have[s]) ? zt_s[kChunk / 4 + s * kST + tid] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float4 rp = __ldcg(&p.rec_p[(size_t)row * p.NC + c]);
    const float4 rq = __ldcg(&p.rec_q[(size_t)row * p.NC + c]);
    const float M = st.x, Zp = st.y, Mq = st.z, Zq = st.w;
    const float sp = exp2p(__fadd_rn(rp.x, -M));
    const float sq = has_draft ? exp2p(__fadd_rn(rq.x, -Mq)) : 0.0f;
    const float2 c1v = make_float2(p.c1, p.c1), nmv = make_float2(-rp.x, -rp.x), nqv = make_float2(-rq.x, -rq.x);
    const float2 spv = make_float2(sp, sp), sqv = make_float2(sq, sq), zqv = make_float2(Zq, Zq), nzpv = make_float2(-Zp, -Zp);
    float rs = 0.0f;
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        if (have[s]) {
            float2 t0, t1;
            exp4(zt[s], c1v, nmv, t0, t1);
            const float2 P0 = __fmul2_rn(make_float2(zt[s].x, zt[s].y), spv);
            const float2 P1 = __fmul2_rn(make_float2(zt[s].z, zt[s].w), spv);
            zt[s] = make_float4(P0.x, P0.y, P1.x, P1.y);
            float4 r4;
            if (has_draft) {
                exp4(zq[s], c1v, nqv, t0, t1);
                const float2 Q0 = __fmul2_rn(make_float2(zq[s].x, zq[s].y), sqv);
                const float2 Q1 = __fmul2_rn(make_float2(zq[s].z, zq[s].w), sqv);
                const float2 w0 = __fmul2_rn(Q0, nzpv), w1 = __fmul2_rn(Q1, nzpv);      // -(Q * Zp), exact sign flip
                const float2 r0 = __ffma2_rn(P0, zqv, w0), r1 = __ffma2_rn(P1, zqv, w1);
                r4 = make_float4(fmaxf(r0.x, 0.0f), fmaxf(r0.y, 0.0f), fmaxf(r1.x, 0.0f), fmaxf(r1.y, 0.0f));
            } else {
                r4 = zt[s];
            }
            zq[s] = r4;
            rs = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(rs, r4.x), r4.y), r4.z), r4.w);
        }
    }
    return rs;
}

__global__ void __launch_bounds__(kST, 3) sampler_draw_kernel(const SamplerParams p) {
    extern __shared__ __align__(128) float4 s_ring[];     // [2][target chunk | draft chunk]
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ float s_red[2][kSW];
    __shared__ float s_rc[kMaxChunks], s_pre[kMaxChunks];
    __shared__ SeqMerge s_seq;
    __shared__ int s_flag, s_cstar, s_tstar[kSW], s_failed;
    __shared__ float s_tau;
    const WaitGuard guard{&s_failed, p.err, WAIT_SAMPLER << 8};
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k1 = p.k + 1, NC = p.NC, G = p.G;
    const int b = blockIdx.x / G, g = blockIdx.x - b * G;
    if (tid == 0) {
        mbar_init(&s_bar[0], 1);
        mbar_init(&s_bar[1], 1);
        s_failed = 0;
        fence_mbar_init();
    }
    grid_dep_wait();
    const int n = merge_rows(p, b, s_seq, g == 0);
    const int row = b * k1 + n;
    const bool has_draft = n < p.k;
    auto issue = [&](int c2, int stage) {       // thread 0
        const uint32_t bytes = (uint32_t)min(kChunk / 4, (p.V - c2 * kChunk) >> 2) * 16u;
        float4* dst = s_ring + stage * (kChunk / 2);
        mbar_expect_tx(&s_bar[stage], has_draft ? 2 * bytes : bytes);
        bulk_g2s(dst, p.target + (size_t)row * p.V + (size_t)c2 * kChunk, bytes, &s_bar[stage]);
        if (has_draft)
            bulk_g2s(dst + kChunk / 4, p.draft + ((size_t)b * p.k + n) * p.V + (size_t)c2 * kChunk, bytes, &s_bar[stage]);
    };
    if (tid == 0 && !p.greedy) {
        issue(g, 0);
        if (g + G < NC) issue(g + G, 1);
    }
    if (g == 0) write_prefix(p, b, n, s_seq);
    if (p.greedy) return;
    const float4 st = s_seq.stat[n];
    float4 zt[kSlots], zq[kSlots];
    bool have[kSlots];
    float rs = 0.0f, hs;
    int c = g, it = 0;
    for (;; c += G, ++it) {
        mbar_wait_far(&s_bar[it & 1], (it >> 1) & 1, guard, 2);
        rs = residual_chunk(p, row, c, has_draft, s_ring + (it & 1) * (kChunk / 2), st, zt, zq, have);
        hs = warp_hs(rs, lane);
        if (lane == 31) s_red[it & 1][warp] = hs;
        __syncthreads();
        if (tid == 0) {
            fence_proxy_async_smem();
            if (c + 2 * G < NC && !*guard.failed) issue(c + 2 * G, it & 1);
            float R = 0.0f;
            for (int w = 0; w < kSW; ++w) R = __fadd_rn(R, s_red[it & 1][w]);
            __stcg(&p.seq_rc[(size_t)b * NC + c], R);
        }
        if (c + G >= NC) break;
    }
    wait_settle(guard);
    if (tid == 0) {
        __threadfence();
        s_flag = atomicAdd(&p.seq_ticket[b], 1) == G - 1;
    }
    __syncthreads();
    if (!s_flag) return;

    // ================================================================ last CTA of the sequence: the draw
    __threadfence();
    if (tid < NC) s_rc[tid] = __ldcg(&p.seq_rc[(size_t)b * NC + tid]);
    __syncthreads();
    if (warp == 0) {
        float R = 0.0f;
        if (lane == 0) {
            p.seq_ticket[b] = 0;
#pragma unroll 8
            for (int c2 = 0; c2 < NC; ++c2) s_pre[c2] = R = __fadd_rn(R, s_rc[c2]);
        }
        R = __shfl_sync(0xffffffffu, R, 0);
        int cstar = -1;
        float tau = 0.0f;
        if (R > 0.0f) {
            float ur = (float)p.u_resid[b];
            if (!(ur >= 0.0f)) ur = 0.0f;
            if (ur >= 1.0f) ur = 0x1.fffffep-1f;
            tau = __fmul_rn(ur, R);
            if (!(tau < R)) tau = 0.0f;
            __syncwarp();
            const unsigned h0 = __ballot_sync(0xffffffffu, lane < NC && s_pre[lane] > tau);
            const unsigned h1 = __ballot_sync(0xffffffffu, lane + 32 < NC && s_pre[lane + 32] > tau);
            cstar = h0 ? __ffs(h0) - 1 : (h1 ? 31 + __ffs(h1) : -1);
        }
        if (lane == 0) {
            s_cstar = cstar;
            s_tau = tau;
        }
    }
    __syncthreads();
    const int cstar = s_cstar;
    const float tau = s_tau, X = cstar > 0 ? s_pre[cstar - 1] : 0.0f;
    const float logZ = logf(st.y);
    if (cstar < 0) {
        // residual mass is zero (p == q on this row): the draft token itself is a valid draw
        if (tid == 0) {
            const int x = has_draft ? p.draft_tokens[b * p.k + n] : -1;
            const bool x_ok = has_draft && x >= 0 && x < p.V;
            const int y = x_ok ? x : 0;
            const float4 rp = __ldcg(&p.rec_p[(size_t)row * NC + y / kChunk]);
            const float sp = exp2p(__fadd_rn(rp.x, -st.x));
            const float ey = exp2p(__fmaf_rn(p.target[(size_t)row * p.V + y], p.c1, -rp.x));
            const float lp = logf(__fmul_rn(ey, sp)) - logZ;
            p.out_tokens[row] = y;
            p.out_logprobs[row] = lp;
            p.features[(size_t)row * kNFeat + 5] = lp;
        }
        return;
    }
    if (cstar != c) {           // the other stage is free: its chunk was consumed before this one
        ++it;
        if (tid == 0 && !*guard.failed) issue(cstar, it & 1);
        mbar_wait_far(&s_bar[it & 1], (it >> 1) & 1, guard, 3);
        rs = residual_chunk(p, row, cstar, has_draft, s_ring + (it & 1) * (kChunk / 2), st, zt, zq, have);
    }
    hs = warp_hs(rs, lane);
    if (lane == 31) s_red[0][warp] = hs;   // (thread 0 read both halves before its ticket)
    __syncthreads();
    float off = 0.0f;
    for (int w = 0; w < warp; ++w) off = __fadd_rn(off, s_red[0][w]);
    const float P = __fadd_rn(X, __fadd_rn(off, hs));
    const float Pprev = __shfl_up_sync(0xffffffffu, P, 1);
    const float Xl = lane == 0 ? __fadd_rn(X, off) : Pprev;
    const unsigned hit = __ballot_sync(0xffffffffu, P > tau);
    if (lane == 0) s_tstar[warp] = hit ? warp * 32 + __ffs(hit) - 1 : kST;
    __syncthreads();
    int tstar = kST;
#pragma unroll
    for (int w = 0; w < kSW; ++w) tstar = min(tstar, s_tstar[w]);
    if (tid != tstar) return;
    float cc = Xl, Py = 0.0f, P_last = 0.0f, P_first = 0.0f;
    int sel = -1, last_pos = -1, first = -1;
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        if (have[s] && sel < 0) {
            const int v0 = cstar * kChunk + (s * kST + tid) * 4;
            const float rr[4] = {zq[s].x, zq[s].y, zq[s].z, zq[s].w};
            const float pp[4] = {zt[s].x, zt[s].y, zt[s].z, zt[s].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (sel < 0) {
                    if (first < 0) {
                        first = v0 + e;
                        P_first = pp[e];
                    }
                    if (rr[e] > 0.0f) {
                        last_pos = v0 + e;
                        P_last = pp[e];
                    }
                    cc = __fadd_rn(cc, rr[e]);
                    if (cc > tau) {
                        sel = v0 + e;
                        Py = pp[e];
                    }
                }
            }
        }
    }
    const int y = sel >= 0 ? sel : (last_pos >= 0 ? last_pos : (first >= 0 ? first : 0));
    const float Pv = sel >= 0 ? Py : (last_pos >= 0 ? P_last : P_first);
    const float lp = logf(Pv) - logZ;
    p.out_tokens[row] = y;
    p.out_logprobs[row] = lp;
    p.features[(size_t)row * kNFeat + 5] = lp;
}

static inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

size_t reject_sample_workspace_bytes(int B, int k) {
    const size_t rows = (size_t)B * (k + 1);
    size_t n = 0;
    n += align256(sizeof(int) * (size_t)B);               // seq_ticket
    n += 2 * align256(sizeof(float4) * rows * kMaxChunks);  // rec_p, rec_q
    n += 2 * align256(sizeof(float) * rows);              // row_px, row_qx
    n += align256(sizeof(float) * (size_t)B * kMaxChunks);  // seq_rc
    return n + 256;
}

int launch_reject_sample(const float* target, const float* draft, const int* draft_tokens, const double* u_accept,
                         const double* u_resid, int B, int k, int V, float temperature, uint8_t* accept_mask,
                         int* accepted_len, int* out_tokens, float* out_logprobs, float* features, void* workspace,
                         cudaStream_t stream) {
    if (B <= 0) return 0;
    if (k < 0 || k > 64) return set_error("asd_reject_sample: k must be in [0, 64]");
    if (V < 4 || (V & 3)) return set_error("asd_reject_sample: V must be a positive multiple of 4");
    const int NC = (V + kChunk - 1) / kChunk;
    if (NC > kMaxChunks) return set_error("asd_reject_sample: V must be <= %d", kMaxChunks * kChunk);
    const bool greedy = !(temperature > 0.0f);
    if (!greedy && k > 0 && draft == nullptr) return set_error("asd_reject_sample: draft_logits required");
    if ((reinterpret_cast<uintptr_t>(target) & 15) || (draft && (reinterpret_cast<uintptr_t>(draft) & 15)))
        return set_error("asd_reject_sample: logits must be 16-byte aligned");
    const size_t rows = (size_t)B * (k + 1);
    if (rows * NC > 0x7fffffffull) return set_error("asd_reject_sample: too many rows");

    SamplerParams p;
    p.target = target;
    p.draft = draft;
    p.draft_tokens = draft_tokens;
    p.u_accept = u_accept;
    p.u_resid = u_resid;
    p.B = B;
    p.k = k;
    p.V = V;
    p.NC = NC;
    p.greedy = greedy;
    p.c1 = greedy ? 0x1.715476p+0f : (1.0f / temperature) * 0x1.715476p+0f;
    p.accept_mask = accept_mask;
    p.accepted_len = accepted_len;
    p.out_tokens = out_tokens;
    p.out_logprobs = out_logprobs;
    p.features = features;
    int dev = 0;
    ASD_CUDA(cudaGetDevice(&dev));
    p.err = device_wait_word(dev);
    if (wait_word_check(p.err, "asd_reject_sample")) {      // reported once
        *static_cast<volatile int*>(p.err) = 0;
        return -1;
    }
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        uint8_t* q = ws + off;
        off += align256(bytes);
        return q;
    };
    p.seq_ticket = reinterpret_cast<int*>(take(sizeof(int) * (size_t)B));
    p.rec_p = reinterpret_cast<float4*>(take(sizeof(float4) * rows * kMaxChunks));
    p.rec_q = reinterpret_cast<float4*>(take(sizeof(float4) * rows * kMaxChunks));
    p.row_px = reinterpret_cast<float*>(take(sizeof(float) * rows));
    p.row_qx = reinterpret_cast<float*>(take(sizeof(float) * rows));
    p.seq_rc = reinterpret_cast<float*>(take(sizeof(float) * (size_t)B * kMaxChunks));

    static int sms[64];
    static std::once_flag once[64];
    constexpr int kRing = 2 * 2 * kChunk * 4;       // bytes: two chunk pairs, or four chunks
    std::call_once(once[dev & 63], [&] {        // a second thread's first launch must not overtake the attributes
        cudaDeviceGetAttribute(&sms[dev & 63], cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(sampler_stats_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRing);
        cudaFuncSetAttribute(sampler_stats_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRing);
        cudaFuncSetAttribute(sampler_draw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRing);
        prefer_max_smem(sampler_draw_kernel);
        prefer_max_smem(sampler_stats_kernel<false>);
        prefer_max_smem(sampler_stats_kernel<true>);
    });
    const size_t items = rows * NC, resident = (size_t)3 * sms[dev & 63];
    // three draw CTAs fit an SM: one wave of them shares the chunks of all sequences
    p.G = greedy ? 1 : std::max(1, std::min(NC, (int)resident / B));
    const unsigned grid = (unsigned)std::min(items, resident);
    // Greedy calls whose items all fit the chip at once: a ticket per sequence and the merge by its last CTA, one launch.  Such
    // calls are bound by the host: V = 151936, B = 4, k = 1: 13.9 us with two launches, 12.7 so; V = 32000, B = 1, k = 4: 14.0 and
    // 12.7, host time alone 13.3 and 11.7.  More items than that: the ring would wait for a ticket per item, and the second
    // launch is cheaper (B = 4, k = 5: 13.9 us, 18.7 with tickets).
    p.fused = greedy && items <= resident;
    if (greedy)
        sampler_stats_kernel<true><<<grid, kST, kRing, stream>>>(p);
    else
        sampler_stats_kernel<false><<<grid, kST, kRing, stream>>>(p);
    ASD_CUDA(cudaGetLastError());
    count_launch(1);
    if (p.fused) return 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)((size_t)B * p.G));
    cfg.blockDim = dim3(kST);
    cfg.dynamicSmemBytes = greedy ? 0 : kRing;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ASD_CUDA(cudaLaunchKernelEx(&cfg, sampler_draw_kernel, p));
    count_kernel(KERNEL_SAMPLER_DRAW);
    return 0;
}

}  // namespace asd
