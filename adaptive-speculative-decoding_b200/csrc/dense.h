// Dense projection of an engine's activations, y fp32 [M][ldc] = x [M][K] * w[N][K]^T, routed by shape and element
// type: the weight-streaming tcgen05 GEMM (gemm.cu) for bf16 operands it accepts, its tensor-bound CTA-pair form (gemm_tc.cu)
// above 256 tokens, of larger matrices whose rows are not too long above 160, the few-token kernel (linear_few.cu) up to 16, the
// CUDA-core kernel (linear_simt.cu) for fp32 engines and every other shape.  Plans and tensor maps are cached per (call site,
// token count); a call site always passes the same buffers.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <unordered_map>

#include "blocks.h"
#include "gemm.h"

namespace asd {

struct DenseRunner {
    int f32 = 0;                 // 1: fp32 operands (always the CUDA-core kernel)
    int tc_linear = 1;
    int few = 1;                 // few tokens on smaller matrices: linear_few.cu
    int tc_min_rows = 0;         // token count from which the tensor-bound CTA-pair GEMM runs (0: pair_from's rule)
    struct Entry {
        GemmPlan pl;
        TcPlan big;
        CUtensorMap tw, tx;
    };
    std::unordered_map<unsigned long long, Entry> cache;

    void clear() { cache.clear(); }

    // the engines' options that are this runner's; false: another's
    bool set_option(const char* name, int value) {
        if (!strcmp(name, "tc_linear")) {
            tc_linear = value;
        } else if (!strcmp(name, "linear_few")) {
            few = value;
        } else if (!strcmp(name, "tc_min_rows")) {
            tc_min_rows = value > 0 ? value : 1 << 30;
            clear();
        } else {
            return false;
        }
        return true;
    }

    // Above 160 tokens the weight-streaming kernel has room for fewer blocks of its wider tiles, and CTA pairs are the better form of
    // larger matrices whose rows are no longer than they have of them.  The pairs take K in one slice here, 5.4 us per 1024 of it
    // however few their tiles are: longer rows stay with the weight-streaming kernel, which splits them over a cluster.  161 tokens, us
    // alone, weight-streaming and pairs: 2048 x 2048 22.6, 18.5; 6144 x 2048 28.6, 18.5; 4096 x 4096 39.5, 29.1; 12288 x 4096 51.3,
    // 30.9; but 1024 x 4096 14.4, 28.8; 2048 x 6144 28.8, 39.6; 512 x 8192 16.5, 51.2; 4096 x 12288 60.0, 73.9 (256 tokens 70.6, 74.1).
    // Their plain launches cost a step some 4 us each: 4096 x 1024 (14.4, 12.4) made steps of 168 and 192 tokens of width 1024 slower
    // (Rivetar 324 -> 329 and 335 -> 340, Mavipel 457 -> 462).  Steps of 168 tokens of width 2048 with and without pairs: Mavipel 682,
    // 746, Lukopel 714, 727, Dikopel 558, 633, Nobonex 591, 685, Rivetar 477, 513, Mezilix 214, 236; of width 4096 4 to 12 % faster.
    bool pair_from(int M, int N, int K) const {
        if (tc_min_rows > 0) return M >= tc_min_rows;
        const long long elements = (long long)N * K;
        return M > 256 || (M > 160 && K <= N && (elements >= 8 << 20 || (elements >= 4 << 20 && K >= 2048)));
    }

    // Few tokens: linear_few.cu, of rows up to 4096.  Its blocks stage all of a token's K, 196 KB at 6144 and hence one block an SM, and in
    // a step the weight-streaming kernel's launches overlap: 16 tokens, width 2048, down projections of 2048 x 6144 here and there,
    // Rivetar 226 and 220 us, Lukopel 289 and 283, Mavipel 373 and 368; Mavipel of width 4096, output projections of 4096 x 6144, 588
    // and 579 (580 without linear_few.cu at all).  Steps of 1 to 16 tokens with it and without: width 1024 4 to 11 % faster in all six
    // families, 2048 3 to 8 %, 4096 0 to 5 %.
    bool few_from(int M, int K) const { return few && K <= 4096 && !(tc_min_rows > 0 && M >= tc_min_rows); }

    int run(const void* x, const void* w, float* y, int M, int N, int K, int ldc, int key, cudaStream_t s) {
        if (!f32 && tc_linear && (K % 8) == 0 && (ldc % 4) == 0 && K >= 64 && N >= 8 &&
            (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
            (reinterpret_cast<uintptr_t>(y) & 15) == 0) {
            if (few_from(M, K) && linear_few_takes(x, w, M, N, K)) return launch_linear_few(x, w, y, M, N, K, ldc, s);
            const unsigned long long k = ((unsigned long long)key << 32) | (unsigned)M;
            auto it = cache.find(k);
            if (it == cache.end()) {
                Entry t;
                if (make_tmap_bf16(&t.tw, w, N, K, K, 128)) return -1;
                if (pair_from(M, N, K)) {   // above the HBM / tensor ridge: 256 weight rows x MT tokens on a CTA pair
                    if (gemm_tc_plan(&t.big, M, N, K, GEMM_OUT_F32, 1, 0, false)) return -1;
                    if (make_tmap_bf16(&t.tx, x, M, K, K, t.big.MT / 2)) return -1;
                } else {
                    if (gemm_plan(&t.pl, M, N, K, GEMM_OUT_F32, 0, 0, 1)) return -1;
                    if (make_tmap_bf16(&t.tx, x, M, K, K, t.pl.MT)) return -1;
                }
                it = cache.emplace(k, t).first;
            }
            if (pair_from(M, N, K))
                return gemm_tc_launch(it->second.big, it->second.tw, it->second.tx, y, ldc, N, 0, s, false, nullptr);
            return gemm_launch(it->second.pl, it->second.tw, it->second.tx, y, ldc, N, true, s, false);
        }
        SimtLinear L;
        L.a = x, L.a_f32 = f32, L.lda = K;
        L.w = w, L.w_f32 = f32, L.ldw = K;
        L.c = y, L.c_f32 = 1, L.ldc = ldc;
        L.M = M, L.N = N, L.K = K;
        return launch_simt_linear(L, s);
    }
};

}  // namespace asd
