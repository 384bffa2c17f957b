// Host-side interface of the one-token step (one_step.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>

namespace asd {

struct OneLayer {
    const __nv_bfloat16 *wqkv, *bqkv, *wo, *wgu, *wdown, *ln1, *ln2;
    __nv_bfloat16 *k_cache, *v_cache;
};
constexpr int kOneMaxLayers = 40;          // they travel as launch parameters

struct OneStep {
    OneLayer layers[kOneMaxLayers];
    int n_layers, h, nh, nkv, hd, nqkv, qdim, ffn, page_size, max_pages;
    float eps;
    const __nv_bfloat16 *embed, *final_norm;
    const float* inv_freq;
    const int *page_table, *tokens, *positions, *token_slot;
    __nv_bfloat16* x_out;                  // [h] bf16(residual x final norm's weight)
    float* sums_out;                       // [one_step_sums()] parts of the residual's sum of squares
    void* work;                            // one_step_bytes() of device memory, zeroed once; one step at a time uses it
    unsigned* sync;                        // (filled by the launch)
    int* err;                              // where a wait that ran out is reported
};

int one_step_sums();
size_t one_step_bytes(int h, int nqkv, int qdim, int ffn);
bool one_step_takes(const OneStep& s);
// 0, -1 (error), or 1: sizes that it does not take after all, nothing launched
int one_step_launch(const OneStep& s, int max_kv_len, cudaStream_t stream);
int preload_one_step();

}  // namespace asd
