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

// Sizes that one_step.cu takes on `grid` CTAs.  Every CTA shows that it has read its input by publishing rows of its own, and the others
// wait for all of these before they overwrite what it read: each must have rows of the hidden size, of gate | up and of QKV (pairs of
// rows).  Of QKV because the O projection overwrites the residual that the QKV projection reads: it has waited for the heads, and the
// heads for every row of QKV.
constexpr int kOsPanel = 16;               // weight rows of a panel
constexpr int kOsMaxPanels = 8;            // of a phase
inline bool one_step_sizes(const OneStep& s, int grid) {
    if (s.n_layers <= 0 || s.n_layers > kOneMaxLayers || (s.hd != 64 && s.hd != 128) || s.nkv <= 0 || s.nh % s.nkv || s.nh > grid) return false;
    if (s.h % 16 || s.qdim % 16 || s.ffn % 16 || s.h < grid || s.ffn / 2 < grid || s.nqkv / 2 < grid || grid > 256) return false;
    auto most = [&](int n) { return (n + grid - 1) / grid; };
    return most(s.h) <= 32 && 2 * most(s.nqkv / 2) <= kOsMaxPanels * kOsPanel && 4 * most(s.ffn / 2) <= kOsMaxPanels * kOsPanel;
}

int one_step_sums();
size_t one_step_bytes(int h, int nqkv, int qdim, int ffn);
bool one_step_takes(const OneStep& s);     // on the current device
// 0, -1 (error), or 1: sizes that it does not take after all or not its turn (grid_turn.h), nothing launched
int one_step_launch(const OneStep& s, int max_kv_len, cudaStream_t stream);
int preload_one_step();

}  // namespace asd
