// Internal declarations shared by the translation units of libasd_b200.so.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>

#include "per_device.h"

#define ASD_NUM_FEATURES 6

namespace asd {

int set_error(const char* fmt, ...);  // records the message, returns -1
void count_launch(int n);
// launches of the kernels that a rule chooses between, by name (asd_kernel_launches): what the tests of those rules look at
enum CountedKernel { KERNEL_GEMM, KERNEL_GEMM_PAIR, KERNEL_GEMM_GROUPED, KERNEL_GEMV, KERNEL_ONE_STEP, KERNEL_LINEAR_FEW, KERNEL_ATTENTION_TC, KERNEL_ATTENTION_FEW, KERNEL_LATENT_TC, KERNEL_LATENT_PROMPT, KERNEL_LATENT_STEP, KERNEL_WINDOW_TC, KERNEL_SAMPLER_DRAW, KERNEL_COUNTED };
void count_kernel(CountedKernel k);                     // count_launch(1) too

#define ASD_CUDA(expr)                                                                        \
    do {                                                                                      \
        cudaError_t _e = (expr);                                                              \
        if (_e != cudaSuccess)                                                                \
            return ::asd::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, __LINE__); \
    } while (0)

// ---- Bounded device waits.  A kernel whose barrier does not complete gives up after some seconds (ptx.cuh, mbar_wait), writes
// (kernel << 8 | place) into a word of mapped host memory and ends.  The host reads that word without touching the device: every
// entry point of an engine does before it launches anything, and so does whoever hands results to the host.
enum WaitKernel { WAIT_GEMM = 1, WAIT_GEMM_PAIR, WAIT_ATTENTION, WAIT_SAMPLER, WAIT_LINEAR, WAIT_LATENT, WAIT_PERSIST, WAIT_WINDOW, WAIT_LATENT_PROMPT, WAIT_LATENT_STEP, WAIT_ONE_STEP, WAIT_KERNELS };
inline const char* wait_kernel_name(int k) {
    static const char* const names[] = {"diagnostic kernel", "weight-streaming GEMM", "CTA-pair GEMM", "paged attention", "sampler", "tcgen05 linear",
                                        "latent attention", "persistent forward", "windowed attention", "latent attention of prompts",
                                        "latent attention of few rows", "one-token step"};
    static_assert(sizeof(names) / sizeof(names[0]) == WAIT_KERNELS, "a name for every kernel that waits");
    return names[k >= 1 && k < WAIT_KERNELS ? k : 0];
}
int* wait_word_alloc();                                 // a zeroed word that every device and stream can write, or nullptr
void wait_word_free(int* word);
int wait_word_check(const int* word, const char* who);  // 0, or the error that names the kernel and the place
int* device_wait_word(int dev = -1);                    // of a device (-1: the current one): calls that belong to no engine
int launch_wait_expiry(int* word, cudaStream_t stream); // a wait that runs out (two seconds), for the tests of what follows
extern thread_local int* g_wait_word;
inline int* wait_word() { return g_wait_word ? g_wait_word : device_wait_word(); }
struct WaitScope {                                      // an engine's word, for the launches of one forward on this host thread
    int* prev;
    explicit WaitScope(int* w) : prev(g_wait_word) { g_wait_word = w; }
    ~WaitScope() { g_wait_word = prev; }
};

// Programmatic launch: the grid may become resident while its predecessor drains.  Only for kernels that begin with
// pdl_enter() or otherwise wait (griddepcontrol.wait) before they touch memory, and that keep ptx.cuh's rules on TMEM.
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Every kernel of a forward pass asks for the same (maximum) shared-memory carve-out: an SM only re-partitions
// L1/shared memory when it is idle, so kernels with different carve-outs cannot be co-resident and a
// programmatically launched GEMM could not start streaming weights next to the attention CTAs.
// ASD_CARVEOUT=0 in the environment leaves the driver's per-kernel choice (for A/B runs).
template <typename F>
inline void prefer_max_smem(F* fn) {
    static const bool on = []() {
        const char* v = getenv("ASD_CARVEOUT");
        return !(v && v[0] == '0');
    }();
    if (on) cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}

// Per-engine tuning knobs (engine options).  They used to be process globals, so an option set on the draft
// engine changed the target's plans; now every engine owns a Tuning and installs it for the duration of one
// forward() on the calling host thread (thread_local pointer), which also makes concurrent forwards of different
// engines from different host threads independent.
struct Tuning {
    int gemm_early_trigger = 0;
    int gemm_headroom = 1;
    int gemm_recv_dedicated = 1;
    int gemm_next_mb = 0;   // L2 budget (MB) for the next kernel's weights; measured neutral, off
    int glue_pdl = 1;       // launch the glue kernels programmatically (they wait on griddepcontrol)
    int attn_wide = 0;
    int attn_dbg = 0;       // diagnostics (tcgen05 attention): 1 = skip the softmax arithmetic, 2 = also skip the fold
    int gemm_big = 1;       // token counts above the HBM/tensor ridge use the 2-CTA tensor-bound GEMM
};
extern thread_local const Tuning* g_tuning;
inline const Tuning& tuning() {
    static const Tuning defaults;
    return g_tuning ? *g_tuning : defaults;
}
struct TuningScope {
    const Tuning* prev;
    explicit TuningScope(const Tuning* t) : prev(g_tuning) { g_tuning = t; }
    ~TuningScope() { g_tuning = prev; }
};

int sm_count();      // multiprocessors of the current device

// sampler.cu
size_t reject_sample_workspace_bytes(int B, int k);
int launch_reject_sample(const float* target, const float* draft, const int* draft_tokens, const double* u_accept,
                         const double* u_resid, int B, int k, int V, float temperature, uint8_t* accept_mask,
                         int* accepted_len, int* out_tokens, float* out_logprobs, float* features, void* workspace,
                         cudaStream_t stream);

// stop_rule.cu
int launch_stop_rule(const double* p, const double* C, int n, int L, double lam, int risk_adjustment, double alpha,
                     double beta, int* k_star, double* J, cudaStream_t stream, const double* lam_rows = nullptr);
int launch_cascade_decide(const float* features, const int* n_tokens, int n, int T, const double* scalars, const float* w1,
                          const float* b1, const float* w2, const float* b2, int fdim, const double* prev_p,
                          const double* C, int L, int stage_idx, int mode, double lam, int risk, double n_obs,
                          double alpha, double beta, double* prob, int* stop, int* k_star, cudaStream_t stream);
int stop_rule_rows_host(const double* p, const double* C, const double* lam, int n, int L, int risk_adjustment,
                        double alpha, double beta, int* k_star, double* J);
int stop_rule_host(const double* p, const double* C, int L, double lam, int risk_adjustment, double alpha,
                   double beta, double* J);
double bayesian_adjustment_host(double p_hat, double n_obs, double alpha, double beta);

}  // namespace asd
