// Process-wide state every other translation unit of libasd_b200.so links against: the thread-local error
// message, the launch counter and the per-thread tuning pointer.  Kept apart from the entry points of the individual
// components so that a library holding only some of them (one model family) still links.
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <atomic>
#include <mutex>
#include <vector>

#include "../../include/asd_b200.h"
#include "asd_internal.h"
#include "ptx.cuh"

namespace asd {

static thread_local char g_err[512] = "";
thread_local const Tuning* g_tuning = nullptr;
static std::atomic<long long> g_launches{0};

int set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return -1;
}
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
static std::atomic<long long> g_kernels[KERNEL_COUNTED];
void count_kernel(CountedKernel k) {
    g_kernels[k].fetch_add(1, std::memory_order_relaxed);
    count_launch(1);
}

int sm_count() {
    static std::atomic<int> counts[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = 0;
    int n = counts[dev & 63].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 1;
        counts[dev & 63].store(n, std::memory_order_relaxed);
    }
    return n;
}

// ---- bounded device waits
thread_local int* g_wait_word = nullptr;

// Words come from pages of 64 (one pinned allocation costs an engine's creation milliseconds); a page stays for the next engines.
static std::mutex g_words_lock;
static std::vector<int*> g_words_free;
constexpr int kWordStride = 16;      // ints: a cache line each

int* wait_word_alloc() {
    std::lock_guard<std::mutex> lock(g_words_lock);
    if (g_words_free.empty()) {
        // an allocation is not a stream operation, but a capture in the default mode would refuse it
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        void* p = nullptr;
        const cudaError_t rc = cudaHostAlloc(&p, 64 * kWordStride * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (rc != cudaSuccess) {
            set_error("allocation of device wait words failed: %s", cudaGetErrorString(rc));
            return nullptr;
        }
        for (int i = 63; i >= 0; --i) g_words_free.push_back(static_cast<int*>(p) + i * kWordStride);
    }
    int* w = g_words_free.back();
    g_words_free.pop_back();
    *static_cast<volatile int*>(w) = 0;
    return w;
}
void wait_word_free(int* word) {        // after the engine's last kernel has ended
    if (!word) return;
    std::lock_guard<std::mutex> lock(g_words_lock);
    g_words_free.push_back(word);
}
int wait_word_check(const int* word, const char* who) {
    const int v = word ? *static_cast<const volatile int*>(word) : 0;
    if (v == 0) return 0;
    return set_error("%s: a bounded wait of an earlier launch ran out (%s, place %d); its results are not valid", who,
                     wait_kernel_name(v >> 8), v & 255);
}
// one CTA that waits on a barrier nobody arrives at, with the shortest limit
__global__ void wait_expiry_kernel(int* err) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int failed;
    const WaitGuard guard{&failed, err, 0, 0};
    mbar_init(&bar, 1);
    failed = 0;
    mbar_wait_timed(&bar, 0, guard, 255);
    wait_settle(guard);
}
int launch_wait_expiry(int* word, cudaStream_t stream) {
    wait_expiry_kernel<<<1, 1, 0, stream>>>(word);
    ASD_CUDA(cudaGetLastError());
    return 0;
}
int* device_wait_word(int dev) {
    static std::atomic<int*> words[64] = {};
    if (dev < 0 && cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    if (dev < 0 || dev >= 64) return nullptr;
    int* w = words[dev].load(std::memory_order_acquire);
    if (w) return w;
    static std::mutex m;
    std::lock_guard<std::mutex> lock(m);
    if (!words[dev].load(std::memory_order_relaxed)) words[dev].store(wait_word_alloc(), std::memory_order_release);
    return words[dev].load(std::memory_order_relaxed);
}

}  // namespace asd

using namespace asd;

extern "C" {

int asd_abi_version(void) { return ASD_B200_ABI_VERSION; }
const char* asd_last_error(void) { return g_err; }
long long asd_launch_count(void) { return g_launches.load(); }
void asd_reset_launch_count(void) { g_launches.store(0); }
long long asd_kernel_launches(const char* name) {
    static const char* const names[KERNEL_COUNTED] = {"gemm", "gemm_pair", "gemm_grouped", "gemv", "one_step", "linear_few", "attention_tc", "attention_few", "latent_tc", "latent_prompt", "latent_step", "window_tc", "sampler_draw"};
    for (int i = 0; name && i < KERNEL_COUNTED; ++i)
        if (!strcmp(name, names[i])) return g_kernels[i].load();
    return set_error("asd_kernel_launches: unknown kernel %s", name ? name : "(null)");
}
int asd_debug_wait_expiry(void* stream) { return launch_wait_expiry(device_wait_word(), static_cast<cudaStream_t>(stream)); }
int asd_wait_error(void) {
    int* w = device_wait_word();
    const int rc = wait_word_check(w, "asd_wait_error");
    if (rc) *static_cast<volatile int*>(w) = 0;
    return rc;
}

}  // extern "C"
