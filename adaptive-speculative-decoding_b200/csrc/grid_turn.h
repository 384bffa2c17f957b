// Grids whose CTAs wait for one another (one_step.cu, forward_persist.cu): one at a time on a device, whatever the streams and engines.
#pragma once
#include <cuda_runtime.h>

#include <mutex>

namespace asd {

int set_error(const char* fmt, ...);     // records the message, returns -1

constexpr int kTurnDevices = 64;
struct GridTurn {
    std::mutex m;
    cudaEvent_t done = nullptr;          // behind the last such grid of the device; lives as long as the process
};
inline GridTurn* grid_turns() {
    static GridTurn turns[kTurnDevices];
    return turns;
}

// `launch` (which returns cudaError_t) behind the last such grid of the current device: two of them would share the SMs between them and
// each wait for CTAs that find no place.  Returns 0, -1 (error), or 1: nothing was launched, a chain of kernels has to do.  That is so for a
// captured step, which could not keep its turn when it is replayed, and where the device refuses the grid as a whole (a context with a part
// of the SMs).
template <typename F>
int grid_in_turn(cudaStream_t stream, F&& launch) {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    int device = 0;
    cudaError_t e = cudaStreamIsCapturing(stream, &capturing);
    if (e == cudaSuccess) e = cudaGetDevice(&device);
    if (e == cudaSuccess && (capturing != cudaStreamCaptureStatusNone || device >= kTurnDevices)) return 1;
    if (e == cudaSuccess) {
        GridTurn& turn = grid_turns()[device];
        std::lock_guard<std::mutex> lock(turn.m);
        if (!turn.done) e = cudaEventCreateWithFlags(&turn.done, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, turn.done, 0);       // (nothing recorded yet: no wait)
        if (e == cudaSuccess) e = launch();
        if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
            cudaGetLastError();          // nobody else's error
            return 1;
        }
        if (e == cudaSuccess) e = cudaEventRecord(turn.done, stream);
    }
    return e == cudaSuccess ? 0 : set_error("launch of a grid that waits for itself: %s", cudaGetErrorString(e));
}

}  // namespace asd
