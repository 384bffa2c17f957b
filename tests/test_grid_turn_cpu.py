"""CPU: grids whose CTAs wait for one another take turns on a device (csrc/grid_turn.h): built with g++ against fake runtime calls."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "adaptive-speculative-decoding_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "grid_turn.h"

static thread_local int device = 0;
static bool capturing = false;
static int events = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "fake"; }
extern "C" cudaError_t cudaGetLastError() { printf("cleared "); return cudaSuccess; }
extern "C" cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
extern "C" cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)(size_t)++events; return cudaSuccess; }
extern "C" cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { printf("wait%zu:%zu ", (size_t)s, (size_t)e); return cudaSuccess; }
extern "C" cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { printf("record%zu:%zu ", (size_t)s, (size_t)e); return cudaSuccess; }
namespace asd { int set_error(const char*, ...) { return -1; } }

static int go(size_t stream, cudaError_t result) {
    return asd::grid_in_turn((cudaStream_t)stream, [&] { printf("launch "); return result; });
}
int main() {
    printf("= %d\n", go(1, cudaSuccess));
    printf("= %d\n", go(2, cudaSuccess));                                  // another stream, the same event
    printf("= %d\n", go(2, cudaErrorInvalidValue));
    capturing = true;
    printf("= %d\n", go(1, cudaSuccess));
    capturing = false;
    device = 1;
    printf("= %d\n", go(3, cudaSuccess));                                  // a device of its own
    device = 64;
    printf("= %d\n", go(3, cudaSuccess));
    device = 0;
    printf("= %d\n", go(1, cudaErrorCooperativeLaunchTooLarge));
    printf("= %d\n", go(1, cudaErrorNotSupported));
    printf("= %d\n", go(1, cudaSuccess));
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("grid_turn")
    src, exe = tmp / "t.cpp", tmp / "t"
    src.write_text(PROGRAM)
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", include, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.splitlines()


def test_one_grid_behind_another(lines):
    """every launch waits for the one before on its device, whatever the stream, and none joins a capture"""
    assert lines[0] == "wait1:1 launch record1:1 = 0"
    assert lines[1] == "wait2:1 launch record2:1 = 0"
    assert lines[2] == "wait2:1 launch = -1"
    assert lines[3] == "= 1"
    assert lines[4] == "wait3:2 launch record3:2 = 0"
    assert lines[5] == "= 1"


def test_a_refused_grid_is_no_error(lines):
    """a grid that finds no room as a whole (fewer SMs than the device has, say) leaves the step to a chain of kernels, and no error behind"""
    assert lines[6] == "wait1:1 launch cleared = 1"
    assert lines[7] == "wait1:1 launch cleared = 1"
    assert lines[8] == "wait1:1 launch record1:1 = 0"


def test_every_such_grid_takes_its_turn():
    """cooperative launches all go through it"""
    found = 0
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        if "cudaLaunchAttributeCooperative" not in text:
            continue
        for part in text.split("cudaLaunchAttributeCooperative;")[1:]:
            found += 1
            assert "grid_in_turn(" in part[:part.index("cudaLaunchKernelEx(")], name
    assert found == 2
