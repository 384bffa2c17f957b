"""What host code does once per device (csrc/per_device.h), under several host threads: built with g++ against fake runtime calls."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(__file__), "..", "adaptive-speculative-decoding_b200", "csrc")

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"

static thread_local int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
static void slowly() { std::this_thread::sleep_for(std::chrono::milliseconds(20)); }

static std::atomic<int> calls{0}, ready[2], overtook{0};
static int launch(asd::PerDeviceOnce& once) {           // as a launch: its attribute first
    ASD_ONCE(once, {
        calls.fetch_add(1);
        slowly();
        ready[device].store(1);
    });
    if (!ready[device].load()) overtook.fetch_add(1);
    return 0;
}
static asd::PerDeviceOnce once, failing;
static int tries = 0;
static int fails_once() {
    ASD_ONCE(failing, if (++tries == 1) return -1);
    return 0;
}
int main() {
    std::vector<std::thread> all;
    for (int i = 0; i < 16; ++i) all.emplace_back([i] { device = i & 1; launch(once); });
    for (auto& t : all) t.join();
    const int first = fails_once(), second = fails_once(), third = fails_once();
    printf("%d %d %d %d %d %d\n", calls.load(), overtook.load(), first, second, third, tries);
}
"""


def run(tmp_path, program):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(program)
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", include, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.split()


def test_no_thread_goes_on_before_the_first_has_finished(tmp_path):
    """one call per device, nobody ahead of it; a call that failed is made again"""
    assert run(tmp_path, PROGRAM) == ["2", "0", "-1", "0", "0", "2"]
