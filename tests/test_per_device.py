"""What host code does once per device (csrc/per_device.h), under several host threads: built with g++ against fake runtime calls."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "adaptive-speculative-decoding_b200", "csrc")

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"

static thread_local int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "fake"; }
namespace asd { int set_error(const char*, ...) { return -1; } }
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
static asd::PerDeviceOnce apart;
static std::atomic<int> second_done{0}, waited{0};
static int across() {                                   // device 0's work ends only after device 1's
    ASD_ONCE(apart, {
        if (device == 1) second_done.store(1);
        for (int i = 0; device == 0 && i < 500 && !second_done.load(); ++i) std::this_thread::sleep_for(std::chrono::milliseconds(10));
        if (device == 0 && !second_done.load()) waited.store(1);
    });
    return 0;
}
static std::atomic<int> asked{0}, half{0};
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr attr, int dev) {
    asked.fetch_add(1);
    slowly();
    if (dev == 2 && half.load() < 2) return cudaErrorUnknown;       // a device that cannot be read at first
    *v = (attr == cudaDevAttrMultiProcessorCount ? 100 : 1000) + dev;
    return cudaSuccess;
}
static void limits() {
    asd::DeviceLimits d;
    if (asd::device_limits(&d) || d.sms != 100 + device || d.smem_optin != 1000 + device) half.fetch_add(1);
}
template <typename F>
static void threads(F f) {
    std::vector<std::thread> all;
    for (int i = 0; i < 16; ++i) all.emplace_back([i, f] { device = i & 1; f(); });
    for (auto& t : all) t.join();
}
int main() {
    threads([] { launch(once); });
    const int first = fails_once(), second = fails_once(), third = fails_once();
    printf("%d %d %d %d %d %d\n", calls.load(), overtook.load(), first, second, third, tries);
    threads(limits);
    printf("%d %d", asked.load(), half.load());
    half = 0;
    device = 2;
    for (int i = 0; i < 4; ++i) limits();
    printf(" %d\n", half.load());
    std::thread a([] { device = 0; across(); });
    std::this_thread::sleep_for(std::chrono::milliseconds(50));
    std::thread b([] { device = 1; across(); });
    a.join(), b.join();
    printf("%d %d\n", second_done.load(), waited.load());
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("per_device")
    src, exe = tmp / "t.cpp", tmp / "t"
    src.write_text(PROGRAM)
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", include, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.splitlines()


def test_no_thread_goes_on_before_the_first_has_finished(lines):
    """one call per device, nobody ahead of it; a call that failed is made again"""
    assert lines[0].split() == ["2", "0", "-1", "0", "0", "2"]


def test_no_thread_sees_half_of_a_devices_limits(lines):
    """two questions a device, both answers for everyone; a device that could not be read is asked again"""
    assert lines[1].split() == ["4", "0", "2"]


def test_devices_do_not_wait_for_one_another(lines):
    """a rank's first launch on one device, held up by kernels that wait for a rank on another, whose first launch is still to come"""
    assert lines[2].split() == ["1", "0"]


def test_every_size_of_shared_memory_is_allowed_once():
    """no launch sets the attribute to its own size: a smaller launch on another thread would take it back in between"""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".h")) or name == "per_device.h":
            continue
        text = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r"cudaFuncSetAttribute\([^;]*MaxDynamicSharedMemorySize|allow_max_smem\(", text):
            before = text[:m.start()]
            opened = max(before.rfind(word) for word in ("ASD_ONCE(", "call_once("))
            depth = 0
            for ch in before[opened:]:
                depth += (ch == "(") - (ch == ")")
            assert opened >= 0 and depth > 0, (name, text.count("\n", 0, m.start()) + 1)
