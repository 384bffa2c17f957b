"""CPU: the error of a wait that ran out names its kernel (csrc/asd_internal.h), built with g++."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(__file__), "..", "adaptive-speculative-decoding_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "asd_internal.h"

int main() {
    using namespace asd;
    for (int k : {WAIT_GEMM, WAIT_GEMM_PAIR, WAIT_ATTENTION, WAIT_SAMPLER, WAIT_LINEAR, WAIT_LATENT, WAIT_PERSIST, WAIT_WINDOW, WAIT_LATENT_PROMPT,
                  WAIT_LATENT_STEP, WAIT_ONE_STEP})
        puts(wait_kernel_name(k));
    for (int k : {0, -1, (int)WAIT_KERNELS, 1 << 20}) puts(wait_kernel_name(k));
}
"""


def test_every_kernel_that_waits_has_its_name(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-I", include, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    names = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.splitlines()
    assert names[:11] == ["weight-streaming GEMM", "CTA-pair GEMM", "paged attention", "sampler", "tcgen05 linear", "latent attention",
                          "persistent forward", "windowed attention", "latent attention of prompts", "latent attention of few rows", "one-token step"]
    assert names[11:] == ["diagnostic kernel"] * 4
