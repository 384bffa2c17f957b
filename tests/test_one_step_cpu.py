"""CPU: the sizes that the one-token step takes (csrc/one_step.h), built with g++, against an account of what every CTA of its grid has."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "adaptive-speculative-decoding_b200", "csrc")

# nh heads and nkv key/value heads of hd; the rows are shared out as one_step.cu does
PROGRAM = r"""
#include <cstdio>
#include "one_step.h"

int main() {
    long long h, nh, nkv, hd, ffn, grid;
    while (scanf("%lld %lld %lld %lld %lld %lld", &h, &nh, &nkv, &hd, &ffn, &grid) == 6) {
        asd::OneStep s = {};
        s.n_layers = 2, s.h = h, s.nh = nh, s.nkv = nkv, s.hd = hd, s.ffn = ffn;
        s.qdim = nh * hd, s.nqkv = (nh + 2 * nkv) * hd;
        printf("%d\n", (int)asd::one_step_sizes(s, grid));
    }
}
"""


@pytest.fixture(scope="module")
def takes(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("one_step")
    src, exe = tmp / "t.cpp", tmp / "t"
    src.write_text(PROGRAM)
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-I", include, "-I", CSRC, str(src), "-o", str(exe)], check=True)

    def ask(sizes):
        text = "\n".join(" ".join(map(str, x)) for x in sizes)
        return [line == "1" for line in subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True, timeout=60).stdout.split()]

    return ask


def shares(n, grid):
    return [n * (c + 1) // grid - n * c // grid for c in range(grid)]


@pytest.mark.parametrize("grid", [132, 148, 160])
def test_every_cta_has_rows_to_publish(takes, grid):
    """a CTA without rows of a matrix publishes nothing in its phase, and nobody knows when it has read the input"""
    sizes = [(h, nh, nkv, hd, ffn, grid) for h in (144, 160, 256, 896, 4736) for nh, nkv in ((1, 1), (2, 1), (4, 2), (8, 1), (14, 2))
             for hd in (64, 128) for ffn in (16, 144, 256, 272, 288, 304, 320, 512, 4864)]
    took = 0
    for size, yes in zip(sizes, takes(sizes)):
        h, nh, nkv, hd, ffn, _ = size
        if yes:
            took += 1
            assert min(shares(h, grid)) > 0 and min(shares(ffn // 2, grid)) > 0, size
            assert min(shares((nh + 2 * nkv) * hd // 2, grid)) > 0, size
    assert took > 20


def test_widths_it_is_made_for(takes):
    assert takes([(896, 14, 2, 64, 4864, 148), (1536, 12, 2, 128, 8960, 148)]) == [True, True]
