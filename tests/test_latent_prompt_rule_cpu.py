"""CPU: which prompts' latent attention goes through head space (csrc/blocks.h: latent_prompt_gain), built with g++, held to measured calls."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "adaptive-speculative-decoding_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "blocks.h"

int main() {
    int heads, R, M, nseq, q, kv;
    while (scanf("%d %d %d %d %d %d", &heads, &R, &M, &nseq, &q, &kv) == 6) printf("%.9g\n", asd::latent_prompt_gain(heads, R, 148, M, nseq, q, kv));
}
"""


@pytest.fixture(scope="module")
def gain(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("latent_rule")
    src, exe = tmp / "t.cpp", tmp / "t"
    src.write_text(PROGRAM)
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-I", include, "-I", CSRC, str(src), "-o", str(exe)], check=True)

    def ask(calls):
        text = "\n".join(" ".join(map(str, c)) for c in calls)
        return [float(x) for x in subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True, timeout=60).stdout.split()]

    return ask


def test_equal_sequences(gain):
    """as the fit over equal calls has it"""
    up = lambda a, b: -(-a // b)
    calls, want = [], []
    for heads in (4, 8, 16, 32, 130):
        for R in (256, 512):
            for n in (1, 4, 16):
                for q in (9, 17, 128, 129, 256):
                    for ctx in (0, 120, 2560):
                        kt, th, tq = up(ctx + q, 128), 1e-3 * heads, min(max(128 // heads, 1), q)
                        here, latent = n * heads * up(q, 128) / 148, n * up(q, tq) * up(heads, 128) * (2 if R > 256 else 1) / 148
                        calls.append((heads, R, n * q, n, q, ctx + q))
                        want.append(12 + 1.85 * th * n * q + 9.06 * latent * kt - (0.512 * th * kt * 128 * n + 2.58 * max(here, 1.0) * kt))
    assert gain(calls) == pytest.approx(want, rel=1e-6, abs=1e-6)


# heads, tokens, sequences, most tokens and positions of one; us of a layer in latent and in head space
UNEQUAL = [
    (32, 195, 24, 172, 1109, 382, 768), (16, 195, 24, 172, 1109, 261, 464), (32, 130, 12, 119, 1659, 379, 570), (32, 792, 32, 761, 761, 622, 859),
    (32, 143, 16, 128, 257, 301, 400), (16, 527, 16, 512, 512, 263, 306), (32, 143, 16, 128, 128, 291, 320), (16, 271, 16, 256, 256, 208, 217),
    (8, 143, 16, 128, 257, 155, 165),
    (16, 1280, 4, 512, 512, 420, 341), (8, 1040, 2, 1024, 1024, 296, 229), (32, 2560, 8, 512, 512, 1201, 953), (16, 960, 3, 512, 2560, 581, 355),
    (32, 480, 3, 256, 2304, 655, 503), (8, 515, 4, 512, 2501, 346, 256),
]


def test_unequal_sequences(gain):
    """one prompt among short ones stays in latent space, prompts of some length each go through head space"""
    for c, g in zip(UNEQUAL, gain([(c[0], 512) + c[1:5] for c in UNEQUAL])):
        assert (g > 0) == (c[6] < c[5]), (c, g)
