"""CPU: every interleaving of the warps that pass a tile of scores on through parity barriers (csrc/latent_step_tc.cu): none may be lapped.
A parity wait only tells odd phases from even ones, so whoever waits must have looked before the phase after the next one completes."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "adaptive-speculative-decoding_b200", "csrc")
WARPS, TILES = 4, 4


def stuck(readers):
    """The product warp commits the scores of a tile (s_full) when `readers` of the four softmax warps have arrived for the tile before
    (s_read); those wait for the scores, the first `readers` of them arrive, and all four meet before the next tile.  Walks all
    interleavings; True if one of them ends with a warp waiting for ever."""
    # committed tiles; per warp: steps done (two a tile: looked, met)
    start = (0, (0,) * WARPS)
    seen, todo = {start}, [start]
    while todo:
        committed, warps = todo.pop()
        nxt = []
        # a phase of s_read is complete when every reader has looked at its tile; the product warp takes these in order and at once
        reads = min((w + 1) // 2 for w in warps[:readers])
        if committed < TILES and (committed == 0 or reads >= committed):
            nxt.append((committed + 1, warps))
        for i, w in enumerate(warps):
            tile = w // 2
            if tile == TILES:
                continue
            if w % 2 == 0:                                             # wait for phase `tile` of s_full, by its parity
                go = committed > 0 and (committed - 1) % 2 == tile % 2
            else:                                                      # the barrier of the four
                go = all(v >= w for v in warps)
            if go:
                nxt.append((committed, warps[:i] + (w + 1,) + warps[i + 1:]))
        if not nxt and (committed < TILES or any(w < 2 * TILES for w in warps)):
            return True
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


def test_the_walk_finds_a_lapped_barrier():
    assert stuck(3) and not stuck(4)


@pytest.mark.parametrize("name", ["latent_step_tc.cu", "latent_prompt_tc.cu"])
def test_scores_wait_for_every_warp_that_looks_for_them(name):
    text = open(os.path.join(CSRC, name)).read()
    assert not stuck(int(re.search(r"mbar_init\(&B->s_read, (\d)\)", text).group(1)))


@pytest.mark.parametrize("name", ["latent_step_tc.cu", "latent_prompt_tc.cu"])
def test_a_warp_arrives_when_all_its_lanes_have_looked(name):
    """lanes look one by one: the one that arrives for its warp does so behind a __syncwarp"""
    lines = [l.split("//")[0].strip() for l in open(os.path.join(CSRC, name))]
    lines = [l for l in lines if l]
    at = [i for i, l in enumerate(lines) if "mbar_arrive(&B->s_read)" in l]
    assert at
    for i in at:
        assert lines[i] == "if (lane == 0) mbar_arrive(&B->s_read);" and lines[i - 1] == "__syncwarp();", lines[i - 1:i + 1]
