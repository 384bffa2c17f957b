"""GPU: the gated recurrence at the edges of its split: 8 key rows x 4 columns of the state per thread, 32 or 16 columns per CTA,
positions staged 4 to 16 at a time (as many as the forward's average run; 1 in steps), 16-byte copies where the sizes allow."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import rivetar_oracle as O  # noqa: E402
from test_rivetar_gpu import close, config, feed, gla, make_engine, rel_err, tokens  # noqa: E402


# one row group, whole groups and a rest of one, sizes that are no multiple of four, the largest group counts of both instances
@pytest.mark.parametrize("dim,vdim,rank", [(8, 4, 8), (72, 36, 1), (65, 34, 3), (128, 128, 32), (260, 32, 5), (512, 33, 2),
                                           (520, 12, 2), (1024, 8, 1)])
def test_state_tiles_and_chunks(dim, vdim, rank):
    cfg = config([gla(heads=2, dim=dim, vdim=vdim, tau=16.0, decay_rank=rank)])
    w = O.random_model(cfg, seed=21)
    ids = tokens(47, 96, 22)
    ref, _ = O.forward(cfg, w, ids)
    eng = make_engine(cfg, w, max_tokens=64)
    one = feed(eng, eng.open_sequence(), ids, [])
    # runs of 1, 2, 4, 5, 16 and 17 positions: the sums of a position do not depend on the cut
    cut = feed(eng, eng.open_sequence(), ids, [1, 2, 4, 5, 16, 17, 1, 1])
    assert rel_err(one, ref)[1] < 2e-4          # as the other tests of this engine: far below one missed position
    assert torch.equal(one, cut)
    close(eng)


# warps with row groups beyond the key size, whole and in part; steps of 16 columns a CTA that the values do not fill
@pytest.mark.parametrize("dim,vdim", [(16, 8), (24, 40), (20, 33), (264, 36), (300, 20), (516, 44)])
def test_row_groups_beyond_the_key_size(dim, vdim):
    cfg = config([gla(heads=2, dim=dim, vdim=vdim, tau=16.0, decay_rank=4)])
    w = O.random_model(cfg, seed=23)
    ids = tokens(24, 96, 24)
    ref, _ = O.forward(cfg, w, ids)
    eng = make_engine(cfg, w, max_tokens=64)
    one = feed(eng, eng.open_sequence(), ids, [])
    cut = feed(eng, eng.open_sequence(), ids, [1, 1, 5, 1, 9, 1])
    assert rel_err(one, ref)[1] < 2e-4          # as above
    assert torch.equal(one, cut)
    close(eng)


def test_chunks_of_an_unequal_batch():
    """one run of 100 positions beside nine single tokens: chunks of the average run (11), which no run of its own has, then a step of
    all of them; bit for bit what every sequence gets alone"""
    cfg = config([gla(heads=2, dim=72, vdim=36, tau=16.0, decay_rank=4)])
    w = O.random_model(cfg, seed=25)
    lens = [1, 1, 1, 100, 1, 1, 1, 1, 1, 1]
    ids = [tokens(n + 7, 96, 26 + i) for i, n in enumerate(lens)]       # six positions before, one after
    eng = make_engine(cfg, w, max_tokens=128, max_seqs=20)
    alone, slots = [], []
    for t, n in zip(ids, lens):
        alone.append(feed(eng, eng.open_sequence(), t, [6, n, 1]))
    for t in ids:
        slots.append(eng.open_sequence())
        eng.reserve(slots[-1], len(t))
        eng.forward_ragged([(slots[-1], 0, t[:6], [5])])
    got = eng.forward_ragged([(s, 6, t[6:6 + n], list(range(n))) for s, t, n in zip(slots, ids, lens)])
    step = eng.forward_ragged([(s, 6 + n, t[6 + n:], [0]) for s, t, n in zip(slots, ids, lens)])
    assert torch.equal(got, torch.cat([a[6:6 + n] for a, n in zip(alone, lens)]))
    assert torch.equal(step, torch.cat([a[6 + n:] for a, n in zip(alone, lens)]))
    close(eng)


# two sequences: 192, 180 and 160 CTAs of 32 columns, 144, 120 and 80 of 48
@pytest.mark.parametrize("heads,dim,vdim", [(24, 128, 128), (30, 20, 66), (40, 72, 48)])
def test_wider_column_tiles(heads, dim, vdim):
    """as many heads and sequences as take 48 columns a CTA: bit for bit what each sequence gets alone, by 32"""
    cfg = config([gla(heads=heads, dim=dim, vdim=vdim, tau=16.0, decay_rank=4)])
    w = O.random_model(cfg, seed=31)
    ids = [tokens(n, 96, 32 + n) for n in (41, 19)]
    eng = make_engine(cfg, w, max_tokens=64, max_seqs=4)
    alone = [feed(eng, eng.open_sequence(), t, []) for t in ids]
    slots = [eng.open_sequence() for _ in ids]
    for s, t in zip(slots, ids):
        eng.reserve(s, len(t))
    got = eng.forward_ragged([(s, 0, t, list(range(len(t)))) for s, t in zip(slots, ids)])
    assert rel_err(got[:41], O.forward(cfg, w, ids[0])[0])[1] < 2e-4        # as above
    assert torch.equal(got, torch.cat(alone))
    close(eng)
