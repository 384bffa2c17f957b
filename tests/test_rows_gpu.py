"""GPU: row kernels at the edges of their split: one, two and four groups of four elements per thread, rows that end inside the
last warp, the widest row kept in registers and the first one that is not."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import test_mezilix_gpu as mz  # noqa: E402
from oracle import mezilix_oracle, rivetar_oracle as O  # noqa: E402
from test_rivetar_gpu import close, config, feed, gla, latent, make_engine, rel_err, tokens  # noqa: E402


@pytest.mark.parametrize("width,ff,q_rank", [(36, 132, 20), (1024, 1028, 1028), (1028, 2052, 132), (2052, 4100, 260), (16384, 36, 8),
                                             (16388, 36, 6)])
def test_closes_norms_and_polynomials_of_odd_widths(width, ff, q_rank):
    cfg = config([gla(heads=1, dim=8, vdim=8, ff=ff), latent(heads=1, dim=8, rot_dim=4, vdim=8, kv_rank=12, q_rank=q_rank, ff=0)],
                 width=width)
    w = O.random_model(cfg, seed=31)
    ids = tokens(9, 96, 32)
    ref, _ = O.forward(cfg, w, ids)
    eng = make_engine(cfg, w)
    one = feed(eng, eng.open_sequence(), ids, [])
    cut = feed(eng, eng.open_sequence(), ids, [4, 1])
    assert rel_err(one, ref)[1] < 2e-4          # as the other tests of this engine
    assert torch.equal(one, cut)                # a row's sums do not depend on the rows beside it
    close(eng)


@pytest.mark.parametrize("width", [36, 1024, 1028, 2052, 16384, 16388, 1026])
def test_pair_embedding_shift_and_depth_weighted_close_of_odd_widths(width):
    cfg = mz.config([mz.layer(heads=1, dim=8, rot_dim=4, vdim=8, kv_rank=12, experts=3, top=2, ff=8),
                     mz.layer(heads=1, dim=8, rot_dim=4, vdim=8, kv_rank=12, experts=0)], width=width)
    w = mezilix_oracle.random_model(cfg, seed=33)
    ids = mz.tokens(9, 96, 34)
    ref, _ = mezilix_oracle.forward(cfg, w, ids)
    eng = mz.make_engine(cfg, w)
    one = mz.feed(eng, eng.open_sequence(), ids, [])
    cut = mz.feed(eng, eng.open_sequence(), ids, [4, 1])
    assert mz.rel_err(one, ref)[1] < 2e-4
    assert torch.equal(one, cut)
    mz.close(eng)
