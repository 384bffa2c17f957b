"""GPU: windowed grouped-query attention on tcgen05 (bf16 engines, 17 query rows a tile and more) at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import rivetar_oracle as O  # noqa: E402
from test_rivetar_gpu import close, config, feed, make_engine, rel_err, tokens, window  # noqa: E402


def launches():
    from asd_b200._lib import lib
    return lib().asd_kernel_launches(b"window_tc")


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,size,keep,layout,page_size,portions", [
    (16, 4, 128, 128, 300, 4, None, 16, [130, 1, 8, 9, 300, 1, 2]),           # a window inside the prompt, kept keys of one tile
    (4, 2, 64, 64, 129, 131, "halves", 8, [257, 128, 64, 16]),                # kept keys of two tiles, the second in part
    (2, 2, 128, 64, 128, 0, None, 128, [127, 129, 17, 16, 199]),              # one head a row group: 128 tokens a tile
    (5, 1, 64, 64, 1, 2, None, 32, [26, 25, 24, 51, 180]),                    # rows that no tile fills; a window of one key
    (3, 3, 128, 128, 100000, 0, "halves", 64, [500, 33]),                     # every key, head size 128, one head a row group
    (128, 1, 64, 64, 90, 200, None, 16, [1, 2, 100, 150]),                    # one token a tile, kept keys beyond the window
])
def test_window_attention_on_tcgen05(heads, kv_heads, dim, vdim, size, keep, layout, page_size, portions):
    """the tcgen05 kernel against the mma.sync kernel of the same engine, both held to the oracle; the pool starts out as NaN,
    none of which may reach a result"""
    cfg = config([window(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, size=size, keep_first=keep, rot_dims=dim, scale=0.3,
                         ff=0, layout=layout)])
    w = O.random_model(cfg, seed=41)
    n = sum(portions)
    ids = tokens(n, 96, 42)
    ref, _ = O.forward(cfg, w, ids)
    outs, group = [], heads // kv_heads
    for mode in (2, 1):
        eng = make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512, max_seq_len=1024, page_size=page_size)
        eng.set_option("attn_tiled", mode)
        eng.cache_pool.fill_(255)
        before = launches()
        outs.append(feed(eng, eng.open_sequence(), ids, portions).cpu())
        want = sum(min(128 // group, p) * group >= 17 for p in portions) if mode == 2 else 0
        assert launches() - before == want
        close(eng)
    assert torch.isfinite(outs[0]).all()
    e_tc, e_mma = rel_err(outs[0], ref)[0], rel_err(outs[1], ref)[0]
    assert e_mma < 4e-2 and e_tc < 1.1 * e_mma + 1e-4, (e_tc, e_mma)


def test_window_attention_on_tcgen05_unequal_prompts():
    """prompts of unequal length and a single token of another sequence in one forward, then a step"""
    cfg = config([window(heads=8, kv_heads=2, dim=128, vdim=128, size=150, keep_first=3, rot_dims=64, scale=0.3, ff=0)])
    w = O.random_model(cfg, seed=43)
    lens = [300, 1, 77]
    ids = [tokens(n + 1, 96, 44 + n) for n in lens]
    refs = [O.forward(cfg, w, t)[0] for t in ids]
    eng = make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512, max_seq_len=512)
    slots = [eng.open_sequence() for _ in lens]
    for s, n in zip(slots, lens):
        eng.reserve(s, n + 1)
    before = launches()
    got = eng.forward_ragged([(s, 0, t[:n], list(range(n))) for s, t, n in zip(slots, ids, lens)]).cpu()
    assert launches() == before + 1
    step = eng.forward_ragged([(s, n, t[n:], [0]) for s, t, n in zip(slots, ids, lens)]).cpu()
    at = 0
    for i, n in enumerate(lens):
        assert rel_err(got[at:at + n], refs[i][:n])[0] < 4e-2
        assert rel_err(step[i:i + 1], refs[i][n:])[0] < 4e-2
        at += n
    close(eng)
