"""GPU: latent attention of few query rows (latent_step_tc.cu) at the edges of its tiles, row groups and key shares."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import test_mezilix_gpu as mz  # noqa: E402
from oracle import mezilix_oracle as O  # noqa: E402


def _config(heads, kv_rank, window, scale):
    return mz.config([mz.layer(heads=heads, dim=16, rot_dim=64, vdim=16, kv_rank=kv_rank, window=window, scale=scale, experts=0)], width=64)


@pytest.mark.parametrize("heads,kv_rank,window,page_size,scale,portions", [
    (16, 512, 1 << 20, 16, 0.3, [63, 1, 1, 1, 2, 60, 1, 1, 2, 3, 4]),     # one key short of a tile, a whole one, one beyond; two row tiles
    (8, 512, 1 << 20, 8, 0.3, [130, 4, 8, 1, 300, 1]),                    # four tokens a row tile; shares of the keys
    (32, 384, 100, 64, 1.0, [90, 1, 1, 40, 2, 1]),                        # a window inside two tiles, a sharp softmax
    (40, 128, 1 << 20, 128, 0.2, [129, 1, 1]),                            # two head groups of a single token, a page of two tiles
    (3, 256, 70, 32, 0.5, [200, 10, 9, 1]),                               # 30 of 32 rows, windows that begin inside a tile
])
def test_latent_attention_of_few_rows(heads, kv_rank, window, page_size, scale, portions):
    """against the fp32 kernel of the same engine, both held to the oracle; the pool starts out as NaN"""
    from asd_b200._lib import lib
    cfg = _config(heads, kv_rank, window, scale)
    w = O.random_model(cfg, seed=81, scale=1.5)
    ids = mz.tokens(sum(portions), 96, 82)
    ref, _ = O.forward(cfg, w, ids)
    outs = []
    for mode in (2, 1):
        eng = mz.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512, max_seq_len=1024, page_size=page_size)
        eng.set_option("attn_tiled", mode)
        if mode == 2:
            eng.cache_pool.fill_(255)
        names = (b"latent_step", b"latent_tc")
        before = [lib().asd_kernel_launches(n) for n in names]
        outs.append(mz.feed(eng, eng.open_sequence(), ids, portions).cpu())
        ran, want, at = [lib().asd_kernel_launches(n) - b for n, b in zip(names, before)], [0, 0], 0
        for p in portions:
            at += p
            hg = min(heads, 32)
            tq = min(32 // hg, p)
            tiles = -(-p // tq) * -(-heads // hg)
            if tiles <= 2 and (hg * tq >= 32 or min(at, window) > 64):
                want[0] += 1
            elif min(128 // min(heads, 128), p) * min(heads, 128) >= 32:       # rows of a tile of latent_attention_tc.cu
                want[1] += 1
        assert ran == (want if mode == 2 else [0, 0])
        eng.check_device()
        mz.close(eng)
    assert torch.isfinite(outs[0]).all()
    e_tc, e_fp32 = mz.rel_err(outs[0], ref)[0], mz.rel_err(outs[1], ref)[0]
    assert e_fp32 < 4e-2 and e_tc < 1.1 * e_fp32 + 1e-4, (e_tc, e_fp32)


def test_few_rows_of_unequal_sequences():
    """single tokens and pairs behind contexts of unequal length: shares that have no keys in the short ones"""
    from asd_b200._lib import lib
    cfg = _config(16, 512, 1 << 20, 0.3)
    w = O.random_model(cfg, seed=83, scale=1.5)
    lens = [(400, 1), (3, 2), (129, 1), (0, 1)]
    ids = [mz.tokens(a + b, 96, 84 + a) for a, b in lens]
    eng = mz.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512, max_seq_len=512, max_seqs=4)
    slots = [eng.open_sequence() for _ in lens]
    for s, t, (a, b) in zip(slots, ids, lens):
        eng.reserve(s, a + b)
        if a:
            eng.forward_ragged([(s, 0, t[:a], [])])
    before = lib().asd_kernel_launches(b"latent_step")
    got = eng.forward_ragged([(s, a, t[a:], list(range(b))) for s, t, (a, b) in zip(slots, ids, lens)]).cpu()
    assert lib().asd_kernel_launches(b"latent_step") - before == 1
    eng.check_device()
    at = 0
    for t, (a, b) in zip(ids, lens):
        assert mz.rel_err(got[at:at + b], O.forward(cfg, w, t)[0][a:])[0] < 4e-2
        at += b
    mz.close(eng)


def test_many_tiles_of_the_narrowest_latent():
    """128 latent columns leave the least time between the scores of two tiles (12 products): 64 sequences of 40 tiles, again and again with
    the same bits, and no wait ran out"""
    from asd_b200._lib import lib
    cfg = _config(16, 128, 1 << 20, 0.3)
    w = O.random_model(cfg, seed=85, scale=1.5)
    n, prompt = 64, 2560
    eng = mz.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512, max_seq_len=prompt + 16, max_seqs=n)
    ids = mz.tokens(prompt + 1, 96, 86)
    slots = [eng.open_sequence() for _ in range(n)]
    for s in slots:
        eng.reserve(s, prompt + 1)
        eng.forward_ragged([(s, 0, ids[:prompt], [])])
    tok = torch.full((n, 1), ids[prompt], dtype=torch.int32, device="cuda")
    at, slot = torch.full((n,), prompt, dtype=torch.int32, device="cuda"), torch.tensor(slots, dtype=torch.int32, device="cuda")
    before = lib().asd_kernel_launches(b"latent_step")
    first = eng.forward_uniform(tok, at, slot, prompt + 1).clone()
    for _ in range(100):
        assert torch.equal(eng.forward_uniform(tok, at, slot, prompt + 1), first)
    assert lib().asd_kernel_launches(b"latent_step") - before == 101
    eng.check_device()
    assert mz.rel_err(first[:1].cpu(), O.forward(cfg, w, ids)[0][-1:])[0] < 4e-2
    mz.close(eng)
