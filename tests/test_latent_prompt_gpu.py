"""GPU: attention of prompts in head space (latent_prompt_tc.cu) at the edges of its tiles, against latent space and the oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import test_mezilix_gpu as mz  # noqa: E402
from oracle import mezilix_oracle as O  # noqa: E402


def _config(heads, kv_rank, window, scale):
    return mz.config([mz.layer(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=kv_rank, window=window, scale=scale, experts=0)], width=64)


@pytest.mark.parametrize("heads,kv_rank,window,page_size,scale,portions", [
    (2, 512, 1 << 20, 16, 0.05, [1, 127, 128, 129, 3]),     # tiles one short of, equal to and one beyond 128 positions
    (3, 200, 1 << 20, 8, 0.3, [385, 17]),                    # a latent that is no multiple of the products' 64, four key tiles
    (2, 512, 100, 128, 2.0, [300, 60, 200]),                # windows that begin and end inside a tile, a sharp softmax
    (1, 192, 128, 24, 0.5, [512, 40]),                       # a window of one tile, pages that divide no tile
])
def test_prompts_in_head_space(heads, kv_rank, window, page_size, scale, portions):
    """the pool starts out as NaN, none of which may reach a result"""
    from asd_b200._lib import lib
    cfg = _config(heads, kv_rank, window, scale)
    w = O.random_model(cfg, seed=71, scale=1.5)
    ids = mz.tokens(sum(portions), 96, 72)
    ref, _ = O.forward(cfg, w, ids)
    outs = []
    for mode in (2, 0):
        eng = mz.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512, max_seq_len=1024, page_size=page_size)
        eng.set_option("latent_prompt", mode)
        if mode == 2:
            eng.cache_pool.fill_(255)
        before = lib().asd_kernel_launches(b"latent_prompt")
        outs.append(mz.feed(eng, eng.open_sequence(), ids, portions).cpu())
        assert lib().asd_kernel_launches(b"latent_prompt") - before == (len(portions) if mode == 2 else 0)
        eng.check_device()
        mz.close(eng)
    assert torch.isfinite(outs[0]).all()
    # two bf16 terms on either side against one rounding each: no further from the oracle than in latent space
    e_head, e_latent = mz.rel_err(outs[0], ref)[0], mz.rel_err(outs[1], ref)[0]
    assert e_latent < 4e-2 and e_head < 1.1 * e_latent + 1e-4, (e_head, e_latent)


def test_unequal_prompts_in_head_space():
    """prompts of unequal length behind contexts of unequal length, one sequence a single token"""
    from asd_b200._lib import lib
    cfg = _config(2, 512, 150, 0.2)
    w = O.random_model(cfg, seed=73, scale=1.5)
    lens = [(5, 200), (130, 1), (0, 77), (64, 128)]
    ids = [mz.tokens(a + b, 96, 74 + b) for a, b in lens]
    refs = [O.forward(cfg, w, t)[0] for t in ids]
    eng = mz.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512, max_seq_len=512, max_seqs=4)
    eng.set_option("latent_prompt", 2)
    slots = [eng.open_sequence() for _ in lens]
    for s, (a, b) in zip(slots, lens):
        eng.reserve(s, a + b)
    eng.forward_ragged([(s, 0, t[:a], []) for s, t, (a, b) in zip(slots, ids, lens) if a])
    before = lib().asd_kernel_launches(b"latent_prompt")
    got = eng.forward_ragged([(s, a, t[a:], list(range(b))) for s, t, (a, b) in zip(slots, ids, lens)]).cpu()
    assert lib().asd_kernel_launches(b"latent_prompt") - before == 1
    eng.check_device()
    at = 0
    for ref, (a, b) in zip(refs, lens):
        assert mz.rel_err(got[at:at + b], ref[a:])[0] < 4e-2
        at += b
    mz.close(eng)


@pytest.mark.parametrize("portion,context,taken", [(8, 0, False), (9, 0, True), (17, 120, True), (17, 495, True), (17, 496, False)])
def test_calls_that_are_taken(portion, context, taken):
    """the rule's borders: tokens a sequence, positions a token; the same result as in latent space"""
    from asd_b200._lib import lib
    cfg = _config(4, 512, 1 << 20, 0.1)
    w = O.random_model(cfg, seed=75)
    ids = mz.tokens(context + portion, 96, 76)
    outs = []
    for mode in (1, 0):
        eng = mz.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=1024, max_seq_len=1024)
        eng.set_option("latent_prompt", mode)
        slot = eng.open_sequence()
        if context:
            mz.feed(eng, slot, ids[:context], [])
        eng.reserve(slot, context + portion)
        before = lib().asd_kernel_launches(b"latent_prompt")
        outs.append(eng.forward_ragged([(slot, context, ids[context:], list(range(portion)))]).double().cpu())
        assert lib().asd_kernel_launches(b"latent_prompt") - before == (1 if taken and mode == 1 else 0)
        mz.close(eng)
    assert ((outs[0] - outs[1]).norm() / outs[1].norm()).item() < 1e-2      # latent space rounds queries and results to bf16 once more
