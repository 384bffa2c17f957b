"""GPU: the Rivetar engine's latent attention on the kernels made for heads of 128 + 64: prompts in head space (latent_prompt_tc.cu), single
tokens on the few-row kernel (latent_step_tc.cu).  The family brings its own sources, weights, scratch and output to both."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import test_rivetar_gpu as rv  # noqa: E402
from oracle import rivetar_oracle as O  # noqa: E402


@pytest.mark.parametrize("heads,kv_rank,rot_dims,layout,loop", [
    (16, 512, 64, None, None),                # interleaved pairs
    (2, 128, 40, "halves", (0, 2, 2)),        # a part of the coordinates rotates; a span run twice, every pass with its own cache
])
def test_latent_attention_of_128_and_64(heads, kv_rank, rot_dims, layout, loop):
    """the same prompts and steps with both kernels and with neither, held to the oracle; the pool starts out as NaN"""
    from asd_b200._lib import lib
    layer = rv.latent(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=kv_rank, q_rank=48, scale=0.07, rot_dims=rot_dims, layout=layout)
    cfg = rv.config([layer, rv.gla(ff=32)], width=64, loop=loop)
    w = O.random_model(cfg, seed=91, scale=1.5)
    portions = [200, 1, 90, 1, 1]
    ids = rv.tokens(sum(portions), 96, 92)
    ref, _ = O.forward(cfg, w, ids)
    runs = loop[2] if loop else 1
    names, outs = (b"latent_prompt", b"latent_step"), []
    for on in (1, 0):
        eng = rv.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512, max_seq_len=512)
        eng.set_option("latent_prompt", 2 * on)
        eng.set_option("latent_step", on)
        eng.cache_pool.fill_(255)
        slot, out, at = eng.open_sequence(), [], 0
        for p in portions:
            eng.reserve(slot, at + p)
            before = [lib().asd_kernel_launches(n) for n in names]
            # head space takes any portion here; a step is asked for without it
            eng.set_option("latent_prompt", 2 * on * (p > 1))
            out.append(eng.forward_ragged([(slot, at, ids[at:at + p], list(range(p)))]).cpu())
            assert [lib().asd_kernel_launches(n) - b for n, b in zip(names, before)] == [on * runs * (p > 1), on * runs * (p == 1)]
            at += p
        outs.append(torch.cat(out))
        rv.close(eng)
    assert torch.isfinite(outs[0]).all()
    # both kernels keep at least the bits of what they stand in for: no further from the oracle than without them
    e_on, e_off = rv.rel_err(outs[0], ref)[0], rv.rel_err(outs[1], ref)[0]
    assert e_off < 5e-2 and e_on < 1.1 * e_off + 1e-4, (e_on, e_off)
