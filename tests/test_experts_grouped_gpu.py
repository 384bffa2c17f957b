"""GPU: the experts' products on CTA pairs (grouped form of the tensor-bound GEMM) at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import test_mezilix_gpu as mz  # noqa: E402
from oracle import mezilix_oracle as O  # noqa: E402


@pytest.mark.parametrize("width,ff,experts,top,tokens,alone", [
    (256, 256, 4, 2, 20, False),        # 10 rows an expert: the smallest tile, boxes cut by the next group throughout
    (256, 256, 4, 2, 300, False),       # 150 rows an expert, one weight tile
    (264, 136, 3, 1, 400, False),       # no size a multiple of a tile; a box of 16 tokens cut by the next group
    (256, 520, 2, 2, 700, False),       # 700 rows an expert: tiles of 256 tokens, the third weight tile half empty
    (256, 256, 9, 1, 577, True),        # one expert takes every token: eight empty groups
])
def test_experts_on_cta_pairs(width, ff, experts, top, tokens, alone):
    """against the single-CTA kernel of the same engine, both held to the oracle"""
    from asd_b200._lib import lib
    cfg = mz.config([mz.layer(heads=1, dim=16, rot_dim=8, vdim=16, kv_rank=24, experts=experts, top=top, ff=ff)], width=width)
    w = O.random_model(cfg, seed=61)
    if alone:
        # equal scores: the first expert here, any in the oracle's topk, so they are all the same one
        w["l0.mlp.router"] = torch.zeros_like(w["l0.mlp.router"])
        for e in range(1, experts):
            for n in ("up", "down"):
                w[f"l0.mlp.e{e}.{n}"] = w[f"l0.mlp.e0.{n}"].clone()
    ids = mz.tokens(tokens, 96, 62)
    ref, _ = O.forward(cfg, w, ids)
    outs = []
    for rows in (1, 1 << 20):
        eng = mz.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=1024, max_seq_len=1024)
        eng.set_option("experts_rows", rows)
        before = lib().asd_kernel_launches(b"gemm_grouped")
        outs.append(mz.feed(eng, eng.open_sequence(), ids, []).cpu())
        assert lib().asd_kernel_launches(b"gemm_grouped") - before == (2 if rows == 1 else 0)
        mz.close(eng)
    e_pair, e_one = mz.rel_err(outs[0], ref)[0], mz.rel_err(outs[1], ref)[0]
    assert e_one < 4e-2 and e_pair < 1.1 * e_one + 1e-4, (e_pair, e_one)


@pytest.mark.parametrize("width,top,tokens,pairs", [
    (2048, 1, 3, False), (2048, 1, 4, True),            # 4M elements: a row an expert, on average
    (1024, 2, 63, False), (1024, 2, 64, True),          # 1M: 32
])
def test_rows_an_expert_from_which_pairs_are_taken(width, top, tokens, pairs):
    """four experts of width x width, the rule's own border on either side; the same result as without pairs"""
    from asd_b200._lib import lib
    cfg = mz.config([mz.layer(heads=1, dim=16, rot_dim=8, vdim=16, kv_rank=24, experts=4, top=top, ff=width)], width=width)
    w = O.random_model(cfg, seed=63)
    ids = mz.tokens(tokens, 96, 64)
    outs = []
    for rows in (0, 1 << 20):
        eng = mz.make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=64, max_seq_len=64)
        eng.set_option("experts_rows", rows)
        before = lib().asd_kernel_launches(b"gemm_grouped")
        outs.append(mz.feed(eng, eng.open_sequence(), ids, []).double().cpu())
        assert lib().asd_kernel_launches(b"gemm_grouped") - before == (2 if pairs and rows == 0 else 0)
        mz.close(eng)
    assert ((outs[0] - outs[1]).norm() / outs[1].norm()).item() < 1e-2      # fp32 sums in another order, one bf16 rounding between
