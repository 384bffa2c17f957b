"""GPU: which kernel a dense projection of a family's engine runs on, by tokens, matrix size and options."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import rivetar_oracle as O  # noqa: E402
from test_rivetar_gpu import close, config, gla, make_engine, tokens  # noqa: E402


@pytest.mark.parametrize("length,pairs", [(160, 0), (161, 2), (256, 2), (257, 3)])
def test_larger_matrices_take_pairs_from_161_tokens(length, pairs):
    """up and down projection of 2048 x 2048 (4M elements) and a smaller input projection (the output projection of 16 columns and
    the head's single row take other kernels)"""
    from asd_b200._lib import lib
    cfg = config([gla(heads=1, dim=16, vdim=16, ff=2048)], width=2048)
    w = O.random_model(cfg, seed=71)
    ids = tokens(length, 96, 72)
    outs = []
    for rows in (0, None):
        eng = make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512)
        if rows is not None:
            eng.set_option("tc_min_rows", rows)         # 0: never
        slot = eng.open_sequence()
        eng.reserve(slot, length)
        before = lib().asd_kernel_launches(b"gemm_pair")
        outs.append(eng.forward_ragged([(slot, 0, ids, [length - 1])]).double().cpu())
        assert lib().asd_kernel_launches(b"gemm_pair") - before == (pairs if rows is None else 0)
        close(eng)
    # the same bf16 operands, fp32 sums in another order: a rounding of the activations apart
    assert ((outs[0] - outs[1]).norm() / outs[0].norm()).item() < 1e-2


@pytest.mark.parametrize("width,ff,length,pairs", [
    (2048, 4096, 161, 1), (2048, 4096, 256, 1), (2048, 4096, 257, 3),       # up projection 4096 x 2048 on pairs, down 2048 x 4096 not
    (1024, 4096, 161, 0), (1024, 4096, 256, 0), (1024, 4096, 257, 3),       # 4096 x 1024: K too short for the plain launch it costs
    (1024, 8192, 161, 1),                                                   # 8M elements
])
def test_long_rows_stay_with_the_weight_streaming_kernel(width, ff, length, pairs):
    """matrices of more columns than rows, which the pairs would take in one slice, not before 257 tokens"""
    from asd_b200._lib import lib
    cfg = config([gla(heads=1, dim=16, vdim=16, ff=ff)], width=width)
    w = O.random_model(cfg, seed=73)
    eng = make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=512)
    slot = eng.open_sequence()
    eng.reserve(slot, length)
    before = lib().asd_kernel_launches(b"gemm_pair")
    eng.forward_ragged([(slot, 0, tokens(length, 96, 74), [length - 1])])
    assert lib().asd_kernel_launches(b"gemm_pair") - before == pairs
    close(eng)


@pytest.mark.parametrize("ff,few", [(4096, 3), (4104, 2)])
def test_few_tokens_of_long_rows_stay_with_the_weight_streaming_kernel(ff, few):
    """input, up and down projection (2048 x ff) and the head for 8 tokens: a block of the few-token kernel would stage all of ff"""
    from asd_b200._lib import lib
    cfg = config([gla(heads=1, dim=16, vdim=16, ff=ff)], width=2048)
    w = O.random_model(cfg, seed=75)
    eng = make_engine(cfg, w, dtype=torch.bfloat16, max_tokens=64)
    slot = eng.open_sequence()
    eng.reserve(slot, 8)
    names = (b"linear_few", b"gemm")
    before = [lib().asd_kernel_launches(n) for n in names]
    eng.forward_ragged([(slot, 0, tokens(8, 96, 76), [7])])
    assert [lib().asd_kernel_launches(n) - b for n, b in zip(names, before)] == [few + 1, 3 - few]
    close(eng)


@pytest.mark.parametrize("family", ["Mezilix", "Rivetar", "Mavipel", "Lukopel", "Dikopel", "Nobonex"])
def test_options_of_dense_projections_hold_for_few_tokens(family):
    """8 tokens of every family's engine: the few-token kernel, without it, and CTA pairs where they are asked for"""
    import importlib
    from asd_b200 import engine
    from asd_b200._lib import lib
    model = importlib.import_module(f"asd_b200.models.{family.lower()}")
    cfg = model.sized_config(256, 3, 2, vocab=512)
    eng = getattr(engine, family + "Engine")(cfg, max_seqs=8, max_seq_len=64, max_tokens=64).load_random(seed=5)
    slots = torch.arange(8, dtype=torch.int32, device="cuda")
    ids = torch.randint(0, 512, (8, 1), generator=torch.Generator().manual_seed(6), dtype=torch.int32).cuda()

    def launches(**options):
        for name, value in options.items():
            eng.set_option(name, value)
        names = (b"linear_few", b"gemm", b"gemm_pair")
        before = [lib().asd_kernel_launches(n) for n in names]
        out = eng.forward_uniform(ids, torch.zeros(8, dtype=torch.int32, device="cuda"), slots, 1).double()
        return [lib().asd_kernel_launches(n) - b for n, b in zip(names, before)], out
    (few, stream, pairs), a = launches()
    assert few > 0 and pairs == 0
    count, b = launches(linear_few=0)
    assert count == [0, stream + few, 0]
    count, c = launches(linear_few=1, tc_min_rows=9)
    assert count == [few, stream, 0]
    count, d = launches(tc_min_rows=8)
    assert count == [0, 0, stream + few]
    # the same bf16 operands, fp32 sums in another order: a rounding of the activations apart
    assert max(((x - a).norm() / a.norm()).item() for x in (b, c, d)) < 2e-2
    eng.close()
