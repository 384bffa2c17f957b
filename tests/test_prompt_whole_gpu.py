"""GPU: one sequence's prompt through an engine that holds fewer tokens a step than the prompt has."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_engine_gpu import _rel, tiny_config  # noqa: E402


# inside max_tokens, one beyond, weight-streaming and CTA-pair forwards, 1024 and a rest
@pytest.mark.parametrize("length", [32, 33, 256, 257, 1024, 1100])
def test_one_prompt_goes_through_whole(length):
    from asd_b200._lib import AsdError
    from asd_b200.engine import QwenEngine
    cfg = tiny_config(num_hidden_layers=2)
    ids = torch.randint(0, cfg.vocab_size, (2, length), generator=torch.Generator().manual_seed(7), dtype=torch.int32).cuda()
    slots = torch.arange(2, dtype=torch.int32, device="cuda")
    small = QwenEngine(cfg, max_seqs=2, max_seq_len=1200, max_tokens=32).load_random(seed=3)
    large = QwenEngine(cfg, max_seqs=2, max_seq_len=1200, max_tokens=4096).load_random(seed=3)
    forwards = []
    entry = small._forward
    small._forward = lambda name, tokens, *a: (forwards.append(tokens.numel()), entry(name, tokens, *a))[1]
    got = small.prefill(ids[:1], slots[:1])
    assert forwards == [min(length, 1024)] + [length - 1024] * (length > 1024)
    assert torch.equal(got, small.prefill_ragged([ids[0].tolist()], slots[:1]))
    assert _rel(got.double().cpu(), large.prefill(ids[:1], slots[:1]).double().cpu()) < 2e-2      # bf16 activations of two layers
    # several prompts at once, and steps, keep to max_tokens
    forwards.clear()
    both = small.prefill(ids, slots)
    assert max(forwards) <= 32 and _rel(both.double().cpu(), large.prefill(ids, slots).double().cpu()) < 2e-2
    if length > 32:
        with pytest.raises(AsdError, match="exceeds max_tokens"):
            small.forward_uniform(ids[:, :17], torch.zeros(2, dtype=torch.int32, device="cuda"), slots, 17)
        with pytest.raises(AsdError, match="exceeds max_tokens"):
            small._uniform(small._prompt_forward, ids[:, :17], torch.zeros(2, dtype=torch.int32, device="cuda"), slots, 17, True, True)
    small.close()
    large.close()


@pytest.mark.parametrize("length,max_tokens,max_seq_len,options", [
    (509, 64, 517, {}), (768, 256, 1024, {}), (768, 256, 1024, {"gemm_big": 0}), (1000, 32, 1024, {"ksplit": 16})])
def test_whole_prompts_without_the_in_cluster_reduction(length, max_tokens, max_seq_len, options):
    """plans of up to 16 K slices, the workspace of a prompt beyond max_tokens holds 8: widths of the 0.5B model"""
    from asd_b200.engine import QwenEngine
    from asd_b200.models.qwen2 import Qwen2Config
    cfg = Qwen2Config(896, 1, 14, 2, 4864, 512, head_dim=64, name="0.5b-layer")
    ids = torch.randint(0, cfg.vocab_size, (1, length), generator=torch.Generator().manual_seed(8), dtype=torch.int32).cuda()
    slots = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = []
    for held, opts in ((max_tokens, {"reduce": 0, **options}), (1024, {})):
        eng = QwenEngine(cfg, max_seqs=1, max_seq_len=max_seq_len, max_tokens=held, fuse_norm=False).load_random(seed=4)
        for name, value in opts.items():
            eng.set_option(name, value)
        out.append(eng.prefill(ids, slots).double().cpu())
        eng.close()
    assert _rel(out[0], out[1]) < 2e-2      # the same products, their fp32 slices added in another order


def test_prompt_tokens_of_an_engine_are_the_callers():
    """0: forwards of max_tokens and no memory beyond; a number of its own; more than a call of the CTA-pair GEMM takes is refused"""
    from asd_b200._lib import AsdError
    from asd_b200.engine import QwenEngine
    cfg = tiny_config(num_hidden_layers=1, intermediate_size=16384)
    ids = torch.randint(0, cfg.vocab_size, (1, 300), generator=torch.Generator().manual_seed(9), dtype=torch.int32).cuda()
    slots = torch.zeros(1, dtype=torch.int32, device="cuda")
    held, outs = [], []
    for asked, largest in ((0, 32), (64, 64), (None, 300)):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        eng = QwenEngine(cfg, max_seqs=1, max_seq_len=1200, max_tokens=32, prompt_tokens=asked)
        held.append(free - torch.cuda.mem_get_info()[0])
        eng.load_random(seed=3)
        forwards, entry = [], eng._forward
        eng._forward = lambda name, tokens, *a: (forwards.append(tokens.numel()), entry(name, tokens, *a))[1]
        outs.append(eng.prefill(ids, slots).double().cpu())
        assert max(forwards) == largest
        eng.close()
    assert held[2] - held[0] > 24 << 20             # 992 tokens of 16384 bf16 activations, at least
    assert max(_rel(o, outs[2]) for o in outs) < 2e-2
    with pytest.raises(AsdError, match="at most 4096"):
        QwenEngine(cfg, max_seqs=1, max_seq_len=1200, max_tokens=32, prompt_tokens=4097)
