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
