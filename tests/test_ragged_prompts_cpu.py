"""CPU: the forwards that prefill_ragged makes of prompts of unequal length, against a token by token account of them."""
import numpy as np
import pytest
import torch

from asd_b200.engine import _BatchOps, _token_ids
from asd_b200.models.qwen2 import tiny_config


class Recorder(_BatchOps):
    """takes forwards and answers with logits that name their token"""

    def __init__(self, max_tokens):
        self.cfg, self.max_tokens, self.device, self.seen = tiny_config(), max_tokens, torch.device("cpu"), {}

    def forward(self, tokens, positions, token_slot, cu_q, seq_slot, max_qlen, max_kv_len, logit_rows, logits_out, want_logits):
        assert all(t.dtype == torch.int32 and t.is_contiguous() for t in (tokens, positions, token_slot, cu_q, seq_slot))
        assert cu_q[0] == 0 and cu_q[-1] == tokens.numel() <= self.max_tokens and cu_q.numel() == seq_slot.numel() + 1
        for i, slot in enumerate(seq_slot.tolist()):
            a, b = cu_q[i].item(), cu_q[i + 1].item()
            assert 0 < b - a <= max_qlen and (token_slot[a:b] == slot).all()
            for t, p in zip(tokens[a:b].tolist(), positions[a:b].tolist()):
                assert p < max_kv_len and len(self.seen.setdefault(slot, [])) == p
                self.seen[slot].append(t)
        assert want_logits == (logit_rows is not None)
        if logit_rows is None:
            return None
        out = torch.zeros(logit_rows.numel(), self.cfg.vocab_size)
        out[torch.arange(logit_rows.numel()), tokens[logit_rows.long()].long()] = 1 + positions[logit_rows.long()].float()
        return out


@pytest.mark.parametrize("lens,max_tokens,chunk", [([5, 1, 9, 9], 64, 0), ([7], 64, 0), ([3, 30, 17], 12, 0), ([1, 2, 3], 64, 1), ([8, 8], 64, 4)])
def test_forwards_of_unequal_prompts(lens, max_tokens, chunk):
    eng = Recorder(max_tokens)
    g = torch.Generator().manual_seed(3)
    prompts = [torch.randint(0, eng.cfg.vocab_size, (n,), generator=g).tolist() for n in lens]
    slots = torch.tensor([7, 2, 5, 0][:len(lens)], dtype=torch.int32)
    out = eng.prefill_ragged(prompts, slots, chunk)
    assert [eng.seen[s] for s in slots.tolist()] == prompts
    for row, p in zip(out, prompts):
        assert row.argmax() == p[-1] and row.max() == len(p)


def test_token_ids():
    for p in ([1, 2, 3], (1, 2, 3), range(1, 4), np.array([1, 2, 3]), torch.tensor([1, 2, 3]), [np.int64(1), 2, torch.tensor(3)], bytes([1, 2, 3])):
        assert _token_ids(p).dtype == np.int32 and _token_ids(p).tolist() == [1, 2, 3]
    assert _token_ids([1.0, 2]).tolist() == [1, 2]
    with pytest.raises(OverflowError):
        _token_ids([1 << 31])
