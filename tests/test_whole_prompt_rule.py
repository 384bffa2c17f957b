"""How many positions a forward of one sequence's prompt takes."""
import pytest

from asd_b200.engine import whole_prompt_tokens


@pytest.mark.parametrize("max_tokens,max_seq_len,tp_size,asked,want", [
    (256, 4096, 1, None, 1024),         # left alone
    (256, 517, 1, None, 517),           # no longer than a sequence
    (2048, 4096, 1, None, 2048),        # max_tokens is more
    (256, 4096, 2, None, 256),          # tensor-parallel ranks keep to max_tokens
    (256, 4096, 1, 0, 256),             # none
    (256, 4096, 1, 300, 300),
])
def test_tokens_of_a_whole_prompt(max_tokens, max_seq_len, tp_size, asked, want):
    assert whole_prompt_tokens(max_tokens, max_seq_len, tp_size, asked) == want
