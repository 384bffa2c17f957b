"""How many positions a forward of one sequence's prompt takes."""
import pytest

from asd_b200.engine import WHOLE_PROMPT_PAGES, whole_prompt_tokens


@pytest.mark.parametrize("max_tokens,max_seq_len,page_size,tp_size,asked,want", [
    (256, 4096, 16, 1, None, 1024),         # left alone
    (256, 517, 16, 1, None, 517),           # no longer than a sequence
    (2048, 4096, 16, 1, None, 2048),        # max_tokens is more
    (256, 4096, 16, 2, None, 256),          # tensor-parallel ranks keep to max_tokens
    (256, 131072, 16, 1, None, 1024),       # 8192 pages, all of which fit a block's share of the page table
    (256, 131073, 16, 1, None, 256),        # one more
    (256, 131072, 8, 1, None, 256),
    (256, 4096, 16, 1, 0, 256),             # none
    (256, 4096, 16, 1, 300, 300),
    (256, 131072, 8, 1, 512, 512),          # as asked
])
def test_tokens_of_a_whole_prompt(max_tokens, max_seq_len, page_size, tp_size, asked, want):
    assert whole_prompt_tokens(max_tokens, max_seq_len, page_size, tp_size, asked) == want


def test_the_pages_of_a_whole_prompt_fit_beside_the_tiles():
    """shared memory of a block: 227 KB; five tiles of 32 KB, barriers, row statistics and alignment take 168192 bytes"""
    assert 168192 + 4 * (WHOLE_PROMPT_PAGES + 2) <= 227 * 1024
