"""Which attention kernel a step's portions get: rules on sizes alone, asked without a GPU."""
import ctypes

import pytest

from aegean_tge_b200.csrc import build


@pytest.fixture(scope="module")
def one_query_tile():
    lib = ctypes.CDLL(build.build_attention(128))
    return lambda tokens, first, seqs, group, kv_heads, ctx: bool(lib.tge_attention_mma_one_query_tile(tokens, first, seqs, group, kv_heads, 1, ctx, 148))


@pytest.mark.parametrize("group,kv_heads", [(7, 4), (5, 8), (6, 2)])
@pytest.mark.parametrize("portions,each", [(1, 300), (3, 40), (6, 128), (16, 64), (20, 64), (64, 32), (12, 100), (8, 300)])
def test_portions_beside_single_tokens_get_the_kernel_that_they_get_alone(one_query_tile, group, kv_heads, portions, each):
    """The single tokens at the head of a step have a kernel of their own; how many they are says nothing about the others."""
    for ctx in (each, 320, 600, 5000):
        alone = one_query_tile(portions * each, 0, portions, group, kv_heads, ctx)
        for lead in (8, 31, 64):
            assert one_query_tile(lead + portions * each, lead, portions, group, kv_heads, ctx) == alone, (ctx, lead)


def test_both_choices_occur(one_query_tile):
    assert one_query_tile(16 * 64, 0, 16, 7, 4, 64) != one_query_tile(20 * 64, 0, 20, 7, 4, 64)
