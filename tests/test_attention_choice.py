"""Which attention kernel a step's portions get: rules on sizes alone, asked without a GPU."""
import ctypes
import random
from types import SimpleNamespace

import pytest

from aegean_tge_b200 import ops

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


@pytest.mark.parametrize("count,kv_heads,longest,cut", [(31, 4, 4096, False), (31, 8, 4096, False), (64, 4, 4096, False), (64, 8, 4096, False),
                                                        (16, 8, 3000, False), (40, 8, 800, False), (16, 4, 4096, True), (40, 4, 4096, True), (8, 8, 4096, True)])
def test_single_tokens_are_cut_where_that_measured_faster_over_drawn_lengths(monkeypatch, count, kv_heads, longest, cut):
    """Requests of lengths drawn up to ``longest`` beside a prompt, on 148 SMs: the same choice for five in six draws."""
    monkeypatch.setattr(ops, "core", lambda: SimpleNamespace(tge_device_sm_count=lambda: 148))
    same = 0
    for seed in range(200):
        rnd = random.Random(seed)
        lengths = [rnd.randrange(64, longest) for _ in range(count)]
        split = ops.choose_leading_split(count, sum(lengths), max(lengths), kv_heads, max(1187, *lengths))
        assert split % 64 == 0 and (split == 0 or split * 148 >= sum(lengths) * kv_heads)
        same += (split > 0) == cut
    assert same >= 167, same
