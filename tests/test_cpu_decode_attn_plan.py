"""The decode attention's cut of rows by their lengths against the grid that the launcher makes (no GPU)."""
import random

import pytest

from penny_b200.parallel import schedule


def _fits(positions, kv_heads, max_len):
    cut = schedule.decode_attn_cut(positions, kv_heads, max_len)
    if cut is None:
        return None
    pieces, extra = cut
    assert all(p >= 1 for p in pieces)
    # every piece of every row has a CTA: one that is missing never arrives at its row's counter
    assert sum(pieces) * kv_heads <= len(positions) * kv_heads + extra, (len(positions), kv_heads, max_len, positions[:8])
    return pieces


@pytest.mark.parametrize("max_len", [1, 256, 257, 511, 512, 513, 768, 1024, 4352, 100000])
@pytest.mark.parametrize("kv_heads", [1, 2, 8])
def test_every_piece_has_a_cta(max_len, kv_heads):
    rng = random.Random(max_len * 8 + kv_heads)
    for B in (1, 2, 3, 7, 18, 19, 37, 64, 130, 300):
        inside = [rng.randrange(max_len) for _ in range(B)]
        # the last position, the first one past the cache (where a step at the last one leaves it), far past it, before it
        for edge in (max_len - 1, max_len, max_len + 1, 2 * max_len + 5, 2 ** 30, -1, -4096):
            _fits([edge] * B, kv_heads, max_len)
            _fits([edge] + inside[1:], kv_heads, max_len)
            _fits([p if rng.random() < 0.5 else edge for p in inside], kv_heads, max_len)
        _fits(inside, kv_heads, max_len)


def test_the_cut_at_the_caches_end():
    # 768 rows in a cache of 768 are three whole pieces of 256; the cache's last position asks for two
    assert _fits([768], 8, 768) == _fits([767], 8, 768) == [2]
    assert _fits([5000], 8, 5001) == [16] and _fits([0], 8, 5001) == [1] and _fits([-7], 8, 5001) == [1]
    assert schedule.decode_attn_cut([100] * 300, 8, 4096) is None  # four rounds of CTAs: whole rows
