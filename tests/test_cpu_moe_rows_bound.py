"""Rows per tile of the MoE layer's grouped GEMMs: no expert, however many rows it gets, has its weights staged more often than
on tiles of 128 rows, and layers that lose by the tiles with the weight on the M side keep the others."""
import pytest


@pytest.mark.parametrize("experts,topk", [(2, 2), (8, 1), (8, 2), (64, 2), (64, 8), (256, 8)])
def test_no_more_tiles_than_of_128_rows(experts, topk):
    from penny_b200.models.moe_ep import expert_rows
    for tokens in list(range(1, 700)) + [1024, 4096]:
        for hidden in (1024, 2048, 4096):
            for width in expert_rows(tokens * topk, experts, hidden, tokens):
                assert width % 16 == 0 and 0 <= width <= 256
                assert width == 0 or -(-tokens // width) <= -(-tokens // 128), (tokens, hidden, width)


@pytest.mark.parametrize("per,hidden,want", [(88, 4096, 256), (88, 2048, 0), (127, 2048, 0), (128, 2048, 256), (128, 1024, 0),
                                             (1024, 1024, 0), (1024, 512, 0), (1, 512, 0), (1, 1024, 16)])
def test_small_layers(per, hidden, want):
    from penny_b200.models.moe_ep import expert_rows
    assert expert_rows(8 * per, 8, hidden, 4 * per) == (want, want)
