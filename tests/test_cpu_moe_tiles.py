"""Tiles of the MoE layer's grouped GEMMs: the rule against the sizes it was measured at."""
import os
import subprocess
import sys

import pytest

from penny_b200.models.moe_ep import expert_tiles


@pytest.mark.parametrize("rows,experts,hidden,ffn,want", [
    (2, 8, 4096, 14336, (256, 2)), (4, 8, 4096, 14336, (256, 2)), (5, 8, 4096, 14336, (256, 0)),  # 64 and 80 tiles
    (100, 4, 4096, 14336, (256, 2)), (129, 4, 4096, 14336, (256, 0)),                             # one row tile at most
    (4, 8, 4096, 1024, (256, 0)), (4, 8, 4096, 1664, (256, 0)), (4, 8, 4096, 2048, (256, 2)),     # K steps to save
    (5120, 8, 4096, 14336, (256, 0)), (5121, 8, 4096, 14336, (512, 0)), (641, 1, 4096, 14336, (512, 0)),
])
def test_expert_tiles(rows, experts, hidden, ffn, want):
    assert expert_tiles(rows, experts, hidden, ffn, 148) == want


def test_no_pairs_where_they_are_switched_off():
    code = "from penny_b200.models.moe_ep import expert_tiles; assert expert_tiles(9000, 8, 4096, 14336, 148) == (256, 0)"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, PENNY_GEMM_PAIR="0"), check=True, timeout=300)
