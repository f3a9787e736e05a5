"""Rows per tile of the MoE layer's grouped GEMMs with the weight on the M side: the rule, with and without pairs."""
import os
import subprocess
import sys

import pytest


@pytest.mark.parametrize("rows,want", [(2, (16, 16)), (48, (16, 16)), (49, (128, 0)), (416, (128, 0)), (417, (0, 0)), (703, (0, 0)),
                                       (704, (256, 256)), (8192, (256, 256))])
def test_expert_rows(rows, want):
    from penny_b200.models.moe_ep import expert_rows
    assert expert_rows(rows, 8) == want


def test_no_pairs_where_they_are_switched_off():
    code = "from penny_b200.models.moe_ep import expert_rows; assert expert_rows(9000, 8) == (0, 0) == expert_rows(2, 8)"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, PENNY_GEMM_PAIR="0"), check=True, timeout=300)
