"""Leaving the tiled GEMM's epilogue after a wait that ran out, on a model of two warps made from the source.

Two warps of a TMEM quarter run the same code and meet at a named barrier.  Every outcome of their bounded waits is
tried: in none may one warp be left at a barrier that the other has passed by."""
import itertools
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc", "gemm_tile_sm100.cuh")


def _steps():
    """What a warp whose rows are finished by its own CTA does in one tile: "vote" (both decide), "alone" (one
    decides whether to leave), "meet" (a barrier)."""
    text = open(SOURCE).read()
    text = text[text.index("for (int tile = worker;", text.index("epilogue (this CTA's 128 rows)")):text.index("teardown")]
    a = text.index("if (owner != cs) {")  # the other CTAs' rows: sent away, and the loop is left
    b = text.index("          break;\n        }", a)
    assert "named_bar" not in text[a:b] and "agree" not in text[a:b]
    text = text[:a] + text[b:].split("}", 1)[1]
    # the barrier stands once for each of the two warps: one waits before its part, one arrives after it
    kinds = {"if (!agree(ok)) break": "vote", "if (!__all_sync(0xffffffffu, ok)) break": "alone", "h == 0) named_bar_sync": "meet"}
    found = re.findall("|".join(re.escape(k) for k in kinds), text)
    assert text.count("break;") == sum(kinds[f] != "meet" for f in found), "a way out of the loop that is not modelled"
    assert text.count("named_bar_sync") == 2 and text.count("h == 1) named_bar_sync") == 1
    return [kinds[f] for f in found]


def test_both_warps_leave_together():
    steps = _steps()
    assert steps[-1] == "meet" and len(steps) >= 2
    waits = sum(s != "meet" for s in steps)
    for outcome in itertools.product(itertools.product([True, False], repeat=waits), repeat=2):
        left = [False, False]
        w = 0
        for s in steps:
            if s == "vote":
                assert not any(left) or all(left), ("one warp votes alone", steps, outcome)
                if not (outcome[0][w] and outcome[1][w]):
                    left = [True, True]
            elif s == "alone":
                left = [gone or not out[w] for gone, out in zip(left, outcome)]
            else:
                assert left[0] == left[1], ("one warp waits for ever", steps, outcome)
            w += s != "meet"
