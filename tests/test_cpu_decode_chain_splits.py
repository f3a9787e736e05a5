"""Cluster rule of the decode linears between folded norms (no GPU)."""
from penny_b200.parallel import schedule


def test_cluster_rule_of_the_chain():
    f = schedule.decode_choose_splits_chain
    assert [f(t, kb) for t, kb in ((48, 64), (32, 64), (32, 224), (224, 64), (1002, 64))] == [5, 7, 7, 1, 1]
    assert f(32, 28) == 4 and f(32, 8) == 1  # ranges of at least six steps
