"""Cluster rule of the decode linears between folded norms (no GPU)."""
from penny_b200.parallel import schedule


def test_cluster_rule_of_the_chain():
    f = schedule.decode_choose_splits_chain
    assert [f(t, kb) for t, kb in ((48, 64), (32, 64), (32, 224), (224, 64), (1002, 64))] == [5, 7, 7, 1, 1]
    assert f(32, 28) == 4 and f(32, 8) == 1  # ranges of at least six steps


def test_no_smaller_clusters_than_the_device_has_room_for():
    f, cap = schedule.decode_choose_splits_chain, schedule.B200_CLUSTER_CTAS
    # timed in the chain: more CTAs win here (64 and 128 tiles 3-5 %, 42 and 63 1.5 %), five CTAs on three SMs alone has
    # three, one, five and three
    assert [f(t, 64) for t in (64, 128, 42, 63)] == [4, 2, 6, 4]
    # filled to the last cluster they lose
    assert [f(t, 64) for t in (44, 90)] == [5, 2] and 44 * 6 == cap[6] and 90 * 3 == cap[3]
    for tiles in range(1, 400):
        for num_kb in (8, 32, 64, 224):
            s = f(tiles, num_kb)
            assert s == 1 or (num_kb // s >= 6 and (tiles * s < cap[s] or tiles * s * 3 <= 148 * 5))
            # a larger cluster only where the device has no room left for it, or its ranges are too short
            assert all(num_kb // r < 6 or tiles * r >= cap[r] for r in range(s + 1, 9))
