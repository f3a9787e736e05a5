"""Token ids on their way into a decode step: copied, and looked at against the embedding's rows (no GPU)."""
import pytest
import torch


@pytest.mark.parametrize("n", [1, 5, 256])
def test_take_ids(n):
    from penny_b200._ext import ops
    dst, ids = torch.full((n,), -5), torch.arange(n) % 7
    assert ops.take_ids(ids, dst, 7 if n >= 7 else n) and torch.equal(dst, ids)
    assert ops.take_ids(ids.to(torch.int32), dst, 1000) and torch.equal(dst, ids)
    assert ops.take_ids(torch.stack([ids, ids], 1)[:, 1], dst, 1000) and torch.equal(dst, ids)  # strided
    for at in {0, n // 2, n - 1}:
        for bad in (7, 2 ** 62, -1, -(2 ** 63)):
            wrong = ids.clone()
            wrong[at] = bad
            assert not ops.take_ids(wrong, dst, 7)
            assert torch.equal(dst, wrong)
    with pytest.raises(RuntimeError):
        ops.take_ids(torch.arange(n + 1) if n > 1 else torch.arange(3), dst, 1000)
    with pytest.raises(RuntimeError, match="take_ids"):
        ops.take_ids(ids, dst.int(), 1000)
