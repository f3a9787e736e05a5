"""Arg-max by packed maxima: ties, NaN, rows of the lowest value, zeros of either sign."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one vector, a partial batch of four, several batches per thread, a width whose odd rows are not aligned to 16 bytes
@pytest.mark.parametrize("cols", [8, 1000, 2048, 16384, 128256, 2049])
@pytest.mark.parametrize("chunked", [False, True])
def test_argmax_edges(cols, chunked):
    from penny_b200._ext import ops
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = torch.randn(10, cols, device="cuda", generator=g).bfloat16()
    x[1] = float("-inf")
    x[2] = float("nan")
    x[3, : cols // 2] = float("nan")
    x[4] = float("-inf")
    x[4, 0] = float("nan")
    x[5, [cols // 3, cols // 3 + 1, cols - 1]] = 50.0  # a tie: the lowest index
    x[6] = -1.0
    x[6, [cols // 2, cols - 1]] = torch.tensor([-0.0, 0.0], device="cuda", dtype=torch.bfloat16)
    x[7] = 2.0
    x[8, cols - 1] = float("inf")
    ws = torch.zeros(ops.argmax_workspace_bytes(10), dtype=torch.uint8, device="cuda") if chunked else None
    val, idx = torch.empty(10, device="cuda"), torch.empty(10, dtype=torch.int64, device="cuda")
    ops.argmax_rows(x, val, idx, 0, ws)
    v = x.float()
    best = torch.where(v.isnan(), torch.full_like(v, float("-inf")), v).max(-1).values
    first = (v == best[:, None]).int().argmax(-1)  # (an all-NaN row: 0)
    assert torch.equal(val, best) and torch.equal(idx, first)


def test_host_tokens_take_the_winners():
    """Pinned host memory gets the ids that next_tokens gets, and is refused where there are none to get."""
    from penny_b200._ext import ops
    rows, cols = 5, 3001
    logits = torch.randn(rows, cols, device="cuda").bfloat16()
    val, idx = torch.empty(rows, device="cuda"), torch.empty(rows, dtype=torch.int64, device="cuda")
    ws = torch.zeros(ops.argmax_workspace_bytes(rows), dtype=torch.uint8, device="cuda")
    nxt, tok = (torch.full((rows,), -1, dtype=torch.int64, device="cuda") for _ in range(2))
    pos, host = torch.arange(rows, dtype=torch.int32, device="cuda"), torch.full((rows,), -1, dtype=torch.int64).pin_memory()
    with pytest.raises(RuntimeError, match="host_tokens"):
        ops.argmax_rows(logits, val, idx, 0, ws, host_tokens=host)
    ops.argmax_rows(logits, val, idx, 7, ws, None, nxt, tok, pos, host)
    torch.cuda.synchronize()
    assert torch.equal(val, logits.float().max(-1).values)
    assert torch.equal(host, idx.cpu()) and torch.equal(nxt, idx) and torch.equal(tok, idx)
    assert pos.tolist() == [r + 1 for r in range(rows)]
    for bad in (host.clone(), host.to(torch.int32).pin_memory(), torch.zeros(rows + 1, dtype=torch.int64).pin_memory()):
        with pytest.raises(RuntimeError, match="host_tokens"):
            ops.argmax_rows(logits, val, idx, 7, ws, None, nxt, tok, pos, bad)
