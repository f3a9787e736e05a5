"""The decode GEMM's row scale and residual epilogue (the norms on either side of a linear)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (rows, columns, K): one row, an odd number with a ragged last slice, whole and just exceeded batch tiles (16, 32, 48, 64,
# 128 rows), two slabs;
# K of one step, of a partial last step, and more K steps than the ring is deep
SHAPES = [(1, 128, 64), (5, 256, 520), (16, 256, 1024), (17, 128, 2048), (33, 512, 1024), (48, 256, 4096), (49, 128, 1024),
          (64, 384, 4096), (128, 256, 2048), (129, 256, 1032)]


def _inputs(B, N, K, parts):
    g = torch.Generator(device="cuda").manual_seed(B * 7 + N + K)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    return r(B, K).bfloat16(), (r(N, K) * K ** -0.5).bfloat16(), r(parts, B).square() * K / parts


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("splits", [0, 1, 3, 8])
def test_residual_epilogue(shape, splits):
    from penny_b200._ext import ops
    B, N, K = shape
    x, w, _ = _inputs(B, N, K, 1)
    res, norm_w = torch.randn(B, N, device="cuda").bfloat16(), torch.rand(N, device="cuda").bfloat16()
    res0 = res.clone()
    z = res.double() + x.double() @ w.double().t()
    out, ss = torch.empty_like(res), torch.full((N // 128, B), float("nan"), device="cuda")
    ops.gemm_decode(x, w, out, False, splits, residual=res, norm_w=norm_w, sumsq_out=ss)
    assert ops.gemm_error() == 0
    # fp32 sums of up to 4096 products of size K ** -0.5: 1e-5 at most; then one bf16 rounding (2 ** -9)
    tol = z.abs() * 2.0 ** -8 + 1e-4
    alone = res0.clone()
    ops.gemm_decode(x, w, torch.empty_like(res), False, splits, residual=alone)  # without a norm behind it
    assert torch.equal(alone, res)
    assert ((res.double() - z).abs() <= tol).all()
    assert ((out.double() - z * norm_w.double()).abs() <= tol * norm_w.double() + 1e-6).all()
    want = z.square().view(B, N // 128, 128).sum(-1).t()
    torch.testing.assert_close(ss.double(), want, rtol=1e-4, atol=1e-4)
    # the stream in fp32, with a copy in bf16
    wide, copy, out2, ss2 = res0.float(), torch.empty_like(res), torch.empty_like(out), torch.empty_like(ss)
    ops.gemm_decode(x, w, out2, False, splits, residual=wide, norm_w=norm_w, sumsq_out=ss2, stream_out=copy)
    assert bool(((wide.double() - z).abs() <= 1e-4).all()) and torch.equal(copy, wide.bfloat16())
    assert torch.equal(copy, res) and torch.equal(out2, out) and torch.equal(ss2, ss)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("silu,parts,splits", [(False, 1, 0), (False, 32, 2), (True, 3, 0), (True, 32, 4)])
def test_row_scale(shape, silu, parts, splits):
    from penny_b200._ext import ops
    B, N, K = shape
    x, w, ss = _inputs(B, N, K, parts)
    scale = torch.rsqrt(ss.double().sum(0) / K + 1e-5)
    want = (x.double() @ w.double().t()) * scale[:, None]
    if silu:
        v = want.view(B, N // 128, 2, 64)
        want = (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(B, N // 2)
    out = torch.empty(B, N // 2 if silu else N, device="cuda", dtype=torch.bfloat16)
    ops.gemm_decode(x, w, out, silu, splits, sumsq=ss, eps=1e-5)
    assert ops.gemm_error() == 0
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4 * scale.max()).all()


@pytest.mark.parametrize("B", [1, 40, 130])
def test_silu_of_large_negative_gates(B):
    """silu(g) * up far out on the negative side, where exp(-g) is near the largest fp32: small, not zero."""
    from penny_b200._ext import ops
    K, gates = 64, torch.arange(64, device="cuda") * 0.5 - 88.5
    x, w = torch.zeros(B, K, device="cuda"), torch.zeros(128, K, device="cuda")
    x[:, 0], w[:64, 0], w[64:, 0] = 1.0, gates, 1.0
    ss, out = torch.full((1, B), float(K), device="cuda"), torch.empty(B, 64, device="cuda", dtype=torch.bfloat16)
    for sumsq, scale in ((None, 1.0), (ss, (1.0 + 1e-5) ** -0.5)):
        ops.gemm_decode(x.bfloat16(), w.bfloat16(), out, True, sumsq=sumsq, eps=1e-5)
        want = torch.nn.functional.silu(gates.double() * scale) * scale
        # one bf16 rounding; the fast exponential is off by 2 + 1.173 * 88.5 ulp (2 ** -16) at most, CUDA's bound for it
        torch.testing.assert_close(out.double(), want.expand(B, 64), rtol=2.0 ** -8 + 2.0 ** -15, atol=0)


@pytest.mark.parametrize("B,N,K", [(1, 4096, 4096), (16, 1024, 2048), (40, 4096, 4096), (64, 8192, 4096), (65, 4096, 4096)])
def test_splits_query_is_what_a_launch_takes(B, N, K):
    """Sums of a launch with splits=0 have the bits of the cluster size that the query names, with and without a fold."""
    from penny_b200._ext import ops
    x, w, ss = _inputs(B, N, K, 1)
    for folded in (False, True):
        def run(splits):
            out = torch.empty(B, N, device="cuda", dtype=torch.bfloat16)
            wide = torch.zeros(B, N, device="cuda")  # (fp32 sums, where another order of adding shows)
            if folded:
                ops.gemm_decode(x, w, out, False, splits, residual=wide)
            else:
                ops.gemm_decode(x, w, out, False, splits)
            return wide if folded else out
        took, named = run(0), ops.gemm_decode_splits(B, N, K, folded)
        assert torch.equal(took, run(named))
        if folded:
            assert [s for s in range(1, 9) if torch.equal(took, run(s))] == [named]


def test_outputs_that_nothing_writes_are_refused():
    from penny_b200._ext import ops
    x, w, _ = _inputs(3, 128, 64, 1)
    out, ss = torch.empty(3, 128, device="cuda", dtype=torch.bfloat16), torch.empty(1, 3, device="cuda")
    norm_w = torch.ones(128, device="cuda", dtype=torch.bfloat16)
    for kw in ({"norm_w": norm_w, "sumsq_out": ss}, {"sumsq_out": ss}, {"stream_out": torch.empty_like(out)}):
        with pytest.raises(RuntimeError, match="beside a residual"):
            ops.gemm_decode(x, w, out, **kw)
    wide = torch.zeros(3, 128, device="cuda")
    with pytest.raises(RuntimeError, match="together"):
        ops.gemm_decode(x, w, out, residual=wide, norm_w=norm_w)
    with pytest.raises(RuntimeError, match="stream_out"):
        ops.gemm_decode(x, w, out, residual=torch.zeros_like(out), stream_out=torch.empty_like(out))


def test_embedding_rows_start_the_stream():
    from penny_b200._ext import ops
    table = torch.randn(50, 512, device="cuda").bfloat16()
    ids = torch.tensor([49, 0, 7, 7, 31], device="cuda")
    w = torch.rand(512, device="cuda").bfloat16()
    res, out = (torch.empty(5, 512, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ss = torch.empty(1, 5, device="cuda")
    ops.norm_prep(table, w, res, out, ss, ids=ids)
    want = table[ids]
    wide = torch.empty(5, 512, device="cuda")
    ops.norm_prep(table, w, wide, out, ss, ids=ids)
    assert torch.equal(wide, want.float())
    assert torch.equal(res, want) and torch.equal(out, (want.float() * w.float()).bfloat16())
    torch.testing.assert_close(ss[0], want.float().square().sum(-1), rtol=1e-5, atol=0)
    # ids in pinned host memory are read when the kernel runs
    host, again = ids.cpu().pin_memory(), torch.empty_like(wide)
    for _ in range(2):
        ops.norm_prep(table, w, again, out, ss, ids=host)
        torch.cuda.synchronize()
        assert torch.equal(again, table[host.cuda()].float())
        host.copy_(torch.tensor([0, 1, 49, 30, 2]))
    with pytest.raises(RuntimeError, match="ids"):
        ops.norm_prep(table, w, again, out, ss, ids=host.clone())  # pageable
