"""Widths of the tiled GEMM beside the powers of two, two accumulators, shared columns of a cluster, an fp32 stream."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (columns of a tile, CTAs or pairs that split K, pairs): remainders of a 32-column pass, of an accumulator, of 74 and 148
# tiles; two accumulators; shares of 16, 32, 48 and 80 columns
SHAPES = [(80, 1, -1), (112, 1, 1), (208, 1, -1), (240, 1, 1), (288, 1, -1), (416, 1, 1), (512, 1, 1), (512, 1, -1),
          (96, 2, -1), (96, 3, 1), (160, 2, 1), (144, 3, -1), (64, 4, -1)]


def _data(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + K)
    return torch.randn(M, K, device="cuda", generator=g).bfloat16(), (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()


def _close(out, want):
    # one rounding to bf16 (8 bits): at most 2^-8 of every value, and so of the 2-norm
    assert ((out.float() - want).norm() / want.norm()).item() < 2 ** -8
    torch.testing.assert_close(out.float(), want, atol=1e-4 * want.std().item(), rtol=2 ** -8)


@pytest.mark.parametrize("bn,cl,pair", SHAPES)
@pytest.mark.parametrize("M", [1, 129, 385])
def test_plain_and_silu(M, bn, cl, pair):
    from penny_b200._ext import ops
    N, K = 1000, 1096
    a, b = _data(M, N, K)
    ss = torch.rand(3, M, device="cuda") * K
    y = (a.float() @ b.float().t()) * torch.rsqrt(ss.sum(0) / K + 1e-5)[:, None]
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(a, b, out, 0, sumsq=ss, block_n=bn, cluster=cl, pair=pair)
    assert ops.gemm_error() == 0
    _close(out, y)
    if cl > 1 and (bn // 2 % 16 or bn // 2 < 16 * cl):  # a share of the activations is whole columns of 16
        with pytest.raises(RuntimeError):
            ops.gemm_tile(a, b, out[:, :N // 2], 1, block_n=bn, cluster=cl, pair=pair)
        return
    act = torch.full((M, N // 2), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(a, b, act, 1, sumsq=ss, block_n=bn, cluster=cl, pair=pair)
    assert ops.gemm_error() == 0
    want = torch.nn.functional.silu(y[:, :N // 2]) * y[:, N // 2:]
    assert ((act.float() - want).norm() / want.norm()).item() < 2 ** -8


@pytest.mark.parametrize("bn,cl,pair", SHAPES + [(0, 0, 0)])
@pytest.mark.parametrize("M,wide", [(1, True), (129, False), (129, True), (385, False)])
def test_residual_of_any_width(M, wide, bn, cl, pair):
    from penny_b200._ext import ops
    N, K = 1152, 712
    a, b = _data(M, N, K)
    res = torch.randn(M, N, device="cuda").to(torch.float32 if wide else torch.bfloat16)
    nw = (1 + 0.1 * torch.randn(N, device="cuda")).bfloat16()
    z = res.float() + a.float() @ b.float().t()
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    stream = torch.full_like(out, float("nan")) if wide else None
    ss = torch.full((N // 16, M), float("nan"), device="cuda")
    rows = ops.gemm_tile(a, b, out, 2, residual=res, norm_w=nw, sumsq_out=ss, stream_out=stream, block_n=bn, cluster=cl, pair=pair)
    assert ops.gemm_error() == 0 and 0 < rows <= N // 16
    if wide:  # fp32 sums in another order: K products of 0.05
        torch.testing.assert_close(res, z, atol=1e-4, rtol=1e-5)
        _close(stream, z)
    else:
        _close(res, z)
    _close(out, z * nw.float())
    torch.testing.assert_close(ss[:rows].sum(0), z.pow(2).sum(1), atol=0, rtol=1e-5)
    assert torch.isnan(ss[rows:]).all()


def test_the_choice_is_kept_per_shape():
    """The same call twice, and one of another shape between them: each the right product."""
    from penny_b200._ext import ops
    for M, N, K in [(256, 768, 1024), (200, 1600, 320), (256, 768, 1024)]:
        a, b = _data(M, N, K)
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        ops.gemm_tile(a, b, out)
        _close(out, a.float() @ b.float().t())
    assert ops.gemm_error() == 0
