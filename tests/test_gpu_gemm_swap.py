"""The tiled GEMM with the weight on the M side (pair=2) against fp32 PyTorch, and the MoE layer around its rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _data(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + K)
    return torch.randn(M, K, device="cuda", generator=g).bfloat16(), (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()


def _close(out, want):
    # one rounding to bf16 (8 bits): at most 2^-8 of every value, and so of the 2-norm
    assert ((out.float() - want).norm() / want.norm()).item() < 2 ** -8


@pytest.mark.parametrize("width", [16, 96, 256])  # rows of a tile: one MMA step, a remainder, the widest
@pytest.mark.parametrize("N,K", [(64, 72), (1000, 320), (1408, 1096)])
@pytest.mark.parametrize("M", [1, 16, 17, 257, 700])
def test_plain_and_silu(M, N, K, width):
    from penny_b200._ext import ops
    a, b = _data(M, N, K)
    ss = torch.rand(3, M, device="cuda") * K
    y = a.float() @ b.float().t()
    z = y * torch.rsqrt(ss.sum(0) / K + 1e-5)[:, None]
    for sumsq, want in ((None, y), (ss, z)):
        out = torch.full((M + 1, N), -7.0, device="cuda", dtype=torch.bfloat16)
        ops.gemm_tile(a, b, out[:M], 0, sumsq=sumsq, block_n=width, pair=2)
        _close(out[:M], want)
        act = torch.full((M + 1, N // 2), -7.0, device="cuda", dtype=torch.bfloat16)
        ops.gemm_tile(a, b, act[:M], 1, sumsq=sumsq, block_n=width, pair=2)
        _close(act[:M], torch.nn.functional.silu(want[:, :N // 2]) * want[:, N // 2:])
        assert (out[M:] == -7).all() and (act[M:] == -7).all()
    assert ops.gemm_error() == 0


@pytest.mark.parametrize("width", [16, 128, 256])
@pytest.mark.parametrize("counts", [[300, 0, 1, 129, 0, 1024], [0, 0], [0, 256, 257], [3, 0, 1, 40], [2400, 15]])
def test_groups(counts, width):
    from penny_b200._ext import ops
    F, K, E = 200, 328, len(counts)
    ends = torch.tensor(counts).cumsum(0) + 3
    ranges = torch.stack([ends - torch.tensor(counts), ends], 1).to(torch.int32)
    rows = int(ends[-1]) + 5
    x, w = _data(rows, E * 2 * F, K)
    for epi in (0, 1):
        out = torch.full((rows, 2 * F if epi == 0 else F), -7.0, device="cuda", dtype=torch.bfloat16)
        ops.gemm_tile(x, w, out, epi, ranges=ranges.cuda(), block_n=width, pair=2)
        assert ops.gemm_error() == 0
        want = torch.full(out.shape, -7.0, device="cuda")
        for e in range(E):
            s, t = ranges[e].tolist()
            y = x[s:t].float() @ w[e * 2 * F:(e + 1) * 2 * F].float().t()
            want[s:t] = y if epi == 0 else torch.nn.functional.silu(y[:, :F]) * y[:, F:]
        _close(out, want)


def test_groups_outside_the_rows():
    from penny_b200._ext import ops
    K, N, M = 320, 256, 100
    ranges = torch.tensor([[-40, 10], [10, 10], [10, 30], [60, 30], [90, 400], [120, 500]], dtype=torch.int32)
    x, w = _data(M, 6 * N, K)
    whole = torch.full((M + 400, N), -7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(x, w, whole[200:200 + M], 0, ranges=ranges.cuda(), pair=2)
    assert ops.gemm_error() == 0
    want = torch.full((M, N), -7.0, device="cuda")
    for g, (s, t) in enumerate([(0, 10), (10, 10), (10, 30), (0, 0), (90, M), (0, 0)]):
        want[s:t] = x[s:t].float() @ w[g * N:(g + 1) * N].float().t()
    _close(whole[200:200 + M], want)
    assert (whole[:200] == -7).all() and (whole[200 + M:] == -7).all()


def test_what_it_does_not_take():
    from penny_b200._ext import ops
    a, b = _data(64, 128, 64)
    out, res = torch.zeros(64, 128, device="cuda").bfloat16(), torch.zeros(64, 128, device="cuda").bfloat16()
    for epi, kw in ((2, dict(residual=res)), (0, dict(cluster=2)), (0, dict(block_n=24)), (0, dict(block_n=272))):
        with pytest.raises(RuntimeError):
            ops.gemm_tile(a, b, out, epi, pair=2, **kw)


@pytest.mark.parametrize("tokens", [24, 25, 208, 209, 351, 352])  # 6, 52 and 88 rows per expert, and one side of each
def test_moe_layer_around_the_rule(tokens):
    from test_gpu_moe_one_rank import _check, _layer
    from penny_b200.models.moe_ep import MoeConfig
    comm, layer = _layer(MoeConfig(hidden=512, ffn=640), tokens)
    try:
        _check(layer, [torch.randn(tokens, 512, device="cuda").bfloat16()])
        assert comm.gemm_error() == 0
    finally:
        comm.close()
