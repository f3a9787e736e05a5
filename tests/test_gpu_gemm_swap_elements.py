"""The tiled GEMM with the weight on the M side, element by element: a store of eight columns with a wrong row or feature shows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(out, want, size):
    """`size`: standard deviation of the products (and of a gate times an up row).  bf16 rounding of every value, and fp32 sums in
    another order, off by some 1e-6 of the products' size."""
    torch.testing.assert_close(out.float(), want, atol=1e-4 * size, rtol=2 ** -8)


@pytest.mark.parametrize("width", [16, 48, 96, 256])
@pytest.mark.parametrize("N,K", [(64, 72), (1000, 320), (1408, 1096)])
@pytest.mark.parametrize("M", [1, 16, 17, 257, 700])
def test_plain_and_silu(M, N, K, width):
    from penny_b200._ext import ops
    from test_gpu_gemm_swap import _data
    a, b = _data(M, N, K)
    ss = torch.rand(3, M, device="cuda") * K
    y = a.double() @ b.double().t()
    z = y * torch.rsqrt(ss.double().sum(0) / K + 1e-5)[:, None]
    for sumsq, want in ((None, y), (ss, z)):
        size = want.std().item() if want.numel() > 1 else 1.0
        out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.gemm_tile(a, b, out, 0, sumsq=sumsq, block_n=width, pair=2)
        _check(out, want.float(), size)
        act = torch.full((M, N // 2), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.gemm_tile(a, b, act, 1, sumsq=sumsq, block_n=width, pair=2)
        up = want[:, N // 2:]
        _check(act, (torch.nn.functional.silu(want[:, :N // 2]) * up).float(), size * (size + up.abs().max().item()))
    assert ops.gemm_error() == 0


@pytest.mark.parametrize("width", [16, 128, 256])
@pytest.mark.parametrize("counts", [[300, 0, 1, 129, 0, 1024], [0, 256, 257], [3, 0, 1, 40], [2400, 15]])
def test_groups(counts, width):
    from penny_b200._ext import ops
    from test_gpu_gemm_swap import _data
    F, K, E = 200, 328, len(counts)
    ends = torch.tensor(counts).cumsum(0)
    rows = int(ends[-1])
    x, w = _data(rows, E * 2 * F, K)
    borders = torch.cat([torch.zeros(1, dtype=ends.dtype), ends]).to(torch.int32)
    y = torch.cat([x[s:t].double() @ w[e * 2 * F:(e + 1) * 2 * F].double().t()
                   for e, (s, t) in enumerate(zip(borders[:-1].tolist(), borders[1:].tolist()))])
    size = y.std().item()
    out = torch.full((rows, 2 * F), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(x, w, out, 0, ranges=borders.cuda(), block_n=width, pair=2)
    _check(out, y.float(), size)
    act = torch.full((rows, F), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(x, w, act, 1, ranges=borders.cuda(), block_n=width, pair=2)
    _check(act, (torch.nn.functional.silu(y[:, :F]) * y[:, F:]).float(), size * (size + y[:, F:].abs().max().item()))
    assert ops.gemm_error() == 0
