"""The streamed GEMM (few rows of activations, flat split over the K steps of all weight tiles) against fp32 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _workspace(rows):
    from penny_b200._ext import ops
    return torch.zeros(ops.gemm_stream_workspace_bytes(rows), dtype=torch.uint8, device="cuda")


def _data(rows, N, K, scale=0.05):
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + N * 3 + K)
    x = torch.randn(rows, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * scale).bfloat16()
    return x, w


def _close(out, want):
    rel = ((out.float() - want).norm() / want.norm()).item()
    assert rel < 4e-3, rel
    torch.testing.assert_close(out.float(), want, atol=2e-2 * want.std().item(), rtol=1e-2)


# one row .. a full accumulator, ragged weight rows and K, one K step, tiles shared by many pairs
@pytest.mark.parametrize("cluster", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("shape", [(1, 4096, 4096), (33, 1000, 264), (64, 128, 64), (7, 257, 1088), (64, 6144, 4096),
                                   (128, 4096, 1792), (129, 3584, 512), (256, 640, 2048), (200, 16032, 512)])
def test_plain(shape, cluster):
    from penny_b200._ext import ops
    rows, N, K = shape
    if cluster > K // 64:
        pytest.skip("more K ranges than K steps")
    x, w = _data(rows, N, K)
    ws = _workspace(rows)
    for _ in range(2):  # the arrival counters are back at zero
        out = torch.full((rows, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.gemm_stream(x, w, out, ws, cluster=cluster)
        assert ops.gemm_error() == 0
        _close(out, x.float() @ w.float().t())


@pytest.mark.parametrize("interleaved", [True, False])
@pytest.mark.parametrize("shape", [(5, 14336, 512), (64, 192, 4096), (160, 1792, 1024)])
def test_silu_and_row_scale(shape, interleaved):
    from penny_b200._ext import ops
    rows, F, K = shape
    x, w = _data(rows, 2 * F, K, 0.02)
    sumsq = torch.rand(3, rows, device="cuda") * K / 3 + 1
    rstd = torch.rsqrt(sumsq.sum(0) / K + 1e-5)
    y = (x.float() @ w.float().t()) * rstd[:, None]
    if interleaved:
        y = y.view(rows, F // 64, 2, 64)
        gate, up = y[:, :, 0].reshape(rows, F), y[:, :, 1].reshape(rows, F)
    else:
        gate, up = y[:, :F], y[:, F:]
    out = torch.full((rows, F), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_stream(x, w, out, _workspace(rows), 1, 64 if interleaved else F, sumsq=sumsq)
    assert ops.gemm_error() == 0
    _close(out, torch.nn.functional.silu(gate) * up)


@pytest.mark.parametrize("shape", [(1, 4096, 512), (37, 512, 1024), (256, 4096, 4096)])
def test_residual_epilogue(shape):
    from penny_b200._ext import ops
    rows, N, K = shape
    x, w = _data(rows, N, K)
    res = torch.randn(rows, N, device="cuda").bfloat16()
    nw = (1 + 0.1 * torch.randn(N, device="cuda")).bfloat16()
    z = res.float() + x.float() @ w.float().t()
    out = torch.full((rows, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ss = torch.full((N // 128, rows), float("nan"), device="cuda")
    ops.gemm_stream(x, w, out, _workspace(rows), 2, residual=res, norm_w=nw, sumsq_out=ss)
    assert ops.gemm_error() == 0
    _close(res, z)
    _close(out, z * nw.float())
    torch.testing.assert_close(ss, z.pow(2).view(rows, N // 128, 128).sum(-1).t(), atol=1e-2, rtol=1e-3)


# all groups, empty groups first / last / between, one live group, a full group; ranges that start anywhere
@pytest.mark.parametrize("counts", [[3, 0, 1, 40, 0, 256, 17, 0], [0, 0, 5, 0], [64] * 6, [0, 0, 0]])
def test_groups(counts):
    from penny_b200._ext import ops
    N, K, E = 384, 704, len(counts)
    ends = torch.tensor(counts).cumsum(0) + 3
    ranges = torch.stack([ends - torch.tensor(counts), ends], 1).to(torch.int32)
    rows = int(ends[-1]) + 5
    x, w = _data(rows, E * N, K)
    out = torch.full((rows, N), -7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_stream(x, w, out, _workspace(256), ranges=ranges.cuda(), max_rows=256)
    assert ops.gemm_error() == 0
    want = torch.full((rows, N), -7.0, device="cuda")
    for e in range(E):
        s, t = ranges[e].tolist()
        want[s:t] = x[s:t].float() @ w[e * N:(e + 1) * N].float().t()
    _close(out, want)


# ------------------------------------------------------------------ tiled GEMM with fused epilogues
TILES = [128, 192, 256, 512, 0]


@pytest.mark.parametrize("cluster", [0, 1, 2, 3, 4])  # pairs that split a tile's K steps
@pytest.mark.parametrize("block_n", TILES)
@pytest.mark.parametrize("shape", [(1152, 768, 1024), (130, 200, 264), (2304, 1280, 512), (7, 64, 64), (256, 512, 8192)])
def test_tile_plain(shape, block_n, cluster):
    from penny_b200._ext import ops
    M, N, K = shape
    if cluster > 1 and (block_n != 512 or cluster > K // 64):
        pytest.skip("clusters are for CTA pairs and as many K steps")
    a, b = _data(M, N, K)
    for _ in range(2):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.gemm_tile(a, b, out, block_n=block_n, cluster=cluster)
        assert ops.gemm_error() == 0
        _close(out, a.float() @ b.float().t())


@pytest.mark.parametrize("block_n", [128, 256, 512])
@pytest.mark.parametrize("shape", [(384, 704, 512), (129, 1792, 320)])
def test_tile_silu_row_scale(shape, block_n):
    from penny_b200._ext import ops
    M, F, K = shape
    a, b = _data(M, 2 * F, K, 0.02)
    sumsq = torch.rand(5, M, device="cuda") * K / 5 + 1
    y = (a.float() @ b.float().t()) * torch.rsqrt(sumsq.sum(0) / K + 1e-5)[:, None]
    out = torch.full((M, F), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(a, b, out, 1, sumsq=sumsq, block_n=block_n, cluster=2)
    assert ops.gemm_error() == 0
    _close(out, torch.nn.functional.silu(y[:, :F]) * y[:, F:])


@pytest.mark.parametrize("block_n", [128, 256, 512])
@pytest.mark.parametrize("shape", [(384, 1024, 512), (1000, 384, 1088)])
def test_tile_residual(shape, block_n):
    from penny_b200._ext import ops
    M, N, K = shape
    a, b = _data(M, N, K)
    res = torch.randn(M, N, device="cuda").bfloat16()
    plain = res.clone()
    nw = (1 + 0.1 * torch.randn(N, device="cuda")).bfloat16()
    z = res.float() + a.float() @ b.float().t()
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ss = torch.full((N // 128, M), float("nan"), device="cuda")
    ops.gemm_tile(a, b, out, 2, residual=res, norm_w=nw, sumsq_out=ss, block_n=block_n, cluster=2)
    ops.gemm_tile(a, b, plain, 2, residual=plain, block_n=block_n)
    assert ops.gemm_error() == 0
    _close(res, z)
    _close(out, z * nw.float())
    _close(plain, z)
    torch.testing.assert_close(ss, z.pow(2).view(M, N // 128, 128).sum(-1).t(), atol=1e-1, rtol=1e-2)


@pytest.mark.parametrize("block_n", [128, 256, 512])
@pytest.mark.parametrize("counts", [[300, 0, 1, 129, 0, 1024], [0, 0], [0, 256, 256]])
def test_tile_groups(counts, block_n):
    from penny_b200._ext import ops
    F, K, E = 384, 320, len(counts)
    ends = torch.tensor(counts).cumsum(0) + 3
    ranges = torch.stack([ends - torch.tensor(counts), ends], 1).to(torch.int32)
    rows = int(ends[-1]) + 5
    x, w = _data(rows, E * 2 * F, K, 0.05)
    out = torch.full((rows, F), -7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(x, w, out, 1, ranges=ranges.cuda(), block_n=block_n)
    assert ops.gemm_error() == 0
    want = torch.full((rows, F), -7.0, device="cuda")
    for e in range(E):
        s, t = ranges[e].tolist()
        y = x[s:t].float() @ w[e * 2 * F:(e + 1) * 2 * F].float().t()
        want[s:t] = torch.nn.functional.silu(y[:, :F]) * y[:, F:]
    _close(out, want)


@pytest.mark.parametrize("tokens", [128, 384])  # streamed and tiled linears
def test_prefill_one_rank_matches_fp32(tokens):
    from penny_b200.models.llama_sp import LlamaSPPrefill
    from penny_b200.models.llama_tp import LlamaConfig
    from penny_b200.parallel.comm import Communicator
    cfg, layers = LlamaConfig.tiny(), 2
    x = torch.randn(tokens, cfg.hidden, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).bfloat16()
    want = LlamaSPPrefill.reference_forward(cfg, x, layers, seed=1)
    comm = Communicator.emulated(1, heap_bytes=64 << 20)
    try:
        m = LlamaSPPrefill(cfg, comm=comm, tokens=tokens, layers=layers, seed=1)
        for _ in range(2):
            got = m.forward(x).float()
            assert ((got - want).norm() / want.norm()).item() < 1.5e-2
    finally:
        comm.close()
