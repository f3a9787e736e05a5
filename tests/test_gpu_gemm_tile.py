"""The tiled GEMM with fused epilogues against fp32 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _data(rows, N, K, scale=0.05):
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + N * 3 + K)
    x = torch.randn(rows, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * scale).bfloat16()
    return x, w


def _close(out, want):
    rel = ((out.float() - want).norm() / want.norm()).item()
    assert rel < 4e-3, rel
    torch.testing.assert_close(out.float(), want, atol=2e-2 * want.std().item(), rtol=1e-2)


TILES = [128, 192, 256, 512, 0]


@pytest.mark.parametrize("cluster", [0, 1, 2, 3, 4])  # pairs or CTAs that split a tile's K steps
@pytest.mark.parametrize("block_n", TILES)
@pytest.mark.parametrize("shape", [(1152, 768, 1024), (130, 200, 264), (2304, 1280, 512), (7, 64, 64), (256, 512, 8192)])
def test_tile_plain(shape, block_n, cluster):
    from penny_b200._ext import ops
    M, N, K = shape
    if cluster > K // 64:
        pytest.skip("a cluster splits at least as many K steps")
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


@pytest.mark.parametrize("cluster", [2, 3, 4])
@pytest.mark.parametrize("block_n", [128, 256, 512])
@pytest.mark.parametrize("shape", [(384, 1024, 512), (1000, 384, 1088)])
def test_tile_residual(shape, block_n, cluster):
    from penny_b200._ext import ops
    M, N, K = shape
    a, b = _data(M, N, K)
    res = torch.randn(M, N, device="cuda").bfloat16()
    plain = res.clone()
    nw = (1 + 0.1 * torch.randn(N, device="cuda")).bfloat16()
    z = res.float() + a.float() @ b.float().t()
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ss = torch.full((N // 128, M), float("nan"), device="cuda")
    ops.gemm_tile(a, b, out, 2, residual=res, norm_w=nw, sumsq_out=ss, block_n=block_n, cluster=cluster)
    ops.gemm_tile(a, b, plain, 2, residual=plain, block_n=block_n)
    assert ops.gemm_error() == 0
    _close(res, z)
    _close(out, z * nw.float())
    _close(plain, z)
    torch.testing.assert_close(ss, z.pow(2).view(M, N // 128, 128).sum(-1).t(), atol=1e-1, rtol=1e-2)


@pytest.mark.parametrize("block_n", [128, 256, 512])
@pytest.mark.parametrize("counts", [[300, 0, 1, 129, 0, 1024], [0, 0], [0, 256, 256], [3, 0, 1, 40]])
@pytest.mark.parametrize("cluster", [0, 2])
def test_tile_groups(counts, block_n, cluster):
    from penny_b200._ext import ops
    if cluster and sum(counts) > 100:
        pytest.skip("clusters want one row tile per group")
    F, K, E = 384, 320, len(counts)
    ends = torch.tensor(counts).cumsum(0) + 3
    ranges = torch.stack([ends - torch.tensor(counts), ends], 1).to(torch.int32)
    rows = int(ends[-1]) + 5
    x, w = _data(rows, E * 2 * F, K, 0.05)
    out = torch.full((rows, F), -7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(x, w, out, 1, ranges=ranges.cuda(), block_n=block_n, cluster=cluster)
    assert ops.gemm_error() == 0
    want = torch.full((rows, F), -7.0, device="cuda")
    for e in range(E):
        s, t = ranges[e].tolist()
        y = x[s:t].float() @ w[e * 2 * F:(e + 1) * 2 * F].float().t()
        want[s:t] = torch.nn.functional.silu(y[:, :F]) * y[:, F:]
    _close(out, want)


@pytest.mark.parametrize("tokens", [128, 384])  # one row tile, and several
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


def test_b_written_by_the_kernel_before():
    """Unless told otherwise the GEMM waits for what wrote either operand, also a kernel that releases it early."""
    from penny_b200._ext import ops
    N, K = 2048, 4096
    a = torch.randn(128, K, device="cuda").bfloat16()
    ones = torch.ones(K, device="cuda", dtype=torch.bfloat16)
    b, h, ss = torch.zeros(N, K, device="cuda", dtype=torch.bfloat16), torch.empty(N, K, device="cuda").bfloat16(), \
        torch.empty(N, device="cuda")
    out = torch.empty(128, N, device="cuda", dtype=torch.bfloat16)
    for i in range(8):
        src = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
        torch.cuda.synchronize()
        ops.norm_prep(src, ones, b, h, ss)  # b = src
        ops.gemm_tile(a, b, out)
        _close(out, a.float() @ src.float().t())


@pytest.mark.parametrize("tokens", [128, 512])
def test_prefill_after_a_weight_update(tokens):
    """A forward right behind the kernels that rewrite its weights, on one stream, uses the new ones."""
    from penny_b200.models.llama_sp import LlamaSPPrefill
    from penny_b200.models.llama_tp import LlamaConfig
    from penny_b200.parallel.comm import Communicator
    cfg = LlamaConfig.tiny()
    x = torch.randn(tokens, cfg.hidden, device="cuda").bfloat16()
    comm = Communicator.emulated(1, heap_bytes=64 << 20)
    try:
        new = LlamaSPPrefill(cfg, comm=comm, tokens=tokens, layers=1, seed=2)
        m = LlamaSPPrefill(cfg, comm=comm, tokens=tokens, layers=1, seed=1)
        want = new.forward(x)
        stale = torch.zeros_like(m.layers[0]["wqkv"])
        for _ in range(20):
            m.layers[0]["wqkv"].copy_(stale)
            torch.cuda.synchronize()
            for k in ("norm1", "norm2", "wo", "wgu", "wd", "wqkv"):  # the first linear's weight last
                m.layers[0][k].copy_(new.layers[0][k])
            assert torch.equal(m.forward(x), want)
    finally:
        comm.close()


@pytest.mark.parametrize("cluster", [0, 2])
def test_tile_groups_outside_the_rows(cluster):
    """Ranges that leave the rows of a are cut to them: nothing is read or written outside."""
    from penny_b200._ext import ops
    K, N, M = 320, 256, 100
    ranges = torch.tensor([[-40, 10], [10, 10], [10, 30], [60, 30], [90, 400], [120, 500]], dtype=torch.int32)
    x, w = _data(M, 6 * N, K)
    whole = torch.full((M + 400, N), -7.0, device="cuda", dtype=torch.bfloat16)
    out = whole[200:200 + M]
    ops.gemm_tile(x, w, out, 0, ranges=ranges.cuda(), block_n=256, cluster=cluster)
    assert ops.gemm_error() == 0
    want = torch.full((M, N), -7.0, device="cuda")
    for g, (s, t) in enumerate([(0, 10), (10, 10), (10, 30), (0, 0), (90, M), (0, 0)]):
        want[s:t] = x[s:t].float() @ w[g * N:(g + 1) * N].float().t()
    _close(out, want)
    assert (whole[:200] == -7).all() and (whole[200 + M:] == -7).all()


def test_tile_norm_weight_must_be_contiguous():
    from penny_b200._ext import ops
    a, b = _data(128, 256, 64)
    res, out, ss = torch.zeros(128, 256, device="cuda").bfloat16(), torch.zeros(128, 256, device="cuda").bfloat16(), \
        torch.zeros(2, 128, device="cuda")
    row = torch.ones(1, 128, device="cuda").bfloat16()
    for nw in (row.expand(2, 128), torch.ones(2, 192, device="cuda").bfloat16()[:, :128]):  # 256 elements, but not in a row
        with pytest.raises(RuntimeError, match="contiguous norm_w"):
            ops.gemm_tile(a, b, out, 2, residual=res, norm_w=nw, sumsq_out=ss)


@pytest.mark.parametrize("backend,local", [("penny", True), ("penny", False), ("nccl", False)])
def test_kernels_per_forward(backend, local, monkeypatch):
    from penny_b200.models import llama_sp
    from penny_b200.models.llama_tp import LlamaConfig
    from penny_b200.parallel.comm import Communicator
    cfg, calls = LlamaConfig.tiny(), []

    class Counted:
        def __init__(self, inner):
            self.inner = inner

        def __getattr__(self, name):
            f = getattr(self.inner, name)
            return (lambda *a, **k: calls.append(name) or f(*a, **k)) if callable(f) else f
    comm = Communicator.emulated(1, heap_bytes=64 << 20)
    try:
        m = llama_sp.LlamaSPPrefill(cfg, comm=comm, tokens=128, layers=3, backend=backend)
        assert m.local == (backend == "penny")
        if m.local and not local:  # the fused GEMM + collective kernels, as several ranks run them
            x = torch.empty(128 * cfg.hidden + 1, device="cuda", dtype=torch.bfloat16)[1:].view(128, cfg.hidden).normal_()
        else:
            x = torch.randn(128, cfg.hidden, device="cuda").bfloat16()
        monkeypatch.setattr(llama_sp, "ops", Counted(llama_sp.ops))
        m.comm = Counted(comm)
        m.forward(x)
        assert len(calls) == (m.kernels_per_forward if m.local == local else 3 * 8), calls
    finally:
        comm.close()


@pytest.mark.parametrize("block_n", [128, 256, 512, 0])
def test_tile_residual_over_several_rounds(block_n):
    """More than two tiles for every CTA or pair, ragged rows: accumulators, sums of squares and the residual that is
    loaded ahead are used again and again, with the norm and without."""
    from penny_b200._ext import ops
    M, N, K = 4200, 2560, 256
    a, b = _data(M, N, K)
    res = torch.randn(M, N, device="cuda").bfloat16()
    plain = res.clone()
    nw = (1 + 0.1 * torch.randn(N, device="cuda")).bfloat16()
    z = res.float() + a.float() @ b.float().t()
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ss = torch.full((N // 128, M), float("nan"), device="cuda")
    ops.gemm_tile(a, b, out, 2, residual=res, norm_w=nw, sumsq_out=ss, block_n=block_n)
    ops.gemm_tile(a, b, plain, 2, residual=plain, block_n=block_n)
    assert ops.gemm_error() == 0
    _close(res, z)
    _close(out, z * nw.float())
    _close(plain, z)
    # the sums are over the product rounded to bf16 plus the residual: 2 * 2^-9 of each of 128 squares at most
    torch.testing.assert_close(ss, z.pow(2).view(M, N // 128, 128).sum(-1).t(), atol=0, rtol=2 ** -8)


def _prefill(cfg, tokens, layers, local, limit):
    from penny_b200.models.llama_sp import LlamaSPPrefill
    from penny_b200.parallel.comm import Communicator
    x = torch.randn(tokens, cfg.hidden, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).bfloat16()
    want = LlamaSPPrefill.reference_forward(cfg, x, layers, seed=1)
    comm = Communicator.emulated(1, heap_bytes=256 << 20, timeout_ms=2000)
    try:
        m = LlamaSPPrefill(cfg, comm=comm, tokens=tokens, layers=layers, seed=1)
        assert m.local
        m.local = local
        for _ in range(2):
            got = m.forward(x).float()
            comm.check()
            assert comm.gemm_error() == 0
            assert ((got - want).norm() / want.norm()).item() < limit
    finally:
        comm.close()


@pytest.mark.parametrize("tokens", [128, 384, 2432])
def test_prefill_one_rank_long_k(tokens):
    """K of 2048 and 4096: at 128 and 384 tokens clusters split it (more than the 26 steps of 64 from which that
    pays); 2432 tokens are several rounds of tiles per SM in gate/up."""
    from penny_b200.models.llama_tp import LlamaConfig
    _prefill(LlamaConfig(hidden=2048, layers=2, heads=16, kv_heads=4, head_dim=128, ffn=4096, vocab=2048), tokens, 2, True, 1.5e-2)


def test_prefill_fused_kernels_on_one_rank():
    """The GEMM + collective kernels that several ranks run (heap slots, flags, gathered-buffer TMA), on one."""
    from penny_b200.models.llama_tp import LlamaConfig
    _prefill(LlamaConfig.tiny(), 512, 2, False, 3e-2)
