"""silu(gate) * up far out on the negative side, where exp(-gate) is near the largest fp32, wherever a decode step computes it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, gates, scale):
    want = torch.nn.functional.silu(gates.double() * scale) * scale
    # one bf16 rounding; the fast exponential is off by 2 + 1.173 * 88.5 ulp (2 ** -16) at most, CUDA's bound for it
    torch.testing.assert_close(got.double(), want.expand(got.shape), rtol=2.0 ** -8 + 2.0 ** -15, atol=0)


# (columns of a tile, CTAs or pairs that split K, pairs)
@pytest.mark.parametrize("bn,cl,pair", [(0, 0, 0), (128, 1, -1), (192, 1, 1), (512, 1, 1), (128, 2, -1), (256, 2, 1)])
@pytest.mark.parametrize("M", [1, 65, 200])
@pytest.mark.parametrize("pairs", [False, True])
def test_tiled_gemm(M, bn, cl, pair, pairs):
    from penny_b200._ext import ops
    K, gates = 256, torch.arange(64, device="cuda") * 0.5 - 88.5
    x, w = torch.zeros(M, K, device="cuda"), torch.zeros(128, K, device="cuda")
    x[:, 0], w[:64, 0], w[64:, 0] = 1.0, gates, 1.0  # (64 features: one block, so both layouts are these rows)
    ss, out = torch.full((1, M), float(K), device="cuda"), torch.empty(M, 64, device="cuda", dtype=torch.bfloat16)
    for sumsq, scale in ((None, 1.0), (ss, (1.0 + 1e-5) ** -0.5)):
        ops.gemm_tile(x.bfloat16(), w.bfloat16(), out, 1, sumsq=sumsq, eps=1e-5, block_n=bn, cluster=cl, pair=pair,
                      silu_pairs=pairs, exact_silu=True)
        assert ops.gemm_error() == 0
        _close(out, gates, scale)


@pytest.mark.parametrize("bn,cl,pair", [(128, 1, -1), (512, 1, 1), (128, 2, -1)])
def test_both_sides_of_the_ordinary_range(bn, cl, pair):
    """Rows whose gates are all inside it, and rows and passes with one outside, an infinity or a NaN among them."""
    from penny_b200._ext import ops
    K, F, M = 64, 192, 96
    gates = torch.linspace(-44, 44, F, device="cuda").bfloat16()
    gates[7], gates[70], gates[71] = float("inf"), float("-inf"), float("nan")
    x, w = torch.zeros(M, K, device="cuda"), torch.zeros(2 * F, K, device="cuda")
    x[:, 0], w[:F, 0], w[F:, 0] = torch.where(torch.arange(M, device="cuda") < 32, 0.5, 1.0), gates.float(), 1.0
    out = torch.empty(M, F, device="cuda", dtype=torch.bfloat16)
    ops.gemm_tile(x.bfloat16(), w.bfloat16(), out, 1, block_n=bn, cluster=cl, pair=pair, exact_silu=True)
    assert ops.gemm_error() == 0
    s = x[:, :1].double()
    want = torch.nn.functional.silu(gates.double() * s) * s
    torch.testing.assert_close(out.double(), want, rtol=2.0 ** -8 + 2.0 ** -15, atol=0, equal_nan=True)


# decode GEMM; tiled GEMM with folded norms; the vendor library's linears; gate/up alone on the tiled GEMM
@pytest.mark.parametrize("batch", [64, 65, 128, 150, 200])
def test_step(batch):
    """A stream of ones through layers of zeros, a norm that picks one element of it: the last layer's gates are its weights."""
    from test_gpu_decode_tiled import _config
    from penny_b200._ext import ops
    from penny_b200.models.llama_tp import LlamaTPDecoder
    m = LlamaTPDecoder(_config(), world=1, max_batch=batch, max_len=90, full_init=True)
    last, gates = m.layers[-1], torch.arange(64, device="cuda") * 0.5 - 88.5
    m.embed.fill_(1.0)
    for L in m.layers:
        for k in ("wqkv", "wo", "wgu", "wdown"):
            L[k].zero_()
    last["norm2"].zero_()
    last["norm2"][0] = 1.0
    last["wgu"][:64, 0], last["wgu"][64:128, 0] = gates.bfloat16(), 1.0
    m.fill_synthetic_kv(70)
    m.capture()
    m.step(torch.zeros(batch, dtype=torch.int64))
    assert ops.gemm_error() == 0
    _close(m.act[:, :64], gates, (1.0 + m.cfg.eps) ** -0.5 if m.fold else 1.0)  # (a norm of its own rounds to bf16: to one)


def test_where_an_exact_silu_is_refused():
    from penny_b200._ext import ops
    x, w = torch.zeros(16, 64, device="cuda").bfloat16(), torch.zeros(128, 64, device="cuda").bfloat16()
    for out, epi, kw in ((torch.empty_like(x), 1, dict(pair=2)), (torch.empty(16, 128, device="cuda").bfloat16(), 0, {})):
        with pytest.raises(RuntimeError):
            ops.gemm_tile(x, w, out, epi, exact_silu=True, **kw)
