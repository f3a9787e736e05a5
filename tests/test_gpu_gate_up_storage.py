"""One storage of gate and up: weights that are written after capture are the ones of the next step, and the tiled GEMM and
silu * up read the decode GEMM's layout (blocks of 64 gate rows and the 64 up rows of the same features)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# decode GEMM; tiled GEMM with folded norms; the vendor library's linears; gate/up alone on the tiled GEMM
@pytest.mark.parametrize("batch", [64, 65, 128, 150, 200])
def test_step_uses_weights_written_after_capture(batch):
    from test_gpu_decode_tiled import _config
    from penny_b200._ext import ops
    from penny_b200.models.llama_tp import LlamaTPDecoder
    m = LlamaTPDecoder(_config(), world=1, max_batch=batch, max_len=90, full_init=True)
    m.fill_synthetic_kv(70)
    m.capture()
    tokens, positions = m.tokens.clone(), m.positions.clone()
    before = m.reference_logits(tokens, positions, m.kcache, m.vcache)
    for L in m.layers:
        for k in ("wqkv", "wo", "wgu", "wdown"):
            L[k].copy_(torch.randn_like(L[k], dtype=torch.float32) * m.cfg.init_std)
    m.lm_head.copy_(torch.randn_like(m.lm_head, dtype=torch.float32) * m.cfg.init_std)
    want = m.reference_logits(tokens, positions, m.kcache, m.vcache)
    assert ((before - want).norm() / want.norm()).item() > 1  # (other weights, other logits)
    for separate in (False, True):
        m.tokens.copy_(tokens)
        m.positions.copy_(positions)
        m.logits.fill_(float("nan"))
        if separate:
            m._step_impl(separate=True)
        else:
            m.step(tokens.cpu())
        assert ops.gemm_error() == 0
        # the bound of test_gpu_decode_tiled.py, for the same layers; norms of their own round the stream to bf16 twice a
        # layer (2^-9 of it each, four times in two layers, carried on at its own size: 2^-8 in quadrature)
        assert ((m.logits.float() - want).norm() / want.norm()).item() < 1.6e-2 + (2 ** -8 if separate else 0)


@pytest.mark.parametrize("batch", [64, 128, 150, 200])
def test_gate_up_is_stored_once(batch):
    from test_gpu_decode_tiled import _config
    from penny_b200.models.llama_tp import LlamaTPDecoder
    m = LlamaTPDecoder(_config(), world=1, max_batch=batch, max_len=40, use_graph=False)
    F, H = m.cfg.ffn, m.cfg.hidden
    assert all(sum(t.numel() == 2 * F * H for t in L.values()) == 1 for L in m.layers)


# (columns of a tile, CTAs or pairs that split K, pairs): strips of 8, 16, 32 and 64 rows, one and two accumulators, shares of a
# cluster that end inside a block
@pytest.mark.parametrize("bn,cl,pair", [(32, 1, -1), (80, 1, -1), (112, 1, 1), (128, 1, -1), (192, 1, 1), (208, 1, -1), (256, 1, 1),
                                        (288, 1, -1), (416, 1, 1), (448, 1, -1), (512, 1, 1), (96, 2, -1), (96, 3, 1),
                                        (160, 2, 1), (256, 3, -1), (0, 0, 0)])
@pytest.mark.parametrize("M,F,K", [(1, 64, 72), (129, 448, 1096), (385, 1216, 712)])
def test_both_layouts_give_the_same_bits(M, F, K, bn, cl, pair):
    from penny_b200._ext import ops
    from penny_b200.models.llama_tp import LlamaTPDecoder
    g = torch.Generator(device="cuda").manual_seed(M + F + K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    gate, up = ((torch.randn(F, K, device="cuda", generator=g) * 0.05).bfloat16() for _ in range(2))
    ss = torch.rand(3, M, device="cuda") * K
    outs = []
    for w, pairs in ((torch.cat([gate, up]), False), (LlamaTPDecoder.interleave_gate_up(gate, up), True)):
        out = torch.full((M + 1, F), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.gemm_tile(x, w, out[:M], 1, sumsq=ss, block_n=bn, cluster=cl, pair=pair, silu_pairs=pairs)
        assert ops.gemm_error() == 0 and torch.isnan(out[M]).all()
        outs.append(out[:M])
    scale = torch.rsqrt(ss.sum(0) / K + 1e-5)[:, None]
    want = torch.nn.functional.silu(x.float() @ gate.float().t() * scale) * (x.float() @ up.float().t() * scale)
    assert ((outs[0].float() - want).norm() / want.norm()).item() < 2 ** -8  # one rounding to bf16
    if (bn, cl) != (0, 0):  # (a choice of its own may split K elsewhere)
        assert torch.equal(outs[0], outs[1])
    assert ((outs[1].float() - want).norm() / want.norm()).item() < 2 ** -8


def test_pairs_are_refused_elsewhere():
    from penny_b200._ext import ops
    x, w = torch.zeros(16, 64, device="cuda").bfloat16(), torch.zeros(192, 64, device="cuda").bfloat16()
    half, ranges = torch.zeros(16, 96, device="cuda").bfloat16(), torch.tensor([0, 16], dtype=torch.int32).cuda()
    whole = torch.zeros(16, 64, device="cuda").bfloat16()
    for w_, out, epi, kw in ((w, half, 1, {}), (w[:128], whole, 1, dict(ranges=ranges)), (w[:128], whole, 1, dict(pair=2)),
                             (w[:64], whole, 0, {})):
        with pytest.raises(RuntimeError):
            ops.gemm_tile(x, w_, out, epi, silu_pairs=True, **kw)


@pytest.mark.parametrize("rows,F", [(1, 64), (150, 1216)])
def test_silu_mul_of_pairs(rows, F):
    from penny_b200._ext import ops
    gate, up = (torch.randn(rows, F, device="cuda").bfloat16() for _ in range(2))
    want, got = torch.empty_like(gate), torch.empty_like(gate)
    ops.silu_mul(torch.cat([gate, up], 1), want)
    ops.silu_mul(torch.stack([gate.view(rows, -1, 64), up.view(rows, -1, 64)], 2).reshape(rows, 2 * F), got, pairs=True)
    assert torch.equal(got, want)
