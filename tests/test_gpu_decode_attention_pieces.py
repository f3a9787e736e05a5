"""Decode attention with the rows cut by their lengths, against whole rows and fp64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


def _positions(kind, B, L):
    g = torch.Generator().manual_seed(B)
    if kind == "empty":
        return torch.zeros(B, dtype=torch.int32)
    if kind == "uniform":
        return torch.full((B,), L - 1, dtype=torch.int32)
    p = torch.randint(0, L, (B,), generator=g, dtype=torch.int32)
    if kind == "one long":
        p = p % 17
        p[B // 2] = L - 1
    return p


# one row in up to sixteen pieces; fewer and more (row, KV head) pairs than half of the CTAs that the GPU holds; more rows
# than a block has threads; lengths around the shortest piece (256)
@pytest.mark.parametrize("B,Hq,Hkv,L", [(1, 8, 2, 5000), (3, 4, 1, 257), (37, 8, 8, 1025), (130, 4, 2, 700), (300, 2, 1, 511)])
@pytest.mark.parametrize("kind", ["empty", "uniform", "mixed", "one long"])
def test_pieces_by_length(B, Hq, Hkv, L, kind):
    from penny_b200._ext import ops
    g = torch.Generator(device="cuda").manual_seed(B + L)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    kc, vc, pos = r(B, Hkv, L, D), r(B, Hkv, L, D), _positions(kind, B, L).cuda()
    need = ops.decode_attn_balanced_splits(B, Hkv)
    for splits in {need, max(1, need - 1)}:  # (room for fewer pieces than the cut may take: whole rows)
        ws = torch.zeros(ops.decode_attn_fused_workspace_bytes(B, Hq, Hkv, need), dtype=torch.uint8, device="cuda")
        for _ in range(2):  # the counters are left at zero
            qkv = r(B, (Hq + 2 * Hkv) * D)
            k1, v1, k2, v2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
            whole, out = (torch.full((B, Hq * D), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
            args = (Hq, Hkv)
            ops.decode_attention_fused(qkv, k1, v1, pos, whole, ws, *args, 1, D ** -0.5, 1e4)
            ops.decode_attention_fused(qkv, k2, v2, pos, out, ws, *args, splits, D ** -0.5, 1e4, balance=True)
            assert torch.equal(k1, k2) and torch.equal(v1, v2)
            # probabilities are rounded to bf16 under other running maxima (2 ** -9 of an average of values of size 1 to 4),
            # the output once more (2 ** -9 of it each)
            torch.testing.assert_close(out.float(), whole.float(), atol=2.0 ** -7, rtol=2.0 ** -7)
    b = int(pos.argmax())
    p, G = int(pos[b]), Hq // Hkv
    ang = p * 1e4 ** (-torch.arange(64, device="cuda", dtype=torch.float64) / 64)
    a, c = qkv[b, :Hq * D].double().view(Hq, 2, 64).unbind(1)
    q = torch.cat([a * ang.cos() - c * ang.sin(), c * ang.cos() + a * ang.sin()], -1).view(Hkv, G, D)
    s = torch.einsum("hgd,htd->hgt", q, k2[b, :, :p + 1].double()) / math.sqrt(D)
    want = torch.einsum("hgt,htd->hgd", s.softmax(-1), v2[b, :, :p + 1].double()).reshape(Hq * D)
    # (as above, and q rounded to bf16 before the scores, angles of up to 5000 rad in fp32)
    torch.testing.assert_close(out[b].double(), want, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("balance", [True, False])
def test_position_past_the_cache(balance):
    """A row that the cache cannot hold attends to all cached rows and itself and is stored nowhere, and the rows' arrival
    counters serve the next launch."""
    from penny_b200._ext import ops
    B, Hq, Hkv, L = 2, 8, 8, 768
    g = torch.Generator(device="cuda").manual_seed(9)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    kf, vf = r(B + 1, Hkv, L, D), r(B + 1, Hkv, L, D)  # (a row of slack behind the caches)
    kc, vc, splits = kf[:B], vf[:B], ops.decode_attn_balanced_splits(B, Hkv)
    ws = torch.zeros(ops.decode_attn_fused_workspace_bytes(B, Hq, Hkv, splits), dtype=torch.uint8, device="cuda")
    for last in (L, L + 300, L - 1):
        pos = torch.tensor([40, last], dtype=torch.int32, device="cuda")
        qkv, k0, v0 = r(B, (Hq + 2 * Hkv) * D), kf.clone(), vf.clone()
        out = torch.full((B, Hq * D), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.decode_attention_fused(qkv, kc, vc, pos, out, ws, Hq, Hkv, splits, D ** -0.5, 1e4, balance=balance)
        for b, p in enumerate(pos.tolist()):
            ang = p * 1e4 ** (-torch.arange(64, device="cuda", dtype=torch.float64) / 64)
            rot = lambda t: torch.cat([t[:, :64] * ang.cos() - t[:, 64:] * ang.sin(), t[:, 64:] * ang.cos() + t[:, :64] * ang.sin()], -1)  # noqa: E731
            q, k, v = (t.view(Hkv, D) for t in qkv[b].double().split(Hkv * D))
            q, k = rot(q), rot(k)
            rows = min(p, L)
            keys = torch.cat([k0[b, :, :rows].double(), k.bfloat16().double()[:, None]], 1)
            vals = torch.cat([v0[b, :, :rows].double(), v[:, None]], 1)
            s = torch.einsum("hd,htd->ht", q, keys) / math.sqrt(D)
            want = torch.einsum("ht,htd->hd", s.softmax(-1), vals).reshape(Hq * D)
            # (tolerance as in test_pieces_by_length)
            torch.testing.assert_close(out[b].double(), want, atol=2e-2, rtol=2e-2)
            if p < L:
                torch.testing.assert_close(kf[b, :, p].double(), k, atol=3e-2, rtol=2e-2)
                assert torch.equal(vf[b, :, p].double(), v)
                k0[b, :, p], v0[b, :, p] = kf[b, :, p], vf[b, :, p]
        assert torch.equal(kf, k0) and torch.equal(vf, v0)  # nothing else was written


def test_decoder_up_to_the_caches_last_row():
    """A cache filled up to its last row: the warm-up's second step has no row left, and none of it shows later."""
    from penny_b200.models.llama_tp import LlamaConfig, LlamaTPDecoder
    for L in (768, 300):
        m = LlamaTPDecoder(LlamaConfig.tiny(), world=1, max_batch=3, max_len=L, full_init=True)
        m.fill_synthetic_kv(L - 1)
        before = [c.clone() for c in m.kcache + m.vcache]
        m.capture()
        for c, old in zip(m.kcache + m.vcache, before):
            assert torch.equal(c[:, :, :L - 1], old[:, :, :L - 1])
        tokens, positions = m.tokens.clone(), m.positions.clone()
        m.step_device()
        want = m.reference_logits(tokens, positions, m.kcache, m.vcache)
        assert (m.logits.float() - want).abs().max().item() < 0.05 * want.std().item() + 0.02
        assert torch.equal(m.positions, positions + 1)


def test_separate_kernels_past_the_cache():
    """rope_append stores no row that the cache does not have; the attention reads the rows that there are."""
    from penny_b200._ext import ops
    B, Hq, Hkv, L = 3, 8, 2, 100
    g = torch.Generator(device="cuda").manual_seed(4)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    kf, vf, qkv = r(B + 1, Hkv, L, D), r(B + 1, Hkv, L, D), r(B, (Hq + 2 * Hkv) * D)
    pos = torch.tensor([L - 1, L, L + 500], dtype=torch.int32, device="cuda")
    k0, v0 = kf.clone(), vf.clone()
    ops.rope_append(qkv, kf[:B], vf[:B], pos, Hq, Hkv, D, 1e4)
    assert not torch.equal(kf[0, :, L - 1], k0[0, :, L - 1])
    k0[0, :, L - 1], v0[0, :, L - 1] = kf[0, :, L - 1], vf[0, :, L - 1]
    assert torch.equal(kf, k0) and torch.equal(vf, v0)
    for splits in (1, 3):
        out = torch.empty(B, Hq * D, device="cuda", dtype=torch.bfloat16)
        ws = torch.empty(ops.decode_attn_workspace_bytes(B, Hq, splits), dtype=torch.uint8, device="cuda")
        ops.decode_attention(qkv, kf[:B], vf[:B], pos, out, ws, Hq, Hkv, splits, D ** -0.5)
        q = qkv[:, :Hq * D].view(B, Hkv, Hq // Hkv, D).double()
        s = torch.einsum("bhgd,bhtd->bhgt", q, kf[:B].double()) / math.sqrt(D)
        want = torch.einsum("bhgt,bhtd->bhgd", s.softmax(-1), vf[:B].double()).reshape(B, Hq * D)
        torch.testing.assert_close(out.double(), want, atol=2e-2, rtol=2e-2)  # (as above)
