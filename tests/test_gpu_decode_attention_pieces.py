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
