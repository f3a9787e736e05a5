"""The public decode call: host tokens in, host tokens out, step after step."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _decoder(use_graph, linears, batch=5, max_len=1500):
    from penny_b200.models.llama_tp import LlamaConfig, LlamaTPDecoder
    m = LlamaTPDecoder(LlamaConfig.tiny(), world=1, max_batch=batch, max_len=max_len, use_graph=use_graph, full_init=True,
                       linears=linears)
    m.fill_synthetic_kv(max_len - 10)
    # (mixed lengths: whole rows and rows of several pieces)
    m.positions.copy_(torch.tensor([1400, 3, 600, 1, 900][:batch], dtype=torch.int32))
    m.capture()
    return m


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("linears", ["penny", "cublas"])
def test_steps_follow_their_tokens(use_graph, linears):
    m = _decoder(use_graph, linears)
    g = torch.Generator().manual_seed(2)
    tokens = torch.randint(0, m.cfg.vocab, (m.B,), generator=g)
    for i in range(4):
        caches, positions = [c.clone() for c in m.kcache + m.vcache], m.positions.clone()
        got = m.step(tokens).clone()
        logits, after = m.logits.clone(), [c.clone() for c in m.kcache + m.vcache]
        assert got.device.type == "cpu" and torch.equal(got, m.next_tokens.cpu()) and torch.equal(got, m.tokens.cpu())
        assert torch.equal(m.positions, positions + 1)
        assert torch.equal(logits.gather(1, got.cuda()[:, None])[:, 0], logits.max(-1).values)
        want = m.reference_logits(tokens.cuda(), positions, m.kcache, m.vcache)
        assert (logits.float() - want).abs().max().item() < 0.05 * want.std().item() + 0.02
        # the same tokens from the device, the same state: the same bits
        for c, old in zip(m.kcache + m.vcache, caches):
            c.copy_(old)
        m.positions.copy_(positions)
        m.tokens.copy_(tokens)
        m.step_device()
        assert torch.equal(m.logits, logits) and torch.equal(m.next_tokens.cpu(), got) and torch.equal(m.positions, positions + 1)
        assert all(torch.equal(c, a) for c, a in zip(m.kcache + m.vcache, after))
        # one step that goes on from what this one returned, then tokens of the caller's own
        tokens = got if i % 2 == 0 else torch.randint(0, m.cfg.vocab, (m.B,), generator=g)


@pytest.mark.parametrize("use_graph", [True, False])
def test_ids_without_an_embedding_row_are_refused(use_graph):
    """Before anything is launched: the state is what it was, and the next step runs."""
    m = _decoder(use_graph, "auto")
    good = torch.arange(m.B)
    positions = m.positions.clone()
    first = m.step(good).clone()
    m.positions.copy_(positions)
    for bad_id in (m.cfg.vocab, -1, 2 ** 62, -(2 ** 63)):
        bad = good.clone()
        bad[m.B - 1] = bad_id
        with pytest.raises(IndexError):
            m.step(bad)
        torch.cuda.synchronize()
        assert torch.equal(m.positions, positions)
    edge = good.clone()
    edge[0] = m.cfg.vocab - 1
    m.step(edge)
    m.positions.copy_(positions)
    assert torch.equal(m.step(good), first)


def _exact_logits(m, tokens, positions):
    """One decode step of `m` in 64 bits, nothing rounded."""
    cfg, D, B = m.cfg, m.cfg.head_dim, tokens.numel()

    def norm(z, w):
        return z * torch.rsqrt(z.pow(2).mean(-1, keepdim=True) + cfg.eps) * w.double()
    ang = positions.double()[:, None] * cfg.rope_theta ** (-torch.arange(D // 2, device="cuda", dtype=torch.float64) * 2 / D)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def rope(t):
        a, b = t[..., :D // 2], t[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    res = m.embed[tokens].double()
    x = norm(res, m.layers[0]["norm1"])
    for li, L in enumerate(m.layers):
        q, k, v = (x @ L["wqkv"].double().t()).split([cfg.heads * D, cfg.kv_heads * D, cfg.kv_heads * D], -1)
        q, k, v = rope(q.view(B, -1, D)), rope(k.view(B, -1, D)), v.view(B, -1, D)
        outs = []
        for b in range(B):
            p = int(positions[b])
            keys, vals = (torch.cat([c[li][b, :, :p].double(), t[b][:, None]], 1) for c, t in ((m.kcache, k), (m.vcache, v)))
            s = torch.einsum("hgd,htd->hgt", q[b].view(cfg.kv_heads, -1, D), keys) * D ** -0.5
            outs.append(torch.einsum("hgt,htd->hgd", s.softmax(-1), vals).reshape(-1))
        res = res + torch.stack(outs) @ L["wo"].double().t()
        gate, up = m.split_gate_up(L["wgu"])
        x = norm(res, L["norm2"])
        res = res + (torch.nn.functional.silu(x @ gate.double().t()) * (x @ up.double().t())) @ L["wdown"].double().t()
        x = norm(res, m.layers[li + 1]["norm1"] if li + 1 < cfg.layers else m.final_norm)
    return x @ m.lm_head.double().t()


@pytest.mark.parametrize("batch", [1, 40])
def test_folded_norms_lose_no_precision(batch):
    """Distance from 64 bits of the step with norms in the GEMM epilogues and of the one with norms of their own."""
    from penny_b200.models.llama_tp import LlamaConfig, LlamaTPDecoder
    cfg = LlamaConfig.tiny()
    cfg.layers, cfg.hidden, cfg.init_std = 8, 1024, 0.05  # (layers that weigh as much as the stream)
    m = LlamaTPDecoder(cfg, world=1, max_batch=batch, max_len=400, use_graph=False, full_init=True)
    m.fill_synthetic_kv(300)
    assert m.fold
    for w in [m.final_norm] + [L[n] for L in m.layers for n in ("norm1", "norm2")]:
        w.copy_(torch.rand_like(w) + 0.5)
    tokens, positions = m.tokens.clone(), m.positions.clone()
    want, far = _exact_logits(m, tokens, positions), {}
    for separate in (True, False):
        m.tokens.copy_(tokens)
        m.positions.copy_(positions)
        m._step_impl(separate=separate)
        far[separate] = ((m.logits.double() - want).norm() / want.norm()).item()
    # about half of the roundings are gone; a tenth for what the ones that are left differ by from batch to batch
    assert far[False] <= 1.1 * far[True] and far[True] < 0.05, far
