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
