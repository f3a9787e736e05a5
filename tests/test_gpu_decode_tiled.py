"""The folded step of one rank with linears on the tiled GEMM."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


def _config(**kw):
    from penny_b200.models.llama_tp import LlamaConfig
    return dataclasses.replace(LlamaConfig.tiny(), hidden=2048, heads=16, kv_heads=4, ffn=1216, vocab=4100, init_std=0.03, **kw)


@pytest.mark.parametrize("batch,on_tiles", [(64, 0), (65, 3), (128, 3), (176, 0), (177, 0), (256, 0)])
def test_step_matches_fp32(batch, on_tiles):
    from penny_b200._ext import ops
    from penny_b200.models.llama_tp import LlamaTPDecoder
    m = LlamaTPDecoder(_config(), world=1, max_batch=batch, max_len=90, full_init=True)
    assert len(m.tiled) == on_tiles and m.fold == (batch <= 128) and m.tiled_gate_up == (batch > 176)
    m.fill_synthetic_kv(70)
    m.positions.copy_(torch.randint(0, 71, (batch,), generator=torch.Generator().manual_seed(batch), dtype=torch.int32))
    m.capture()
    tokens, positions = m.tokens.clone(), m.positions.clone()
    kc, vc = [c.clone() for c in m.kcache], [c.clone() for c in m.vcache]
    want = m.reference_logits(tokens, positions, kc, vc)
    for host in (False, True):
        m.tokens.copy_(tokens)
        m.positions.copy_(positions)
        m.logits.fill_(float("nan"))
        if host:
            got = m.step(tokens.cpu())
            assert torch.equal(got.cuda(), m.next_tokens)
        else:
            m.step_device()
        assert ops.gemm_error() == 0
        # The step on the decode GEMM (64 rows) is 1.05e-2 of the 2-norm from this reference, which rounds at places of its
        # own; half as much again for batches that differ.  Differences of that size spread like a normal variable: a
        # million of them stay within six times it, a rounding of the logits beside it (2^-9 of up to 8 std).
        diff, std = (m.logits.float() - want), want.std().item()
        assert (diff.norm() / want.norm()).item() < 1.6e-2
        assert diff.abs().max().item() < (6 * 1.6e-2 + 8 * 2 ** -9) * std
        assert torch.equal(m.positions, positions + 1) and torch.equal(m.logits.float().argmax(-1), m.next_tokens)


@pytest.mark.parametrize("batch", [96, 180])  # norms folded; gate/up alone
def test_no_further_from_fp64_than_with_norms_of_their_own(batch):
    from test_gpu_decode_step import _exact_logits
    from penny_b200.models.llama_tp import LlamaTPDecoder
    m = LlamaTPDecoder(_config(layers=4), world=1, max_batch=batch, max_len=90, use_graph=False, full_init=True)
    m.fill_synthetic_kv(70)
    for w in [m.final_norm] + [L[n] for L in m.layers for n in ("norm1", "norm2")]:
        w.copy_(torch.rand_like(w) + 0.5)
    tokens, positions = m.tokens.clone(), m.positions.clone()
    want, far = _exact_logits(m, tokens, positions), {}
    for separate in (True, False):
        m.tokens.copy_(tokens)
        m.positions.copy_(positions)
        m._step_impl(separate=separate)
        far[separate] = ((m.logits.double() - want).norm() / want.norm()).item()
    assert far[False] <= 1.1 * far[True] and far[True] < 0.05, far


def test_small_layers_and_several_ranks_stay_as_they_are():
    from penny_b200.models.llama_tp import LlamaConfig, LlamaTPDecoder
    assert not LlamaTPDecoder.tiled_linears(LlamaConfig.tiny(), 200)
    assert len(LlamaTPDecoder.tiled_linears(LlamaConfig.llama3_8b(), 128)) == 3
    m = LlamaTPDecoder(_config(), world=1, max_batch=100, max_len=40, linears="penny", use_graph=False)
    assert not m.tiled and m.fold and "wgu_cat" not in m.layers[0]
