"""The end of a greedy decode step on one GPU: LM head of a large batch, arg-max that hands the tokens on."""
import dataclasses
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 128256), (5, 2049), (64, 40000), (256, 131080), (3, 7)])
def test_argmax_hands_tokens_on(rows, cols):
    from penny_b200._ext import ops
    logits = torch.randn(rows, cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(cols)).bfloat16()
    ws = torch.zeros(ops.argmax_workspace_bytes(rows), dtype=torch.uint8, device="cuda")
    val, idx = torch.empty(rows, device="cuda"), torch.empty(rows, dtype=torch.int64, device="cuda")
    nxt, tok = torch.zeros_like(idx), torch.zeros_like(idx)
    pos = torch.arange(rows, dtype=torch.int32, device="cuda")
    for step in range(1, 3):
        ops.argmax_rows(logits, val, idx, 0, ws, None, nxt, tok, pos)
        best = logits.float().max(-1).values
        first = (logits.float() == best[:, None]).int().argmax(-1)  # ties: the lowest index
        assert torch.equal(val, best) and torch.equal(idx, first) and torch.equal(nxt, idx) and torch.equal(tok, idx)
        assert torch.equal(pos, torch.arange(rows, dtype=torch.int32, device="cuda") + step)


@pytest.mark.parametrize("batch", [192, 200])  # the vendor library's LM head and this library's
def test_lm_head_of_a_large_batch(batch):
    from penny_b200.models.llama_tp import LlamaConfig, LlamaTPDecoder
    cfg = dataclasses.replace(LlamaConfig.tiny(), vocab=1 << 16)
    m = LlamaTPDecoder(cfg, world=1, max_batch=batch, max_len=40, use_graph=True, full_init=True)
    m.fill_synthetic_kv(20)
    m.capture()
    tokens, positions = m.tokens.clone(), m.positions.clone()
    m.step_device()
    torch.cuda.synchronize()
    want = m.reference_logits(tokens, positions, m.kcache, m.vcache)
    err = (m.logits.float() - want).abs().max().item()
    assert err < 0.05 * want.std().item() + 0.02, err
    assert torch.equal(m.positions, positions + 1) and torch.equal(m.next_tokens, m.tokens)


def test_gemm_error_outlives_a_captured_first_gemm():
    """The first GEMM of a process is a captured one: its error word is zero before any replay, and a replay
    leaves an error that is already there to be read."""
    code = """if True:
        import dataclasses, torch
        from penny_b200._ext import ops
        from penny_b200.models.llama_tp import LlamaConfig, LlamaTPDecoder
        cfg = dataclasses.replace(LlamaConfig.tiny(), vocab=1 << 16)
        m = LlamaTPDecoder(cfg, world=1, max_batch=200, max_len=40)
        m.fill_synthetic_kv(20)
        m.capture()
        assert ops.gemm_error() == 0
        ops.gemm_error_word().fill_(7)
        m.step_device()
        assert ops.gemm_error() == 7 and ops.gemm_error() == 0
    """
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], cwd=root, check=True, timeout=300)


@pytest.mark.parametrize("batch,own", [(192, 0), (193, 1), (256, 1), (257, 0), (512, 0)])
def test_which_head_and_how_many_kernels(batch, own, monkeypatch):
    from penny_b200.models import llama_tp
    cfg = dataclasses.replace(llama_tp.LlamaConfig.tiny(), vocab=1 << 16)
    m = llama_tp.LlamaTPDecoder(cfg, world=1, max_batch=batch, max_len=24, use_graph=False, full_init=True)
    m.fill_synthetic_kv(8)
    tokens, positions = m.tokens.clone(), m.positions.clone()
    calls, inner = [], llama_tp.ops

    class Counted:
        def __getattr__(self, name):
            return lambda *a, **k: calls.append(name) or getattr(inner, name)(*a, **k)
    monkeypatch.setattr(llama_tp, "ops", Counted())
    m.step_device()
    monkeypatch.undo()
    assert calls.count("gemm_tile") == own and len(calls) == m.kernels_per_step
    want = m.reference_logits(tokens, positions, m.kcache, m.vcache)
    err = (m.logits.float() - want).abs().max().item()
    assert err < 0.05 * want.std().item() + 0.02, err
