"""A MoE layer of many experts where nearly all rows meet the same two: few rows per expert on average, many tiles of one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [24, 64, 65, 190])
def test_nearly_all_rows_at_two_experts(tokens):
    from test_gpu_moe_one_rank import _check, _layer
    from penny_b200.models.moe_ep import MoeConfig, expert_rows
    cfg = MoeConfig(hidden=1024, ffn=640, experts=64)
    assert min(expert_rows(tokens * cfg.topk, cfg.experts, cfg.hidden, tokens)) >= min(tokens, 128)
    comm, layer = _layer(cfg, tokens)
    try:
        g = torch.Generator(device="cuda").manual_seed(tokens)
        common = torch.randn(1, cfg.hidden, device="cuda", generator=g)
        x = (torch.randn(tokens, cfg.hidden, device="cuda", generator=g) + 0.5 * common).bfloat16()
        layer.router[0][:2] += (0.02 * common).bfloat16()
        picked = (x.float() @ layer.router[0].float().t()).topk(cfg.topk).indices
        assert (picked < 2).float().mean().item() > 0.9
        _check(layer, [x])
        assert comm.gemm_error() == 0
    finally:
        comm.close()
