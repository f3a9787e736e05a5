"""The MoE layer of a world of one in one native call, at the borders of its kernels' choices, against fp32 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# clusters for a handful of rows; routing in one block (up to 1024 tokens) or two launches; pair tiles
@pytest.mark.parametrize("tokens", [4, 5, 1024, 1032, 2700])
@pytest.mark.parametrize("topk", [1, 2])
def test_one_rank(tokens, topk):
    from penny_b200.models.moe_ep import MoeConfig, MoeEPLayer
    from penny_b200.parallel.comm import Communicator
    comm = Communicator.emulated(1, heap_bytes=256 << 20, timeout_ms=3000)
    try:
        cfg = MoeConfig(hidden=256, ffn=640, experts=8, topk=topk)
        layer = MoeEPLayer(cfg, comm, tokens=tokens)
        g = torch.Generator(device="cuda").manual_seed(tokens)
        x = torch.randn(tokens, cfg.hidden, device="cuda", generator=g).bfloat16()
        want = layer.reference([x], layer.w13[0], layer.w2[0], layer.router[0])[0]
        for replaced in (False, True):  # also with experts that are not views of one tensor
            if replaced:
                layer.w13[0][1] = layer.w13[0][1].clone()
            got = layer.forward([x])[0]
            comm.check()
            assert comm.gemm_error() == 0
            torch.testing.assert_close(got.float(), want, atol=3e-3, rtol=3e-2)
    finally:
        comm.close()
