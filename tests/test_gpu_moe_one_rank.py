"""The MoE layer of a world of one in one native call, at the borders of its kernels' choices, against fp32 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# routing in one block (up to 1024 tokens) or two launches; pair tiles
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


def _layer(cfg, tokens, world=1, **kw):
    from penny_b200.models.moe_ep import MoeEPLayer
    from penny_b200.parallel.comm import Communicator
    comm = Communicator.emulated(world, heap_bytes=256 << 20, timeout_ms=3000)
    return comm, MoeEPLayer(cfg, comm, tokens=tokens, **kw)


def _check(layer, xs):
    w13, w2 = sum(layer.w13, []), sum(layer.w2, [])
    for got, want in zip(layer.forward(xs), layer.reference(xs, w13, w2, layer.router[0])):
        torch.testing.assert_close(got.float(), want, atol=3e-3, rtol=3e-2)


@pytest.mark.parametrize("world", [1, 2])
def test_weights_are_those_of_the_lists(world):
    """Entries replaced, given other memory, swapped or written to after construction: every forward uses what the
    lists hold then, without a copy of the experts, and what they no longer hold is freed."""
    from penny_b200.models.moe_ep import MoeConfig
    cfg = MoeConfig(hidden=512, ffn=1024, experts=8, topk=2)
    comm, layer = _layer(cfg, 64, world, cap_factor=float(world))
    try:
        xs = [torch.randn(64, cfg.hidden, device="cuda").bfloat16() for _ in range(world)]
        fresh = lambda t: torch.randn_like(t) * 0.02  # noqa: E731
        _check(layer, xs)
        layer.w13[0][1].copy_(fresh(layer.w13[0][1]))
        _check(layer, xs)
        layer.w13[0][2].data = fresh(layer.w13[0][2])
        _check(layer, xs)
        layer.w2[-1][0], layer.w2[-1][1] = layer.w2[-1][1], layer.w2[-1][0]
        _check(layer, xs)
        both = sum(t.numel() for t in sum(layer.w13 + layer.w2, [])) * 2
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        layer.forward(xs)
        assert torch.cuda.max_memory_allocated() - before < both // 4
        for lists in (layer.w13, layer.w2):
            for mats in lists:
                mats[:] = [fresh(t) for t in mats]
        del mats, lists
        assert torch.cuda.memory_allocated() < before + both // 4  # (the tensors that the lists held are gone)
        _check(layer, xs)
    finally:
        comm.close()


def test_router_of_any_strides():
    from penny_b200.models.moe_ep import MoeConfig
    comm, layer = _layer(MoeConfig(hidden=256, ffn=640), 40)
    try:
        x = torch.randn(40, 256, device="cuda").bfloat16()
        wide = torch.zeros(8, 257, device="cuda", dtype=torch.bfloat16)
        wide[:, 1:] = layer.router[0]
        for router in (layer.router[0].t().contiguous().t(), wide[:, 1:]):  # column-major; padded and unaligned
            layer.router[0] = router
            _check(layer, [x])
    finally:
        comm.close()


@pytest.mark.parametrize("world", [1, 2])
def test_more_tokens_than_built_for_are_refused(world):
    from penny_b200.models.moe_ep import MoeConfig
    comm, layer = _layer(MoeConfig(hidden=256, ffn=640), 40, world, cap_factor=float(world))
    try:
        xs = [torch.randn(41 if v == 0 else 40, 256, device="cuda").bfloat16() for v in range(world)]
        with pytest.raises(RuntimeError, match="built for 40 tokens"):
            layer.forward(xs)
        _check(layer, [x[:40] for x in xs])
    finally:
        comm.close()


@pytest.mark.parametrize("experts", [256, 264])  # the most groups of a launch, and more
def test_many_experts(experts):
    from penny_b200.models.moe_ep import MoeConfig
    comm, layer = _layer(MoeConfig(hidden=256, ffn=256, experts=experts), 200)
    try:
        _check(layer, [torch.randn(200, 256, device="cuda").bfloat16()])
    finally:
        comm.close()


@pytest.mark.parametrize("world", [1, 2])
def test_fewer_tokens_than_built_for(world, monkeypatch):
    """A call's tiles follow its own rows: a layer built for a prefill batch decodes on the tiles of a small one."""
    from penny_b200.models import moe_ep
    cfg = moe_ep.MoeConfig(hidden=256, ffn=640)
    comm, layer = _layer(cfg, 3000, world, cap_factor=float(world))
    asked, rule = [], moe_ep.expert_tiles
    monkeypatch.setattr(moe_ep, "expert_tiles", lambda rows, *a: asked.append((rows, rule(rows, *a)[0])) or rule(rows, *a))
    try:
        for tokens in (3000, 5, 700, 1):
            asked.clear()
            _check(layer, [torch.randn(tokens, cfg.hidden, device="cuda").bfloat16() for _ in range(world)])
            comm.check()
            assert sum(r for r, _ in asked) == world * tokens * cfg.topk
            assert all(t == (512 if r > 640 * layer.epr else 256) for r, t in asked)
            assert tokens == 3000 or {t for _, t in asked} == {256}
    finally:
        comm.close()


@pytest.mark.parametrize("experts,tokens", [(8, 2), (8, 3), (4, 2), (4, 64), (4, 65), (2, 33)])
def test_down_projection_in_clusters(experts, tokens):
    """Around the borders of the rule for two CTAs per tile of the down projection (long K)."""
    from penny_b200.models.moe_ep import MoeConfig, expert_tiles
    cfg = MoeConfig(hidden=512, ffn=2048, experts=experts)
    comm, layer = _layer(cfg, tokens)
    try:
        assert expert_tiles(2 * tokens, experts, 512, 2048, layer.sms)[1] == (0 if tokens == 65 else 2)
        _check(layer, [torch.randn(tokens, cfg.hidden, device="cuda").bfloat16()])
        assert comm.gemm_error() == 0
    finally:
        comm.close()
