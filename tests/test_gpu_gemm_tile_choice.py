"""gemm_tile without block_n: what the caller settles of the launch (pairs or single CTAs, CTAs that share K) is kept."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,epi", [(1, 1000, 1096, 0), (129, 4096, 4096, 0), (300, 28672, 4096, 1), (128, 4096, 14336, 2),
                                       (4096, 14336, 4096, 0)])
@pytest.mark.parametrize("pair", [-1, 1])
@pytest.mark.parametrize("cluster", [0, 1, 2, 4])
def test_choice_keeps_what_is_given(M, N, K, epi, pair, cluster):
    from penny_b200._ext import ops
    block_n, took, shared = ops.gemm_tile_choice(M, N, K, epi, pair=pair, cluster=cluster)
    assert block_n % 16 == 0 and 64 <= block_n <= 512 and took == pair
    assert shared == cluster if cluster else 1 <= shared <= 4


def test_a_cluster_that_nothing_can_share_is_left():
    from penny_b200._ext import ops
    assert ops.gemm_tile_choice(700, 512, 256, groups=3, cluster=2)[2] == 1  # (a group may have two row tiles)


@pytest.mark.parametrize("epi", [0, 1, 2])
def test_a_ring_has_three_stages(epi):
    """Single CTAs from 448 columns on have room for two, which is slower than any narrower tile."""
    from penny_b200._ext import ops
    for M in (65, 128, 384, 640, 1152, 2048, 4096):
        for N, K in [(12288, 8192), (8192, 28672), (28672, 4096), (4096, 14336), (6144, 4096)]:
            block_n, pair, _ = ops.gemm_tile_choice(M, N, K, epi)
            assert pair == 1 or block_n < 448


@pytest.mark.parametrize("pair,cluster", [(1, 0), (-1, 0), (1, 2), (-1, 2), (-1, 4), (0, 3), (0, 1)])
@pytest.mark.parametrize("M,groups", [(1, 0), (385, 0), (100, 2)])
def test_products(M, groups, pair, cluster):
    from penny_b200._ext import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    N, K, E = 1152, 712, max(1, groups)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = (torch.randn(E * N, K, device="cuda", generator=g) * 0.05).bfloat16()
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ends = [M * (e + 1) // E for e in range(E)]
    ranges = torch.tensor([0] + ends, dtype=torch.int32).cuda() if groups else None
    ops.gemm_tile(a, b, out, 0, ranges=ranges, pair=pair, cluster=cluster)
    assert ops.gemm_error() == 0
    want = torch.cat([a[s:t].float() @ b[e * N:(e + 1) * N].float().t() for e, (s, t) in enumerate(zip([0] + ends, ends))])
    # one rounding to bf16 (8 bits), and fp32 sums in another order
    torch.testing.assert_close(out.float(), want, atol=1e-4 * want.std().item(), rtol=2 ** -8)


def test_the_bits_are_those_of_the_shape_it_names():
    """An fp32 residual, where another order of adding shows: a cluster that is given is the one that ran."""
    from penny_b200._ext import ops
    M, N, K = 64, 1024, 4096
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b = torch.randn(M, K, device="cuda", generator=g).bfloat16(), torch.randn(N, K, device="cuda", generator=g).bfloat16()
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)

    def run(**kw):
        wide = torch.zeros(M, N, device="cuda")
        ops.gemm_tile(a, b, out, 2, residual=wide, **kw)
        assert ops.gemm_error() == 0
        return wide
    fixed = [run(block_n=128, pair=-1, cluster=c) for c in (1, 2, 3, 4)]
    for c in (1, 2, 3, 4):
        got = run(pair=-1, cluster=c)
        assert [torch.equal(got, f) for f in fixed] == [c == d for d in (1, 2, 3, 4)]


@pytest.mark.parametrize("pair", [-2, 3])
@pytest.mark.parametrize("block_n", [0, 128])
def test_other_values_of_pair_are_refused(pair, block_n):
    from penny_b200._ext import ops
    a = torch.zeros(16, 64, device="cuda").bfloat16()
    with pytest.raises(RuntimeError):
        ops.gemm_tile(a, a, torch.empty(16, 16, device="cuda", dtype=torch.bfloat16), pair=pair, block_n=block_n)
