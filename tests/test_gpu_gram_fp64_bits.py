"""The FP64-pipe Gram gives the same bits every time, and a symmetric matrix."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,k", [(4000, 20), (3001, 51)])
def test_same_bits(ctx, N, k):
    from kernel_evd_gb300 import api
    g = torch.Generator("cuda").manual_seed(k)
    F = torch.randn((N, k), dtype=torch.float64, device="cuda", generator=g)
    s = torch.rand(N, dtype=torch.float64, device="cuda", generator=g) + 0.5
    G = api.weighted_gram(ctx, F, s)
    assert torch.equal(G, G.T)
    for _ in range(30):
        assert torch.equal(api.weighted_gram(ctx, F, s), G)
