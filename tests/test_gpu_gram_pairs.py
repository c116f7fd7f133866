"""Weighted Grams of an FP32 factor on CTA pairs: even and odd counts of column
tiles, ragged last tiles, row counts off the stage and the flush, one and two
Grams.  Per entry, with S = sum_i |w_i F_ia F_ib|: two-term f16 splits err by
2^-20 S, and the FP32 accumulator rounds 360 times (3 products of 120 K steps)
between two flushes, each by at most 2^-23 S."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,k", [(1057, 641), (1025, 768), (4099, 1000), (70001, 700), (2049, 1921), (3000, 1813), (3333, 2048)])
def test_against_fp64(ctx, N, k):
    from kernel_evd_gb300 import api
    gen = torch.Generator(device="cuda").manual_seed(N + k)
    F = torch.randn((N, k), device="cuda", generator=gen) * torch.logspace(0, -3, k, device="cuda")
    s = torch.rand(N, dtype=torch.float64, device="cuda", generator=gen) + 0.1
    s2 = torch.rand(N, dtype=torch.float64, device="cuda", generator=gen) + 0.1
    got = (*api.weighted_gram2(ctx, F, s, s2), api.weighted_gram(ctx, F, s))
    Fd = F.double()
    for G, w in zip(got, (s, s2, s)):
        Y = Fd * w[:, None]
        S = Y.abs().T @ Y.abs()
        assert bool(((G - Y.T @ Y).abs() <= (2.0 ** -20 + 360 * 2.0 ** -23) * S).all())
        assert torch.equal(G, G.T)
    assert torch.equal(got[0], got[2])
