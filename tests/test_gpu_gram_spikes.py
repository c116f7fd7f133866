"""FP64 Gram: columns so uneven that fixed point would lose digits go to the FP64 pipe
without a product in digits first, others do not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,k,spike", [(300000, 70, True), (300000, 70, False), (270001, 33, True)])
def test_route(ctx, N, k, spike):
    from kernel_evd_gb300 import api
    g = torch.Generator("cuda").manual_seed(N + k)
    F = torch.randn((N, k), dtype=torch.float64, device="cuda", generator=g)
    if spike:
        F[12345, k // 2] = 1e7
    s = torch.rand(N, dtype=torch.float64, device="cuda", generator=g) + 0.5
    api.profile_enable(ctx, True)
    G = api.weighted_gram(ctx, F, s)
    digits = "gram_f64_tc" in api.profile_read(ctx)
    api.profile_enable(ctx, False)
    assert digits == (not spike)
    Y = F * s[:, None]
    ref = sum(y.T @ y for y in Y.split(1 << 12))
    size = sum(y.abs().T @ y.abs() for y in Y.split(1 << 12))
    assert bool(((G - ref).abs() <= 2.0 ** -53 * (2 ** 12 + 2 ** 11) * size).all())
