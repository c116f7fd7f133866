"""The exact median where a histogram bin holds more than 2^32 pairs: states at the
corners of a simplex (one distance for nearly all pairs), states that nearly all
coincide (also with more than 2^32 pairs per CTA), and Gaussian states, whose
median is checked by counting FP64 distances below and up to it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_simplex(ctx):
    from kernel_evd_gb300 import api
    X = torch.eye(64, device="cuda")[torch.arange(100000, device="cuda") % 64].contiguous()
    assert api.pair_median(ctx, X) == 2.0   # 4.9e9 of 5.0e9 pairs


@pytest.mark.parametrize("N,apart", [(100000, 2000), (1200000, 1200)])
def test_coinciding(ctx, N, apart):
    from kernel_evd_gb300 import api
    X = torch.zeros((N, 4), device="cuda")
    X[:apart] = torch.randn((apart, 4), generator=torch.Generator().manual_seed(1)).cuda()
    assert api.pair_median(ctx, X) == 0.0


def test_gaussian(ctx):
    from kernel_evd_gb300 import api
    N = 200000
    X = torch.randn((N, 64), generator=torch.Generator().manual_seed(2)).cuda()
    m = api.pair_median(ctx, X)
    # FP32 distances of 64 terms: a difference, a product and a sum each, 66 x 2^-24 < 4e-6
    lo, hi = m * (1 - 4e-6), m * (1 + 4e-6)
    Xd = X.double()
    sq = (Xd * Xd).sum(1)
    below = upto = 0
    for a in range(0, N, 4000):
        D = torch.addmm(sq[None], Xd[a:a + 4000], Xd.T, alpha=-2.0) + sq[a:a + 4000, None]
        below += int((D < lo).sum())
        upto += int((D <= hi).sum())
    rank = (N * (N - 1) // 2 - 1) // 2   # of the lower median; every pair counted twice, a state against itself once
    assert (below - N) // 2 <= rank < (upto - N) // 2
