"""States with an infinity or a NaN are never pivots, in any form of a round, and leave the
other states' rows as they are without them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("b", [1, 3, 8, 9, 64])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_never_a_pivot(ctx, prec, b, value):
    from kernel_evd_gb300 import api
    N, d, k = 300, 5, 40
    g = torch.Generator().manual_seed(b)
    X = torch.randn((N, d), generator=g)
    bad = [0, 7, 150, 299]   # in the first and the last rows too
    X[bad, torch.arange(4)] = value
    f = api.rpcholesky(ctx, X.cuda(), 0.2, k, block=b, seed=3, precision=prec)
    assert f.rank == k and not set(bad) & set(f.piv.tolist())
    good = np.setdiff1d(np.arange(N), bad)
    F, Xg = f.factor.double().cpu()[good], X[good].double()
    assert bool(torch.isfinite(F).all())
    # the pivots' columns are those of the good states alone
    K = torch.exp(-0.2 * torch.cdist(Xg, X[f.piv].double(), compute_mode="donot_use_mm_for_euclid_dist") ** 2)
    assert float((K - F @ f.factor.double().cpu()[f.piv].T).abs().max()) < (1e-10 if prec == "fp64" else 1e-4)
