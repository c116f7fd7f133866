"""Plain FP64 rounds of few proposals (b <= 8) against the FP64 oracle: pivots
bit-identical, factor and trace errors to 1e-10, as for the general round.
Sizes at the edges of the 16-row blocks, of the 32-lane sums and of the four
pivot widths (1, 2, 4, 8)."""
import numpy as np
import pytest
import torch

from oracle import ks, rpchol

pytestmark = pytest.mark.gpu
SCALE = 1.0 / 30.0


@pytest.fixture(scope="module")
def states():
    return ks.seeded_mode(3000, warm_time=100.0).astype(np.float32)


@pytest.mark.parametrize("N,d,k,b", [(16, 64, 16, 1), (17, 33, 9, 2), (777, 64, 100, 1), (1000, 31, 65, 3),
                                     (3000, 64, 120, 5), (2999, 7, 40, 8), (31, 64, 30, 8)])
def test_small_rounds_match_oracle(ctx, states, N, d, k, b):
    from kernel_evd_gb300 import api
    X = np.ascontiguousarray(states[:N, :d])
    ref = rpchol.rpcholesky(X.astype(np.float64), SCALE, k, b, seed=40 + b, n_rounds=6 * k)
    F = torch.full((N, k + 3), 7.0, dtype=torch.float64, device="cuda")   # a row stride of its own
    g = api.rpcholesky(ctx, torch.from_numpy(X).cuda(), SCALE, k, block=b, seed=40 + b, max_rounds=6 * k,
                       precision="fp64", F=F)
    assert g.rank == ref["F"].shape[1]
    np.testing.assert_array_equal(g.piv, ref["piv"])
    np.testing.assert_array_equal(g.accepted, ref["hm"])
    np.testing.assert_allclose(g.err, ref["err"], rtol=1e-10, atol=1e-14)
    np.testing.assert_allclose(g.factor.cpu().numpy(), ref["F"], rtol=0, atol=1e-10)
    assert bool((F[:, g.rank:] == 7.0).all())   # nothing is written past the rank
