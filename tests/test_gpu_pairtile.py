"""Calibration sums at the edges of the pair tiles (half tiles of 64 rows, groups
that get no tile, ragged features, scale counts around the fours the kernel
reduces together), single and batched, against FP64 on the same states.  The
tolerance is the FP32 form's: ex2.approx (2^-22) and FP32 sums of 2,048 terms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(X, scales):
    X = X.double()
    D = torch.cdist(X, X, compute_mode="donot_use_mm_for_euclid_dist").square()
    m = torch.ones_like(D, dtype=torch.bool).tril(-1)
    return np.array([float(torch.exp(-s * D)[m].sum()) for s in scales])


@pytest.mark.parametrize("N,d,n", [(2, 5, 1), (64, 64, 3), (65, 63, 4), (128, 1, 5), (129, 130, 8), (1000, 64, 41),
                                   (2049, 66, 64)])
def test_sums(ctx, N, d, n):
    from kernel_evd_gb300 import api
    g = torch.Generator().manual_seed(N * 1000 + d)
    X = torch.randn((N, d), generator=g).cuda()
    scales = 2.0 ** np.linspace(-8, 1, n) / (2.0 * d)
    ref = _exact(X, scales)
    out = api.calibrate(ctx, X, scales)
    np.testing.assert_allclose(out, ref, rtol=4e-6, atol=1e-300)
    np.testing.assert_allclose(api.calibrate_batched(ctx, [X, X[: N // 2 + 1].contiguous()], [scales, scales])[0], out,
                               rtol=1e-13)
    np.testing.assert_allclose(api.calibrate_noalloc(X, scales), out, rtol=1e-13)
