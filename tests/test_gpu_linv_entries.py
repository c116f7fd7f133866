"""F from /linv entry by entry: the error of F(i, n) against extended precision,
relative to sum_k |K(i, k)| |Linv(n, k)|, which FP64 arithmetic keeps small for every
entry, however small the entry is against its row."""
import numpy as np
import pytest
import torch

from oracle import ks

pytestmark = pytest.mark.gpu
LD = np.longdouble


def _case(ctx, N, d, r, mul):
    """states, scale (mul over what the calibration selects), pivots and Linv."""
    from kernel_evd_gb300 import api
    X = ks.seeded_mode(N, M=d, seed=d + r, warm_time=150.0).astype(np.float32)
    Xt = torch.from_numpy(X).cuda()
    scale = mul / (0.17 * api.pair_median(ctx, Xt))
    piv = api.rpcholesky(ctx, Xt, scale, r, block=32, seed=3).piv
    S = torch.from_numpy(X[piv]).cuda().double()
    D = torch.cdist(S, S, compute_mode="donot_use_mm_for_euclid_dist")
    L = torch.linalg.cholesky(torch.exp(-scale * D * D))
    Linv = torch.linalg.solve_triangular(L, torch.eye(len(piv), dtype=torch.float64, device="cuda"), upper=False)
    return X, Xt, scale, piv, np.tril(Linv.cpu().numpy())


def _errors(ctx, X, Xt, scale, piv, Linv, precision="fp64"):
    """|F - exact| / sum |K| |Linv| of 24 rows, and their largest exponent scale D."""
    from kernel_evd_gb300 import api
    F = api.factor_from_linv(ctx, Xt, scale, piv, np.asfortranarray(Linv), precision=precision)
    at = np.random.default_rng(1).choice(X.shape[0], 24, replace=False)
    E = LD(scale) * sum((X[at, None, f].astype(LD) - X[piv][None, :, f].astype(LD)) ** 2 for f in range(X.shape[1]))
    K, L = np.exp(-E), Linv.astype(LD)
    ref = np.stack([(K[:, :n + 1] * L[n, :n + 1]).sum(1) for n in range(len(piv))], axis=1)
    size = np.abs(K).astype(float) @ np.abs(Linv).T
    return np.abs(F[torch.from_numpy(at).cuda()].cpu().numpy().astype(LD) - ref).astype(float) / size, float(E.max())


@pytest.mark.parametrize("N,d,r", [(3000, 64, 600), (3000, 64, 200), (2500, 32, 333), (3000, 128, 257)])
def test_calibrated_scale(ctx, N, d, r):
    # K and the result are each within a rounding or two of 2^-53 of S
    err, _ = _errors(ctx, *_case(ctx, N, d, r, 1.0))
    assert np.sqrt((err ** 2).mean()) <= 2.0 ** -52
