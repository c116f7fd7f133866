"""FP64 products in exact slices (Gram, F from /linv, U) against extended
precision, at the edges of tiles (128 x 64), stages (32 terms) and integer
blocks (128 terms), and the calls that keep the FP64 pipe (uneven columns, not
finite, large scales).

Gram entries are checked relative to sqrt(G_ii G_jj): Y = diag(s) F is rounded
once per entry (2^-53, at random), the sum is exact and is rounded once per row
split: 1e-15 covers both."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gram_err(G, F, s, cols):
    Y = F[:, cols].astype(np.longdouble) * s[:, None].astype(np.longdouble)
    R = Y.T @ Y
    sc = np.sqrt(np.outer(np.diag(R), np.diag(R)))
    return float((np.abs(G[np.ix_(cols, cols)] - R) / sc).max())


@pytest.mark.parametrize("N,k", [(1000, 129), (4097, 64), (33, 600), (31, 577), (130000, 9), (2049, 128), (1153, 193)])
def test_gram(ctx, N, k):
    from kernel_evd_gb300 import api
    rng = np.random.default_rng(N + k)
    F = rng.standard_normal((N, k)) * np.exp(-3 * rng.random((N, k))) * 10.0 ** (-8 * rng.random(k))
    s = np.exp(0.5 * rng.standard_normal(N))
    ld = torch.zeros((N, k + 3), dtype=torch.float64, device="cuda")
    ld[:, :k] = torch.from_numpy(F)
    G = api.weighted_gram(ctx, ld[:, :k], torch.from_numpy(s).cuda(), k=k).cpu().numpy()
    cols = rng.choice(k, min(k, 24), replace=False)
    assert _gram_err(G, F, s, cols) < 1e-15
    np.testing.assert_array_equal(G, G.T)


def test_gram_uneven_column_and_nan(ctx):
    from kernel_evd_gb300 import api
    rng = np.random.default_rng(0)
    F = rng.standard_normal((300000, 6))
    F[17, 2] = 1e7
    s = np.ones(300000)
    G = api.weighted_gram(ctx, torch.from_numpy(F).cuda(), torch.from_numpy(s).cuda()).cpu().numpy()
    assert _gram_err(G, F, s, np.arange(6)) < 1e-13      # the FP64 pipe's sequential sums
    F[5, 1] = np.nan
    G = api.weighted_gram(ctx, torch.from_numpy(F).cuda(), torch.from_numpy(s).cuda()).cpu().numpy()
    assert np.isnan(G[1, 3]) and np.isfinite(G[0, 3])


@pytest.mark.parametrize("N,d,r,scale,precision", [(1000, 20, 330, 0.05, "fp64"), (1025, 64, 321, 0.01, "mixed"),
                                                   (3000, 3, 193, 9.0, "fp64"), (1500, 130, 300, 0.004, "fp64")])
def test_factor_from_linv(ctx, N, d, r, scale, precision):
    from kernel_evd_gb300 import api
    rng = np.random.default_rng(r)
    X = rng.standard_normal((N, d)).astype(np.float32)
    X[r // 2] = X[1]                                      # a coincident pair: K = 1 exactly
    piv = rng.choice(N, r, replace=False)
    Linv = np.tril(rng.standard_normal((r, r))) * 10.0 ** (-3 * rng.random((r, 1)))
    junk = Linv + np.triu(np.full((r, r), 1e30), 1)       # the strict upper part is never read
    F = api.factor_from_linv(ctx, torch.from_numpy(X).cuda(), scale, piv, junk, precision=precision).cpu().numpy()
    Xl = X.astype(np.longdouble)
    D = ((Xl[:, None, :] - Xl[piv][None, :, :]) ** 2).sum(-1) if N * r * d < 3e7 else \
        sum((Xl[:, None, f] - Xl[piv][None, :, f]) ** 2 for f in range(d))
    K = np.exp(-np.longdouble(scale) * D)
    at = rng.choice(N, 60, replace=False)
    R = K[at] @ Linv.astype(np.longdouble).T
    size = np.abs(K[at]) @ np.abs(Linv.T)                 # the sum's own scale
    tol = 2e-15 if precision == "fp64" else 2.0 ** -24 + 1e-14
    err = np.abs(F[at] - R) / (size if precision == "fp64" else np.maximum(np.abs(R), 1e-9 * size))
    # K carries exp's argument to about scale D 2^-52 and its own rounding
    assert float(err.max()) < tol * (1 + 4 * float((scale * D[at]).min(axis=1).max()))
    bad = np.tril(Linv)
    bad[5, 3] = np.nan
    F = api.factor_from_linv(ctx, torch.from_numpy(X).cuda(), scale, piv, bad, precision=precision).cpu().numpy()
    assert np.isnan(F[:, 5]).all() and np.isfinite(F[:, 4]).all()


@pytest.mark.parametrize("N,k,k_out", [(3000, 300, 1), (20001, 65, 65), (5000, 160, 100)])
def test_u(ctx, N, k, k_out):
    """U = Dtil^{-1} F Z of the FP64 EVD (FP32 output) from its own Z and dtil."""
    from kernel_evd_gb300 import api
    rng = np.random.default_rng(k)
    F = np.abs(rng.standard_normal((N, k))) * 2.0 ** (-6 * np.arange(k) / k)
    e = api.bistochastic_evd(ctx, torch.from_numpy(F).cuda(), k_out=k_out if k_out <= k else k, dump=True)
    ref = (F @ e.dump["Z"]) / e.dump["dtil"][:, None]
    U = e.U.cpu().numpy()
    np.testing.assert_allclose(U, ref, rtol=1e-6, atol=1e-7 * np.abs(ref).max())
