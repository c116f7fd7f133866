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
    """|F - exact| / S of 24 rows, S = sum |K| |Linv|, where S is well inside the range of
    FP64, and the largest exponent scale D that counts there."""
    from kernel_evd_gb300 import api
    F = api.factor_from_linv(ctx, Xt, scale, piv, np.asfortranarray(Linv), precision=precision)
    at = np.random.default_rng(1).choice(X.shape[0], 24, replace=False)
    E = LD(scale) * sum((X[at, None, f].astype(LD) - X[piv][None, :, f].astype(LD)) ** 2 for f in range(X.shape[1]))
    K, L = np.exp(-E), Linv.astype(LD)
    ref = np.stack([(K[:, :n + 1] * L[n, :n + 1]).sum(1) for n in range(len(piv))], axis=1)
    size = np.abs(K).astype(float) @ np.abs(Linv).T
    err = np.abs(F[torch.from_numpy(at).cuda()].cpu().numpy().astype(LD) - ref).astype(float)
    live = size > 1e-290
    return err[live] / size[live], min(float(E.max()), 668.0)


@pytest.mark.parametrize("N,d,r", [(3000, 64, 600), (3000, 64, 200), (2500, 32, 333), (3000, 128, 257)])
def test_calibrated_scale(ctx, N, d, r):
    # K and the result are each within a rounding or two of 2^-53 of S
    err, _ = _errors(ctx, *_case(ctx, N, d, r, 1.0))
    assert np.sqrt((err ** 2).mean()) <= 2.0 ** -52


@pytest.mark.parametrize("N,d,r,mul", [(3000, 64, 400, 1.5), (3000, 64, 600, 4.0), (3000, 64, 600, 20.0),
                                       (3000, 32, 333, 1e4)])
def test_wide_kernels(ctx, N, d, r, mul):
    # an FP64 evaluation: the exponent scale D of an entry to a rounding per feature, in
    # the root of their number, and a sum of r terms alike
    X, Xt, scale, piv, Linv = _case(ctx, N, d, r, mul)
    err, top = _errors(ctx, X, Xt, scale, piv, Linv)
    assert np.sqrt((err ** 2).mean()) <= 2.0 ** -53 * (np.sqrt(d) * top + np.sqrt(len(piv)))


@pytest.mark.parametrize("mul", [1.0, 2.0, 8.0])
def test_fp32_output(ctx, mul):
    # the FP64 sum rounded to FP32, entries below the FP32 range aside
    X, Xt, scale, piv, Linv = _case(ctx, 3000, 64, 400, mul)
    F = {}
    for p in ("fp64", "mixed"):
        from kernel_evd_gb300 import api
        F[p] = api.factor_from_linv(ctx, Xt, scale, piv, np.asfortranarray(Linv), precision=p).double()
    size = torch.exp(-scale * torch.cdist(Xt.double(), Xt[torch.from_numpy(piv).cuda()].double(),
                                          compute_mode="donot_use_mm_for_euclid_dist") ** 2)
    size = size @ torch.from_numpy(np.abs(Linv).T.copy()).cuda()
    far = (F["mixed"] - F["fp64"]).abs() > 2.0 ** -24 * F["fp64"].abs() * (1 + 1e-6) + 2.0 ** -28 * size + 2.0 ** -149
    assert not bool(far.any())


def test_uneven_panel(ctx):
    # the second panel (33,554 rows each) alone has rows far from all landmarks but one
    from kernel_evd_gb300 import api
    r, N = 1000, 40000
    g = torch.Generator("cuda").manual_seed(3)
    X = torch.randn((N, 8), device="cuda", generator=g)
    X[36000:] *= 12.0
    piv = np.arange(0, 33 * r, 33)
    Linv = torch.eye(r, dtype=torch.float64) + 1e-3 * torch.randn((r, r), dtype=torch.float64,
                                                                  generator=torch.Generator().manual_seed(1)).tril()
    F = api.factor_from_linv(ctx, X, 0.05, piv, np.asfortranarray(Linv.numpy()), precision="fp64")
    D = torch.cdist(X.double(), X[torch.from_numpy(piv).cuda()].double(), compute_mode="donot_use_mm_for_euclid_dist")
    K = torch.exp(-0.05 * D * D)
    S = K @ Linv.abs().T.cuda()
    live = S > 1e-290
    # exponents up to 668 to a rounding per feature, sums of r terms
    assert bool(((F - K @ Linv.T.cuda()).abs() <= 2.0 ** -53 * (668 * 10 + r) * S)[live].all())
