"""The FP64 products in digits over more than one panel of rows, short last panels
included: Gram (panels of 2^20 rows), F from /linv (256 MiB of K) and U (2 GiB of
digits), against FP64 products on rows of every panel."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,k", [((1 << 20) + 1, 7), ((1 << 20) + 1000, 9), ((1 << 21) + 192, 5)])
def test_gram(ctx, N, k):
    from kernel_evd_gb300 import api
    g = torch.Generator("cuda").manual_seed(N)
    F = torch.randn((N, k), dtype=torch.float64, device="cuda", generator=g)
    F[1 << 20:] += 3.0   # the rows past the first panel weigh
    s = torch.rand(N, dtype=torch.float64, device="cuda", generator=g) + 0.5
    G = api.weighted_gram(ctx, F, s)
    ref = sum(y.T @ y for y in (F * s[:, None]).split(1 << 14))
    d = torch.sqrt(torch.diagonal(ref))
    # FP64 sums of 2^14 terms and of their sums: 2^-53 a term at worst
    assert bool(((G - ref).abs() <= 2.0 ** -53 * (2 ** 14 + 2 ** 8) * d[:, None] * d[None, :]).all())


def test_factor_from_linv(ctx):
    from kernel_evd_gb300 import api
    r, N, d, scale = 1000, 34054, 16, 0.02
    g = torch.Generator("cuda").manual_seed(1)
    X = torch.randn((N, d), device="cuda", generator=g)
    piv = np.arange(0, 34 * r, 34)
    Linv = torch.randn((r, r), dtype=torch.float64, device="cuda", generator=g).tril()
    F = api.factor_from_linv(ctx, X, scale, piv, np.asfortranarray(Linv.cpu().numpy()), precision="fp64")
    S = X[torch.from_numpy(piv).cuda()].double()
    for a in (0, 33000, 33554, N - 200):   # 33,554 rows a panel
        D = torch.cdist(X[a:a + 200].double(), S, compute_mode="donot_use_mm_for_euclid_dist")
        K = torch.exp(-scale * D * D)
        assert bool(((F[a:a + 200] - K @ Linv.T).abs() <= 2.0 ** -53 * (r + 100) * (K @ Linv.abs().T)).all())


def test_u(ctx):
    from kernel_evd_gb300 import api
    N, k, k_out = 900000, 300, 8   # 894,784 rows a panel
    g = torch.Generator("cuda").manual_seed(2)
    F = torch.rand((N, k), dtype=torch.float64, device="cuda", generator=g) * torch.rand(k, dtype=torch.float64, device="cuda", generator=g)
    e = api.bistochastic_evd(ctx, F, k_out=k_out, dump=True)
    Z, dt = torch.from_numpy(np.ascontiguousarray(e.dump["Z"])).cuda(), torch.from_numpy(e.dump["dtil"]).cuda()
    for a in (0, 894000, 894784, N - 200):
        f = F[a:a + 200]
        ref = (f @ Z) / dt[a:a + 200, None]
        size = (f @ Z.abs()) / dt[a:a + 200, None]
        assert bool(((e.U[a:a + 200].double() - ref).abs() <= 2.0 ** -24 * ref.abs() + 2.0 ** -44 * size).all())
