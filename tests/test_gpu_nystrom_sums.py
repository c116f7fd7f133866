"""The sums of the out-of-sample kernel.  States whose one near landmark is up to
e^-87 away and has small coefficients: K cancels in the quotient, which is the
landmark's own value.  And the sums over many landmarks against FP64 sums of the
same FP32 kernel values (kernel_block forms them by the same operations): what is
left is the output's rounding, and 2^-40 of the sums of magnitudes (plain FP32 sums
would be 2^-24 of those off)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 320])   # both forms of the kernel
def test_far_states(ctx, n):
    from kernel_evd_gb300 import api
    g = torch.Generator().manual_seed(4)
    X = torch.zeros((2000, 2))
    X[:1999, 0] = 3 * torch.rand(1999, generator=g)
    X[1999, 0] = 50.0
    scale = 0.5
    X = X.cuda()
    fac = api.rpcholesky(ctx, X, scale, 8, block=4, seed=1, precision="fp64")
    assert 1999 in fac.piv
    m = api.NystromModel(ctx, X, fac, k_out=4)
    own = m(X[1999:])[0].double()
    live = own.abs() > 1e-6 * own.abs().max()
    assert int(live.sum()) >= 1
    for a in (1.0, 60.0, 74.0, 78.0, 82.0, 85.0, 87.0):
        Y = torch.zeros((n, 2), device="cuda")
        Y[:, 0] = 50.0 + (a / scale) ** 0.5
        U = m(Y).double()
        assert bool(((U - own).abs() <= 2.0 ** -23 * own.abs())[:, live].all()), a
    m.close()


@pytest.mark.parametrize("d,k,k_out,prec", [(64, 700, 32, "mixed"), (64, 400, 64, "fp64"), (33, 300, 8, "fp64")])
def test_sums_against_fp64(ctx, d, k, k_out, prec):
    from kernel_evd_gb300 import api
    from oracle import ks
    X = torch.from_numpy(ks.seeded_mode(5000, warm_time=100.0).astype(np.float32)[:, :d].copy()).cuda()
    N, scale = 4600, 1.0 / 30.0
    fac = api.rpcholesky(ctx, X[:N].contiguous(), scale, k, block=32, seed=5, precision=prec)
    F = fac.factor.contiguous()
    piv = torch.from_numpy(fac.piv).cuda()
    e = api.bistochastic_evd(ctx, F, k_out=k_out, dump=True)
    m = api.NystromModel(ctx, X[:N].contiguous(), fac, k_out=k_out)
    U = m(X[N:].contiguous()).double()
    m.close()
    rhs = torch.from_numpy(np.concatenate([e.dump["Z"], e.dump["c1"][:, None]], axis=1)).cuda()
    W = torch.linalg.solve_triangular(F[piv].double().tril().T, rhs, upper=True)
    K = api.kernel_block(ctx, X, scale, piv, row0=N, nrows=X.shape[0] - N, precision="mixed").double()
    P, size = K @ W, K @ W.abs()
    ref = P[:, :-1] / P[:, -1:]
    sums = (size[:, :-1] + ref.abs() * size[:, -1:]) / P[:, -1:]
    assert bool(((U - ref).abs() <= 2.0 ** -24 * ref.abs() + 2.0 ** -40 * sums).all())
