"""Out-of-sample kernel at the edges of its tiles: ragged features, several
feature chunks, fewer landmark steps than groups, one and four states per
thread row.  On training rows it reproduces the U of the EVD it was built from
(same coefficients, FP32 outputs): 2e-6 of max|U|, as in test_gpu_serve.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,d,k,k_out,n", [(400, 3, 20, 5, 9), (400, 130, 33, 32, 1), (900, 64, 513, 33, 305),
                                           (900, 257, 70, 64, 304), (5000, 20, 300, 1, 4999), (64, 16, 1, 1, 64)])
def test_training_rows(ctx, N, d, k, k_out, n):
    from kernel_evd_gb300 import api
    g = torch.Generator().manual_seed(N + d)
    # a curve in d dimensions plus a little noise: a spectrum without clusters
    t = torch.linspace(0, 3, N)[:, None]
    X = (torch.cos(t * torch.arange(1, d + 1) / d) + 0.02 * torch.randn((N, d), generator=g)).float().cuda()
    scale = 4.0 / d
    fac = api.rpcholesky(ctx, X, scale, k, block=min(k, 16), seed=5, precision="fp64")
    k_out = min(k_out, fac.rank)
    e = api.bistochastic_evd(ctx, fac.factor.contiguous(), k_out=k_out)
    m = api.NystromModel(ctx, X, fac, k_out=k_out)
    at = torch.randperm(N, generator=g)[:n].cuda()
    lead = min(k_out, 4)   # the leading columns: the others' coefficients may be ill-conditioned
    U, ref = m(X[at].contiguous())[:, -lead:].double(), e.U[at][:, -lead:].double()
    sgn = torch.sign((U * ref).sum(0))
    assert float((U * sgn - ref).abs().max()) <= 2e-6 * float(e.U[:, -lead:].abs().max())
    whole = m(X)   # a state's values do not depend on its batch
    assert torch.equal(whole[at], m(X[at].contiguous()))
    m.close()
