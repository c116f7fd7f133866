"""The one-pass median over all pairs equals the radix selection over the same
pairs given explicitly, bit for bit: smooth data, data with many ties (the
bracket overflows) and data whose median lies between two clusters."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,N,d", [("normal", 4100, 64), ("normal", 4097, 3), ("normal", 4003, 130),
                                      ("ties", 4050, 5), ("clusters", 4200, 16), ("inf", 4010, 4)])
def test_equals_radix_selection(ctx, kind, N, d):
    from kernel_evd_gb300 import api
    g = torch.Generator().manual_seed(N)
    X = torch.randn((N, d), generator=g)
    if kind == "ties":
        X = torch.round(X)
    elif kind == "clusters":
        X[: N // 2] = 0.01 * X[: N // 2]
        X[N // 2:] = 0.01 * X[N // 2:] + 5.0
    elif kind == "inf":
        X[: N // 2] *= 1e30
    X = X.cuda().contiguous()
    i = torch.tril_indices(N, N, -1, device="cuda")
    ref = api.pair_median(ctx, X, pairs=(i[0].contiguous(), i[1].contiguous()))
    assert np.float64(api.pair_median(ctx, X)).tobytes() == np.float64(ref).tobytes()
