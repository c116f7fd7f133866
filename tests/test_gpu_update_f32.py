"""The FP32-pipe residual update (factor strides the tensor-core update cannot
read, both column widths) and the round factorisation up to b = 128, by backward
error: for the pivots S_q of round q, K(:, S_q) - F F(S_q)^T in FP64 against the
first-order bound of FP32 rounding.  With u = 2^-24:

  G_i = K - F F_S^T (old columns)   |e| <= u ((d + 2) / e + 3 + r + b): distances in
        FP32 (t e^-t <= 1/e), expf to 2 ulp, an FMA chain with |F_i| |F_s| <= 1
  F_i = fl(G_i L^-T), L^-1 rounded  |e| <= u (m + 1) |F_i| |L^T| |L^-T|, times L^T
  F_S = fl(G_S L^-T) carries e too, which F_i meets as e times |F_i L^-1|_1
"""
import numpy as np
import pytest
import torch

from oracle import ks

pytestmark = pytest.mark.gpu
SCALE = 1.0 / 30.0
U = 2.0 ** -24


@pytest.fixture(scope="module")
def states():
    return ks.seeded_mode(3000, warm_time=100.0).astype(np.float32)


@pytest.mark.parametrize("N,d,k,b", [(3000, 64, 101, 1), (2999, 64, 203, 32), (129, 64, 67, 32), (1000, 63, 130, 33),
                                     (2048, 30, 199, 64), (3000, 64, 301, 65), (2500, 64, 331, 128)])
def test_against_fp64(ctx, states, N, d, k, b):
    from kernel_evd_gb300 import api
    X = np.ascontiguousarray(states[:N, :d])
    F = torch.full((N, k + (1 if k % 2 == 0 else 2)), 7.0, device="cuda")   # an odd stride
    g = api.rpcholesky(ctx, torch.from_numpy(X).cuda(), SCALE, k, block=b, seed=5, precision="mixed", F=F)
    assert bool((F[:, g.rank:] == 7.0).all()) and int(g.accepted.sum()) == g.rank
    Xd = torch.from_numpy(X).cuda().double()
    Fd, piv, r = g.factor.double(), torch.from_numpy(g.piv).cuda(), 0
    for m in (int(a) for a in g.accepted if a > 0):
        S = piv[r:r + m]
        K = torch.exp(-SCALE * torch.cdist(Xd, Xd[S], compute_mode="donot_use_mm_for_euclid_dist") ** 2)
        L = torch.linalg.cholesky(K[S] - Fd[S, :r] @ Fd[S, :r].T)
        Li = torch.linalg.inv(L)
        Fq = Fd[:, r:r + m]
        e = U * ((d + 2) / np.e + 3 + r + b)
        w = (Fq @ Li).abs().sum(1, keepdim=True)
        # both F_i and F_S are rounded products
        inv = U * (m + 1) * Fq.abs() @ (L.T.abs() @ Li.T.abs() @ L.T.abs())
        bound = e * (1 + w) + inv + inv[S].T.abs().amax() * (1 + w)
        err = (K - Fd[:, :r + m] @ Fd[S, :r + m].T).abs()
        assert bool((err <= bound).all()), (r, float((err / bound).max()))
        r += m
    assert abs(g.trace_error - float((1.0 - (Fd * Fd).sum(1)).clamp_min(0).mean())) < 1e-6
