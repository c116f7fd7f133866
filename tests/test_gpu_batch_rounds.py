"""Batched factorisations run in chunks of rounds and keep their workspaces with
the context: runs that end by the round limit inside, at and after a chunk, early
stops, one row, odd factor strides, and a second batch of other sizes give what
each job gives alone, bit for bit."""
import numpy as np
import pytest
import torch

from oracle import ks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [True, False])
def test_round_limits(use_graph):
    from kernel_evd_gb300 import api
    ctx = api.Context()
    X = torch.from_numpy(ks.seeded_mode(3000, warm_time=60.0).astype(np.float32)).cuda()
    batches = [  # (rows, k, b, max_rounds)
        [(3000, 301, 32, 1), (2999, 300, 32, 3), (700, 128, 16, 4), (1, 1, 8, 5), (3000, 64, 64, 40)],
        [(129, 200, 32, 8), (3000, 400, 64, 200), (2000, 99, 129, 2), (3000, 200, 32, 9), (500, 7, 1, 12), (1500, 33, 5, 7)],
        [(3000, 301, 32, 5)],
    ]
    for batch in batches:
        Xs = [X[:n].contiguous() for n, _, _, _ in batch]
        got = api.rpcholesky_batched(ctx, Xs, [1.0 / 30.0] * len(batch), [j[1] for j in batch], [j[2] for j in batch],
                                     seeds=range(3, 3 + len(batch)), max_rounds=[j[3] for j in batch],
                                     use_graph=use_graph)
        for q, (n, k, b, limit) in enumerate(batch):
            ref = api.rpcholesky(ctx, Xs[q], 1.0 / 30.0, k_max=k, block=b, seed=3 + q, max_rounds=limit,
                                 precision="mixed")
            assert (got[q].rank, got[q].rounds, got[q].trace_error) == (ref.rank, ref.rounds, ref.trace_error)
            np.testing.assert_array_equal(got[q].piv, ref.piv)
            assert torch.equal(got[q].factor, ref.factor)
