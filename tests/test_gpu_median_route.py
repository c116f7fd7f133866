"""The bracketed median at sizes where it is the form in use, against the radix
selection over the same pairs given explicitly, bit for bit, and with so many ties
that the sample turns the bracket down before its pass (then no slower than the
radix selection's three passes alone)."""
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,d,ties", [(9500, 3, False), (7100, 17, False), (4800, 64, False), (2900, 300, False),
                                      (7100, 17, True)])
def test_equals_radix_selection(ctx, N, d, ties):
    from kernel_evd_gb300 import api
    X = torch.randn((N, d), generator=torch.Generator().manual_seed(N))
    X = (torch.round(X) if ties else X).cuda().contiguous()
    i = torch.tril_indices(N, N, -1, device="cuda")
    ref = api.pair_median(ctx, X, pairs=(i[0].contiguous(), i[1].contiguous()))
    assert np.float64(api.pair_median(ctx, X)).tobytes() == np.float64(ref).tobytes()


def test_ties_skip_the_pass(ctx):
    from kernel_evd_gb300 import api

    def best(X):
        t = []
        for _ in range(7):
            t0 = time.perf_counter()
            api.pair_median(ctx, X)
            t.append(time.perf_counter() - t0)
        return min(t)
    g = torch.Generator().manual_seed(5)
    X = torch.round(torch.randn((100000, 16), generator=g)).cuda()
    # past N = 160,000 there is no bracket: three passes, 2.62 times the pairs
    Y = torch.round(torch.randn((161800, 16), generator=g)).cuda()
    assert best(X) < 1.15 * best(Y) / 2.618
