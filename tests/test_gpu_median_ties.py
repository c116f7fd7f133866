"""The bracketed median where the bracket is a power of two of bits wide: the
distances around the median are 1 and v2, and the median, v2, is the last value of
the bracket."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v2", [2, 4, 16])
def test_last_value_of_the_bracket(ctx, v2):
    from kernel_evd_gb300 import api
    # states at the origin, far off, at distance 1 and at distance v2 of the origin:
    # 47.0 % of the pairs at 0, 2.7 % in [1, v2), 2.3 % at v2, the rest far
    n0, far, n1, n2 = 3340, 2394, 142, 124
    X = torch.zeros((n0 + far + n1 + n2, 64))
    X[n0:n0 + far, 63] = 1000.0
    X[n0 + far:n0 + far + n1, 0] = 1.0
    X[n0 + far + n1:, :v2] = 1.0
    X = X[torch.randperm(X.shape[0], generator=torch.Generator().manual_seed(3))].cuda().contiguous()
    assert api.pair_median(ctx, X) == float(v2)
