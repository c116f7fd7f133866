"""The two forms of the out-of-sample kernel for large batches, a 16-CTA cluster or one
CTA per 32 states, and the form for small ones give a state the same bits; and few
landmarks take less time than many."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(ctx, d, r, k_out):
    from kernel_evd_gb300 import api
    g = torch.Generator("cuda").manual_seed(d + r)
    X = 0.5 * torch.randn((4000, d), device="cuda", generator=g) + torch.linspace(0, 3, 4000, device="cuda")[:, None]
    fac = api.rpcholesky(ctx, X, 0.4 / d, r, block=32, seed=1, precision="fp64")
    return api.NystromModel(ctx, X, fac, k_out=k_out), g


@pytest.mark.parametrize("d,r,k_out", [(64, 1, 1), (64, 33, 8), (130, 100, 33), (3, 16, 5), (64, 513, 64), (257, 300, 2)])
def test_forms_agree(ctx, d, r, k_out):
    m, g = _model(ctx, d, r, k_out)
    Y = torch.randn((16003, d), device="cuda", generator=g)
    whole = m(Y)   # one CTA
    for n in (310, 500, 290):   # clusters from 3 landmark steps on, one CTA, the small form
        for a in (0, 7777, 16003 - n):
            part = m(Y[a:a + n].contiguous())
            assert torch.equal(part.view(torch.int32), whole[a:a + n].contiguous().view(torch.int32))
    m.close()


def test_few_landmarks_are_quick(ctx):
    def best(r):
        m, g = _model(ctx, 64, r, 8)
        Y = torch.randn((65536, 64), device="cuda", generator=g)
        m(Y)
        times = []
        for _ in range(5):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            m(Y)
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        m.close()
        return min(times)
    assert best(96) < 0.6 * best(480)
