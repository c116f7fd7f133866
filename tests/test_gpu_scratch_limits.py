"""Calls that fit the device only when a context gives back the workspaces that it keeps
from other calls: the rest of the memory is taken first, but for a little."""
import contextlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
MIB = 1 << 20


@contextlib.contextmanager
def _only(mib):
    """Leaves mib MiB of the device's free memory."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hold = [torch.empty((torch.cuda.mem_get_info()[0] - mib * MIB) // (2 * MIB) * (2 * MIB), dtype=torch.uint8,
                        device="cuda")]
    try:
        yield
    finally:
        hold.clear()
        torch.cuda.empty_cache()


def _states(N, d=64, seed=0):
    t = torch.linspace(0, 30, N, device="cuda")[:, None]
    noise = torch.randn((N, d), device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    return (torch.cos(t * torch.arange(1, d + 1, device="cuda") / d) + 0.3 * noise).contiguous()


def test_median_buffer():
    from kernel_evd_gb300 import api
    X, Y = _states(1000000), _states(40000)
    F = torch.empty((X.shape[0], 64), device="cuda")
    with api.Context(0) as warm:   # modules and library handles
        ref = api.rpcholesky(warm, X, 0.05, 64, 64, seed=1, F=F).piv
        api.pair_median(warm, Y)
    with api.Context(0) as ctx:
        with _only(310):
            api.pair_median(ctx, Y)   # keeps about 190 MiB
            piv = api.rpcholesky(ctx, X, 0.05, 64, 64, seed=1, F=F).piv   # K(:, S): 244 MiB
    assert np.array_equal(piv, ref)


def test_batch_workspaces():
    from kernel_evd_gb300 import api
    small, big = [_states(200000, seed=s) for s in range(3)], [_states(700000)]
    with api.Context(0) as warm:
        ref = api.rpcholesky_batched(warm, big, [0.05], 64, 64)[0].piv
        api.rpcholesky_batched(warm, small, [0.05] * 3, 64, 64)
    with api.Context(0) as ctx:
        api.rpcholesky_batched(ctx, small, [0.05] * 3, 64, 64)   # keeps about 170 MiB
        with _only(110 + 172):   # the factor, and too little beside it
            piv = api.rpcholesky_batched(ctx, big, [0.05], 64, 64)[0].piv   # about 190 MiB
    assert np.array_equal(piv, ref)


def test_model_beside_batch_workspaces():
    from kernel_evd_gb300 import api
    X, small = _states(3000, 1024), [_states(200000)]
    with api.Context(0) as ctx:
        fac = api.rpcholesky(ctx, X, 0.002, 1000, 64, seed=1)
        api.NystromModel(ctx, X, fac, k_out=8).close()
        api.rpcholesky_batched(ctx, small, [0.05], 64, 64)
        with _only(3):
            api.NystromModel(ctx, X, fac, k_out=8).close()   # landmarks: 4 MB


@pytest.mark.parametrize("leave", [524, 526, 528])
def test_digit_panels_without_room(leave):
    # the kernel panel, Linv and the first digit panel fit, the digits of Linv do not: the
    # FP64 pipe's panel takes the digit panel's place
    from kernel_evd_gb300 import api
    X = _states(40000)
    r, scale = 1000, 0.05
    piv = np.arange(0, 40000, 40)
    with api.Context(0) as ctx:
        Linv = np.asfortranarray(np.tril(np.random.default_rng(1).standard_normal((r, r))))
        ref = api.factor_from_linv(ctx, X, scale, piv, Linv, precision="mixed").double()
    with api.Context(0) as ctx:
        with _only(leave + 154):   # 154: the factor
            out = api.factor_from_linv(ctx, X, scale, piv, Linv, precision="mixed")
    out = out.double()
    size = torch.exp(-scale * torch.cdist(X.double(), X[torch.from_numpy(piv).cuda()].double()) ** 2)
    size = size @ torch.from_numpy(np.abs(Linv).T.copy()).cuda()
    assert bool(((out - ref).abs() <= 2.0 ** -23 * ref.abs() + 2.0 ** -40 * size).all())
