"""Calls that run beside others: the handles of a device share the GPU in the choice of points
per CTA, and a handle carries a choice for calls that bring none.  Marked gpu.
"""
import numpy as np
import pytest
import torch

from tests._cases import make_case

pytestmark = pytest.mark.gpu


def _spec(si, E):
    from optifax_gb300 import solver as sv
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(np.asarray(a).astype(d))).cuda()
    return sv.PulseSpec(E=t(E, np.complex64), alpha=t(si.alpha, np.float32), beta=t(si.beta, np.float32),
                        G=t(si.G, np.float32), w0=si.w0, bdiffw0=si.bdiffw0, h=si.h, dt=si.dt, max_err=si.max_err,
                        min_err=si.min_err, sel=si.sel, n_steps=si.n_steps)


def _field(si, E, cta_points=0):
    from optifax_gb300 import solver as sv
    return sv.propagate([_spec(si, E)], cta_points=cta_points)[0][0].cpu().numpy()


@pytest.mark.parametrize("N", [4096, 16384])
def test_many_handles_take_the_narrow_shape(N):
    """One pulse on each of 150 handles fills the GPU at 4096 points per CTA."""
    from optifax_gb300 import _native as nat
    win, si, E = make_case(N=N, length=0.02e-3, power=2.0)
    narrow, wide = _field(si, E[0], 4096), _field(si, E[0])
    assert not np.array_equal(wide, narrow)              # alone: spread over more CTAs, another rounding
    others = [nat.Context(0) for _ in range(149)]
    try:
        assert np.array_equal(_field(si, E[0]), narrow)
    finally:
        for o in others:
            o.close()
    assert np.array_equal(_field(si, E[0]), wide)


def test_the_handle_carries_the_choice():
    """optifax_opo_mex_batch has no argument for it: alone and in a batch the same bits."""
    from optifax_gb300 import _native as nat
    from optifax_gb300 import solver as sv
    N = 4096
    win, si, E = make_case(N=N, length=0.02e-3, power=2.0)
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(np.asarray(a).astype(d))).cuda()
    chunks = sv.n_chunks(si.n_steps, si.sel)

    def mex(k):
        return sv.opo_mex_batch(t(np.repeat(E, k, axis=0), np.complex64), t(si.alpha, np.float32),
                                t(si.G if k == 1 else np.stack([si.G] * k), np.float32), si.w0, si.bdiffw0, si.h, si.n_steps,
                                si.dt, t(si.beta, np.float32), si.max_err, si.min_err, si.sel,
                                torch.zeros((k, chunks, N), dtype=torch.complex64, device="cuda"),
                                torch.zeros(si.n_steps, dtype=torch.float32, device="cuda"))[0].cpu().numpy()
    ctx = sv.context(0)
    wide, narrow = mex(1)[0], _field(si, E[0], 4096)
    assert not np.array_equal(wide, narrow)
    try:
        ctx.set_cta_points(4096)
        assert np.array_equal(mex(1)[0], narrow)
        assert all(np.array_equal(a, narrow) for a in mex(3))
        assert np.array_equal(_field(si, E[0]), narrow)
        ctx.set_cta_points(1024)                           # 4 CTAs a pulse
        assert np.array_equal(mex(1)[0], _field(si, E[0], 1024))
        with pytest.raises(nat.OptifaxError, match="one wave"):
            mex(60)
    finally:
        ctx.set_cta_points(0)
    assert np.array_equal(mex(1)[0], wide)
    for bad in (-1, 100, 256, 3000, 8192):
        with pytest.raises(nat.OptifaxError):
            ctx.set_cta_points(bad)
