"""The crystal pass's own choice of points per CTA, and the error class away from its
common path.  Marked gpu.

A call without a choice of the caller spreads a pulse over more CTAs while the GPU holds
the whole call at once.  Every shape computes the same pass: the step schedule is that of
4096 points per CTA and the fields differ by FP32 rounding only (each is within 1e-4 of
the FP64 oracle in test_parity_gpu.py; two FP32 passes of ~100 steps differ by ~1e-6).
"""
import numpy as np
import pytest
import torch

from tests._cases import make_case, rel_l2

pytestmark = pytest.mark.gpu


def _spec(si, E, **kw):
    from optifax_gb300 import solver as sv
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(np.asarray(a).astype(d))).cuda()
    return sv.PulseSpec(E=t(E, np.complex64), alpha=t(si.alpha, np.float32), beta=t(si.beta, np.float32),
                        G=t(si.G, np.float32), w0=si.w0, bdiffw0=si.bdiffw0, h=si.h, dt=si.dt,
                        max_err=kw.pop("max_err", si.max_err), min_err=kw.pop("min_err", si.min_err), sel=si.sel,
                        n_steps=si.n_steps, trace_cap=20000, **kw)


def _run(specs, method, variant, cta_points=0):
    from optifax_gb300 import solver as sv
    outs, st = sv.propagate(specs, method=method, variant=variant, cta_points=cta_points)
    st = sv.decode_stats(st)
    return [o.cpu().numpy() for o in outs], st, [p.trace.cpu().numpy()[:s["attempts"]] for p, s in zip(specs, st)]


@pytest.mark.parametrize("N", [2048, 4096, 8192, 16384, 32768])
@pytest.mark.parametrize("kind", ["heun", "rk23", "nee"])
def test_spread_computes_the_same_pass(N, kind):
    from optifax_gb300 import _native as nat
    if N == 32768 and kind != "heun":
        pytest.skip("no kernel of this schedule at this size")
    method = nat.RK23 if kind == "rk23" else nat.HEUN
    variant = {"heun": nat.VARIANT_BATCH_XTAL, "rk23": nat.VARIANT_ODE23, "nee": nat.VARIANT_NEE}[kind]
    win, si, E = make_case(N=N, length=0.02e-3, power=2.0)
    a, sa, ta = _run([_spec(si, E[0])], method, variant)
    b, sb, tb = _run([_spec(si, E[0])], method, variant, cta_points=min(N, 4096))
    assert sa[0]["status"] == 0 and np.array_equal(ta[0][:, :2], tb[0][:, :2])
    assert rel_l2(a[0], b[0]) <= 1e-5
    # too many for the wide shapes: the narrow one, bit for bit
    many, sm, _ = _run([_spec(si, E[0]) for _ in range(160)], method, variant)
    assert all(np.array_equal(m, b[0]) for m in many)


@pytest.mark.parametrize("N", [512, 4096])
def test_error_class_off_the_common_path(oracle, N):
    """Bounds that the approximate class cannot decide (zero, or equal to what the pass
    meets) and vanishing or non-finite fields, against the oracle's decisions."""
    from optifax_gb300 import _native as nat
    win, si, E = make_case(N=N, length=0.01e-3, power=2.0)
    for hi, lo in ((0.05, 0.0), (0.0, 0.0), (1e-3, 1e-3), (5e-2, 5e-2)):
        _, st, tr = _run([_spec(si, E[0], max_err=hi, min_err=lo)], nat.HEUN, nat.VARIANT_BATCH_XTAL)
        ref = oracle.run(E[0], si.alpha, si.G, si.beta, w0=si.w0, bdiffw0=si.bdiffw0, h=si.h, n_steps=si.n_steps,
                         dt=si.dt, max_err=float(np.float32(hi)), min_err=float(np.float32(lo)), sel=si.sel,
                         trace_cap=20000)
        assert np.array_equal(tr[0][:, :2], ref.trace[0][:, :2]), (hi, lo)
    z, st, tr = _run([_spec(si, np.zeros(N))], nat.HEUN, nat.VARIANT_BATCH_XTAL)
    assert st[0]["status"] == 0 and not z[0].any() and np.all((tr[0][:, 2] & 7) == 0)
    bad = E[0].copy()
    bad[N // 3] = np.nan
    _, st, tr = _run([_spec(si, bad)], nat.HEUN, nat.VARIANT_BATCH_XTAL)
    assert st[0]["status"] & 1 and np.all(tr[0][:, 2] & 4)
