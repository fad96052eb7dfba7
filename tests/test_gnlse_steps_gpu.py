"""Fibre step growth: the next step is the accepted one divided in FP64 by an FP32 factor.
Marked gpu.

Steps are integers of about 2^34 to 2^37, so the quotients by neighbouring FP32 factors are
thousands of units apart: a step that is one of them, to the unit, came from that division.
"""
import numpy as np
import pytest

from oracle import gnlse_oracle as go

pytestmark = pytest.mark.gpu

UNITS = 1 << 40                  # of the fibre's length


@pytest.mark.parametrize("n", [512, 4096])
def test_growth_divides_in_fp64(n):
    from optifax_gb300 import gnlse
    T = np.arange(-n // 2, n // 2) * (8e-12 / 4096)
    w0 = 2 * np.pi * 299792458.0 / 835e-9
    A = np.sqrt(1000.0) / np.cosh(T / 28.4e-15)
    ops = gnlse.fibre_operators(T, w0, 0.11, [-1.183e-26, 8.1e-41, -9.5e-56], 0.0, 0.18, go.raman_response(T))
    r = gnlse.propagate(ops, A, 0.08, 2, w0=w0, trace_cap=10000)
    tr = r.trace[0].cpu().numpy()[:r.stats[0]["attempts"]]
    z, grown = 0, 0
    for i in range(len(tr) - 1):
        h, ok, nxt = int(tr[i, 0]), bool(tr[i, 1]), int(tr[i + 1, 0])
        if not ok:
            continue
        z += h
        clean = i == 0 or bool(tr[i - 1, 1])                # no failed attempt before it
        if not clean or nxt in (UNITS // 10, UNITS - z, 5 * h):
            continue
        f = np.float32(h / nxt)
        near = [f]
        for _ in range(3):
            near += [np.nextafter(near[0], np.float32(0)), np.nextafter(near[-1], np.float32(8))]
            near.sort()
        assert nxt in [int(float(h) / float(t)) for t in near], (i, h, nxt)
        grown += 1
    assert grown >= 20


def test_field_error_over_a_power_scan():
    """Fields of 1 to 10 kW pulses over 5 mm against the FP64 oracle on the GPU's own steps.  The
    bound is what transforms in three radix-16 passes had on these pulses (mean 2.70e-7): the
    four passes of radix 8 may not cost precision."""
    from optifax_gb300 import gnlse
    import torch
    n, w0, betas = 4096, 2 * np.pi * 299792458.0 / 835e-9, [-1.183e-26, 8.1e-41, -9.5e-56]
    T = np.arange(-n // 2, n // 2) * (6e-12 / 4096)
    A = (np.sqrt(np.linspace(1e3, 1e4, 90))[:, None] / np.cosh(T / 28.4e-15)).astype(np.complex64)
    RT = go.raman_response(T)
    r = gnlse.propagate(gnlse.fibre_operators(T, w0, 0.11, betas, 0.0, 0.18, RT), torch.from_numpy(A).cuda(), 5e-3, 5,
                        w0=w0, trace_cap=1000)
    ops = go.gnlse_ops(T, w0, 0.11, betas, 0.0, 0.18, RT)
    errs = []
    for b in range(len(A)):
        steps = [(int(h), int(a)) for h, a in r.trace[b].cpu().numpy()[:r.stats[b]["attempts"]]]
        ref = go.propagate(ops, A[b].astype(np.complex128), 5e-3, 5, forced=steps)
        errs.append(np.linalg.norm(r.AT[b].cpu().numpy() - ref.AT) / np.linalg.norm(ref.AT))
    assert np.mean(errs) <= 2.7e-7, (np.mean(errs), np.max(errs))
