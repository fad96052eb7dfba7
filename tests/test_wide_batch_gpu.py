"""Wide-state batches of 8192 points on both sides of the shape's change.  Marked gpu.

The GPU holds 14 clusters of 16 CTAs of 512 points and 15 of 8 of 1024: a call of 15 pulses
takes the second shape.  Equal pulses on one schedule take a single pulse's steps, and the
shapes differ by rounding (tolerances of the single-pulse tests against the FP64 oracle).
"""
import numpy as np
import pytest
import torch

from tests._cases import make_case, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry,variant,tol", [("propagate_fp64", 0, 1e-11), ("propagate_fp64", 5, 1e-11),
                                               ("propagate_f32x2", 0, 1e-10)])
def test_both_shapes_compute_the_same_pass(entry, variant, tol):
    from optifax_gb300 import solver as sv
    win, si, E = make_case(N=8192, length=0.01e-3, power=2.0)
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(np.asarray(a).astype(d))).cuda()

    def run(B):
        A, st, tr = getattr(sv, entry)(t(np.repeat(E, B, axis=0), np.complex128), t(si.alpha, np.float64),
                                       t(si.beta, np.float64), t(si.G, np.float64), w0=si.w0, bdiffw0=si.bdiffw0, h=si.h,
                                       dt=si.dt, n_steps=si.n_steps, max_err=si.max_err, min_err=si.min_err, sel=si.sel,
                                       variant=variant, trace_cap=10000)
        return A.cpu().numpy(), st, tr
    one, s1, t1 = run(1)
    for B, wide in ((14, True), (15, False)):
        A, st, tr = run(B)
        assert st["status"] == 0 and np.array_equal(tr[:, :2], t1[:, :2])
        for a in A:
            assert rel_l2(a, one[0]) <= tol
            assert np.array_equal(a, one[0]) == wide
