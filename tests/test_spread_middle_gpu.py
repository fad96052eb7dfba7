"""The middle spread, which mixed calls and medium batches take.  Marked gpu.

Nine pulses of 16384 points do not fit the GPU at 16 CTAs each (7 clusters do) and fit at 8
(15), so the whole call runs at the middle level: 16384 points on 8 CTAs of 2048, 4096 on 4 of
1024, 2048 on one CTA (two of 1024 points take longer and twice the SMs).  Every shape
computes the same pass (tolerance as in test_spread_gpu.py).
"""
import numpy as np
import pytest
import torch

from tests._cases import make_case, rel_l2
from tests.test_spread_gpu import _run, _spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["heun", "rk23", "nee"])
def test_a_mixed_call_takes_the_middle_level(kind):
    from optifax_gb300 import _native as nat
    method = nat.RK23 if kind == "rk23" else nat.HEUN
    variant = {"heun": nat.VARIANT_BATCH_XTAL, "rk23": nat.VARIANT_ODE23, "nee": nat.VARIANT_NEE}[kind]
    cases = {N: make_case(N=N, length=0.02e-3, power=2.0) for N in (2048, 4096, 16384)}
    sizes = [16384] * 9 + [4096] * 2 + [2048] * 2
    out, st, tr = _run([_spec(cases[N][1], cases[N][2][0]) for N in sizes], method, variant)
    for N in cases:
        si, E = cases[N][1], cases[N][2]
        same = [i for i, n in enumerate(sizes) if n == N]
        narrow, sn, tn = _run([_spec(si, E[0])], method, variant, cta_points=min(N, 4096))
        widest, _, _ = _run([_spec(si, E[0])], method, variant)
        for i in same:
            assert st[i]["status"] == 0 and np.array_equal(tr[i][:, :2], tn[0][:, :2]), N
            assert rel_l2(out[i], narrow[0]) <= 1e-5
            assert np.array_equal(out[i], out[same[0]])
        assert not np.array_equal(out[same[0]], widest[0]), N
        assert np.array_equal(out[same[0]], narrow[0]) == (N == 2048), N
        if kind == "heun" and N > 2048:
            asked, _, _ = _run([_spec(si, E[0])], method, variant, cta_points=2048 if N == 16384 else 1024)
            assert np.array_equal(out[same[0]], asked[0])
