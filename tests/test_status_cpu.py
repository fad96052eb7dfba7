"""Statistics of passes on the host: a wait that ran out is an error, other status bits are
the caller's to look at."""
import ctypes

import pytest
import torch

from optifax_gb300 import _native as nat
from optifax_gb300 import solver as sv


def _stats(*status):
    rows = []
    for s in status:
        st = nat.OptifaxPulseStats()
        st.status, st.attempts = s, 7
        rows.append(torch.frombuffer(bytearray(bytes(st)), dtype=torch.int32))
    assert ctypes.sizeof(nat.OptifaxPulseStats) == nat.STATS_BYTES
    return torch.stack(rows)


def test_a_wait_that_ran_out_raises():
    with pytest.raises(nat.OptifaxError, match=r"ran out.*\[1\]"):
        sv.decode_stats(_stats(0, nat.PULSE_TIMEOUT | nat.PULSE_NAN))


def test_other_status_bits_are_returned():
    got = sv.decode_stats(_stats(0, nat.PULSE_NAN, nat.PULSE_ATTEMPT_LIMIT))
    assert [g["status"] for g in got] == [0, 1, 2] and got[0]["attempts"] == 7


def test_choice_of_points_needs_a_handle():
    assert nat.load().optifax_set_cta_points(None, 0) == 5
