"""The crystal pass's bounded waits, run out by a short limit and something that nobody sends
(wait_kernels.cu): every CTA of the cluster agrees, the field is NaN, the status says so, the
GPU stays usable.  Marked gpu.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "optifax_gb300", "csrc")
POINTS = [512, 1024, 1024, 16384, 1024]                    # of kinds 0 to 4
SHORT = 2000                                               # looks of 4 us: about 8 ms


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("waits") / "wait_kernels.so")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode=arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "--expt-relaxed-constexpr", "-I" + CSRC, os.path.join(HERE, "wait_kernels.cu"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _pass(lib, kind, clusters, expected):
    from optifax_gb300 import _native as nat
    status = (ctypes.c_int * clusters)()
    flag = ctypes.c_int()
    out = np.ones(2 * POINTS[kind] * clusters, dtype=np.float32)
    rc = lib.wait_pass(kind, clusters, expected, SHORT, status, out.ctypes.data_as(ctypes.c_void_p),
                       ctypes.byref(flag))
    assert rc == 0
    return [s & nat.PULSE_TIMEOUT for s in status], out, flag.value


@pytest.mark.parametrize("kind", range(5))
@pytest.mark.parametrize("clusters", [1, 3])
def test_schedule_that_expects_one_cluster_more(lib, kind, clusters):
    status, out, flag = _pass(lib, kind, clusters, clusters + 1)
    assert all(status) and np.isnan(out).all() and flag == 1
    status, out, flag = _pass(lib, kind, clusters, clusters)           # and the next launch runs
    assert not any(status) and not out.any() and flag == 0


def test_flags_agree_across_a_cluster(lib):
    def run(what):
        out = np.zeros((2, 128), dtype=np.int32)
        assert lib.wait_flags(what, SHORT, out.ctypes.data_as(ctypes.c_void_p)) == 0
        return out
    assert np.all(run(0) == 3)                                         # the OR of both
    a = run(1)                                                         # CTA 0 waits for nothing
    assert np.all(a[0] == 8 + 128)                                     # its wait ran out, for every thread
    assert np.all(a[1] == 64 + 128)                                    # CTA 1 met its last barrier and sees it
    assert np.all(run(2) == 8 + 128)                                   # one knows: both end in the same attempt
