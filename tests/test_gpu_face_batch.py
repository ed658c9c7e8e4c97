"""The batched face calls' shared scratch: sizes below, at and above what it
keeps between calls, several threads at once, and a device reset between
calls.  GPU only.  The same call on the same faces gives the same bits, so
every result is compared exactly with the one a single whole batch gave."""
import subprocess
import sys
import threading

import numpy as np
import pytest

from flowpsi_b200 import inviscid_riemann_flux, roe_jacobian
from tests.helpers import face_states

pytestmark = pytest.mark.gpu


def _all(n, seed=0):
    return face_states(n, seed)


def test_sizes_and_threads_agree(need_gpu):
    n = 700000  # 109 MB of scratch for a flux, 151 MB for FP64 Jacobians
    qL, qR, an, area = _all(n)
    F = inviscid_riemann_flux("roe", qL, qR, an, area)
    J = roe_jacobian(qL, qR, an, area, 1, as_double=True)
    for m in (1, 31, 128, 129, 5000, 400000):
        s = slice(n - m, n)
        assert np.array_equal(F[s], inviscid_riemann_flux("roe", qL[s], qR[s], an[s], area[s]))
    bad = []

    def work(k):
        for i in range(20):
            m = 1 + (7919 * (k + 1) * (i + 1)) % 9000
            s = slice(1000 * k, 1000 * k + m)
            f = inviscid_riemann_flux("roe", qL[s], qR[s], an[s], area[s])
            j = roe_jacobian(qL[s], qR[s], an[s], area[s], 1, as_double=True)
            if not (np.array_equal(f, F[s]) and np.array_equal(j, J[s])):
                bad.append((k, i))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_calls_work_after_a_device_reset(need_gpu):
    code = """
import ctypes, numpy as np
from flowpsi_b200 import inviscid_riemann_flux
from tests.helpers import face_states
a = face_states(300, 1)
f = inviscid_riemann_flux("hllc", *a)
rt = ctypes.CDLL("libcudart.so.12")
assert rt.cudaDeviceReset() == 0
assert np.array_equal(f, inviscid_riemann_flux("hllc", *a))
print("ok")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
