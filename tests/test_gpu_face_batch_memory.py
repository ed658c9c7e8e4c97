"""The device memory that the batched face calls keep between calls is bounded
and given back when a context is destroyed.  GPU only; in a process of its
own, which nothing else takes memory in."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import ctypes as C, numpy as np
from flowpsi_b200 import FlowPsi, cases, inviscid_riemann_flux
from tests.helpers import face_states
rt = C.CDLL("libcudart.so.12")
def free():
    f, t = C.c_size_t(), C.c_size_t()
    assert rt.cudaMemGetInfo(C.byref(f), C.byref(t)) == 0
    return f.value
def context():
    c = cases.farfield_cube(4)
    FlowPsi(c.mesh, c.params).close()
n = 400_000  # 76 MB of scratch for a flux
a = face_states(n, 0)
context()
inviscid_riemann_flux("roe", *(v[:10] for v in a))  # kernels loaded
context()
f0 = free()
F = inviscid_riemann_flux("roe", *a)
kept = f0 - free()
assert 25e6 < kept < 160e6, kept
context()
left = f0 - free()
assert left < 8e6, left
assert np.array_equal(F, inviscid_riemann_flux("roe", *a))
print("ok")
"""


def test_kept_memory_is_given_back(need_gpu):
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
