"""Runs test code in a child process whose CUDA runtime is tests/fake_cudart.c,
so that the library's host code can be looked at without a GPU: what it
launches, allocates and waits for, and what it does when a call fails.

The code sees ``calls``, a list of Call records, ``names(pattern)``, the
kernels launched so far whose mangled name contains the pattern, and ``on``, a
list of functions; each is given a call before it takes effect and may return
the CUDA error that the call then gives.
"""
import os
import subprocess
import sys
import tempfile
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
SRC = Path(__file__).resolve().parent / "fake_cudart.c"

PRELUDE = """
import ctypes as C, os
from collections import namedtuple
import numpy as np
Call = namedtuple("Call", "what name stream p q n args")
calls, on = [], []
_T = C.CFUNCTYPE(C.c_int, C.c_char_p, C.c_char_p, *[C.c_uint64] * 4, C.c_void_p)
def _hook(what, name, stream, p, q, n, args):
    c = Call(what.decode(), name.decode(), stream, p, q, n, args)
    calls.append(c)
    for f in on:
        e = f(c)
        if e:
            return e
    return 0
_cb = _T(_hook)
_fake = C.CDLL(os.environ["LD_PRELOAD"])
_fake.fake_set_hook(_cb)
def names(pattern):
    return [c.name for c in calls if c.what == "launch" and pattern in c.name]
from flowpsi_b200 import FlowPsi, FpsiError, cases
"""


def run(code: str) -> str:
    """the child's output; fails with it when the code raises"""
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    with tempfile.TemporaryDirectory() as d:
        so = Path(d) / "fake_cudart.so"
        subprocess.run(["gcc", "-O1", "-shared", "-fPIC", f"-I{cuda}/include", str(SRC), "-o", str(so)], check=True)
        r = subprocess.run([sys.executable, "-c", PRELUDE + code], cwd=ROOT, capture_output=True, text=True,
                           timeout=300, env={**os.environ, "LD_PRELOAD": str(so)})
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
