"""The line solver's quotients and their guards as they are compiled
(flowpsi_b200/csrc/line_quotient.cuh, built here with the host compiler): every
quotient that the guards let stand is a / b bit for bit, in both precisions,
and operands outside the ranges do not pass."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HEADER = Path(__file__).resolve().parent.parent / "flowpsi_b200" / "csrc" / "line_quotient.cuh"
SRC = """
#include "HEADER"
#include <cstdint>
using namespace fpsi::dev;
template <class T> static void eval(int64_t n, const T* a, const T* b, T* q, uint8_t* ok) {
  for (int64_t i = 0; i < n; ++i) {
    q[i] = quotient<T>(a[i], b[i], T(1) / b[i]);
    ok[i] = pivot_ok(b[i]) && !tiny<T>(key_min(~0u, a[i]));
  }
}
template <class T> static int smallest_is_tiny(int64_t n, const T* a) {
  uint32_t k = ~0u;
  for (int64_t i = 0; i < n; ++i) k = key_min(k, a[i]);
  return tiny<T>(k);
}
extern "C" {
void eval4(int64_t n, const float* a, const float* b, float* q, uint8_t* ok) { eval(n, a, b, q, ok); }
void eval8(int64_t n, const double* a, const double* b, double* q, uint8_t* ok) { eval(n, a, b, q, ok); }
int tiny4(int64_t n, const float* a) { return smallest_is_tiny(n, a); }
int tiny8(int64_t n, const double* a) { return smallest_is_tiny(n, a); }
}
"""
# mantissa bits, pivot range, smallest dividend, smallest subnormal
FORMAT = {np.float32: (24, (-100, 28), -90, -149), np.float64: (53, (-300, 300), -600, -1074)}


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotient")
    (d / "q.cpp").write_text(SRC.replace("HEADER", str(HEADER)))
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", str(d / "q.cpp"), "-o",
                    str(d / "q.so")], check=True)
    return C.CDLL(str(d / "q.so"))


def _eval(lib, a, b):
    assert a.shape == b.shape and a.dtype == b.dtype
    q, ok = np.empty_like(a), np.empty(a.size, np.uint8)
    p = lambda v: v.ctypes.data_as(C.c_void_p)
    getattr(lib, f"eval{a.itemsize}")(C.c_int64(a.size), p(a), p(b), p(q), p(ok))
    return q, ok.astype(bool)


def _draw(r, t, n, lo, hi):
    """n values with exponents lo..hi and mantissas near a power of two or any"""
    bits = FORMAT[t][0] - 1
    any_ = r.integers(0, 2**bits, n)
    m = np.choose(r.integers(0, 4, n), [any_, any_ % 8, 2**bits - 1 - any_ % 8, any_])
    s = r.choice([-1.0, 1.0], n)
    return np.ldexp((s * (1.0 + m / 2.0**bits)).astype(t), r.integers(lo, hi + 1, n).astype(np.int32)).astype(t)


def _operands(r, t, n):
    _, (lo, hi), small, _ = FORMAT[t]
    top = 127 if t is np.float32 else 1023
    b = np.concatenate([_draw(r, t, n, lo, hi - 1), _draw(r, t, n, lo, lo + 1), _draw(r, t, n, hi - 1, hi - 1)])
    a = np.concatenate([_draw(r, t, n, small, 20), _draw(r, t, n, small, small + 2), _draw(r, t, n, -20, top)])
    with np.errstate(over="ignore", under="ignore"):  # dividends whose quotient is a short number, or nearly
        near = (b * _draw(r, t, b.size, -30, 30)).astype(t)
    return np.concatenate([a, a, near]), np.concatenate([b, r.permutation(b), b])


@pytest.mark.parametrize("t", [np.float32, np.float64])
@pytest.mark.parametrize("seed", range(3))
def test_what_the_guards_let_stand_is_the_division(lib, t, seed):
    r = np.random.default_rng(seed)
    a, b = _operands(r, t, 60000)
    q, ok = _eval(lib, a, b)
    assert np.array_equal(ok, (a == 0) | (np.abs(a) >= np.ldexp(t(1), FORMAT[t][2])))  # every b is in its range
    with np.errstate(over="ignore"):
        want = a / b
    # an overflow anywhere ends in a NaN, which the caller finds
    stands = ok & ~np.isnan(q)
    assert np.array_equal(q[stands], want[stands])
    assert np.isinf(want).any() and np.isnan(q[ok & np.isinf(want)]).all()


@pytest.mark.parametrize("t", [np.float32, np.float64])
def test_operands_outside_the_ranges_do_not_pass(lib, t):
    _, (lo, hi), small, sub = FORMAT[t]
    one = t(1)
    down = lambda x: np.nextafter(x, t(0))
    up = lambda x: np.nextafter(x, t(np.inf))
    two = lambda e: np.ldexp(one, e)
    bs = np.array([two(lo), two(hi), down(two(lo)), up(two(hi)), t(0), t(np.inf), t(np.nan)], t)
    for s in (1, -1):
        assert _eval(lib, np.ones(7, t), t(s) * bs)[1].tolist() == [True, True] + 5 * [False]
    # dividends: at the bound, one step below it, and every binade down to the
    # smallest subnormal; a zero passes
    fine = np.array([two(small), up(two(small)), one, t(0), -t(0)], t)
    bad = np.array([down(two(small))] + [two(e) for e in range(sub, small)]
                   + [down(two(e)) for e in range(sub + 1, small)], t)
    for s in (1, -1):
        assert _eval(lib, t(s) * fine, np.ones(fine.size, t))[1].all()
        v = t(s) * bad
        assert not _eval(lib, v, np.ones(v.size, t))[1].any()


@pytest.mark.parametrize("t", [np.float32, np.float64])
def test_the_smallest_dividend_of_several_decides(lib, t):
    f = getattr(lib, f"tiny{np.dtype(t).itemsize}")

    def call(*v):
        a = np.array(v, t)
        return f(C.c_int64(a.size), a.ctypes.data_as(C.c_void_p))

    sub = np.ldexp(t(1), FORMAT[t][3])
    assert call(1, 2, 0, -3) == 0
    assert call(1, 0, sub, -3) == 1 and call(-sub, 0) == 1 and call(0, 0) == 0
