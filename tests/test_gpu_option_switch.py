"""Options that change between a residual and what is built from it: the
assembly uses the last residual's state with the options in force, as a new
context that was given those options from the start.  GPU only."""
import numpy as np
import pytest

from flowpsi_b200 import FlowPsi, cases
from flowpsi_b200._native import FLUX
from tests.helpers import block_rel

pytestmark = pytest.mark.gpu

# FP32 blocks: both sides evaluate the same formulas in FP64 and round once
# (the bars of test_gpu_viscous.py)
TOL = {"ref": 1e-6, "fp64": 1e-11}


def _case(flux, prec):
    c = cases.boundary_layer_block(6, 8, 4, dy0=1e-3, growth=1.3, viscous=1, precision=prec, solver="sgs")
    c.params.flux = FLUX[flux]
    return c


def _states(g, c):
    T, p, u = c.initial_state(g.geometry()["cellcenter"])
    r = np.random.default_rng(5)
    a = (T * (1.0 + 0.1 * r.random(T.size)), p, u)
    b = (2.5 * T * (1.0 + 0.1 * r.random(T.size)), p, u * (1.0 + 0.1 * r.random(u.shape)))
    return a, b


def _blocks(g):
    g.assemble()
    return g.blocks()


def _compare(got, want, prec):
    for k in ("fjp", "fjm"):
        inner = np.abs(want[k]).reshape(len(want[k]), -1).max(1) > 0
        assert block_rel(got[k][inner], want[k][inner]) < TOL[prec], k


@pytest.mark.parametrize("prec", ["ref", "fp64"])
def test_viscosity_follows_the_state_of_an_inviscid_residual(need_gpu, prec):
    """viscous on state A, inviscid on state B, viscous again: the KEC flux
    keeps the gradient records of B, the viscosities have to be B's too"""
    c = _case("kec", prec)
    g = FlowPsi(c.mesh, c.params)
    A, B = _states(g, c)
    p = g.params
    g.set_state(*A)
    g.residual()
    p.viscous = 0
    g.set_params(p)
    g.set_state(*B)
    g.residual()
    p.viscous = 1
    g.set_params(p)
    got = _blocks(g)
    # the time step is the inviscid residual's: the new context switches as well
    d = _case("kec", prec)
    d.params.viscous = 0
    f = FlowPsi(d.mesh, d.params)
    f.set_state(*B)
    f.residual()
    d.params.viscous = 1
    f.set_params(d.params)
    _compare(got, _blocks(f), prec)
    f.close(), g.close()


@pytest.mark.parametrize("prec", ["ref", "fp64"])
def test_viscous_blocks_after_an_inviscid_residual(need_gpu, prec):
    """viscous on state A, inviscid (Roe: no gradient records) on state B,
    viscous again: the face Jacobians are those of a viscous context on B"""
    c = _case("roe", prec)
    g = FlowPsi(c.mesh, c.params)
    A, B = _states(g, c)
    p = g.params
    g.set_state(*A)
    g.residual()
    p.viscous = 0
    g.set_params(p)
    g.set_state(*B)
    g.residual()
    p.viscous = 1
    g.set_params(p)
    got = _blocks(g)
    d = _case("roe", prec)
    f = FlowPsi(d.mesh, d.params)
    f.set_state(*B)
    f.residual()
    _compare(got, _blocks(f), prec)
    f.close(), g.close()


@pytest.mark.parametrize("prec", ["ref", "fp64"])
def test_face_records_follow_the_gas(need_gpu, prec):
    """gamma changed between an inviscid residual and the assembly: the face
    Jacobians are those of the new gas (the face states' pressures,
    temperatures and velocities, first order here, do not depend on it)"""
    c = cases.farfield_cube(6, precision=prec, limiter="zero")
    g = FlowPsi(c.mesh, c.params)
    st = c.initial_state(g.geometry()["cellcenter"])
    g.set_state(*st)
    g.residual()
    p = g.params
    p.gamma = 1.3
    g.set_params(p)
    got = _blocks(g)
    d = cases.farfield_cube(6, precision=prec, limiter="zero")
    d.params.gamma = 1.3
    f = FlowPsi(d.mesh, d.params)
    f.set_state(*st)
    f.residual()
    want = _blocks(f)
    # interior faces: a boundary state may depend on gamma
    inner = d.mesh.arrays().cr >= 0
    for k in ("fjp", "fjm"):
        assert block_rel(got[k][inner], want[k][inner]) < TOL[prec], k
    f.close(), g.close()


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_line_solve_from_a_given_start_after_a_diverged_one(need_gpu, prec):
    """an infinite relaxation factor leaves NaN everywhere, in the line
    layout's padding too; a solve from a given start afterwards is a new
    context's, its measured residual and its stopping test included"""
    def mk():
        c = cases.boundary_layer_block(5, 7, 3, dy0=1e-3, growth=1.3, precision=prec, solver="lsgs")
        c.params.lsgs_max_iter, c.params.lsgs_abs_tol, c.params.lsgs_rel_tol = 30, 0.0, 1e-2
        g = FlowPsi(c.mesh, c.params)
        g.set_lines(c.lines)
        g.set_state(*c.initial_state(g.geometry()["cellcenter"]))
        return g

    g, f = mk(), mk()
    x0 = 1e-3 * np.random.default_rng(1).standard_normal((g.ncells, 5))
    p = g.params
    w, p.lsgs_relaxation = p.lsgs_relaxation, np.inf
    g.set_params(p)
    g.residual()
    g.assemble()
    assert np.isnan(g.linear_solve()).any()
    p.lsgs_relaxation = w
    g.set_params(p)
    out = []
    for s in (g, f):
        s.residual()
        s.assemble()
        out.append(s.linear_solve(x0, info=True))
    (dg, ig), (df, jf) = out
    assert 0 < jf["iterations"] < 30 and np.isfinite(jf["resid"])
    assert ig == jf and np.array_equal(dg, df)
    f.close(), g.close()
