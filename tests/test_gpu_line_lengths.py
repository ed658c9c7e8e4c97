"""Line solves at the lengths where their walk changes: less than a stage's
rows, whole stages, a remainder, mixed lengths and single cells in one group
of 32 lines, and lines too long for the forward results to stay in shared
memory.  GPU only, against the oracle on the same lines and colours, with the
bars of test_gpu_lsgs.py (FP64 1e-8 of max|dq|; FP32 blocks within twice the
oracle's own FP32 distance from its FP64 result)."""
import numpy as np
import pytest

from flowpsi_b200 import FlowPsi, cases
from flowpsi_b200.solver import GeneratedMesh, bc
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _case(ny, prec):
    c = cases.farfield_cube(2, precision=prec)
    U0 = 0.5 * np.sqrt(cases.GAMMA * cases.RTILDE * 300.0)
    mesh = GeneratedMesh("hex", n=(5, ny, 3), L=(1.0, ny / 5.0, 0.6), bc_side=(0,) * 6,
                         bcs=[bc("farfield", u=(U0, 0.0, 0.0))])
    c.params.solver, c.params.lsgs_max_iter = 1, 4
    return mesh, c


def _lines(mesh, ny, mixed):
    lines = mesh.lines_along(1)
    if not mixed:
        return lines
    # cut every column at its own places; some pieces are left out (single
    # cells then)
    out = []
    for i, l in enumerate(lines):
        cuts = sorted({(7 * i + 3 * k) % ny for k in range(i % 4)} | {0, ny})
        out += [l[a:b] for a, b in zip(cuts[:-1], cuts[1:]) if (a + i) % 5]
    return out


def _dq64(ny, state, lines, colours):
    mesh, c = _case(ny, "fp64")
    o = Oracle(mesh, c.params)
    o.set_state(*state)
    o.residual()
    o.assemble()
    return o.lsgs_solve(lines, colours)[0]


@pytest.mark.parametrize("prec", ["fp64", "ref", "mixed"])
@pytest.mark.parametrize("ny,mixed", [(2, False), (3, False), (4, False), (9, False),
                                      (23, True), (64, True), (400, False)])
def test_line_lengths_match_oracle(need_gpu, ny, mixed, prec):
    mesh, c = _case(ny, prec)
    g, o = FlowPsi(mesh, c.params), Oracle(mesh, c.params)
    g.set_lines(_lines(mesh, ny, mixed))
    lines, colours = g.line_list()
    state = c.initial_state(o.geometry()["cellcenter"])
    for s in (g, o):
        s.set_state(*state)
        s.residual()
        s.assemble()
    dg, do = g.linear_solve(), o.lsgs_solve(lines, colours)[0]
    if prec != "fp64":
        d64 = _dq64(ny, state, lines, colours)
    for k in range(5):
        if prec == "fp64":
            assert np.abs(dg[:, k] - do[:, k]).max() <= 1e-8 * np.abs(do[:, k]).max(), k
        else:
            e_orc, e_gpu = (np.abs(d[:, k] - d64[:, k]).max() for d in (do, dg))
            assert e_gpu <= 2.0 * e_orc + 1e-6 * np.abs(d64[:, k]).max(), k
    g.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_zero_right_hand_side_stays_zero(need_gpu, prec):
    """a uniform freestream: the residual is at rounding level or zero, every
    dividend of the line solves tiny"""
    mesh, c = _case(21, prec)
    g = FlowPsi(mesh, c.params)
    g.set_lines(mesh.lines_along(1))
    nc = g.ncells
    u = np.zeros((nc, 3))
    u[:, 0] = 0.5 * np.sqrt(cases.GAMMA * cases.RTILDE * 300.0)
    g.set_state(np.full(nc, 300.0), np.full(nc, 1e5), u)
    g.residual()
    g.assemble()
    dq = g.linear_solve()
    assert np.isfinite(dq).all()
    assert np.abs(dq[:, 0]).max() <= 1e-6 and np.abs(dq[:, 4]).max() <= 1e-3  # of 300 K, 1e5 Pa
    g.close()


@pytest.mark.parametrize("prec", ["ref", "mixed"])
@pytest.mark.parametrize("size", [1e-16, 1e-15, 1e-7])
def test_small_domains_match_oracle(need_gpu, size, prec):
    """areas so small that the FP32 blocks' pivots lie below the range of the
    stored reciprocals (2^-100; most of them, some, none): the factoring and
    the solves take their divisions there.  Bars as above."""
    def mk(p):
        mesh, c = _case(9, p)
        U0 = 0.5 * np.sqrt(cases.GAMMA * cases.RTILDE * 300.0)
        return GeneratedMesh("hex", n=(5, 9, 3), L=(size, 1.8 * size, 0.6 * size), bc_side=(0,) * 6,
                             bcs=[bc("farfield", u=(U0, 0.0, 0.0))]), c

    mesh, c = mk(prec)
    g = FlowPsi(mesh, c.params)
    g.set_lines(mesh.lines_along(1))
    lines, colours = g.line_list()
    o, o64 = Oracle(mesh, c.params), Oracle(*(lambda m, k: (m, k.params))(*mk("fp64")))
    cc = o.geometry()["cellcenter"] / size
    state = (300.0 + 20.0 * np.sin(5 * cc[:, 0]), 1e5 + 5e3 * np.cos(4 * cc[:, 1]),
             50.0 + 30.0 * np.sin(3 * cc + [0.0, 1.0, 2.0]))
    for s in (g, o, o64):
        s.set_state(*state)
        s.residual()
        s.assemble()
    dg, do, d64 = g.linear_solve(), o.lsgs_solve(lines, colours)[0], o64.lsgs_solve(lines, colours)[0]
    for k in range(5):
        e_orc, e_gpu = (np.abs(d[:, k] - d64[:, k]).max() for d in (do, dg))
        assert e_gpu <= 2.0 * e_orc + 1e-6 * np.abs(d64[:, k]).max(), k
    g.close()
