"""Line solves whose colours have more groups of 32 lines than the device has
multiprocessors, and fewer, in one system: their launches differ in shared
memory.  GPU only, against the oracle on the same lines and colours (bars of
test_gpu_line_lengths.py), and as a captured step against launched ones."""
import numpy as np
import pytest

from flowpsi_b200 import FlowPsi, cases
from flowpsi_b200.solver import GeneratedMesh, bc

pytestmark = pytest.mark.gpu

N = 110  # 6,050 columns of two cells in one colour: 190 groups; 95 in the others


def uneven_lines(mesh, n):
    """the columns of an n x 2 x n block; of every other one half the columns
    fall apart into single cells"""
    lines = mesh.lines_along(1)
    return [l for i, l in enumerate(lines) if (i % n + i // n) % 2 == 0 or i % 4 < 2]


def _solver(prec, graphs):
    U0 = 0.5 * np.sqrt(cases.GAMMA * cases.RTILDE * 300.0)
    mesh = GeneratedMesh("hex", n=(N, 2, N), L=(1.0, 0.02, 1.0), bc_side=(0,) * 6,
                         bcs=[bc("farfield", u=(U0, 0.0, 0.0))])
    c = cases.farfield_cube(2, precision=prec)
    p = c.params
    p.solver, p.lsgs_max_iter, p.step_graphs = 1, 3, graphs
    g = FlowPsi(mesh, p)
    g.set_lines(uneven_lines(mesh, N))
    state = c.initial_state(g.geometry()["cellcenter"])
    g.set_state(*state)
    return g, mesh, p, state


@pytest.mark.parametrize("prec", ["fp64", "ref", "mixed"])
def test_colours_on_both_sides_of_the_multiprocessors(need_gpu, prec):
    from oracle import Oracle

    g, mesh, p, state = _solver(prec, 1)
    lines, colours = g.line_list()
    groups = [(np.sum(colours == k) + 31) // 32 for k in range(colours.max() + 1)]
    assert max(groups) > 148 > min(groups)

    def dq(s):
        s.set_state(*state)
        s.residual()
        s.assemble()
        return s.linear_solve() if s is g else s.lsgs_solve(lines, colours)[0]

    dg, do = dq(g), dq(Oracle(mesh, p))
    if prec != "fp64":
        p64 = cases.farfield_cube(2, precision="fp64").params
        p64.solver, p64.lsgs_max_iter = 1, 3
        d64 = dq(Oracle(mesh, p64))
    for k in range(5):
        if prec == "fp64":
            assert np.abs(dg[:, k] - do[:, k]).max() <= 1e-8 * np.abs(do[:, k]).max(), k
        else:
            e_orc, e_gpu = (np.abs(d[:, k] - d64[:, k]).max() for d in (do, dg))
            assert e_gpu <= 2.0 * e_orc + 1e-6 * np.abs(d64[:, k]).max(), k
    g.close()


@pytest.mark.parametrize("prec", ["fp64", "ref", "mixed"])
def test_captured_steps_with_such_colours(need_gpu, prec):
    out = []
    for graphs in (0, 1):
        g = _solver(prec, graphs)[0]
        out.append((g.run(5), g.get_state()))
        g.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
