"""A context keeps its instantiated step graph between runs and writes each
run's own step into it: runs whose options changed in between (values only, or
the launches themselves) against a new context's, bit for bit.  GPU only."""
import numpy as np
import pytest

from flowpsi_b200 import FlowPsi, cases

pytestmark = pytest.mark.gpu

# sweeps, cflmax, flux, steps
SEQ = [(5, 1e4, 0, 4), (5, 1e4, 0, 5), (5, 20.0, 0, 4), (2, 20.0, 0, 4), (2, 20.0, 1, 3), (0, 1e4, 1, 6), (5, 1e4, 0, 4)]


def _set(p, sweeps, cfl, flux):
    p.gauss_seidel_iter, p.cflmax, p.flux = sweeps, cfl, flux


@pytest.mark.parametrize("prec", ["mixed", "ref", "fp64"])
@pytest.mark.parametrize("solver", [0, 1])  # SGS, LSGS
def test_runs_with_changed_options(need_gpu, solver, prec):
    def mk():
        c = cases.farfield_cube(11, precision=prec)
        c.params.solver, c.params.lsgs_max_iter = solver, 2
        return c

    c = mk()
    g = FlowPsi(c.mesh, c.params)
    state = c.initial_state(g.geometry()["cellcenter"])
    for k, (sweeps, cfl, flux, steps) in enumerate(SEQ):
        p = g.params
        _set(p, sweeps, cfl, flux)
        g.set_params(p)
        g.set_state(*state)
        hist, q = g.run(steps), g.get_state()
        d = mk()
        _set(d.params, sweeps, cfl, flux)
        f = FlowPsi(d.mesh, d.params)
        f.set_state(*state)
        assert f.run(steps) == hist, k
        for a, b in zip(f.get_state(), q):
            assert np.array_equal(a, b), k
        f.close()
    g.close()
