"""A step's norms are finished by one block of its assembly and written to the
run's history by the device; residual() finishes them in a kernel of its own.
Both are the same sums in the same order, so they agree bit for bit: with
fewer partials than the finishing block's threads, than its chains, and more,
in runs of launches (2 steps) and of replayed graphs, with and without the
compact face records, and for the step after a longer run.  GPU only."""
import pytest

from flowpsi_b200 import FlowPsi, cases

pytestmark = pytest.mark.gpu


def _case(n, form):
    if form == "lsgs":
        c = cases.farfield_cube(n, precision="mixed")
        c.params.solver, c.params.lsgs_max_iter = 1, 2
        return c
    c = cases.farfield_cube(n, precision=form)
    return c


@pytest.mark.parametrize("form", ["mixed", "ref", "fp64", "lsgs"])
@pytest.mark.parametrize("n", [2, 7, 32, 33, 41])  # partials: 1, 2, 128, 141, 270
def test_history_is_the_residuals_norms(need_gpu, n, form):
    c = _case(n, form)
    g = FlowPsi(c.mesh, c.params)
    state = c.initial_state(g.geometry()["cellcenter"])
    want = []
    g.set_state(*state)
    for _ in range(6):
        want.append(g.residual()[1])
        got = g.newton_step()
        assert {k: got[k] for k in want[-1]} == want[-1]
    for steps in (6, 2, 4):
        g.set_state(*state)
        assert g.run(steps) == want[:steps], steps
    g.close()
