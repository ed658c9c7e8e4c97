"""The training pass at graph sizes where its split changes: less than one
64-cell tile, a remainder, one, three and four tiles per block.  GPU only.
Against the torch CPU replica; the bars are those of test_gpu_learned.py (loss
1e-5, gradients 1e-3 of a group's norm and 3e-3 of its largest entry, from
single activations that the two summation orders round to neighbouring BF16
values, measured on 216 cells), times sqrt(216 / cells) on smaller graphs,
over which one flipped activation is averaged less."""
import numpy as np
import pytest

from flowpsi_b200 import FlowPsi, cases
from flowpsi_b200.learned import LearnedStart
from flowpsi_b200.solver import GeneratedMesh, bc
from oracle import gnn_oracle as G
from tests.test_gpu_learned import _random_head

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(2, 2, 2), (3, 3, 2), (20, 20, 20), (29, 29, 29)])
def test_gradient_over_sizes(need_gpu, n):
    case = cases.farfield_tets(2, precision="ref")
    mesh = GeneratedMesh("kuhn", n=n, jitter=0.1, bc_side=(0,) * 6,
                         bcs=[bc("farfield", u=(170.0, 0.0, 0.0))])
    g = FlowPsi(mesh, case.params)
    g.keep_blocks(True)
    g.set_state(*case.initial_state(g.geometry()["cellcenter"]))
    g.residual()
    g.assemble()
    g.sweeps(3)
    dq = g.get_iterate()
    g.assemble()
    model = LearnedStart(seed=5)
    model.add_snapshot(g, dq)
    w = _random_head(model)
    loss, grad = model.loss_grad(0)
    f, t, _, _ = model.snapshot(0)
    a = mesh.arrays()
    A = G.neighbour_mean_matrix(a.ncells, np.asarray(a.cl), np.asarray(a.cr))
    loss_o, grad_o, _ = G.loss_and_grad(w, f, t, A)
    k = max(1.0, np.sqrt(216 / a.ncells))
    assert abs(loss - loss_o) <= 1e-5 * k * loss_o
    for name, lo, hi in G.groups():
        go, gg = grad_o[lo:hi], grad[lo:hi]
        assert np.linalg.norm(gg - go) <= 1e-3 * k * np.linalg.norm(go) + 1e-12, name
        assert np.abs(gg - go).max() <= 3e-3 * k * np.abs(go).max() + 1e-12, name
    model.close()
    g.close()
