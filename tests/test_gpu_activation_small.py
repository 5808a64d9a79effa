"""Activations around the size up to which the host writes the records: the
same bits as a potential built with the activation, and a solver over two
potentials, which reads the activation back, starts from the same state."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n_cells", [1, 127, 128, 129])
def test_a_potential_and_a_solver_see_the_same_activation(n_cells, dtype, cuda_device):
    m = meshgen.grid(5, 5, 5)
    cells, rest = m.cells[:n_cells], m.cells[n_cells:]
    rng = np.random.default_rng(n_cells)
    act = 0.1 * rng.normal(size=(n_cells, 6))
    U = torch.tensor(0.01 * rng.normal(size=m.points.shape), dtype=dtype, device=cuda_device)
    grads, starts = [], []
    for late in (False, True):
        pot = ag.StableNeoHookeanMuscle(cells, 1.0, 4.0, points=m.points, dtype=dtype,
                                        activation=None if late else act)
        if late:
            pot.eval(U, grad=True)
            pot.set_activation(0.5 * act)
            pot.set_activation(act)
        grads.append(pot.eval(U, grad=True)["grad"])
        mesh = meshgen.TetMesh(m.points, m.cells)
        mesh.point_data["FixedMask"] = np.zeros((m.n_points, 3), bool)
        mesh.point_data["FixedValue"] = np.zeros((m.n_points, 3))
        b = ag.ModelBuilder(dtype=dtype)
        b.add_vertices(mesh)
        b.add_fixed(mesh)
        b.add_potential(pot)
        b.add_potential(ag.StableNeoHookean(rest, 1.0, 4.0, points=m.points, dtype=dtype))
        model = b.finalize()
        if late:  # the model's own copy of the potential, too
            pot.set_activation(act)
        sv = ag.PNCG().solver(ag.ForwardProblem(model))
        sv.reset(U)
        starts.append(sv.read_gradient()[0])
    assert torch.equal(grads[0], grads[1]) and torch.equal(starts[0], starts[1])
    assert bool(starts[0].any())
