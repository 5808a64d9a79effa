"""The FP32 resident iterations' sums against FP64 sums of the solver's own
stored gradient and diagonal, on a mesh of one tile, where no rounding error
averages out over CTAs.  A thread's own three products or absolute values are
added in FP32 (at most 2.5 roundings each, independent between threads);
everything above is float-float.  Over 150 free vertices of uneven weight that
leaves an error of about 0.1 units of rounding, 0.35 at most (2.5 / sqrt(150)
times 1.7 for the weights); trees in plain FP32 make it 0.7."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen

pytestmark = pytest.mark.gpu

UNIT = 2.0**-24


@pytest.mark.parametrize("refresh_ratio", [0.0, 0.5])
def test_same_sign_sums_keep_their_low_words(refresh_ratio, cuda_device):
    m = meshgen.grid(4, 4, 6)
    rng = np.random.default_rng(3)
    mesh = meshgen.TetMesh(m.points, m.cells)
    mesh.cell_data["mu"], mesh.cell_data["lambda"] = rng.uniform(1, 2, m.n_cells), rng.uniform(3, 5, m.n_cells)
    mask = meshgen.face_mask(m, 2, "min")[:, None].repeat(3, 1)
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, np.zeros((m.n_points, 3))
    b = ag.ModelBuilder(dtype=torch.float32)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    b.add_potential(ag.StableNeoHookean.from_pyvista(mesh))
    fm = meshgen.TetMesh(m.points, m.cells)
    fm.point_data["Force"] = meshgen.lumped_gravity(m, 0.02)
    fm.point_data["GlobalPointId"] = np.arange(m.n_points)
    b.add_potential(ag.ExternalForce.from_pyvista(fm))
    model = b.finalize()
    opt = ag.PNCG(ag.ConvergenceCriteria(max_steps=10**6, rtol=0.0), refresh_ratio=refresh_ratio)
    sv = opt.solver(ag.ForwardProblem(model))
    sv.reset(ag.Forward(model, ag.PNCG()).state.u)
    free = ~mask
    err = []
    for _ in range(40):
        sv.iterate(1)
        g, d = (t.double().numpy()[free] for t in sv.read_gradient())
        red = sv.read_reductions()
        if refresh_ratio == 0.0:  # a refresh replaces the stored gradient after its norm was taken
            err.append(red["grad_norm"] ** 2 / np.sum(g * g) - 1.0)
        err.append(np.count_nonzero(d > 0) / red["precond_fill_inv"] / np.sum(np.abs(d)) - 1.0)
    assert np.sqrt(np.mean(np.square(err))) <= 0.35 * UNIT
