"""A batch's tails in its passes (up to a tile per SM) and in kernels of their
own (above): both add the same partials in the same order, so a model's
iterates in a batch on one side of the rule are bit for bit those in the same
batch with one more model, which puts it on the other side."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from apple_gb300.batch import BatchedForward

pytestmark = pytest.mark.gpu

# grid cells per model with 25 elements per tile, by their tiles; one more model of 2 tiles
BATCHES = {151: [(5, 4, 36), (5, 2, 2), (2, 2, 2), (1, 1, 1)], 152: [(5, 4, 36), (5, 2, 2), (5, 2, 2)]}
ONE_MORE = (5, 1, 2)


def _model(dims, material, dtype, seed):
    m = meshgen.grid(*dims)
    rng = np.random.default_rng(seed)
    mesh = meshgen.TetMesh(m.points, m.cells)
    mesh.cell_data["mu"] = rng.uniform(1, 2, m.n_cells)
    if material != "arap":
        mesh.cell_data["lambda"] = rng.uniform(3, 5, m.n_cells)
    mask = meshgen.face_mask(m, 2, "min")[:, None].repeat(3, 1)
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, np.zeros((m.n_points, 3))
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    pot = {"arap": ag.Arap, "snh": ag.StableNeoHookean}[material].from_pyvista(mesh, dtype=dtype, tile_elems=25)
    b.add_potential(pot)
    fm = meshgen.TetMesh(m.points, m.cells)
    fm.point_data["Force"] = meshgen.lumped_gravity(m, 0.02)
    fm.point_data["GlobalPointId"] = np.arange(m.n_points)
    b.add_potential(ag.ExternalForce.from_pyvista(fm, dtype=dtype))
    return b.finalize(), pot.info()[0]


@pytest.mark.parametrize("mode", ["f32", "f32_correction", "f64", "arap"])
@pytest.mark.parametrize("tiles", sorted(BATCHES))
def test_one_more_model_changes_no_bit(tiles, mode, cuda_device):
    dtype = torch.float64 if mode == "f64" else torch.float32
    built = [_model(d, "arap" if mode == "arap" else "snh", dtype, k)
             for k, d in enumerate(BATCHES[tiles] + [ONE_MORE])]
    models = [m for m, _ in built]
    assert sum(t for _, t in built[:-1]) == tiles and sum(t for _, t in built) > 152
    runs = []
    for ms in (models[:-1], models):
        opt = ag.PNCG(ag.ConvergenceCriteria(max_steps=10**6, rtol=0.0),
                      refresh_ratio=0.5 if mode == "f32_correction" else 0.0)
        bf = BatchedForward(ms, opt)
        bf.reset()
        bf.iterate(9)
        bf.step()
        runs.append(bf.read())
    (sol_a, u_a), (sol_b, u_b) = runs
    for k in range(len(models) - 1):
        assert sol_a[k] == sol_b[k] and sol_a[k].n_steps == 10
        assert torch.equal(u_a[k], u_b[k])
