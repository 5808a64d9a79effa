"""Resident PNCG iterations at the edges of their launch rule: one tile, at
most one tile per SM, at most two, and more (the three-kernel iteration),
in FP32 with and without the reference-state correction and in FP64.  A fixed
number of iterations against the FP64 oracle's, and the same run cut into
single steps bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from oracle import fem_oracle as O

pytestmark = pytest.mark.gpu

# (grid cells, elements per tile): 1, 152, 159, 304, 305, 608, 610 tiles
SIZES = [((2, 2, 3), 1024), ((5, 4, 38), 25), ((5, 4, 38), 24), ((5, 4, 76), 25), ((5, 5, 61), 25),
         ((5, 4, 152), 25), ((5, 5, 122), 25)]
STEPS = 12


def _model(dims, tile_elems, material, dtype, force):
    m = meshgen.grid(*dims)
    rng = np.random.default_rng(7)
    mu, lam = rng.uniform(1, 2, m.n_cells), rng.uniform(3, 5, m.n_cells)
    act = 0.05 * rng.normal(size=(m.n_cells, 6)) if material == "muscle" else None
    mesh = meshgen.TetMesh(m.points, m.cells)
    mesh.cell_data["mu"], mesh.cell_data["lambda"] = mu, lam
    extra = {}
    if act is not None:
        mesh.cell_data["activation"] = act
        extra["activation"] = act
    mask = np.zeros((m.n_points, 3), bool)
    mask[meshgen.face_mask(m, 2, "min")] = True
    mask[meshgen.face_mask(m, 0, "max"), 1] = True  # one component only
    values = np.where(mask, 0.01, 0.0)
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, values
    cls = ag.StableNeoHookeanMuscle if material == "muscle" else ag.StableNeoHookean
    mat = O.Material.STABLE_NEO_HOOKEAN_MUSCLE if material == "muscle" else O.Material.STABLE_NEO_HOOKEAN
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    b.add_potential(cls.from_pyvista(mesh, dtype=dtype, tile_elems=tile_elems))
    ext = None
    if force:
        fm = meshgen.TetMesh(m.points, m.cells)
        fm.point_data["Force"] = meshgen.lumped_gravity(m, 0.02)
        fm.point_data["GlobalPointId"] = np.arange(m.n_points)
        b.add_potential(ag.ExternalForce.from_pyvista(fm, dtype=dtype))
        ext = O.ExternalForce(np.arange(m.n_points), fm.point_data["Force"])
    ora = O.FemPotential.from_mesh(mat, m.points, m.cells, mu=mu, lam=lam, **extra)
    return m, b.finalize(), O.Model(O.DofMap(m.n_points, mask, values), [ora], ext)


@pytest.mark.parametrize("mode", ["f32", "f32_correction", "f64"])
@pytest.mark.parametrize("size", range(len(SIZES)))
def test_iterations_match_the_oracle_and_single_steps(size, mode, cuda_device):
    dtype = torch.float64 if mode == "f64" else torch.float32
    dims, tile_elems = SIZES[size]
    m, model, om = _model(dims, tile_elems, "muscle" if size % 2 else "snh", dtype, force=size != 2)
    u0 = ag.Forward(model, ag.PNCG()).state.u
    runs = []
    for single in (False, True):
        opt = ag.PNCG(ag.ConvergenceCriteria(max_steps=10**6, rtol=0.0),
                      refresh_ratio=0.5 if mode == "f32_correction" else 0.0)
        sv = opt.solver(ag.ForwardProblem(model))
        sv.reset(u0)
        if single:
            for _ in range(STEPS):
                sv.step()
        else:
            sv.iterate(5)
            sv.iterate(STEPS - 5)
        u = torch.empty_like(u0)
        st = sv.read(u)
        g, d = sv.read_gradient()
        runs.append((u.cpu(), g, d, sv.read_direction(), st))
    assert runs[0][4].n_steps == STEPS
    assert runs[0][4] == runs[1][4]
    for a, b in zip(runs[0][:4], runs[1][:4]):
        assert torch.equal(a, b)
    ref, _ = O.solve_model(om, rtol=0.0, max_steps=STEPS)
    diag = np.linalg.norm(m.points.max(0) - m.points.min(0))
    # the kernels' bars for displacements: 1e-4 of the diagonal in FP32, 1e-9 in FP64
    err = np.abs(runs[0][0].double().numpy() - ref).max()
    assert err <= (1e-9 if dtype == torch.float64 else 1e-4) * diag
