"""Which meshes iterate in one cooperative launch, and that form on meshes whose
tiles are full and get cut: several rounds of warp groups per warp, whole tiles
beside cut ones, and in FP64 cut tiles in pairs.  PNCG against the FP64 C
restatement of the reference, the adjoint CG against its other form."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from oracle import build_c
from oracle import fem_oracle as O

pytestmark = pytest.mark.gpu

STEPS = 12
# default tiles: grid cells -> tiles (160 to 6,393 warp groups, about 20 per tile)
FULL = {(10, 10, 10): 8, (12, 12, 140): 152, (12, 12, 141): 153, (24, 24, 48): 205, (18, 18, 123): 303,
        (16, 16, 156): 305}
# 25 elements per tile, at the edges of the rule
SMALL = {(2, 2, 3): 3, (5, 4, 38): 152, (5, 4, 76): 304, (5, 5, 61): 305}
MOST = 304


def _mesh(dims, extra=0):
    m = meshgen.grid(*dims, h=1.0 / dims[0])
    # points that no cell uses, last in the vertex order
    pts = np.concatenate([m.points, np.repeat(m.points.max(0, keepdims=True), extra, 0)])
    rng = np.random.default_rng(11)
    mesh = meshgen.TetMesh(pts, m.cells)
    mesh.cell_data["mu"], mesh.cell_data["lambda"] = rng.uniform(1, 2, m.n_cells), rng.uniform(3, 5, m.n_cells)
    mask = np.zeros((pts.shape[0], 3), bool)
    mask[: m.n_points][meshgen.face_mask(m, 2, "min")] = True
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, np.where(mask, 0.01, 0.0)
    return m, mesh, mask, rng


def _model(m, mesh, dtype, material="snh", tile_elems=0, force=None):
    cls = {"snh": ag.StableNeoHookean, "muscle": ag.StableNeoHookeanMuscle, "arap": ag.Arap}[material]
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    pot = cls.from_pyvista(mesh, dtype=dtype, tile_elems=tile_elems)
    b.add_potential(pot)
    if force is not None:
        fm = meshgen.TetMesh(mesh.points, m.cells)
        fm.point_data["Force"] = force
        fm.point_data["GlobalPointId"] = np.arange(mesh.points.shape[0])
        b.add_potential(ag.ExternalForce.from_pyvista(fm, dtype=dtype))
    return b.finalize(), pot


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("material", ["snh", "muscle", "arap"])
@pytest.mark.parametrize("dims", list(SMALL))
def test_the_form_follows_the_number_of_tiles(dims, material, dtype, cuda_device):
    m, mesh, mask, rng = _mesh(dims)
    if material == "muscle":
        mesh.cell_data["activation"] = 0.01 * rng.normal(size=(m.n_cells, 6))
    model, pot = _model(m, mesh, dtype, material, tile_elems=25)
    assert pot.info()[0] == SMALL[dims]
    sv = ag.PNCG().solver(ag.ForwardProblem(model))
    fits = SMALL[dims] <= MOST
    assert sv.info() == {"resident_iterations": fits and material != "arap", "resident_adjoint": None}
    u0 = model.init().u
    sv.reset(u0)
    sv.adjoint(torch.ones_like(u0), max_iter=2)
    assert sv.info()["resident_adjoint"] == fits


@pytest.mark.parametrize("mode", ["f32", "f32_correction", "f64"])
@pytest.mark.parametrize("dims", list(FULL))
def test_iterations_on_full_tiles_match_the_oracle(dims, mode, cuda_device):
    dtype = torch.float64 if mode == "f64" else torch.float32
    m, mesh, mask, _ = _mesh(dims)
    force = meshgen.lumped_gravity(m, 0.02)
    model, pot = _model(m, mesh, dtype, force=force)
    assert pot.info()[0] == FULL[dims]
    opt = ag.PNCG(ag.ConvergenceCriteria(max_steps=10**6, rtol=0.0),
                  refresh_ratio=0.5 if mode == "f32_correction" else 0.0)
    sv = opt.solver(ag.ForwardProblem(model))
    assert sv.info()["resident_iterations"] == (FULL[dims] <= MOST)
    u0 = model.init().u
    runs = []
    for cuts in ((STEPS,), (5, STEPS - 5), (1,) * STEPS):
        sv.reset(u0)
        for n in cuts:
            sv.iterate(n)
        u = torch.empty_like(u0)
        runs.append((sv.read(u), u))
    for st, u in runs[1:]:
        assert st == runs[0][0] and torch.equal(u, runs[0][1])
    assert runs[0][0].n_steps == STEPS
    dhdX, dV = O.region_compute_grad(m.points, m.cells)
    cm = build_c.CModel(1, m.cells, dhdX, dV, mesh.cell_data["mu"], mesh.cell_data["lambda"], m.n_points,
                        mask=mask.astype(np.uint8), force=force)
    ref, _ = cm.pncg(np.where(mask, 0.01, 0.0), max_steps=STEPS, rtol=0.0)
    diag = np.linalg.norm(m.points.max(0) - m.points.min(0))
    # the kernels' bars for displacements: 1e-4 of the diagonal in FP32, 1e-9 in FP64
    err = np.abs(runs[0][1].double().cpu().numpy() - ref).max()
    assert err <= (1e-9 if dtype == torch.float64 else 1e-4) * diag


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("material", ["snh", "muscle", "arap"])
@pytest.mark.parametrize("dims", [(10, 10, 10), (12, 12, 141), (24, 24, 48)])
def test_both_forms_of_the_adjoint(dims, material, dtype, cuda_device):
    """With more points than its tiles have places the CG runs as a kernel per
    pass; points that no cell uses change nothing else.  In FP32 the bits are
    the same; in FP64 the sums above a warp are in another order, and 12
    iterations keep the difference at a few thousand roundings."""
    lam = []
    m = meshgen.grid(*dims)
    for extra in (0, 256 * FULL[dims] - m.n_points + 1):
        m, mesh, mask, rng = _mesh(dims, extra)
        if material == "muscle":
            mesh.cell_data["activation"] = 0.01 * rng.normal(size=(m.n_cells, 6))
        model, _ = _model(m, mesh, dtype, material)
        n = mesh.points.shape[0]
        u = np.where(mask, 0.01, 0.01 * mesh.points * [0.2, -0.3, 1.0] + 0.01)
        rhs = np.zeros((n, 3))
        rhs[: m.n_points] = np.random.default_rng(5).normal(size=(m.n_points, 3))
        sv = ag.PNCG().solver(ag.ForwardProblem(model))
        sv.reset(torch.tensor(u, dtype=dtype, device=cuda_device))
        got, st = sv.adjoint(torch.tensor(rhs, dtype=dtype, device=cuda_device), rtol=0.0, max_iter=STEPS)
        assert st.n_iter == STEPS and sv.info()["resident_adjoint"] == (extra == 0)
        assert not bool(got[m.n_points:].any())
        lam.append(got[: m.n_points])
    if dtype == torch.float32:
        assert torch.equal(lam[0], lam[1])
    else:
        torch.testing.assert_close(lam[0], lam[1], rtol=0.0, atol=1e-12 * float(lam[0].abs().max()))
