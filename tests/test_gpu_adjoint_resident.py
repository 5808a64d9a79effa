"""The adjoint CG at the edges of its one-launch form: one tile, at most one
tile per SM, at most two, and more (the three-kernel iteration), with points
that no cell uses, in every material.  A fixed number of CG iterations at a
mildly strained state against the same iterations over the FP64 oracle's
Hessian products, and the same bits from every solve."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from oracle import fem_oracle as O

pytestmark = pytest.mark.gpu

# (grid cells, elements per tile): 1, 152, 159, 304, 305 tiles
SIZES = [((2, 2, 3), 1024), ((5, 4, 38), 25), ((5, 4, 38), 24), ((5, 4, 76), 25), ((5, 5, 61), 25)]
STEPS = 12
TOL = {torch.float64: 1e-8, torch.float32: 2e-4}  # the adjoint's bars against an FP64 solve


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("material", ["arap", "snh", "muscle"])
@pytest.mark.parametrize("size", range(len(SIZES)))
def test_cg_iterations_match_the_oracle(size, material, dtype, cuda_device):
    dims, tile_elems = SIZES[size]
    m = meshgen.grid(*dims)
    extra_points = np.array([[9.0, 9.0, 9.0], [8.0, 9.0, 9.0]]) if size == 2 else np.zeros((0, 3))
    pts = np.concatenate([m.points, extra_points])
    n = pts.shape[0]
    rng = np.random.default_rng(size)
    mu, lam = rng.uniform(1, 2, m.n_cells), rng.uniform(2, 3, m.n_cells)
    mesh = meshgen.TetMesh(pts, m.cells)
    mesh.cell_data["mu"] = mu
    kw = {}
    if material != "arap":
        mesh.cell_data["lambda"] = kw["lam"] = lam
    if material == "muscle":
        mesh.cell_data["activation"] = kw["activation"] = 0.01 * rng.normal(size=(m.n_cells, 6))
    mask = np.zeros((n, 3), bool)
    mask[: m.n_points][meshgen.face_mask(m, 2, "min")] = True
    mask[m.n_points - 1, 1] = True  # one component only
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, np.zeros((n, 3))
    cls = {"arap": ag.Arap, "snh": ag.StableNeoHookean, "muscle": ag.StableNeoHookeanMuscle}[material]
    mat = {"arap": O.Material.ARAP, "snh": O.Material.STABLE_NEO_HOOKEAN,
           "muscle": O.Material.STABLE_NEO_HOOKEAN_MUSCLE}[material]
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    b.add_potential(cls.from_pyvista(mesh, dtype=dtype, tile_elems=tile_elems))
    model = b.finalize()
    U = torch.tensor(np.where(mask, 0.0, 0.01 * pts * [0.2, -0.3, 1.0]), dtype=dtype, device=cuda_device)
    rhs = torch.tensor(rng.normal(size=(n, 3)), dtype=dtype, device=cuda_device)
    rhs[m.n_points:] = 0.0  # nothing acts on the loose points
    sv = ag.PNCG().solver(ag.ForwardProblem(model))
    sv.reset(U)
    got, st = sv.adjoint(rhs, rtol=0.0, max_iter=STEPS)
    again, _ = sv.adjoint(rhs, rtol=0.0, max_iter=STEPS)
    assert st.n_iter == STEPS and torch.equal(got, again)

    ora = O.FemPotential.from_mesh(mat, pts, m.cells, mu=mu, **kw)
    u, r = U.double().cpu().numpy(), np.where(mask, 0.0, rhs.double().cpu().numpy())
    d = ora.hess_diag(u)
    minv = np.where(mask | (d == 0.0), 0.0, 1.0 / np.where(d == 0.0, 1.0, d))
    lam_ref, p, rz, beta = np.zeros_like(r), np.zeros_like(r), float((r * minv * r).sum()), 0.0
    for _ in range(STEPS):
        p = minv * r + beta * p
        q = np.where(mask, 0.0, ora.hess_prod(u, p))
        alpha = rz / float((p * q).sum())
        lam_ref, r = lam_ref + alpha * p, r - alpha * q
        new = float((r * minv * r).sum())
        beta, rz = new / rz, new
    err = np.linalg.norm(got.double().cpu().numpy() - lam_ref) / np.linalg.norm(lam_ref)
    assert err <= TOL[dtype]
