"""ForwardProblem over free components: the maps folded into the evaluation
give the bits of the separate maps around the full evaluation, for every
method, material and dtype, with per-component fixed DOFs, external forces,
everything fixed or nothing; arguments the folded form does not take go
through the separate maps as before."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _problem(dtype, material, fixed):
    m = meshgen.grid(3, 4, 5)
    rng = np.random.default_rng(0)
    mesh = ag.with_lame(meshgen.TetMesh(m.points, m.cells), rng.uniform(1, 2, m.n_cells), rng.uniform(3, 5, m.n_cells))
    mask = {"none": np.zeros((m.n_points, 3), bool), "all": np.ones((m.n_points, 3), bool),
            "some": rng.random((m.n_points, 3)) < 0.3}[fixed]
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, 0.01 * rng.normal(size=(m.n_points, 3))
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    b.add_potential({"arap": ag.Arap, "snh": ag.StableNeoHookean}[material].from_pyvista(mesh, dtype=dtype))
    fm = meshgen.TetMesh(m.points, m.cells)
    fm.point_data["Force"] = rng.normal(size=(m.n_points, 3))
    fm.point_data["GlobalPointId"] = np.arange(m.n_points)
    b.add_potential(ag.ExternalForce.from_pyvista(fm, dtype=dtype))
    model = b.finalize()
    u = torch.tensor(0.02 * rng.normal(size=(m.n_points, 3)), dtype=dtype, device="cuda")
    p = torch.tensor(rng.normal(size=model.n_free), dtype=dtype, device="cuda")
    return ag.ForwardProblem(model), ag.ModelState(u=u), p


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("material", ["snh", "arap"])
@pytest.mark.parametrize("fixed", ["none", "some", "all"])
def test_folded_maps_equal_separate_maps(fixed, material, dtype, cuda_device):
    problem, state, p = _problem(dtype, material, fixed)
    model, dm = problem.model, problem.model.dof_map
    full = dm.to_full_grad(p)
    assert torch.equal(problem.grad(state), dm.to_free_grad(model.grad(state.u)))
    assert torch.equal(problem.hess_diag(state), dm.to_free_hess_diag(model.hess_diag(state.u)))
    assert torch.equal(problem.hess_prod(state, p), dm.to_free_grad(model.hess_prod(state.u, full)))
    assert torch.equal(problem.hess_quad(state, p), model.hess_quad(state.u, full))


def test_other_arguments_take_the_separate_maps(cuda_device):
    problem, state, p = _problem(torch.float32, "snh", "some")
    ref = problem.hess_prod(state, p)
    assert torch.equal(problem.hess_prod(state, p.double()), ref)  # converted
    assert torch.equal(problem.hess_prod(state, torch.stack([p, p], 1)[:, 0]), ref)  # strided
    assert torch.equal(problem.hess_prod(state, p.reshape(1, -1)), ref)
    with pytest.raises(ValueError):
        problem.hess_prod(state, p[1:])
    with pytest.raises(TypeError):
        problem.grad(ag.ModelState(u=state.u.double()))
    with pytest.raises(TypeError):
        problem.grad(ag.ModelState(u=state.u.cpu()))


def test_eval_stores_what_the_methods_accumulate(cuda_device):
    problem, state, _ = _problem(torch.float32, "snh", "some")
    pot = next(iter(problem.model.warp_model.potentials.values()))
    g = torch.full_like(state.u, 2.0)
    pot.grad(state.u, g)
    e = torch.full((1,), 3.0, dtype=torch.float64, device=cuda_device)
    pot.fun(state.u, e)
    out = pot.eval(state.u, grad=True, fun=True)
    assert torch.allclose(g - 2.0, out["grad"], rtol=0, atol=1e-6 * float(out["grad"].abs().max()) + 4e-7)
    assert abs(e.item() - 3.0 - out["fun"].item()) <= 1e-12 * abs(e.item())
    empty = ag.StableNeoHookean(np.zeros((0, 4), np.int32), np.zeros(0), np.zeros(0), points=np.zeros((5, 3)))
    u = torch.zeros((5, 3), device=cuda_device)
    r = empty.eval(u, u, fun=True, grad=True, hess_diag=True, hess_prod=True, hess_quad=True)
    assert all(torch.count_nonzero(v) == 0 for v in r.values())
