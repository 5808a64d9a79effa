"""Where ForwardProblem may fold the free map into the evaluation and where it
has to ask the model: a WarpModel of another class keeps its own methods, and
a missing direction is refused as the map refuses it."""

from __future__ import annotations

import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from apple_gb300.model import WarpModel

pytestmark = pytest.mark.gpu


class _Doubled(WarpModel):
    """A user's model: every quantity twice."""

    def _eval(self, flags, u, p=None, **out):
        super()._eval(flags, u, p, **out)
        for t in out.values():
            if t is not None:
                t.mul_(2.0)


def _problem():
    m = meshgen.grid(2, 2, 3)
    mesh = ag.with_lame(meshgen.TetMesh(m.points, m.cells), 1.0, 2.0)
    mask = meshgen.face_mask(m, 2, "min")[:, None].repeat(3, 1)
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, 0.0 * mask
    b = ag.ModelBuilder()
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    b.add_potential(ag.StableNeoHookean.from_pyvista(mesh))
    model = b.finalize()
    return model, ag.ForwardProblem(model)


def test_a_warp_model_of_another_class_is_asked(cuda_device):
    model, problem = _problem()
    g = torch.Generator(device=cuda_device).manual_seed(0)
    u = 0.01 * torch.randn((model.n_points, 3), generator=g, device=cuda_device)
    p = torch.randn(model.n_free, generator=g, device=cuda_device)
    state = ag.ModelState(u=u)

    def all_four():
        return [problem.grad(state), problem.hess_diag(state), problem.hess_prod(state, p),
                problem.hess_quad(state, p).reshape(1)]

    plain = all_four()
    model.warp_model.__class__ = _Doubled
    for a, b in zip(plain, all_four()):
        assert torch.equal(2.0 * a, b)
    model.warp_model.__class__ = WarpModel
    model.grad = lambda u: torch.ones_like(u)  # a replaced bound method counts too
    assert torch.equal(problem.grad(state), torch.ones_like(plain[0]))


@pytest.mark.parametrize("method", ["hess_prod", "hess_quad"])
def test_a_missing_direction_is_refused(method, cuda_device):
    model, problem = _problem()
    state = ag.ModelState(u=torch.zeros((model.n_points, 3), device=cuda_device))
    with pytest.raises(TypeError):
        getattr(problem, method)(state, None)
