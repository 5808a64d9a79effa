"""A model's outputs that share a buffer receive their sum (zero, then
accumulate): the gradient after a step to first order, g + H p, in one call."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import _lib, meshgen
from apple_gb300.fem import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _warp_model(dtype):
    m = meshgen.grid(4, 3, 5)
    mesh = ag.with_lame(meshgen.TetMesh(m.points, m.cells), 1.0, 2.0)
    mesh.point_data["FixedMask"] = np.zeros((m.n_points, 3), bool)
    mesh.point_data["FixedValue"] = np.zeros((m.n_points, 3))
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    for _ in range(2):
        b.add_potential(ag.StableNeoHookean.from_pyvista(mesh, dtype=dtype))
    fm = meshgen.TetMesh(m.points, m.cells)
    fm.point_data["Force"] = np.random.default_rng(0).normal(size=(m.n_points, 3))
    fm.point_data["GlobalPointId"] = np.arange(m.n_points)
    b.add_potential(ag.ExternalForce.from_pyvista(fm, dtype=dtype))
    return b.finalize().warp_model


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("first, second", [("grad", "hess_prod"), ("grad", "hess_diag"), ("hess_diag", "hess_prod")])
def test_two_vectors_in_one_buffer(first, second, dtype, cuda_device):
    wm = _warp_model(dtype)
    g = torch.Generator(device=cuda_device).manual_seed(0)
    u, p = (0.05 * torch.randn((wm.n_points, 3), generator=g, device=cuda_device, dtype=dtype) for _ in range(2))
    names = ["grad", "hess_diag", "hess_prod"]
    flags = {"grad": _lib.GRAD, "hess_diag": _lib.HESS_DIAG, "hess_prod": _lib.HESS_PROD}

    def run(**out):
        f = 0
        for k in out:
            f |= flags[k]
        _lib.call("agb_model_eval", wm.handle, f, ptr(u), ptr(p), None, *[ptr(out.get(k)) for k in names], None,
                  stream_ptr(u.device))

    a, b, both = torch.empty_like(u), torch.empty_like(u), torch.full_like(u, 7.0)
    run(**{first: a, second: b})
    run(**{first: both, second: both})
    assert torch.equal(both, a + b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_two_scalars_in_one_buffer(dtype, cuda_device):
    wm = _warp_model(dtype)
    g = torch.Generator(device=cuda_device).manual_seed(0)
    u, p = (0.05 * torch.randn((wm.n_points, 3), generator=g, device=cuda_device, dtype=dtype) for _ in range(2))

    def run(e, q):
        _lib.call("agb_model_eval", wm.handle, _lib.FUN | _lib.HESS_QUAD, ptr(u), ptr(p), ptr(e), None, None, None,
                  ptr(q), stream_ptr(u.device))

    a, b, both = (torch.full((1,), 7.0, dtype=torch.float64, device=cuda_device) for _ in range(3))
    run(a, b)
    run(both, both)
    torch.testing.assert_close(both, a + b, rtol=1e-14, atol=0.0)
