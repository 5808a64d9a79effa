"""The fused evaluation over tiles of a few warp groups, which run with as many
warps as the largest tile has batches of elements; in FP64, where small tiles
leave their groups half empty, a batch is a full warp of elements.  Against the
FP64 oracle, from one element to eight batches a tile."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from oracle import fem_oracle as O

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 1e-9, torch.float32: 1e-5}  # the kernels' bars against the oracle


# the long grid has more than two tiles per SM
@pytest.mark.parametrize("tile_elems", [1, 8, 32, 33, 64, 100, 160, 256, 300])
@pytest.mark.parametrize("dims", [(3, 3, 4), (8, 8, 160)])
@pytest.mark.parametrize("material", ["arap", "snh", "muscle"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_against_the_oracle(dtype, material, dims, tile_elems, cuda_device):
    if tile_elems == 1 and dims != (3, 3, 4):
        pytest.skip("51,200 tiles of one element")
    m = meshgen.grid(*dims)
    rng = np.random.default_rng(1)
    mu, lam = rng.uniform(1, 2, m.n_cells), None if material == "arap" else rng.uniform(3, 5, m.n_cells)
    extra = {"activation": 0.05 * rng.normal(size=(m.n_cells, 6))} if material == "muscle" else {}
    cls = {"arap": ag.Arap, "snh": ag.StableNeoHookean, "muscle": ag.StableNeoHookeanMuscle}[material]
    mat = {"arap": O.Material.ARAP, "snh": O.Material.STABLE_NEO_HOOKEAN,
           "muscle": O.Material.STABLE_NEO_HOOKEAN_MUSCLE}[material]
    pot = cls(m.cells, mu, lam, points=m.points, dtype=dtype, tile_elems=tile_elems, **extra)
    ora = O.FemPotential.from_mesh(mat, m.points, m.cells, mu=mu, lam=lam, **extra)
    h = m.points[1, 0]
    U = torch.tensor(m.points @ (0.05 * rng.normal(size=(3, 3))) + 0.03 * h * rng.normal(size=m.points.shape),
                     dtype=dtype, device=cuda_device)
    P = torch.tensor(rng.normal(size=m.points.shape), dtype=dtype, device=cuda_device)
    u, p = U.double().cpu().numpy(), P.double().cpu().numpy()
    ref = {"fun": ora.fun(u), "grad": ora.grad(u), "hess_diag": ora.hess_diag(u), "hess_prod": ora.hess_prod(u, p),
           "hess_quad": ora.hess_quad(u, p)}
    everything = dict(fun=True, grad=True, hess_diag=True, hess_prod=True, hess_quad=True)
    for asked in (everything, {"grad": True}, {"grad": True, "hess_prod": True}, {"fun": True}):
        got = pot.eval(U, P, **asked)
        for k, v in got.items():
            a, b = v.double().cpu().numpy(), np.asarray(ref[k])
            assert np.linalg.norm((a - b).ravel()) <= TOL[dtype] * np.linalg.norm(b.ravel()), (asked, k)
        again = pot.eval(U, P, **asked)
        assert all(torch.equal(again[k], got[k]) for k in got)
