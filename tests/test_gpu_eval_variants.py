"""The fused evaluation at the edges of its launch rule: one tile, at most one
tile per SM (16 warps per tile; 8 in FP64), at most two (8 warps) and more
(4 warps), for one, two and three vectors and for scalars alone, against the
FP64 oracle; the same values whatever else is asked for, and the same bits on
every call."""

from __future__ import annotations

import itertools

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from oracle import fem_oracle as O

pytestmark = pytest.mark.gpu

# (grid cells, elements per tile): 1, 152, 159, 304, 305 tiles
SIZES = [((2, 2, 3), 1024), ((5, 4, 38), 25), ((5, 4, 38), 24), ((5, 4, 76), 25), ((5, 5, 61), 25)]
VECTORS = ("grad", "hess_diag", "hess_prod")
TOL = {torch.float64: 1e-9, torch.float32: 1e-5}  # the kernels' bars against the oracle


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("material", ["arap", "snh", "muscle"])
@pytest.mark.parametrize("size", range(len(SIZES)))
def test_every_combination(size, material, dtype, cuda_device):
    dims, tile_elems = SIZES[size]
    m = meshgen.grid(*dims)
    rng = np.random.default_rng(size)
    mu, lam = rng.uniform(1, 2, m.n_cells), rng.uniform(3, 5, m.n_cells)
    act = 0.05 * rng.normal(size=(m.n_cells, 6)) if material == "muscle" else None
    cls = {"arap": ag.Arap, "snh": ag.StableNeoHookean, "muscle": ag.StableNeoHookeanMuscle}[material]
    mat = {"arap": O.Material.ARAP, "snh": O.Material.STABLE_NEO_HOOKEAN,
           "muscle": O.Material.STABLE_NEO_HOOKEAN_MUSCLE}[material]
    extra = {} if act is None else {"activation": act}
    pot = cls(m.cells, mu, None if material == "arap" else lam, points=m.points, dtype=dtype, tile_elems=tile_elems,
              **extra)
    ora = O.FemPotential.from_mesh(mat, m.points, m.cells, mu=mu, lam=None if material == "arap" else lam, **extra)
    h = m.points[1, 0]
    U = torch.tensor(m.points @ (0.05 * rng.normal(size=(3, 3))) + 0.03 * h * rng.normal(size=m.points.shape),
                     dtype=dtype, device=cuda_device)
    P = torch.tensor(rng.normal(size=m.points.shape), dtype=dtype, device=cuda_device)
    u, p = U.double().cpu().numpy(), P.double().cpu().numpy()
    ref = {"fun": ora.fun(u), "grad": ora.grad(u), "hess_diag": ora.hess_diag(u), "hess_prod": ora.hess_prod(u, p),
           "hess_quad": ora.hess_quad(u, p)}
    everything = pot.eval(U, P, fun=True, grad=True, hess_diag=True, hess_prod=True, hess_quad=True)
    for k, v in everything.items():
        a, b = v.double().cpu().numpy(), np.asarray(ref[k])
        assert np.linalg.norm((a - b).ravel()) <= TOL[dtype] * np.linalg.norm(b.ravel()), k
    again = pot.eval(U, P, fun=True, grad=True, hess_diag=True, hess_prod=True, hess_quad=True)
    assert all(torch.equal(again[k], everything[k]) for k in everything)
    for n in range(len(VECTORS) + 1):
        for names in itertools.combinations(VECTORS, n):
            for scalars in ((), ("fun",), ("hess_quad",), ("fun", "hess_quad")):
                if not names and not scalars:
                    continue
                got = pot.eval(U, P, **{k: True for k in names + scalars})
                for k in names:
                    a, b = got[k].double().cpu().numpy(), ref[k]
                    assert np.linalg.norm((a - b).ravel()) <= TOL[dtype] * np.linalg.norm(b.ravel()), (names, k)
                for k in scalars:
                    assert abs(got[k].item() - ref[k]) <= TOL[dtype] * abs(ref[k]), (names, scalars, k)


def test_launch_sizes_are_the_edges():
    tiles = []
    for dims, tile_elems in SIZES:
        m = meshgen.grid(*dims)
        tiles.append(ag.StableNeoHookean(m.cells, 1.0, 1.0, points=m.points, tile_elems=tile_elems).info()[0])
    assert tiles == [1, 152, 159, 304, 305]
