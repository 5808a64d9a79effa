"""FP64 evaluation over cut tiles (GB300): tiles of 16 warp groups and more are
cut when their pieces fit the SMs two at a time.  Against the FP64 oracle, for
one tile in pieces, for tiles that stay whole beside cut ones and at the limit,
from a potential on its own and from a model of two potentials that share
vertices."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from oracle import fem_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-9  # the FP64 kernels' bar against the oracle

# grid cells, elements per tile: 2, 160 and 304 tiles
SIZES = [((4, 4, 10), 1024), ((12, 12, 140), 640), ((20, 20, 96), 640)]


@pytest.mark.parametrize("material", ["arap", "snh", "muscle"])
@pytest.mark.parametrize("size", range(len(SIZES)))
def test_pieces(size, material, cuda_device):
    dims, tile_elems = SIZES[size]
    m = meshgen.grid(*dims)
    rng = np.random.default_rng(size)
    mu, lam = rng.uniform(1, 2, m.n_cells), rng.uniform(3, 5, m.n_cells)
    act = 0.05 * rng.normal(size=(m.n_cells, 6))
    cls = {"arap": ag.Arap, "snh": ag.StableNeoHookean, "muscle": ag.StableNeoHookeanMuscle}[material]
    mat = {"arap": O.Material.ARAP, "snh": O.Material.STABLE_NEO_HOOKEAN,
           "muscle": O.Material.STABLE_NEO_HOOKEAN_MUSCLE}[material]

    def pair(sel):
        extra = {"activation": act[sel]} if material == "muscle" else {}
        la = None if material == "arap" else lam[sel]
        pot = cls(m.cells[sel], mu[sel], la, points=m.points, dtype=torch.float64, tile_elems=tile_elems, **extra)
        return pot, O.FemPotential.from_mesh(mat, m.points, m.cells[sel], mu=mu[sel], lam=la, **extra)

    U = torch.tensor(m.points @ (0.05 * rng.normal(size=(3, 3))) + 0.02 * rng.normal(size=m.points.shape) *
                     m.points[1, 0], dtype=torch.float64, device=cuda_device)
    P = torch.tensor(rng.normal(size=m.points.shape), dtype=torch.float64, device=cuda_device)
    u, p = U.cpu().numpy(), P.cpu().numpy()

    def check(got, oras):
        for k, v in got.items():
            args = (u, p) if k in ("hess_prod", "hess_quad") else (u,)
            b = sum(np.asarray(getattr(o, k)(*args)) for o in oras)
            a = v.cpu().numpy()
            assert np.linalg.norm((a - b).ravel()) <= TOL * np.linalg.norm(b.ravel()), k

    want = dict(fun=True, grad=True, hess_diag=True, hess_prod=True, hess_quad=True)
    pot, ora = pair(slice(None))
    check(pot.eval(U, P, **want), [ora])
    half = m.n_cells // 3
    a, b = pair(slice(0, half)), pair(slice(half, None))
    if size == 0:  # one model over two potentials that share vertices
        mesh = meshgen.TetMesh(m.points, m.cells)
        mesh.point_data["FixedMask"] = np.zeros((m.n_points, 3), bool)
        mesh.point_data["FixedValue"] = np.zeros((m.n_points, 3))
        builder = ag.ModelBuilder(dtype=torch.float64)
        builder.add_vertices(mesh)
        builder.add_fixed(mesh)
        builder.add_potential(a[0])
        builder.add_potential(b[0])
        model = builder.finalize()
        check({k: getattr(model, k)(U, P) if k in ("hess_prod", "hess_quad") else getattr(model, k)(U) for k in want},
              [a[1], b[1]])
    else:
        check(a[0].eval(U, P, **want), [a[1]])
