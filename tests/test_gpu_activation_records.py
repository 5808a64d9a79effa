"""Activation records written on the device, at the edges of their launch: one
cell, around the 256-thread blocks, and more cells than one wave of the grid,
against the FP64 oracle's gradient at the new activation."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from oracle import fem_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n_cells", [1, 255, 256, 257, 312_500])
def test_records_follow_the_activation(n_cells, dtype, cuda_device):
    n = max(2, int(np.ceil((n_cells / 5) ** (1 / 3))))
    m = meshgen.grid(n, n, n)
    cells = m.cells[:n_cells]
    rng = np.random.default_rng(n_cells)
    mu, lam = rng.uniform(1, 2, n_cells), rng.uniform(3, 5, n_cells)
    # the vertex space covers every grid point, loaded by a cell or not
    pot = ag.StableNeoHookeanMuscle(cells, mu, lam, points=m.points, dtype=dtype, activation=None)
    u = 0.02 / n * rng.normal(size=m.points.shape)
    U = torch.tensor(u, dtype=dtype, device=cuda_device)
    for k in range(2):  # the second one replaces the first in place
        act = 0.1 * rng.normal(size=(n_cells, 6))
        pot.set_activation(act)
        act[:] = np.nan  # the caller's array is not read again
        g = pot.eval(U, grad=True)["grad"].double().cpu().numpy()
    ora = O.FemPotential.from_mesh(O.Material.STABLE_NEO_HOOKEAN_MUSCLE, m.points, cells, mu=mu, lam=lam,
                                   activation=pot.activation)
    ref = ora.grad(U.double().cpu().numpy())
    tol = 1e-9 if dtype == torch.float64 else 1e-5  # the kernels' bars against the oracle
    assert np.linalg.norm(g - ref) <= tol * np.linalg.norm(ref)
