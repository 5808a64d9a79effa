"""The material gradients are tensors of their own: each can be changed in
place under autograd without touching the other (a regulariser added to one
while the other is saved for a backward)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cls", [ag.StableNeoHookean, ag.StableNeoHookeanMuscle])
def test_in_place_under_autograd(cls, cuda_device):
    m = meshgen.grid(2, 2, 2)
    pot = cls(m.cells, 1.0, 4.0, points=m.points)
    rng = np.random.default_rng(0)
    u, w = (torch.tensor(0.1 * rng.normal(size=m.points.shape), dtype=torch.float32, device=cuda_device)
            for _ in range(2))
    out = pot.grad_param_vjp(u, w)
    before = {k: v.clone() for k, v in out.items()}
    theta = torch.full((m.n_cells,), 2.0, device=cuda_device, requires_grad=True)
    loss = (theta * out["lambda"]).sum()
    out["mu"] += 0.5 * theta
    loss.backward()
    assert torch.equal(theta.grad, before["lambda"])
    assert torch.equal(out["mu"].detach(), before["mu"] + 1.0)
