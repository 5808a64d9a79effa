"""The batch starts from each model's own ``init()`` (on the host, the C
library replaced by a recorder)."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import _lib, meshgen
from apple_gb300.batch import BatchedForward
from apple_gb300.model import DofMap, Model


class _Library:
    def __getattr__(self, name):
        return lambda *args: 0


@pytest.fixture(autouse=True)
def library(monkeypatch):
    lib = _Library()

    monkeypatch.setattr(_lib, "call", lambda name, *args: 0)  # handles stay null: nothing to destroy later
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(_lib, "_lib", lib)


def _parts(n):
    m = meshgen.grid(1, 1, n)
    mesh = ag.with_lame(meshgen.TetMesh(m.points, m.cells), 1.0, 2.0)
    mask = meshgen.face_mask(m, 2, "min")[:, None].repeat(3, 1)
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, 0.25 * mask
    b = ag.ModelBuilder(dtype=torch.float32)
    finalize = b.dof.finalize
    b.dof.finalize = lambda dtype: finalize(dtype=dtype, device="cpu")
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    b.add_potential(ag.StableNeoHookean.from_pyvista(mesh))
    return b.finalize(), torch.tensor(0.25 * mask, dtype=torch.float32)


class _Warm(Model):
    def init(self):
        s = super().init()
        return dataclasses.replace(s, u=s.u + 1.0)


class _Lifted(DofMap):
    def to_full(self, free):
        return super().to_full(free) + 2.0


def test_plain_and_overridden_models():
    (a, fixed_a), (b, fixed_b), (c, fixed_c) = (_parts(n) for n in (1, 2, 3))
    b.__class__ = _Warm
    c.dof_map.__class__ = _Lifted
    bf = BatchedForward([a, b, c])
    u = bf.initial_u(device="cpu")
    expect = torch.cat([fixed_a, fixed_b + 1.0, fixed_c + 2.0])
    assert torch.equal(u, expect)
    assert torch.equal(u, torch.cat([m.init().u for m in (a, b, c)]))
    # a replaced bound method counts too
    a.init = lambda: dataclasses.replace(Model.init(a), u=torch.full_like(fixed_a, 3.0))
    assert torch.equal(bf.initial_u(device="cpu")[: fixed_a.shape[0]], torch.full_like(fixed_a, 3.0))


def test_the_result_is_the_callers_own():
    a, fixed = _parts(2)
    bf = BatchedForward([a])
    u = bf.initial_u(device="cpu")
    u += 5.0
    assert torch.equal(bf.initial_u(device="cpu"), fixed)
    assert np.allclose(a.init().u.numpy(), fixed.numpy())
