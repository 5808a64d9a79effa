"""The batch's device loop runs two iterations a body, the second skipped when
the first ended the run (GB300).  However a run is cut, into even or odd
lengths or single steps, the iterates are the same bits: across reference-state
refreshes (FP32, asked for often), across meshes that end early, with meshes of
one tile and of several, and for ARAP, whose body holds one iteration."""

import numpy as np
import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from apple_gb300.batch import BatchedForward

pytestmark = pytest.mark.gpu

TOTAL = 60


def _model(dims, material, dtype):
    m = meshgen.grid(*dims)
    lam, mu = meshgen.lame_converter(1e4, 0.45)
    mesh = ag.with_lame(meshgen.TetMesh(m.points, m.cells), mu, lam)
    mask = np.zeros((m.n_points, 3), bool)
    mask[meshgen.face_mask(m, 2, "min")] = True
    mesh.point_data["FixedMask"] = mask
    mesh.point_data["FixedValue"] = np.zeros((m.n_points, 3))
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    b.add_potential(material.from_pyvista(mesh, dtype=dtype))
    fm = meshgen.TetMesh(m.points, m.cells)
    fm.point_data["Force"] = meshgen.lumped_gravity(m, 1000.0)
    fm.point_data["GlobalPointId"] = np.arange(m.n_points)
    b.add_potential(ag.ExternalForce.from_pyvista(fm, dtype=dtype))
    return b.finalize()


@pytest.mark.parametrize("material,dtype", [(ag.StableNeoHookean, torch.float32), (ag.StableNeoHookean, torch.float64),
                                            (ag.Arap, torch.float32)])
@pytest.mark.parametrize("count", [1, 3])
def test_however_the_run_is_cut(cuda_device, material, dtype, count):
    # 6 tets, one tile of 750, several tiles and several vertex chunks
    models = [_model(d, material, dtype) for d in [(6, 6, 9), (1, 1, 1), (5, 5, 5)][:count]]
    crit = ag.ConvergenceCriteria(max_steps=10**6, rtol=1e-4)
    runs = {}
    for name, cuts in {"steps": None, "one": (TOTAL,), "even": (2,) * (TOTAL // 2), "odd": (1, 3, 5, 7) * 3 + (9, 3),
                       "mixed": (2, 1, 4, 3, 50)}.items():
        bf = BatchedForward(models, ag.PNCG(crit, refresh_ratio=0.8))
        bf.reset()
        if cuts is None:
            for _ in range(TOTAL):
                bf.step()
        else:
            assert sum(cuts) == TOTAL
            for c in cuts:
                bf.iterate(c)
        runs[name] = bf.read()
    sols, us = runs.pop("steps")
    assert max(s.n_steps for s in sols) > 8
    for name, (s2, u2) in runs.items():
        for a, b, p, q in zip(sols, s2, us, u2):
            assert a.n_steps == b.n_steps and a.result == b.result, name
            assert torch.equal(p, q), name
