"""A grid barrier whose wait runs out: the launch ends, the error is reported,
and after a reset the solver computes what one without the failure does.  The
limit is set to nothing, so a CTA gives up at its first look unless it is the
last to arrive."""

from __future__ import annotations

import pytest
import torch

import apple_gb300 as ag
from apple_gb300 import _lib, meshgen

pytestmark = pytest.mark.gpu

DEFAULT_NS = 2_000_000_000


def _model(dims, tile_elems, dtype):
    m = meshgen.grid(*dims)
    mesh = ag.with_lame(meshgen.TetMesh(m.points, m.cells), 1.0, 4.0)
    mask = meshgen.face_mask(m, 2, "min")[:, None].repeat(3, 1)
    mesh.point_data["FixedMask"], mesh.point_data["FixedValue"] = mask, 0.01 * mask
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    b.add_potential(ag.StableNeoHookean.from_pyvista(mesh, dtype=dtype, tile_elems=tile_elems))
    return b.finalize()


def _limit(sv, ns):
    _lib.call("agb_solver_set_wait_limit", sv.handle, ns)


# 76 and 159 tiles: one and two tiles per SM
@pytest.mark.parametrize("dims, tile_elems", [((5, 4, 19), 25), ((5, 4, 38), 24)])
@pytest.mark.parametrize("mode", ["f32", "f32_correction", "f64"])
def test_iterations_report_a_wait_that_ran_out(mode, dims, tile_elems, cuda_device):
    model = _model(dims, tile_elems, torch.float64 if mode == "f64" else torch.float32)
    opt = lambda: ag.PNCG(ag.ConvergenceCriteria(max_steps=10**6, rtol=0.0),  # noqa: E731
                          refresh_ratio=0.5 if mode == "f32_correction" else 0.0)
    u0 = ag.Forward(model, ag.PNCG()).state.u

    def run(sv):
        sv.reset(u0)
        sv.iterate(12)
        u = torch.empty_like(u0)
        return sv.read(u), u

    a, b = opt(), opt()
    expected = run(a.solver(ag.ForwardProblem(model)))
    sv = b.solver(ag.ForwardProblem(model))
    for drive in (lambda: sv.iterate(50), lambda: [sv.step() for _ in range(50)]):
        sv.reset(u0)
        _limit(sv, 0)
        drive()
        with pytest.raises(RuntimeError, match="device guard"):
            sv.read()
        drive()  # the failed solve stays ended
        with pytest.raises(RuntimeError, match="device guard"):
            sv.read()
        _limit(sv, DEFAULT_NS)
        got = run(sv)
        assert got[0] == expected[0] and torch.equal(got[1], expected[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_the_adjoint_reports_a_wait_that_ran_out(dtype, cuda_device):
    model = _model((5, 4, 38), 24, dtype)
    u0 = ag.Forward(model, ag.PNCG()).state.u
    rhs = torch.ones_like(u0)
    opt = ag.PNCG()
    sv = opt.solver(ag.ForwardProblem(model))
    sv.reset(u0)
    expected, st = sv.adjoint(rhs, rtol=0.0, max_iter=12)
    _limit(sv, 0)
    with pytest.raises(RuntimeError, match="barrier"):
        sv.adjoint(rhs, rtol=0.0, max_iter=12)
    _limit(sv, DEFAULT_NS)
    got, again = sv.adjoint(rhs, rtol=0.0, max_iter=12)
    assert torch.equal(got, expected) and again == st


def test_a_negative_limit_is_refused(cuda_device):
    model = _model((2, 2, 3), 24, torch.float32)
    opt = ag.PNCG()
    sv = opt.solver(ag.ForwardProblem(model))
    with pytest.raises(RuntimeError):
        _limit(sv, -1)
