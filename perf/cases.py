"""The work that this package is measured on: one case is one call (or one
group of calls) a program makes through the public entry points.

``listed()`` are the standing cases, ``draw(rng)`` more of the same ranges.
``prepare`` builds what a program holds before the call, ``run`` makes one
pass, ``work`` counts the bytes and operations the pass cannot do without and
``exact`` restates its outputs in float64 torch, without the package's code.

Kinds of cases:

* ``problem``  the five methods of ``ForwardProblem`` one after another, each
               through the free/fixed DOF map: what an optimizer outside the
               package calls once per iteration of its own;
* ``fused``    one ``eval`` of a potential with all five quantities;
* ``steps``    ``Forward.step()`` with a fixed budget of PNCG iterations, as
               an interactive or time-stepped program runs it every frame;
* ``batch``    ``BatchedForward.solve()`` of many uneven meshes, the same
               budget for each;
* ``adjoint``  the adjoint CG at a deformed state and the material gradients
               from it: the backward of an inverse problem;
* ``muscle``   one evaluation of an activation fit: new activations from the
               host, energy, gradient and diagonal, and the pull-back to
               stiffness and activation.
"""

from __future__ import annotations

import functools
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import apple_gb300 as ag
from apple_gb300 import meshgen
from apple_gb300.batch import BatchedForward

_DTYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # the smallest calls: an outer optimizer on the 5,000-tet cube, where launches and
        # host latency count
        dict(name="problem_cube_5k", kind="problem", mesh="grid", nx=10, ny=10, nz=10, material="snh", dtype="f32"),
        # the same calls with ARAP on an irregular Delaunay ball (random vertex order)
        dict(name="problem_ball_arap", kind="problem", mesh="ball", interior=20000, shell=3000, material="arap",
             dtype="f32"),
        # all five quantities in one pass on the 1.5M-tet grid: the largest evaluation
        dict(name="fused_grid_1500k", kind="fused", mesh="grid", nx=50, ny=50, nz=120, material="snh", dtype="f32"),
        # the reference's default precision
        dict(name="fused_grid_138k_f64", kind="fused", mesh="grid", nx=24, ny=24, nz=48, material="snh", dtype="f64"),
        # the cube under gravity, solved with a budget of iterations per frame
        dict(name="steps_cube_5k", kind="steps", mesh="grid", nx=10, ny=10, nz=10, material="snh", dtype="f32",
             load="gravity", steps=40),
        # an ordinary mesh
        dict(name="steps_grid_138k", kind="steps", mesh="grid", nx=24, ny=24, nz=48, material="snh", dtype="f32",
             load="stretch", steps=40),
        # the headline mesh
        dict(name="steps_grid_1500k", kind="steps", mesh="grid", nx=50, ny=50, nz=120, material="snh", dtype="f32",
             load="stretch", steps=40),
        # ARAP on the 64x64x96 grid: the largest mesh, its line search by element passes
        dict(name="steps_grid_1966k_arap", kind="steps", mesh="grid", nx=64, ny=64, nz=96, material="arap",
             dtype="f32", load="stretch", steps=20),
        # a solve in the reference's default precision
        dict(name="steps_grid_138k_f64", kind="steps", mesh="grid", nx=24, ny=24, nz=48, material="snh", dtype="f64",
             load="stretch", steps=20),
        # many uneven meshes at once
        dict(name="batch_24", kind="batch", count=24, low=4, high=24, shapes=1, material="snh", dtype="f32", steps=20),
        # the backward of an inverse problem
        dict(name="adjoint_grid_138k", kind="adjoint", mesh="grid", nx=24, ny=24, nz=48, material="snh", dtype="f32",
             steps=40),
        # one evaluation of an activation fit, activations from the host
        dict(name="muscle_grid_138k", kind="muscle", mesh="grid", nx=24, ny=24, nz=48, material="muscle",
             dtype="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid_dims(rng, lo, hi):
    """Grid dimensions with about lo..hi tets (log-uniform), odd ones among them, aspect up to 4."""
    cells = _log(rng, lo, hi) / 5.0
    ax, ay = rng.uniform(0.5, 2.0), rng.uniform(0.5, 2.0)
    s = (cells / (ax * ay)) ** (1.0 / 3.0)
    return [max(2, int(round(v))) for v in (s * ax, s * ay, s)]


def draw(rng):
    kind = rng.choice(["problem", "fused", "steps", "steps", "batch", "adjoint", "muscle"])
    dtype = "f64" if rng.random() < 0.2 else "f32"
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 24), low=rng.randint(3, 6), high=rng.randint(8, 24),
                    shapes=rng.randint(2, 10**6), material=rng.choice(["snh", "snh", "arap"]), dtype="f32",
                    steps=rng.randint(5, 20))
    if kind == "muscle":
        material = "muscle"
    elif kind == "adjoint":
        material = rng.choice(["snh", "snh", "arap"])
    else:
        material = rng.choice(["snh", "snh", "arap", "muscle"])
    most = 2e5 if dtype == "f64" else 1e6
    case = dict(kind=kind, material=material, dtype=dtype)
    if rng.random() < 0.25:
        n = _log(rng, 100, 20000)
        case.update(mesh="ball", interior=n, shell=max(20, n // 7))
    else:
        nx, ny, nz = _grid_dims(rng, 300, most)
        case.update(mesh="grid", nx=nx, ny=ny, nz=nz)
    if kind == "steps":
        case.update(load=rng.choice(["gravity", "stretch"]), steps=rng.randint(5, 40))
    if kind == "adjoint":
        case.update(steps=rng.randint(10, 40))
    return case


# ---------------------------------------------------------------------------
# meshes and inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def _grid(nx, ny, nz):
    m = meshgen.grid(nx, ny, nz, h=1.0 / nx)
    return m.points, m.cells, 1.0 / nx


@functools.lru_cache(maxsize=8)
def _ball(interior, shell):
    m = meshgen.ball(interior, shell, seed=0)
    return m.points, m.cells, (4.2 / m.points.shape[0]) ** (1.0 / 3.0)


def _geometry(case):
    """(points, cells, edge length) of the case's mesh."""
    if case["mesh"] == "ball":
        return _ball(case["interior"], case["shell"])
    return _grid(case["nx"], case["ny"], case["nz"])


def _materials(case, n_cells, rng):
    """mu, lambda, activation per cell: stiffnesses scaled by U(0.5, 2) per cell as in an inverse fit."""
    lam0, mu0 = meshgen.lame_converter(1e4, 0.45)
    theta = rng.uniform(0.5, 2.0, n_cells)
    mu, lam = mu0 * theta, lam0 * theta
    if case["material"] == "arap":
        return mu, None, None
    act = 0.05 * rng.standard_normal((n_cells, 6)) if case["material"] == "muscle" else None
    return mu, lam, act


def _boundary(points, load):
    """Fixed mask and values: the lower end held, the upper one held too or displaced along z."""
    z = points[:, 2]
    lo, hi = z.min(), z.max()
    tol = 0.05 * (hi - lo) if np.unique(z).size > 0.5 * z.size else 1e-9
    mask = np.zeros(points.shape, bool)
    values = np.zeros(points.shape)
    mask[z <= lo + tol] = True
    if load == "stretch":
        top = z >= hi - tol
        mask[top] = True
        values[top, 2] = 0.08 * (z[top] - lo)
    return mask, values


def _deformed(points, h, rng):
    """A moderately deformed state: an affine map of about 5% strain and a jitter of 5% of the edge length."""
    A = 0.05 * rng.standard_normal((3, 3))
    return points @ A.T + 0.05 * h * rng.standard_normal(points.shape)


def _mesh(points, cells, mu, lam, act):
    m = meshgen.TetMesh(points, cells)
    m.cell_data["mu"] = mu
    if lam is not None:
        m.cell_data["lambda"] = lam
    if act is not None:
        m.cell_data["activation"] = act
    return m


_CLASSES = {"snh": ag.StableNeoHookean, "arap": ag.Arap, "muscle": ag.StableNeoHookeanMuscle}


def _force(points, cells, g):
    return meshgen.lumped_gravity(meshgen.TetMesh(points, cells), 50.0, g)


def _build(points, cells, material, dtype, mu, lam, act, mask, values, force=None):
    """(model, potential)"""
    mesh = _mesh(points, cells, mu, lam, act)
    mesh.point_data["FixedMask"] = mask
    mesh.point_data["FixedValue"] = values
    b = ag.ModelBuilder(dtype=dtype)
    b.add_vertices(mesh)
    b.add_fixed(mesh)
    pot = _CLASSES[material].from_pyvista(mesh, dtype=dtype)
    b.add_potential(pot)
    if force is not None:
        fm = meshgen.TetMesh(points, cells)
        fm.point_data["Force"] = force
        fm.point_data["GlobalPointId"] = np.arange(points.shape[0])
        b.add_potential(ag.ExternalForce.from_pyvista(fm, dtype=dtype))
    return b.finalize(), pot


def _batch_shapes(case):
    rng = np.random.default_rng(case["shapes"])
    return [tuple(int(v) for v in rng.integers(case["low"], case["high"] + 1, 3)) for _ in range(case["count"])]


def _setting(case, seed):
    """What prepare and exact share: the case's numbers on the host, made from the seed alone."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        models = []
        for shape in _batch_shapes(case):
            points, cells, h = _grid(*shape)
            mu, lam, act = _materials(case, cells.shape[0], rng)
            mask, values = _boundary(points, "gravity")
            g = rng.standard_normal(3)
            models.append(dict(points=points, cells=cells, mu=mu, lam=lam, act=act, mask=mask, values=values,
                               u0=np.where(mask, values, 0.0), force=_force(points, cells, 9.8 * g / np.linalg.norm(g))))
        return models
    points, cells, h = _geometry(case)
    mu, lam, act = _materials(case, cells.shape[0], rng)
    s = dict(points=points, cells=cells, mu=mu, lam=lam, act=act, force=None)
    kind = case["kind"]
    s["mask"], s["values"] = _boundary(points, case.get("load", "gravity"))
    if kind == "steps":
        if case["load"] == "gravity":
            s["force"] = _force(points, cells, (0.0, 0.0, -9.8))
        z = points[:, 2]
        u0 = np.zeros(points.shape)
        if case["load"] == "stretch":
            u0[:, 2] = 0.08 * (z - z.min())
        u0 += rng.uniform(-0.01, 0.01, points.shape) * h
        s["u0"] = np.where(s["mask"], s["values"], u0)
        return s
    u = _deformed(points, h, rng)
    w = rng.standard_normal(points.shape)
    if kind == "adjoint":  # a mild strain, where the Hessian is positive definite as at an equilibrium
        u = np.where(s["mask"], s["values"], 0.1 * u)
    np_dtype = np.float64 if case["dtype"] == "f64" else np.float32
    s["u"], s["w"] = u.astype(np_dtype), w.astype(np_dtype)
    if kind == "problem":
        s["w"] = np.where(s["mask"], 0, s["w"]).astype(np_dtype)
    return s


def prepare(case, seed):
    dtype = _DTYPES[case["dtype"]]
    dev = torch.device("cuda")
    kind = case["kind"]
    s = _setting(case, seed)
    if kind == "batch":
        make = lambda m: _build(m["points"], m["cells"], case["material"], dtype, m["mu"], m["lam"], m["act"],  # noqa: E731
                                m["mask"], m["values"], m["force"])[0]
        with ThreadPoolExecutor(8) as pool:
            models = list(pool.map(make, s))
        opt = ag.PNCG(ag.ConvergenceCriteria(max_steps=case["steps"], rtol=1e-6))
        return dict(kind=kind, batch=BatchedForward(models, opt))
    if kind in ("fused", "muscle"):
        mesh = _mesh(s["points"], s["cells"], s["mu"], s["lam"], s["act"] if kind == "fused" else None)
        pot = _CLASSES[case["material"]].from_pyvista(mesh, dtype=dtype)
        return dict(kind=kind, pot=pot, act=s["act"], u=torch.tensor(s["u"], device=dev),
                    w=torch.tensor(s["w"], device=dev))
    model, pot = _build(s["points"], s["cells"], case["material"], dtype, s["mu"], s["lam"], s["act"], s["mask"],
                        s["values"], s["force"])
    if kind == "problem":
        problem = ag.ForwardProblem(model)
        state = ag.ModelState(u=torch.tensor(s["u"], device=dev))
        p = model.dof_map.to_free(torch.tensor(s["w"], device=dev))
        return dict(kind=kind, problem=problem, state=state, p=p)
    if kind == "steps":
        opt = ag.PNCG(ag.ConvergenceCriteria(max_steps=case["steps"], rtol=1e-9 if case["dtype"] == "f64" else 1e-6))
        start = ag.ModelState(u=torch.tensor(s["u0"], dtype=dtype, device=dev))
        return dict(kind=kind, forward=ag.Forward(model, opt, start), start=start)
    # adjoint: the solver at the state whose loss gradient is pulled back
    opt = ag.PNCG()
    solver = opt.solver(ag.ForwardProblem(model))
    u = torch.tensor(s["u"], device=dev)
    solver.reset(u)
    return dict(kind=kind, model=model, opt=opt, solver=solver, pot=pot, u=u, w=torch.tensor(s["w"], device=dev),
                steps=case["steps"])


def run(state):
    kind = state["kind"]
    if kind == "problem":
        problem, at, p = state["problem"], state["state"], state["p"]
        return {"fun": problem.fun(at), "grad": problem.grad(at), "hess_diag": problem.hess_diag(at),
                "hess_prod": problem.hess_prod(at, p), "hess_quad": problem.hess_quad(at, p)}
    if kind == "fused":
        return state["pot"].eval(state["u"], state["w"], fun=True, grad=True, hess_diag=True, hess_prod=True,
                                 hess_quad=True)
    if kind == "steps":
        forward = state["forward"]
        forward.state = state["start"]
        solution = forward.step()
        return {"u": forward.state.u, "energy": solution.energy}
    if kind == "batch":
        solutions, u = state["batch"].solve()
        return {"u": torch.cat(u), "energy": torch.tensor([s.energy for s in solutions])}
    if kind == "adjoint":
        lam, _ = state["solver"].adjoint(state["w"], rtol=1e-9, max_iter=state["steps"])
        return {"lam": lam, **state["pot"].grad_param_vjp(state["u"], lam)}
    pot, u = state["pot"], state["u"]
    pot.set_activation(state["act"])
    out = pot.eval(u, fun=True, grad=True, hess_diag=True)
    return {**out, **pot.grad_param_vjp(u, state["w"])}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _sizes(case):
    if case["kind"] == "batch":
        nt = nv = 0
        for nx, ny, nz in _batch_shapes(case):
            nt += 5 * nx * ny * nz
            nv += (nx + 1) * (ny + 1) * (nz + 1)
        return nt, nv
    if case["mesh"] == "ball":
        points, cells, _ = _ball(case["interior"], case["shell"])
        return cells.shape[0], points.shape[0]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return 5 * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)


def work(case):
    """Element data (nine entries of dhdX, the Lame parameters, four corner ids; the activation) read once
    per pass over the mesh, vertex fields read or written once; operations per element counted from the
    formulae (F, PK1, Hessian terms, corner products)."""
    nt, nv = _sizes(case)
    r = 8 if case["dtype"] == "f64" else 4
    elem = r * (10 if case["material"] == "arap" else 11) + 16 + (6 * r if case["material"] == "muscle" else 0)
    vec = 3 * r * nv
    # one deformation gradient and invariants ~90; per method ~60-150 more; ARAP's SVD ~500
    svd = 500 if case["material"] == "arap" else 0
    kind = case["kind"]
    if kind == "problem":
        return {"bytes": 5 * elem * nt + 10 * vec, "flops": (850 + 5 * svd) * nt}
    if kind == "fused":
        return {"bytes": elem * nt + 5 * vec, "flops": (600 + svd) * nt}
    if kind in ("steps", "batch"):  # each iteration one pass over the elements and seven vertex fields
        return {"bytes": case["steps"] * (elem * nt + 7 * vec), "flops": case["steps"] * (700 + svd) * nt}
    if kind == "adjoint":
        per = elem * nt + 7 * vec
        return {"bytes": case["steps"] * per + elem * nt + 2 * vec, "flops": (case["steps"] * (330 + svd) + 300) * nt}
    return {"bytes": 48 * nt + 2 * elem * nt + 5 * vec + 8 * r * nt, "flops": 1000 * nt}


# ---------------------------------------------------------------------------
# float64 restatement
# ---------------------------------------------------------------------------
def _eigh3(A):
    """Eigenvalues (ascending) and vectors of symmetric 3x3 matrices by cyclic Jacobi rotations."""
    a = [[A[:, i, j].clone() for j in range(3)] for i in range(3)]
    one, zero = torch.ones_like(a[0][0]), torch.zeros_like(a[0][0])
    v = [[one.clone() if i == j else zero.clone() for j in range(3)] for i in range(3)]
    for _ in range(6):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            x = a[p][q]
            theta = (a[q][q] - a[p][p]) / torch.where(x == 0, one, 2.0 * x)
            t = torch.where(theta >= 0, one, -one) / (theta.abs() + (theta * theta + 1.0).sqrt())
            t = torch.where(x == 0, zero, t)
            c = 1.0 / (t * t + 1.0).sqrt()
            s = t * c
            a[p][p], a[q][q] = a[p][p] - t * x, a[q][q] + t * x
            a[p][q] = a[q][p] = zero
            rp, rq = a[r][p], a[r][q]
            a[r][p] = a[p][r] = c * rp - s * rq
            a[r][q] = a[q][r] = s * rp + c * rq
            for k in range(3):
                v[k][p], v[k][q] = c * v[k][p] - s * v[k][q], s * v[k][p] + c * v[k][q]
    w, order = torch.stack([a[0][0], a[1][1], a[2][2]], 1).sort(1)
    V = torch.stack([torch.stack(row, 1) for row in v], 1)
    return w, V.gather(2, order[:, None, :].expand(-1, 3, -1))


class _Fem:
    """One potential in float64: F per element, energy, gradient, clamped diagonal, products."""

    def __init__(self, material, points, cells, mu, lam, act):
        dev = torch.device("cuda")
        f = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        self.arap = material == "arap"
        self.n = points.shape[0]
        self.cells = torch.tensor(np.asarray(cells, np.int64), device=dev)
        X = f(points)[self.cells]
        Dm = (X[:, 1:] - X[:, :1]).transpose(1, 2)
        self.dV = torch.linalg.det(Dm) / 6.0
        D = torch.linalg.inv(Dm)
        self.A = None
        if act is not None:
            a = f(act)
            self.A = torch.eye(3, device=dev, dtype=torch.float64) + torch.stack(
                [a[:, 0], a[:, 3], a[:, 4], a[:, 3], a[:, 1], a[:, 5], a[:, 4], a[:, 5], a[:, 2]], -1).reshape(-1, 3, 3)
        self.D0 = torch.cat([-D.sum(1, keepdim=True), D], 1)
        self.D = self.D0 if self.A is None else self.D0 @ self.A
        self.mu, self.lam = f(mu) * self.dV, None if lam is None else f(lam) * self.dV

    def field(self, w, D=None):
        return w[self.cells].transpose(1, 2) @ (self.D if D is None else D)

    def scatter(self, M):
        f = M @ self.D.transpose(1, 2)
        return self._sum(f.transpose(1, 2))

    def _sum(self, corner):
        out = torch.zeros((self.n, 3), dtype=torch.float64, device=corner.device)
        return out.index_add_(0, self.cells.reshape(-1), corner.reshape(-1, 3))

    @staticmethod
    def cof(F):
        c = lambda a, b: torch.linalg.cross(F[:, :, a], F[:, :, b])  # noqa: E731
        return torch.stack([c(1, 2), c(2, 0), c(0, 1)], 2)

    def at(self, u):
        """The element state at u that the methods below read."""
        eye = torch.eye(3, dtype=torch.float64, device=u.device)
        self.F = (eye if self.A is None else self.A) + self.field(u)
        if self.arap:
            lam, V = _eigh3(self.F.transpose(1, 2) @ self.F)
            s = lam.clamp_min(1e-300).sqrt()
            FV = self.F @ V
            # the smallest singular value carries the sign of det F
            s = torch.cat([s[:, :1] * torch.linalg.det(self.F).sign()[:, None], s[:, 1:]], 1)
            self.U, self.V, self.s = FV / s[:, None, :], V, s
        else:
            self.C = self.cof(self.F)
            self.J1 = torch.linalg.det(self.F) - 1.0
        return self

    def fun(self):
        if self.arap:
            return 0.5 * (self.mu * ((self.s - 1) ** 2).sum(1)).sum()
        I2 = (self.F**2).sum((1, 2))
        return (0.5 * self.mu * (I2 - 3.0) - self.mu * self.J1 + 0.5 * self.lam * self.J1**2).sum()

    def pk1(self):
        if self.arap:
            return self.mu[:, None, None] * (self.U * (self.s - 1)[:, None, :]) @ self.V.transpose(1, 2)
        return self.mu[:, None, None] * (self.F - self.C) + (self.lam * self.J1)[:, None, None] * self.C

    def grad(self):
        return self.scatter(self.pk1())

    def twists(self):
        """lambda_k and the pairs (i, j) of ARAP's twist modes."""
        out = []
        for i, j in ((1, 0), (1, 2), (0, 2)):
            out.append((i, j, 2.0 / (self.s[:, i] + self.s[:, j]).clamp_min(2.0)))
        return out

    def hess_diag(self):
        nn = (self.D**2).sum(2)[:, :, None]
        if self.arap:
            b = self.D @ self.V  # (n, 4, 3): V^T D_a
            d = nn.expand(-1, -1, 3).clone()
            for i, j, l in self.twists():
                w = (self.U[:, None, :, i] * b[:, :, j, None] - self.U[:, None, :, j] * b[:, :, i, None]) / math.sqrt(2)
                d = d - l[:, None, None] * w**2
            return self._sum((self.mu[:, None, None] * d).clamp_min(0.0))
        w = self.D @ self.C.transpose(1, 2)
        return self._sum((self.lam[:, None, None] * w**2 + self.mu[:, None, None] * nn).clamp_min(0.0))

    def along(self, p):
        """Per element: the Hessian applied to dF = grad p, and dF."""
        dF = self.field(p)
        if self.arap:
            W = self.U.transpose(1, 2) @ dF @ self.V
            M = dF.clone()
            for i, j, l in self.twists():
                q = l * (W[:, i, j] - W[:, j, i]) / 2.0
                M = M - q[:, None, None] * (self.U[:, :, i, None] * self.V[:, None, :, j]
                                            - self.U[:, :, j, None] * self.V[:, None, :, i])
            return self.mu[:, None, None] * M, dF
        x = lambda A, B, a, b: torch.linalg.cross(A[:, :, a], B[:, :, b])  # noqa: E731
        F = self.F
        H = torch.stack([x(F, dF, a, b) + x(dF, F, a, b) for a, b in ((1, 2), (2, 0), (0, 1))], 2)
        k = lambda v: v[:, None, None]  # noqa: E731
        a1 = (self.C * dF).sum((1, 2))
        return k(self.lam * a1) * self.C + k(self.mu) * dF + k(self.lam * self.J1 - self.mu) * H, dF

    def hess_prod(self, p):
        return self.scatter(self.along(p)[0])

    def hess_quad(self, p):
        M, dF = self.along(p)
        return (M * dF).sum((1, 2)).clamp_min(0.0).sum()

    def material_vjp(self, w):
        W = self.field(w)
        if self.arap:
            return {"mu": (self.pk1() * W).sum((1, 2)) / self.mu * self.dV}
        return {"mu": self.dV * ((self.F - self.C) * W).sum((1, 2)), "lambda": self.dV * self.J1 * (self.C * W).sum((1, 2))}

    def activation_vjp(self, w):
        W0 = self.field(w, self.D0)
        F0 = self.F @ torch.linalg.inv(self.A)
        H = self.along(w)[0]
        Z = F0.transpose(1, 2) @ H + W0.transpose(1, 2) @ self.pk1()
        return torch.stack([Z[:, 0, 0], Z[:, 1, 1], Z[:, 2, 2], Z[:, 0, 1] + Z[:, 1, 0], Z[:, 0, 2] + Z[:, 2, 0],
                            Z[:, 1, 2] + Z[:, 2, 1]], 1)


def _fem(material, s):
    return _Fem(material, s["points"], s["cells"], s["mu"], s["lam"], s["act"])


def _pncg(material, s, steps, rtol):
    """PNCG with the Jacobi preconditioner, Dai-Kou beta and Armijo backtracking: (u, energy)."""
    fem = _fem(material, s)
    dev = torch.device("cuda")
    free = ~torch.tensor(s["mask"], device=dev)
    force = torch.zeros((fem.n, 3), dtype=torch.float64, device=dev)
    if s["force"] is not None:
        force = torch.tensor(s["force"], device=dev)
    x = torch.tensor(s["u0"], dtype=torch.float64, device=dev)
    energy = lambda: fem.fun() - (force * x).sum()  # noqa: E731
    fem.at(x)
    f, g, d = energy(), (fem.grad() - force) * free, fem.hess_diag() * free
    precond = lambda: torch.where(d > 0, 1.0 / d.clamp_min(1e-300), d.sum().new_tensor(1.0) / d[d > 0].mean()) * free  # noqa: E731
    P = precond()
    p = -P * g
    g0 = g.norm()
    for _ in range(steps):
        if g.norm() <= rtol * g0:
            break
        slope = (g * p).sum()
        t = float(-slope / fem.hess_quad(p))
        old, gold = x, g
        for halving in range(9):
            x = old + t * p
            fem.at(x)
            fn = energy()
            if fn - f <= 1e-4 * t * slope or halving == 8:
                break
            t *= 0.5
        f, g, d = fn, (fem.grad() - force) * free, fem.hess_diag() * free
        P = precond()
        y = g - gold
        yp = (y * p).sum()
        b = float((P * g * y).sum() / yp - (P * y * y).sum() / yp * (p * g).sum() / yp)
        if not math.isfinite(b) or abs(b) > 10.0:
            b = 0.0
        if not float(-(P * g * g).sum() + b * (p * g).sum()) < 0.0:
            b = 0.0
        p = -P * g + b * p
    return x, f


def exact(case, seed):
    kind, material = case["kind"], case["material"]
    dev = torch.device("cuda")
    s = _setting(case, seed)
    if kind == "batch":
        done = [_pncg(material, m, case["steps"], 1e-6) for m in s]
        return {"u": torch.cat([u for u, _ in done]), "energy": torch.stack([e for _, e in done])}
    if kind == "steps":
        u, e = _pncg(material, s, case["steps"], 1e-9 if case["dtype"] == "f64" else 1e-6)
        return {"u": u, "energy": float(e)}
    u = torch.tensor(s["u"], device=dev).double()
    w = torch.tensor(s["w"], device=dev).double()
    fem = _fem(material, s).at(u)
    if kind == "problem":
        free = torch.tensor(~s["mask"].reshape(-1), device=dev)
        cut = lambda v: v.reshape(-1)[free]  # noqa: E731
        return {"fun": fem.fun(), "grad": cut(fem.grad()), "hess_diag": cut(fem.hess_diag()),
                "hess_prod": cut(fem.hess_prod(w)), "hess_quad": fem.hess_quad(w)}
    if kind == "fused":
        return {"fun": fem.fun().reshape(1), "grad": fem.grad(), "hess_diag": fem.hess_diag(),
                "hess_prod": fem.hess_prod(w), "hess_quad": fem.hess_quad(w).reshape(1)}
    if kind == "muscle":
        return {"fun": fem.fun().reshape(1), "grad": fem.grad(), "hess_diag": fem.hess_diag(),
                **fem.material_vjp(w), "activation": fem.activation_vjp(w)}
    # adjoint: the same number of conjugate-gradient steps
    free = ~torch.tensor(s["mask"], device=dev)
    minv = free / fem.hess_diag()
    r = w * free
    lam, p = torch.zeros_like(r), torch.zeros_like(r)
    rz, beta = (r * minv * r).sum(), 0.0
    for _ in range(case["steps"]):
        p = minv * r + beta * p
        q = fem.hess_prod(p) * free
        alpha = rz / (p * q).sum()
        lam, r = lam + alpha * p, r - alpha * q
        new = (r * minv * r).sum()
        beta, rz = new / rz, new
    return {"lam": lam, **fem.material_vjp(lam)}
