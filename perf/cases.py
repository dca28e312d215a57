"""The workloads this framework's speed is measured on: what its users have it do, through its public entry points.

A program builds its bodies once (meshes, materials, boundary conditions) and then steps many states through
them, so ``prepare`` keeps one body per case and makes the states (and materials, loads or right-hand sides)
from the seed; ``run`` hands one of them in, calls the framework and takes the whole result.

Kinds of case
  step        one body of tetrahedra (corotational or linear) or hexahedra, plain FP64 or mixed precision
  batch       many uneven bodies in one handle
  rollout     a differentiable rollout: forward, then the reverse sweep to materials and initial state
  compliance  a step, then the constraint columns of its system solved (with compliance warping)
  cg          the CG solver on a caller's sparse matrix

Meshes are the cube grids of ``opensurgsim_gb300.mesh`` (5 tetrahedra a cube, interior nodes jittered), clamped
at z = 0. States are those of a body in use: bent, twisted and rippled by a few per cent of strain and
moving at some tenths of a metre per second.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from opensurgsim_gb300 import _lib, autograd, mesh
from opensurgsim_gb300.body import Body, CgSolver

DT = 1e-3
ALPHA, BETA = 0.01, 0.001
GRAVITY = (0.0, 0.0, -9.81)
TOL = 1e-10


def listed():
    """The listed cases; each comment says what in real use the case stands for."""
    return [
        # A tool-sized body in a haptics loop: the state comes from the host and goes back every step.
        dict(name="step fp64 3x3x4", kind="step", a=3, b=3, c=4, element=0, precision=0, steps=1, host=True, bar=False),
        # The reference's own single-organ scale, plain FP64, read back for drawing after each step.
        dict(name="step fp64 10x10x10", kind="step", a=10, b=10, c=10, element=0, precision=0, steps=1, host=True,
             bar=False),
        # The same organ in mixed precision, several physics steps a frame as one captured graph.
        dict(name="step mixed 10x10x10", kind="step", a=10, b=10, c=10, element=0, precision=1, steps=5, host=False,
             bar=False),
        # A finely meshed organ with odd dimensions in plain FP64.
        dict(name="step fp64 23x31x37", kind="step", a=23, b=31, c=37, element=0, precision=0, steps=1, host=False,
             bar=False),
        # A finely meshed organ in mixed precision (80,000 tetrahedra).
        dict(name="step mixed 20x20x40", kind="step", a=20, b=20, c=40, element=0, precision=1, steps=1, host=False,
             bar=False),
        # The large compression bar: 1.28M tetrahedra, every element its own moduli, one face driven.
        dict(name="bar mixed 40x40x160", kind="step", a=40, b=40, c=160, element=0, precision=1, steps=1, host=False,
             bar=True),
        # The element of the reference's performance tests: a block of hexahedra, two graph steps.
        dict(name="hex mixed 64", kind="step", a=63, b=63, c=63, element=2, precision=1, steps=2, host=False, bar=False),
        # The throughput workload: many uneven bodies, mixed precision, graph steps.
        dict(name="batch mixed 64", kind="batch", count=64, lo=500, hi=50000, precision=1, steps=1),
        # A scene of small organs in plain FP64 as one batch.
        dict(name="batch fp64 24", kind="batch", count=24, lo=500, hi=8000, precision=0, steps=1),
        # Identification: gradients of a short rollout to every element's modulus and the initial state.
        dict(name="rollout mixed 20x20x40", kind="rollout", a=20, b=20, c=40, precision=1, steps=4, every=2),
        # Contacts on an organ: a step, then its compliance along the contact normals.
        dict(name="compliance fp64 10x10x10", kind="compliance", a=10, b=10, c=10, precision=0, columns=12),
        # The linear solver by itself on a system the caller assembled.
        dict(name="cg 15x17x19", kind="cg", a=15, b=17, c=19),
    ]


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(["step", "step", "step", "batch", "rollout", "compliance", "cg"])

    def dims(lo, hi):
        side = math.exp(rng.uniform(math.log(lo), math.log(hi))) ** (1.0 / 3.0)
        a = max(2, round(side * rng.uniform(0.6, 1.2)))
        b = max(2, round(side * rng.uniform(0.7, 1.3)))
        return a, b, max(2, round(side ** 3 / (a * b)))

    if kind == "step":
        element = rng.choice([0, 0, 0, 1, 2])
        precision = rng.choice([0, 1])
        a, b, c = dims(30, 20000 if precision == 0 else 100000)
        host = a * b * c < 2000 and rng.random() < 0.5
        steps = rng.choice([1, 2, 5]) if a * b * c < 20000 else 1
        return dict(kind=kind, a=a, b=b, c=c, element=element, precision=precision, steps=steps, host=host,
                    bar=element == 0 and rng.random() < 0.3)
    if kind == "batch":
        precision = rng.choice([0, 1])
        lo = rng.randint(200, 1000)
        return dict(kind=kind, count=rng.randint(3, 48), lo=lo, hi=lo * rng.randint(4, 40 if precision else 8),
                    precision=precision, steps=rng.choice([1, 2]))
    if kind == "rollout":
        precision = rng.choice([0, 1, 1])
        a, b, c = dims(100, 1500 if precision == 0 else 16000)
        return dict(kind=kind, a=a, b=b, c=c, precision=precision, steps=rng.randint(2, 4), every=rng.randint(1, 3))
    a, b, c = dims(100, 4000)
    if kind == "compliance":
        return dict(kind=kind, a=a, b=b, c=c, precision=rng.choice([0, 1]), columns=rng.randint(1, 24))
    return dict(kind=kind, a=a, b=b, c=c)


# ---- the bodies and the states ---------------------------------------------------------------------------------


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


@functools.lru_cache(maxsize=64)
def _meshes(key):
    """The case's meshes (a list of one, or of a batch's) and their grids' dimensions."""
    c = dict(key)
    if c["kind"] == "batch":
        scenes = mesh.scenes_batch(count=c["count"], lo=c["lo"], hi=c["hi"], seed=3)
        return [s.mesh for s in scenes]
    if c.get("element") == 2:
        s = mesh.scene_hex_cube(c["a"], c["b"], c["c"], young=15.3e3, poisson=0.45, density=980.0)
        return [s.mesh]
    if c.get("bar"):
        return [mesh.scene_bar_compression(c["a"], c["b"], c["c"]).mesh]
    return [mesh.scene_cube(c["a"], c["b"], c["c"]).mesh]


def _tolerance(case):
    if case.get("element") == 2 and case["precision"] == 0:
        return 1e-3  # the reference's performance tests
    return 1e-12 if case["kind"] == "rollout" else TOL


@functools.lru_cache(maxsize=64)
def _body(key):
    """The body a program keeps for this case."""
    c = dict(key)
    ms = _meshes(key)
    return Body(ms if c["kind"] == "batch" else ms[0], rayleigh_mass=ALPHA, rayleigh_stiffness=BETA, gravity=GRAVITY,
                cg_tolerance=_tolerance(c), precision=c["precision"], element_type=c.get("element", 0))


def _state(case, m, rng):
    """Positions and velocities (N, 3) of one body in use, from a numpy generator; clamped nodes at rest."""
    X = m.nodes
    lo, hi = X.min(axis=0), X.max(axis=0)
    t = (X - lo) / (hi - lo)
    L = float(hi[2] - lo[2])
    z = t[:, 2:3]
    bend = rng.uniform(-0.03, 0.03, size=2) * L
    twist = rng.uniform(-0.05, 0.05)
    ripple = rng.uniform(-0.005, 0.005, size=X.shape) * m.h
    u = np.zeros_like(X)
    u[:, :2] += bend * z ** 2
    u[:, :2] += twist * z * (X - (lo + hi) / 2)[:, [1, 0]] * np.array([-1.0, 1.0])
    u[:, 2:3] -= rng.uniform(0.0, 0.02) * L * z
    sway = rng.uniform(-0.3, 0.3, size=3)
    v = sway * z + rng.normal(0.0, 0.01, size=X.shape)
    fixed = np.zeros(3 * X.shape[0], dtype=bool)
    fixed[m.bc_dofs] = True
    if case.get("bar"):
        u *= 0.1  # early in its ramp: moduli two decades apart beside each other leave no room for more
    clamped = t[:, 2] == 0.0
    x = X + np.where(clamped[:, None], 0.0, u + ripple)
    v = np.where(fixed.reshape(-1, 3), 0.0, v)
    if case.get("bar"):
        # The far face is driven along z at the ramp's speed; the bar behind it follows.
        speed = -0.2 * L / (50 * DT) * rng.uniform(0.2, 1.0)
        top = t[:, 2] == 1.0
        v = np.where(clamped[:, None], 0.0, np.where(top[:, None], 0.0, v))
        v[:, 2] += np.where(clamped, 0.0, speed * t[:, 2])
    return x, v


def _states(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    xs, vs = zip(*(_state(case, m, rng) for m in _meshes(_key(case))))
    return np.concatenate(xs).ravel(), np.concatenate(vs).ravel()


def _contacts(case, seed):
    """Constraint columns (n, k): unit contact normals at points of elements, in barycentric coordinates."""
    m = _meshes(_key(case))[0]
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    B = np.zeros((m.num_dofs, case["columns"]))
    for k in range(case["columns"]):
        nodes = m.tets[rng.integers(m.num_tets)]
        w = rng.dirichlet(np.ones(4))
        d = rng.normal(size=3)
        d /= np.linalg.norm(d)
        for node, wi in zip(nodes, w):
            B[3 * node:3 * node + 3, k] += wi * d
    return B


@functools.lru_cache(maxsize=16)
def _spring_matrix(key):
    """A caller's system matrix in CSC: M/dt + (dt + beta) K of the mesh's edges as springs."""
    m = _meshes(key)[0]
    pairs = np.concatenate([m.tets[:, [i, j]] for i in range(4) for j in range(i + 1, 4)])
    pairs = np.unique(np.sort(pairs, axis=1), axis=0)
    d = m.nodes[pairs[:, 1]] - m.nodes[pairs[:, 0]]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    stiff = np.random.Generator(np.random.PCG64(5)).uniform(200.0, 2000.0, size=len(pairs))
    block = (DT + BETA) * stiff[:, None, None] * d[:, :, None] * d[:, None, :]
    I, J = pairs[:, 0], pairs[:, 1]
    n = m.num_dofs
    mass = 1e-3 / DT
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.full(n, mass)]
    for r, c, s in ((I, J, -1.0), (J, I, -1.0), (I, I, 1.0), (J, J, 1.0)):
        for i in range(3):
            for j in range(3):
                rows.append(3 * r + i)
                cols.append(3 * c + j)
                vals.append(s * block[:, i, j])
    rows, cols, vals = (np.concatenate(v) for v in (rows, cols, vals))
    at = cols.astype(np.int64) * n + rows
    slots, where = np.unique(at, return_inverse=True)
    data = np.bincount(where, weights=vals, minlength=slots.size)
    colptr = np.searchsorted(slots, np.arange(n + 1, dtype=np.int64) * n).astype(np.int32)
    return colptr, (slots % n).astype(np.int32), data


@functools.lru_cache(maxsize=16)
def _solver(key):
    s = CgSolver(*_spring_matrix(key))
    s.set_tolerance(TOL)
    return s


def prepare(case, seed):
    """The body (or solver) the program keeps, and one set of inputs made from the seed."""
    key = _key(case)
    if case["kind"] == "cg":
        n = _meshes(key)[0].num_dofs
        rng = np.random.Generator(np.random.PCG64(seed))
        return dict(case=case, solver=_solver(key), b=rng.normal(size=n))
    body = _body(key)
    x, v = _states(case, seed)
    s = dict(case=case, body=body, x=x, v=v)
    if case["kind"] == "compliance":
        s["B"] = _contacts(case, seed)
    elif not case.get("host"):
        s["x"], s["v"] = torch.from_numpy(x).cuda(), torch.from_numpy(v).cuda()
        if case["kind"] != "rollout":
            s["xv"], s["vv"] = autograd.state_views(body)
    if case["kind"] == "rollout":
        g = torch.Generator().manual_seed(seed + 2)
        E = body.num_tets
        s["log_young"] = (math.log(1e5) + 0.3 * torch.randn(E, generator=g, dtype=torch.float64)).cuda()
        s["gx"] = torch.randn(body.n, generator=g, dtype=torch.float64).cuda()
        s["gv"] = (0.1 * torch.randn(body.n, generator=g, dtype=torch.float64)).cuda()
    return s


def run(s):
    """One pass through the framework's entry points; the whole result."""
    case = s["case"]
    if case["kind"] == "cg":
        return s["solver"].solve(s["b"])[0]
    body = s["body"]
    if case["kind"] == "rollout":
        leaves = [s[k].detach().requires_grad_() for k in ("log_young", "x", "v")]
        xT, vT = autograd.rollout(body, *leaves, DT, case["steps"], checkpoint_every=case["every"])
        grads = torch.autograd.grad([xT, vT], leaves, [s["gx"], s["gv"]])
        return dict(x=xT.detach(), v=vT.detach(), g_young=grads[0], g_x=grads[1], g_v=grads[2])
    if case["kind"] == "compliance":
        body.set_state(s["x"], s["v"])
        body.step(DT, 1)
        x, v = body.state()
        return dict(x=x, v=v, X=body.apply_compliance(s["B"], warping=True)[0])
    if case.get("host"):
        body.set_state(s["x"], s["v"])
        body.step(DT, case["steps"])
        x, v = body.state()
        return dict(x=x, v=v)
    s["xv"].copy_(s["x"])
    s["vv"].copy_(s["v"])
    torch.cuda.current_stream().synchronize()  # the body steps on its own stream
    graph = case["kind"] == "batch" or (case["precision"] == 1 and case["steps"] > 1)
    body.step(DT, case["steps"], _lib.STEP_GRAPH if graph else 0)
    return dict(x=s["xv"].clone(), v=s["vv"].clone())


# ---- the work a pass cannot do without -------------------------------------------------------------------------


def _iterations(case, young=1e5, h=0.01):
    """CG iterations of one solve of these grids, from the condition number's growth with (dt c / h)^2."""
    if case.get("element") == 2:
        return 40 if case["precision"] else 5
    if case["kind"] == "cg":
        return 60
    if case.get("bar"):
        return 450
    return 9 + 69 * DT * math.sqrt(young / 1000.0) / h


def work(case):
    """Inputs read once, results written once; element updates and CG products as multiply-adds."""
    if case["kind"] == "batch":
        dims = mesh.batch_dims(case["count"], case["lo"], case["hi"], 3)
    else:
        dims = [(case["a"], case["b"], case["c"])]
    nodes = sum((a + 1) * (b + 1) * (c + 1) for a, b, c in dims)
    cubes = sum(a * b * c for a, b, c in dims)
    hexes = case.get("element") == 2
    elements = cubes if hexes else 5 * cubes
    n = 3 * nodes
    nnz = 9.0 * nodes * (26.0 if hexes else 12.7)
    its = _iterations(case)
    steps = case.get("steps", 1)
    solve = 2.0 * nnz * its + 12.0 * n * its
    if case["kind"] == "cg":
        return dict(bytes=16.0 * n + 12.0 * nnz, flops=solve)
    mesh_bytes = elements * ((8 if hexes else 4) * 4 + 24) + 24.0 * nodes
    update = 4.0 * nnz if hexes else 3000.0 * elements
    flops = steps * (update + solve)
    moved = mesh_bytes + 32.0 * n
    if case["kind"] == "rollout":
        flops *= 3.0
        moved += 16.0 * elements + 32.0 * n
    if case["kind"] == "compliance":
        flops += case["columns"] * solve
        moved += 16.0 * n * case["columns"]
    return dict(bytes=float(moved), flops=float(flops))


# ---- the same in 64 bits, in plain torch -----------------------------------------------------------------------


def _skew(w):
    z = torch.zeros_like(w[..., 0])
    return torch.stack([torch.stack([z, -w[..., 2], w[..., 1]], -1), torch.stack([w[..., 2], z, -w[..., 0]], -1),
                        torch.stack([-w[..., 1], w[..., 0], z], -1)], -2)


class _Plain:
    """One implicit-Euler step of a body (or of a batch's bodies side by side) written out with dense element
    matrices: Fem3DElementCorotationalTetrahedron / Fem3DElementTetrahedron / Fem3DElementCube in OdeSolverEulerImplicit."""

    def __init__(self, case):
        ms = _meshes(_key(case))
        self.element = case.get("element", 0)
        up = lambda v, t=torch.float64: torch.as_tensor(np.ascontiguousarray(v), dtype=t).cuda()  # noqa: E731
        offs = np.cumsum([0] + [m.num_nodes for m in ms])
        X = up(np.concatenate([m.nodes for m in ms]))
        self.T = up(np.concatenate([m.tets + o for m, o in zip(ms, offs)]), torch.int64)
        young, nu, self.rho = (up(np.concatenate([getattr(m, k) for m in ms])) for k in ("young", "poisson", "density"))
        self.X, self.n, self.nu, self.log_young = X, 3 * X.shape[0], nu, torch.log(young)
        self.free = torch.ones(self.n, dtype=torch.bool, device="cuda")
        self.free[up(np.concatenate([m.bc_dofs + 3 * o for m, o in zip(ms, offs)]), torch.int64)] = False
        self.E, self.npe = self.T.shape
        self.dof = (3 * self.T[:, :, None] + torch.arange(3, device="cuda")).reshape(self.E, -1)
        if self.element == 2:
            self._hexes()
        else:
            P = X[self.T]
            V = torch.cat([P.transpose(1, 2), torch.ones(self.E, 1, 4, dtype=P.dtype, device="cuda")], 1)
            self.g = torch.linalg.inv(V)[:, :, :3].contiguous()
            self.vol = torch.linalg.det(P[:, 1:] - P[:, :1]) / 6.0
            m0 = torch.ones(4, 4, dtype=P.dtype, device="cuda") + torch.eye(4, dtype=P.dtype, device="cuda")
            self.mass = (self.rho * self.vol / 20.0)[:, None, None] * m0
        weight = (self.rho * self.vol / self.npe)[:, None].expand(-1, self.npe)
        nodal = torch.zeros(X.shape[0], dtype=X.dtype, device="cuda").index_add_(0, self.T.reshape(-1), weight.reshape(-1))
        self.gravity = (nodal[:, None] * torch.tensor(GRAVITY, dtype=X.dtype, device="cuda")).reshape(-1)

    def _moduli(self, log_young):
        y = torch.exp(log_young)
        return y * self.nu / ((1 + self.nu) * (1 - 2 * self.nu)), y / (2 * (1 + self.nu))

    def _hexes(self):
        eps = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                            [-1, 1, 1]], dtype=torch.float64, device="cuda")
        lam, mu = self._moduli(self.log_young)
        P = self.X[self.T]
        K = torch.zeros(self.E, 8, 3, 8, 3, dtype=torch.float64, device="cuda")
        self.mass = torch.zeros(self.E, 8, 8, dtype=torch.float64, device="cuda")
        self.vol = torch.zeros(self.E, dtype=torch.float64, device="cuda")
        I3 = torch.eye(3, dtype=torch.float64, device="cuda")
        for s in eps / math.sqrt(3.0):
            f = 1 + eps * s
            N = f.prod(1) / 8
            dN = torch.stack([eps[:, k] * f[:, (k + 1) % 3] * f[:, (k + 2) % 3] for k in range(3)], 1) / 8
            Jm = torch.einsum("ak,eai->eki", dN, P)
            det = torch.linalg.det(Jm)
            g = torch.einsum("eik,ak->eai", torch.linalg.inv(Jm), dN)
            gg = torch.einsum("eai,ebj->eaibj", g, g)
            Kg = lam[:, None, None, None, None] * gg + mu[:, None, None, None, None] * gg.permute(0, 1, 4, 3, 2)
            Kg = Kg + mu[:, None, None, None, None] * torch.einsum("eab,ij->eaibj", torch.einsum("eai,ebi->eab", g, g), I3)
            K += det[:, None, None, None, None] * Kg
            self.mass += (det * self.rho)[:, None, None] * (N[:, None] * N[None, :])
            self.vol += det
        self.Khex = K.reshape(self.E, 24, 24)

    def tangent(self, x, log_young):
        """Element tangents (E, D, D), forces (E, D) and rotations at positions x (n,)."""
        xe = x[self.dof].reshape(self.E, self.npe, 3)
        q = self.X[self.T]
        if self.element == 2:
            return self.Khex, -torch.einsum("eij,ej->ei", self.Khex, (xe - q).reshape(self.E, -1)), None
        p, q, g = xe - xe[:, :1], q - q[:, :1], self.g
        lam, mu = (m * self.vol for m in self._moduli(log_young))
        I3 = torch.eye(3, dtype=x.dtype, device=x.device)
        gg = torch.einsum("eai,ebj->eaibj", g, g)
        lam, mu = lam[:, None, None, None, None], mu[:, None, None, None, None]
        K0 = lam * gg + mu * gg.permute(0, 1, 4, 3, 2) + mu * torch.einsum("eak,ebk,ij->eaibj", g, g, I3)
        if self.element == 1:
            K = K0.reshape(self.E, 12, 12)
            return K, -torch.einsum("eij,ej->ei", K, (p - q).reshape(self.E, 12)), None
        F = torch.einsum("eai,eaj->eij", p, g)
        R = F
        for _ in range(14):  # the polar factor
            R = 0.5 * (R + torch.linalg.inv(R).transpose(1, 2))
        S = torch.einsum("eki,ekj->eij", R, F)
        S = 0.5 * (S + S.transpose(1, 2))
        G = (S.diagonal(dim1=1, dim2=2).sum(1)[:, None, None] * I3 - S) @ R.transpose(1, 2)
        w = p @ R - q
        Krot = torch.einsum("eki,eaibj,elj->eakbl", R, K0, R)
        Ry = torch.einsum("eik,eak->eai", R, torch.einsum("eaibj,ebj->eai", Krot, w))
        T = torch.einsum("eij,eajk,elk->eail", R, torch.einsum("eaibj,ebjk->eaik", K0, _skew(w)), R) - _skew(Ry)
        turn = torch.linalg.cross(g[:, :, None, :].expand(-1, 4, 3, 3), R[:, None, :, :].expand(-1, 4, 3, 3))  # g_b x r_q
        turn = torch.einsum("ekl,ebql->ebqk", torch.linalg.inv(G), turn)
        K = (Krot + torch.einsum("eaik,ebqk->eaibq", T, turn)).reshape(self.E, 12, 12)
        f = -torch.einsum("eij,ej->ei", K, (p - q @ R.transpose(1, 2)).reshape(self.E, 12))
        return K, f, R

    def _mass(self, u):
        return torch.einsum("eab,ebi->eai", self.mass, u.reshape(self.E, self.npe, 3)).reshape(self.E, -1)

    def _gather(self, ue):
        out = torch.zeros(self.n, dtype=ue.dtype, device=ue.device)
        return out.index_add_(0, self.dof.reshape(-1), ue.reshape(-1))

    def parts(self, x, v, log_young):
        """Element shares of the right-hand side (without gravity) and of the system, read through its lower triangle."""
        K, f, R = self.tangent(x, log_young)
        ve = v[self.dof]
        rhs = f - (DT + BETA) * torch.einsum("eij,ej->ei", K, ve) - ALPHA * self._mass(ve)
        lower = self.dof[:, :, None] >= self.dof[:, None, :]
        return rhs, torch.where(lower, K, K.transpose(1, 2)), R

    def apply(self, Ks, u):
        ue = u[self.dof]
        return self._gather((1.0 / DT + ALPHA) * self._mass(ue) + (DT + BETA) * torch.einsum("eij,ej->ei", Ks, ue))

    def solve(self, Ks, b):
        """The system's solution by CG, to the last digits."""
        b = torch.where(self.free, b, 0.0)
        d = (1.0 / DT + ALPHA) * self.mass.diagonal(dim1=1, dim2=2)[:, :, None].expand(-1, -1, 3).reshape(self.E, -1)
        d = self._gather(d + (DT + BETA) * Ks.diagonal(dim1=1, dim2=2))
        return _cg(lambda p: torch.where(self.free, self.apply(Ks, p), 0.0), b, d)

    def step(self, x, v, log_young=None):
        rhs, Ks, R = self.parts(x, v, self.log_young if log_young is None else log_young)
        dv = self.solve(Ks, self._gather(rhs) + self.gravity)
        return x + DT * (v + dv), v + dv, dv, Ks, R


def _cg(apply, b, diagonal):
    x, r = torch.zeros_like(b), b.clone()
    z = r / diagonal
    p, rz, stop = z.clone(), r @ z, 1e-28 * float(b @ b)
    for it in range(6000):
        q = apply(p)
        a = rz / (p @ q)
        x += a * p
        r -= a * q
        if it % 20 == 19 and float(r @ r) <= stop:
            break
        z = r / diagonal
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return x


def _slerp(a, b, t):
    d = (a * b).sum(1)
    th = torch.arccos(torch.clamp(d.abs(), max=1.0))
    near = d.abs() >= 1.0 - torch.finfo(torch.float64).eps
    st = torch.where(near, 1.0, torch.sin(th))
    s0 = torch.where(near, 1.0 - t, torch.sin((1.0 - t) * th) / st)
    s1 = torch.where(near, t, torch.sin(t * th) / st)
    return s0[:, None] * a + torch.where(d < 0, -s1, s1)[:, None] * b


def _node_rotations(plain, R):
    """Each node's running average of its elements' rotations, in element order."""
    w = 0.5 * torch.sqrt(torch.clamp(1.0 + R.diagonal(dim1=1, dim2=2).sum(1), min=1e-300))  # turned by far less than pi
    axis = torch.stack([R[:, 2, 1] - R[:, 1, 2], R[:, 0, 2] - R[:, 2, 0], R[:, 1, 0] - R[:, 0, 1]], 1) / (4.0 * w[:, None])
    quat = torch.cat([w[:, None], axis], 1)
    node = plain.T.reshape(-1)
    order = torch.argsort(node, stable=True)
    count = torch.bincount(node)
    first = torch.cumsum(count, 0) - count
    of = torch.arange(plain.E, device="cuda")[:, None].expand(-1, plain.npe).reshape(-1)[order]
    q = quat[of[first]]
    for k in range(1, int(count.max())):
        has = count > k
        q[has] = _slerp(q[has], quat[of[first[has] + k]], torch.full_like(q[has][:, 0], 1.0 - 1.0 / (k + 1)))
    w, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                        1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                        1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)


def exact(case, seed):
    """What ``run`` returns, by plain torch in 64 bits."""
    if case["kind"] == "cg":
        colptr, rowidx, data = _spring_matrix(_key(case))
        n = colptr.size - 1
        A = torch.sparse_csr_tensor(torch.from_numpy(colptr.astype(np.int64)), torch.from_numpy(rowidx.astype(np.int64)),
                                    torch.from_numpy(data), size=(n, n)).cuda()  # symmetric: CSC is CSR
        b = torch.from_numpy(np.random.Generator(np.random.PCG64(seed)).normal(size=n)).cuda()
        rows = np.repeat(np.arange(n), np.diff(colptr))
        diagonal = torch.from_numpy(data[rows == rowidx]).cuda()
        return _cg(lambda p: A @ p, b, diagonal)
    plain = _Plain(case)
    x, v = (torch.from_numpy(s).cuda() for s in _states(case, seed))
    if case["kind"] == "rollout":
        return _exact_rollout(plain, case, x, v, seed)
    if case["kind"] == "compliance":
        x1, v1, _, Ks, R = plain.step(x, v)
        W = _node_rotations(plain, R)
        cols = []
        for b in torch.from_numpy(_contacts(case, seed)).cuda().T:
            b = torch.where(plain.free, (b.reshape(-1, 1, 3) @ W).reshape(-1), 0.0)
            y = plain.solve(Ks, b)
            cols.append((W @ y.reshape(-1, 3, 1)).reshape(-1))
        return dict(x=x1, v=v1, X=torch.stack(cols, 1))
    for _ in range(case["steps"]):
        x, v = plain.step(x, v)[:2]
    return dict(x=x, v=v)


def _exact_rollout(plain, case, x, v, seed):
    g = torch.Generator().manual_seed(seed + 2)
    log_young = (math.log(1e5) + 0.3 * torch.randn(plain.E, generator=g, dtype=torch.float64)).cuda()
    lx = torch.randn(plain.n, generator=g, dtype=torch.float64).cuda()
    lv = (0.1 * torch.randn(plain.n, generator=g, dtype=torch.float64)).cuda()
    states = []
    for _ in range(case["steps"]):
        x1, v1, dv, Ks, _ = plain.step(x, v, log_young)
        states.append((x, v, dv, Ks))
        x, v = x1, v1
    out = dict(x=x, v=v, g_young=torch.zeros_like(log_young))
    for x, v, dv, Ks in reversed(states):
        # S dv = rhs: with S m = dt lx + lv, the reverse of the solve is the gradient of m . (rhs - S dv).
        m = plain.solve(Ks, DT * lx + lv)
        leaves = [t.detach().requires_grad_() for t in (x, v, log_young)]
        with torch.enable_grad():
            rhs, K, _ = plain.parts(*leaves)
            me, de = m[plain.dof], dv[plain.dof]
            psi = (me * rhs).sum() - (DT + BETA) * (me * torch.einsum("eij,ej->ei", K, de)).sum()
            gx, gv, gy = torch.autograd.grad(psi, leaves)
        lx, lv = lx + gx, DT * lx + lv + gv
        out["g_young"] += gy
    return dict(out, g_x=lx, g_v=lv)
