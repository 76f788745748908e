"""The work this framework does for its users, as measurable cases.

A case is one call that a particle-in-cell program makes again and again,
through the public entry points (``PicMethod.step``, the depositors, the
pushers, ``DifferentiableTrajectory``), on the package's own synthetic
workloads (a 1 x 1 x 4 cm box of jittered tetrahedra, electron beams and
bunches, ``pyrticle_b200.problems``):

* ``step``: LSRK4 steps of the whole store, each followed by one rho/j
  deposition (plain or normalising, FP64 or mixed, orders 1-4);
* ``push``: the steps alone (a program that deposits less often);
* ``average``: steps with the field-averaging pusher;
* ``grid``: a step whose deposition goes over a brick grid and is remapped;
* ``adjoint``: a short differentiable trajectory, forward and backward.

The beams drift along z, so the meshes that are stepped are z-periodic (a
section of a beam line): a state can be stepped any number of times. One
``PicMethod`` serves all states of a case, as in a user's program; every state
has its own particles, drawn from the seed.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from pyrticle_b200 import meshgen
from pyrticle_b200.adjoint import DifferentiableTrajectory
from pyrticle_b200.cloud import PicMethod
from pyrticle_b200.deposition.grid import GridDepositor
from pyrticle_b200.deposition.grid_base import SingleBrickGenerator
from pyrticle_b200.deposition.shape import (NormalizedShapeFunctionDepositor,
                                            ShapeFunctionDepositor)
from pyrticle_b200.discretization import Discretization
from pyrticle_b200.problems import stable_dt
from pyrticle_b200.pusher import AverageParticlePusher, MonomialParticlePusher
from pyrticle_b200.tools import PolynomialShapeFunction
from pyrticle_b200.units import SIUnitsWithNaturalConstants as U

CM = 1e-2
BOX = (1 * CM, 1 * CM, 4 * CM)
F64 = torch.float64


def _case(name, kind, nx, nz, order, n, radius_cm, **more):
    c = {"kind": kind, "nx": nx, "nz": nz, "order": order, "n": n, "radius_cm": radius_cm,
         "depositor": "plain", "precision": "fp64", "beam": "beam", "fields": "focusing",
         "steps": 1}
    c.update(more)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a first look at a set-up, a few thousand particles
        _case("step_2k", "step", 8, 32, 2, 2000, 0.1),
        # the small workload (config0): ten steps of a call, default depositor
        _case("step_10k_x10", "step", 8, 32, 2, 10_000, 0.1, steps=10),
        # the same size in the chosen form, one step a call (fields change
        # between calls in a coupled program)
        _case("step_10k_norm_mixed", "step", 8, 32, 2, 10_007, 0.1, depositor="normalized",
              precision="mixed"),
        # an ordinary production step, charge-exact, all FP64 (config3's mesh)
        _case("step_1m_norm_fp64", "step", 16, 64, 3, 1_000_003, 0.1, depositor="normalized"),
        # a dense bunch on an order-4 mesh in the chosen form (config4's shape)
        _case("step_2m_o4_bunch_mixed", "step", 24, 48, 4, 2_000_000, 0.05, beam="bunch",
              precision="mixed"),
        # a large FP64 step with the default depositor (config2's mesh)
        _case("step_4m_plain_fp64", "step", 32, 128, 3, 4_000_000, 0.08, fields="fourier"),
        # the largest: config2 in the chosen form
        _case("step_16m_norm_mixed", "step", 32, 128, 3, 16_000_000, 0.08, fields="fourier",
              depositor="normalized", precision="mixed"),
        # steps without a deposition (a program that deposits every few steps)
        _case("push_4m_o3_fp64", "push", 16, 64, 3, 4_000_000, 0.1),
        # the averaging pusher, five shape averages a step
        _case("average_100k", "average", 8, 32, 2, 100_000, 0.1),
        # the grid depositor with its remap, in its default precision and in
        # the chosen form (config1's ratio of grid points to cubes)
        _case("grid_500k_fp64", "grid", 16, 64, 3, 500_000, 0.1),
        _case("grid_200k_mixed", "grid", 8, 32, 2, 200_001, 0.15, precision="mixed"),
        # gradients of a short trajectory (config3)
        _case("adjoint_300k_x10", "adjoint", 16, 64, 3, 300_000, 0.1, steps=10),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | rng.randint(0, 1)

    kind = rng.choice(["step"] * 5 + ["push", "average", "grid", "adjoint"])
    nx = rng.choice([6, 8, 10, 12, 16])
    nz = 4 * nx
    order = rng.choice([1, 2, 2, 3, 3, 4]) if nx <= 12 else rng.choice([2, 3])
    if kind == "grid":
        nx, nz, order = min(nx, 10), 4 * min(nx, 10), min(order, 3)
    # shape radii of 0.8 to 2.4 cube edges
    radius = round(rng.uniform(0.8, 2.4) / nx, 4)
    hi = {"step": 4_000_000, "push": 8_000_000, "average": 200_000, "grid": 1_000_000,
          "adjoint": 500_000}[kind]
    n = log_int(1000, hi)
    # at most 4e9 (particle, node position) pairs a pass
    per = _pairs(_case(None, kind, nx, nz, order, 1, radius))
    n = max(1000, min(n, int(4e9 / max(per, 1.0))))
    more = {}
    if kind == "step":
        more["depositor"] = rng.choice(["plain", "normalized"])
        more["precision"] = rng.choice(["fp64", "mixed"])
        more["beam"] = rng.choice(["beam", "beam", "bunch"])
        more["fields"] = rng.choice(["focusing", "fourier"])
    elif kind == "push":
        more["precision"] = rng.choice(["fp64", "mixed"])
        more["fields"] = rng.choice(["focusing", "fourier"])
    elif kind == "grid":
        more["precision"] = rng.choice(["fp64", "mixed"])
    elif kind == "adjoint":
        more["steps"] = rng.randint(2, 10)
    if kind in ("step", "push") and n < 50_000:
        more["steps"] = rng.randint(1, 10)
    return _case(None, kind, nx, nz, order, n, radius, **more)


# ------------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=2)
def _discretization(nx, nz, order, periodic):
    mesh = meshgen.box_mesh((nx, nx, nz), (0.0, 0.0, 0.0), BOX, jitter=0.15, seed=0,
                            periodic=(False, False, periodic))
    return Discretization(mesh, order)


@functools.lru_cache(maxsize=3)
def _method(kind, nx, nz, order, radius_cm, depositor, precision):
    """The program's PicMethod: mesh tables, depositor and pusher."""
    # the deposition adjoint and the grid have their particles inside the box
    discr = _discretization(nx, nz, order, kind in ("step", "push", "average"))
    if kind == "grid":
        dep = GridDepositor(SingleBrickGenerator(dims=(4 * nx, 4 * nx, 4 * nz)),
                            precision=precision)
    elif depositor == "normalized":
        dep = NormalizedShapeFunctionDepositor(precision=precision)
    else:
        dep = ShapeFunctionDepositor(precision=precision)
    pusher = AverageParticlePusher() if kind == "average" else MonomialParticlePusher()
    method = PicMethod(discr, U, dep, pusher, 3, 3)
    method.depositor.set_shape_function(None, PolynomialShapeFunction(radius_cm * CM, 3, 2))
    return method


def _method_of(case):
    return _method(case["kind"], case["nx"], case["nz"], case["order"], case["radius_cm"],
                   case["depositor"], case["precision"])


def _particles(case, seed):
    """Positions and momenta [n, 3] of an electron beam (or bunch) along z."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]

    def uniform():
        return torch.rand(n, generator=g, device="cuda", dtype=F64)

    def normal():
        return torch.randn(n, generator=g, device="cuda", dtype=F64)

    x = torch.empty((n, 3), device="cuda", dtype=F64)
    if case["beam"] == "bunch":
        gamma = 5.0
        for d, sigma, mid in ((0, 0.1, 0.5), (1, 0.1, 0.5), (2, 0.05, 2.0)):
            x[:, d] = CM * (mid + torch.clamp(sigma * normal(), -0.4, 0.4))
    else:
        gamma = 2.0
        r = 0.25 * CM * torch.sqrt(uniform())
        th = 2 * math.pi * uniform()
        x[:, 0] = 0.5 * CM + r * torch.cos(th)
        x[:, 1] = 0.5 * CM + r * torch.sin(th)
        x[:, 2] = CM * (0.5 + 3.0 * uniform())
    pz = U.EL_MASS * U.VACUUM_LIGHT_SPEED() * math.sqrt(gamma ** 2 - 1)
    p = torch.empty_like(x)
    p[:, 0] = 1e-3 * pz * normal()
    p[:, 1] = 1e-3 * pz * normal()
    p[:, 2] = pz
    return x, p


# static fields at the nodes: a uniform Bz and a linear radial E ("focusing"),
# or Bz and plane waves of E and B ("fourier")
BZ, GRADIENT = 0.1, 1e6


def _fields(case, nodes):
    f = torch.zeros((6, nodes.shape[0]), device="cuda", dtype=F64)
    f[5] = BZ
    if case["fields"] == "focusing":
        f[0] = -GRADIENT * (nodes[:, 0] - 0.5 * CM)
        f[1] = -GRADIENT * (nodes[:, 1] - 0.5 * CM)
        return f
    rng = np.random.default_rng(2)
    for which in (0, 1):
        for _ in range(8):
            amp = rng.normal(0, 1e4) * (1.0 if which == 0 else 1.0 / U.VACUUM_LIGHT_SPEED())
            k = rng.normal(size=3)
            k *= 2 * math.pi / rng.uniform(0.2 * CM, 2 * CM) / np.linalg.norm(k)
            pol = np.cross(k, rng.normal(size=3))
            pol /= np.linalg.norm(pol)
            phase = rng.uniform(0, 2 * math.pi)
            wave = amp * torch.cos(nodes @ torch.as_tensor(k, device="cuda") + phase)
            for d in range(3):
                f[3 * which + d] += float(pol[d]) * wave
    return f


@functools.lru_cache(maxsize=2)
def _field_tensor(fields, nx, nz, order, periodic):
    nodes = torch.as_tensor(np.ascontiguousarray(_discretization(nx, nz, order, periodic).nodes),
                            device="cuda")
    return _fields({"fields": fields}, nodes)


def _cotangents(case, seed, nn):
    """Weights of a linear observable of (rho, j)."""
    g = torch.Generator(device="cuda").manual_seed(seed + 7919)
    grho = torch.randn(nn, generator=g, device="cuda", dtype=F64)
    gj = torch.randn((3, nn), generator=g, device="cuda", dtype=F64) / U.VACUUM_LIGHT_SPEED()
    return grho, gj


def prepare(case, seed):
    method = _method_of(case)
    x, p = _particles(case, seed)
    n = case["n"]
    mesh = method.discretization.mesh
    state = {"case": case, "method": method, "dt": stable_dt(mesh)}
    if case["kind"] == "adjoint":
        nodes = torch.as_tensor(np.ascontiguousarray(method.discretization.nodes), device="cuda")
        basis = torch.zeros((2, 6, nodes.shape[0]), device="cuda", dtype=F64)
        basis[0, 5] = 1.0
        basis[1, 0] = -(nodes[:, 0] - 0.5 * CM)
        basis[1, 1] = -(nodes[:, 1] - 0.5 * CM)
        state["traj"] = DifferentiableTrajectory(
            method, torch.full((n,), -U.EL_CHARGE, device="cuda", dtype=F64),
            torch.full((n,), U.EL_MASS, device="cuda", dtype=F64), state["dt"], case["steps"],
            checkpoint_every=5, basis=basis)
        state["x0"] = x.T.contiguous().requires_grad_()
        state["p0"] = p.T.contiguous().requires_grad_()
        state["theta"] = torch.tensor([BZ, GRADIENT], device="cuda", dtype=F64).requires_grad_()
        state["cotangents"] = _cotangents(case, seed, nodes.shape[0])
        return state
    state["fields"] = _field_tensor(case["fields"], case["nx"], case["nz"], case["order"],
                                    case["kind"] != "grid")
    particles = method.make_state()
    method.add_particles_from_arrays(particles, x.cpu().numpy(), p.cpu().numpy(),
                                     np.full(n, -U.EL_CHARGE), np.full(n, U.EL_MASS))
    state["particles"] = particles
    return state


# --------------------------------------------------------------------- run

def run(state):
    case, method = state["case"], state["method"]
    if case["kind"] == "adjoint":
        leaves = (state["x0"], state["p0"], state["theta"])
        rho, j = state["traj"](*leaves)
        gx, gp, gt = torch.autograd.grad((rho, j), leaves, state["cotangents"])
        return {"rho": rho, "j": j, "grad_x0": gx, "grad_p0": gp, "grad_theta": gt}
    particles = state["particles"]
    if case["kind"] == "grid":
        # deposition and remap of the present particles: the particle side of
        # a step that another pusher made
        rho, j = method.depositor.deposit_densities_device(particles)
        return {"rho": rho, "j": j}
    out = method.step(particles, state["fields"], state["dt"], steps=case["steps"],
                      deposit=case["kind"] != "push",
                      precision=1 if case["precision"] == "mixed" else 0)
    got = {"x": particles.x, "p": particles.p, "el": particles.el}
    if out is not None:
        got["rho"], got["j"] = out
    return got


# -------------------------------------------------------------------- work

def _elements(case):
    return 6 * case["nx"] ** 2 * case["nz"]


def _positions(case):
    """Distinct node positions of a tetrahedral mesh, about order^3 / 6 an element."""
    return _elements(case) * case["order"] ** 3 / 6.0


def _targets(case):
    return 64.0 * case["nx"] ** 2 * case["nz"] if case["kind"] == "grid" else _positions(case)


def _pairs(case):
    """(particle, target point) pairs within the shape radius, about."""
    return case["n"] * 4.19 * case["radius_cm"] ** 3 * _targets(case) / 4.0


def work(case):
    n, np_ = case["n"], (case["order"] + 1) * (case["order"] + 2) * (case["order"] + 3) // 6
    nodes = _elements(case) * np_
    kind, steps = case["kind"], case["steps"]
    pairs = _pairs(case)
    # a stage reads and writes x, p and the two residuals and reads q, m and
    # the element; about 250 + 12 np operations (interpolation, force, update)
    stage_b, stage_f = 216.0 * n, (250.0 + 14.0 * np_) * n
    # a deposition reads x, v, q, writes rho and j; 15 operations a pair, the
    # normalising one 11 more
    dep_b, dep_f = 60.0 * n + 32.0 * nodes, 15.0 * pairs
    fields_b = 48.0 * nodes
    if kind == "adjoint":
        return {"bytes": steps * 5 * 3 * stage_b + 2 * dep_b + fields_b,
                "flops": steps * 5 * 4 * stage_f + 2.2 * dep_f}
    if kind == "grid":
        # the deposition, and a matrix-vector product per element and component
        points = 64.0 * case["nx"] ** 2 * case["nz"]
        return {"bytes": dep_b + 8.0 * points * (np_ + 4),
                "flops": dep_f + 8.0 * points * np_}
    if kind == "push":
        return {"bytes": steps * (5 * stage_b + 144.0 * n) + fields_b,
                "flops": steps * 5 * stage_f}
    if case["depositor"] == "normalized":
        dep_f += 11.0 * pairs
    if kind == "average":
        stage_f += 24.0 * pairs
    return {"bytes": steps * (5 * stage_b + dep_b + 144.0 * n) + fields_b,
            "flops": steps * (5 * stage_f + dep_f)}


# ------------------------------------------- the same results, in plain torch

LSRK_A = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
          -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0)
LSRK_B = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
          1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
          2277821191437.0 / 14882151754819.0)


def _velocity(p):
    c = U.VACUUM_LIGHT_SPEED()
    p2 = (p * p).sum(1, keepdim=True)
    return c * p / torch.sqrt(U.EL_MASS ** 2 * c ** 2 + p2)


def _lorentz(v, e, b):
    return -U.EL_CHARGE * (e + torch.linalg.cross(v, b))


class _Near:
    """Sources binned into cubes of at least the radius, to be met cube by cube."""

    def __init__(self, y, radius, period):
        self.dims = [max(1, int(b / (radius * (1 + 1e-9)))) for b in BOX]
        self.radius, self.period = radius, period
        key = self.key(y)
        self.order = torch.argsort(key)
        self.y = y[self.order]
        cubes = self.dims[0] * self.dims[1] * self.dims[2]
        self.starts = np.concatenate(
            [[0], torch.cumsum(torch.bincount(key, minlength=cubes), 0).cpu().numpy()])

    def key(self, y):
        k = [torch.clamp((y[:, d] * (self.dims[d] / BOX[d])).long(), 0, self.dims[d] - 1)
             for d in range(3)]
        return k[0] + self.dims[0] * (k[1] + self.dims[1] * k[2])

    def near(self, cube):
        """Indexes into self.y that the points of a cube may reach, and z shifts."""
        cx, r = cube % self.dims[0], cube // self.dims[0]
        cy, cz = r % self.dims[1], r // self.dims[1]
        for z in (cz - 1, cz, cz + 1):
            shift = 0.0
            if z < 0 or z >= self.dims[2]:
                if not self.period:
                    continue
                shift = -BOX[2] if z < 0 else BOX[2]
                z %= self.dims[2]
            for yy in range(max(cy - 1, 0), min(cy + 2, self.dims[1])):
                row = self.dims[0] * (yy + self.dims[1] * z)
                s = int(self.starts[row + max(cx - 1, 0)])
                t = int(self.starts[row + min(cx + 1, self.dims[0] - 1) + 1])
                if t > s:
                    yield s, t, shift

    def sums(self, x, visit, most=32 << 20):
        """For the targets x, cube by cube: visit(rows, source indexes, d) with
        d [rows, sources, 3] from target to source."""
        key = self.key(x)
        order = torch.argsort(key)
        cubes = self.dims[0] * self.dims[1] * self.dims[2]
        ends = torch.cumsum(torch.bincount(key, minlength=cubes), 0).cpu().numpy()
        b = 0
        for cube in range(cubes):
            e = int(ends[cube])
            if e > b:
                parts = list(self.near(cube))
                if parts:
                    at = torch.cat([torch.arange(s, t, device=x.device) for s, t, _ in parts])
                    src = torch.cat([self.y[s:t] + torch.tensor([0.0, 0.0, z], device=x.device)
                                     for s, t, z in parts])
                    step = max(1, most // len(at))
                    for r in range(b, e, step):
                        rows = order[r:min(r + step, e)]
                        visit(rows, self.order[at], x[rows], src)
            b = e


def _shape(radius, x, y):
    """t = radius - r^2 / radius, at least 0, for all pairs: the shape is N t^2."""
    r2 = torch.zeros((len(x), len(y)), device=x.device, dtype=F64)
    for d in range(3):
        r2 += (x[:, d, None] - y[None, :, d]) ** 2
    return torch.clamp(radius - r2 / radius, min=0.0)


def _deposit(points, x, w, v, radius, period):
    """rho [points], j [3, points] of particles with weights w."""
    out = torch.zeros((4, len(points)), device=x.device, dtype=F64)
    cols = torch.cat([w[:, None], w[:, None] * v], dim=1)

    def visit(rows, at, a, b):
        out[:, rows] = (_shape(radius, a, b) ** 2 @ cols[at]).T

    _Near(x, radius, period).sums(points, visit)
    return out[0], out[1:]


def exact(case, seed):
    if case["fields"] != "focusing" or case["kind"] == "push" or _pairs(case) > 3e9:
        return None
    method = _method_of(case)
    discr = method.discretization
    nodes = torch.as_tensor(np.ascontiguousarray(discr.nodes), device="cuda")
    radius = case["radius_cm"] * CM
    # S(r) = N (a - r^2/a)^2 integrates to one over space
    norm = 105.0 / (32.0 * math.pi * radius ** 5)
    q = -U.EL_CHARGE
    x, p = _particles(case, seed)
    weights = None
    if case["kind"] == "average" or case["depositor"] == "normalized":
        ldis = discr.element_groups[0].local_discretization
        weights = torch.as_tensor(
            np.outer(discr.mesh.jacobians, ldis.mass_matrix().sum(axis=1)).ravel(), device="cuda")
    axis = torch.tensor([0.5 * CM, 0.5 * CM, 0.0], device="cuda", dtype=F64)
    if case["kind"] == "grid":
        return _exact_grid(case, method, x, p, norm)
    period = case["kind"] != "adjoint"
    theta = torch.tensor([BZ, GRADIENT], device="cuda", dtype=F64)
    if case["kind"] == "adjoint":
        x0, p0 = x.T.contiguous().requires_grad_(), p.T.contiguous().requires_grad_()
        theta.requires_grad_()
        x, p = x0.T, p0.T

    def force(x, p):
        v = _velocity(p)
        if case["kind"] == "average":
            e, b = _averaged(case, nodes, weights, x, radius)
        else:
            e = -theta[1] * (x - axis) * torch.tensor([1.0, 1.0, 0.0], device="cuda")
            b = theta[0] * torch.tensor([0.0, 0.0, 1.0], device="cuda", dtype=F64).expand_as(x)
        return v, _lorentz(v, e, b)

    dt = stable_dt(discr.mesh)
    for _ in range(case["steps"]):
        kx = kp = 0.0
        for a, b in zip(LSRK_A, LSRK_B):
            fx, fp = force(x, p)
            kx, kp = a * kx + dt * fx, a * kp + dt * fp
            x, p = x + b * kx, p + b * kp
            if period:
                x = torch.stack([x[:, 0], x[:, 1], torch.remainder(x[:, 2], BOX[2])], dim=1)
    v = _velocity(p)
    with torch.no_grad():
        w = torch.full((len(x),), q * norm, device="cuda", dtype=F64)
        if case["depositor"] == "normalized":
            integral = torch.zeros(len(x), device="cuda", dtype=F64)

            def visit(rows, at, a, b):
                integral[rows] = _shape(radius, a, b) ** 2 @ weights[at]

            _Near(nodes, radius, period).sums(x, visit)
            w = q / integral
        rho, j = _deposit(nodes, x, w, v, radius, period)
    if case["kind"] != "adjoint":
        return {"x": None, "p": None, "el": None, "rho": rho, "j": j}
    grho, gj = _cotangents(case, seed, len(nodes))
    g = torch.cat([grho[:, None], gj.T], dim=1)
    gx, gv = torch.zeros_like(x), torch.zeros_like(x)
    with torch.no_grad():
        def visit(rows, at, a, b):
            t = _shape(radius, a, b)
            gv[rows] = q * norm * (t ** 2 @ g[at][:, 1:])
            h = t * (g[at][:, 0][None, :] + v[rows] @ g[at][:, 1:].T)
            gx[rows] = q * norm * 4 / radius * (h @ b - h.sum(1, keepdim=True) * a)

        _Near(nodes, radius, period).sums(x, visit)
    grads = torch.autograd.grad((x, v), (x0, p0, theta), (gx, gv))
    return {"rho": rho, "j": j, "grad_x0": grads[0], "grad_p0": grads[1], "grad_theta": grads[2]}


def _averaged(case, nodes, weights, x, radius):
    """E and B at x as their averages over the nodes, weighted by S |J| w."""
    cols = torch.cat([torch.ones((len(nodes), 1), device="cuda", dtype=F64),
                      _fields(case, nodes).T], dim=1) * weights[:, None]
    out = torch.zeros((len(x), 7), device="cuda", dtype=F64)

    def visit(rows, at, a, b):
        out[rows] = _shape(radius, a, b) ** 2 @ cols[at]

    _Near(nodes, radius, True).sums(x, visit)
    return out[:, 1:4] / out[:, :1], out[:, 4:] / out[:, :1]


def _exact_grid(case, method, x, p, norm):
    """Deposition onto the brick points, then each element's interpolation
    matrix times its weighted points."""
    dep = method.depositor
    brick = dep.bricks[0]
    radius = case["radius_cm"] * CM
    dims = [4 * case["nx"], 4 * case["nx"], 4 * case["nz"]]
    axes = [(torch.arange(m, device="cuda", dtype=F64) + 0.5) * (b / m)
            for m, b in zip(dims, BOX)]
    assert len(brick) == dims[0] * dims[1] * dims[2]
    z, y, xx = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    points = torch.stack([xx.ravel(), y.ravel(), z.ravel()], dim=1)
    w = torch.full((len(x),), -U.EL_CHARGE * norm, device="cuda", dtype=F64)
    rho, j = _deposit(points, x, w, _velocity(p), radius, False)
    grid = torch.cat([rho[None], j])
    np_ = method.discretization.nodes_per_element
    counts = np.diff(np.asarray(dep.eog["starts"], dtype=np.int64))
    element = torch.as_tensor(np.repeat(np.arange(len(counts)), counts), device="cuda")
    at = torch.as_tensor(np.asarray(dep.eog["grid_nodes"], dtype=np.int64), device="cuda")
    pw = torch.as_tensor(np.asarray(dep.eog["weights"]), device="cuda")
    mats = torch.as_tensor(np.asarray(dep.eog["matrices"]), device="cuda").view(-1, np_)
    out = torch.zeros((4, len(counts), np_), device="cuda", dtype=F64)
    for k in range(4):
        out[k].index_add_(0, element, mats * (pw * grid[k][at])[:, None])
    out = out.reshape(4, -1)
    return {"rho": out[0], "j": out[1:]}
