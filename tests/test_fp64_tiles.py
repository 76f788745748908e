"""The FP64 pair sums by tiles (deposition, normalised deposition) against a
brute-force sum over all (particle, node) pairs: meshes with fewer positions
than one tile, with a partial last tile and block, with too few and with
enough blocks to fill the device, periodic along all axes with a radius just
below half a period (rows of bins in several pieces), one particle to several
chunks of them."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import _lib, meshgen  # noqa: E402
from pyrticle_b200.cloud import PicMethod  # noqa: E402
from pyrticle_b200.deposition.shape import (NormalizedShapeFunctionDepositor,  # noqa: E402
                                            ShapeFunctionDepositor)
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.pusher import MonomialParticlePusher  # noqa: E402
from pyrticle_b200.tools import PolynomialShapeFunction  # noqa: E402
from pyrticle_b200.units import SIUnitsWithNaturalConstants as U  # noqa: E402

pytestmark = pytest.mark.gpu

F64 = torch.float64
TOL = 1e-12  # the parity tolerance of the FP64 form


def rel(a, b):
    return float(torch.linalg.norm(a - b) / torch.linalg.norm(b))


def setup(depositor, cubes, order, n, periodic, radius, alpha):
    mesh = meshgen.box_mesh(cubes, (0, 0, 0), (0.01, 0.012, 0.014), seed=7,
                            periodic=(periodic,) * 3)
    m = PicMethod(Discretization(mesh, order), U, depositor, MonomialParticlePusher(), 3, 3)
    m.depositor.set_shape_function(None, PolynomialShapeFunction(radius, 3, alpha))
    rng = np.random.default_rng(n)
    x = rng.uniform(0.001, 0.999, (n, 3)) * np.array([0.01, 0.012, 0.014])
    p = U.EL_MASS * U.VACUUM_LIGHT_SPEED() * rng.normal(0, 1, (n, 3))
    s = m.make_state()
    m.add_particles_from_arrays(s, x, p, rng.uniform(0.5, 1.5, n) * U.EL_CHARGE,
                                np.full(n, U.EL_MASS))
    return m, s


def shape(m, s, radius, alpha, periodic):
    """S [nodes, particles] and whether the pair is within the radius."""
    nodes = torch.as_tensor(np.ascontiguousarray(m.discretization.nodes), device="cuda")
    r2 = torch.zeros((len(nodes), len(s)), dtype=F64, device="cuda")
    for d, ext in enumerate((0.01, 0.012, 0.014)):
        diff = nodes[:, d, None] - s.x[d][None]
        if periodic:
            diff = diff - ext * torch.round(diff / ext)
        r2 += diff * diff
    t = torch.clamp(radius - r2 / radius, min=0)
    return m.depositor.shape_function.normalizer * t ** alpha, r2 <= radius * radius


MESHES = [((1, 1, 2), 1), ((3, 3, 3), 2), ((9, 9, 9), 3)]


@pytest.mark.parametrize("cubes,order", MESHES)
@pytest.mark.parametrize("n", [1, 127, 1000])
@pytest.mark.parametrize("periodic,radius,alpha", [(False, 0.003, 2), (True, 0.00499, 2),
                                                   (False, 0.02, 2), (True, 0.002, 3)])
def test_plain(cubes, order, n, periodic, radius, alpha):
    if periodic and cubes[0] == 1:
        cubes = (2, 2, 2)
    m, s = setup(ShapeFunctionDepositor(), cubes, order, n, periodic, radius, alpha)
    S, _ = shape(m, s, radius, alpha, periodic)
    v = m.velocities_device(s)
    rho, j = m.depositor.deposit_densities_device(s)
    m.check_status()
    # (a node that no particle reaches has exactly zero in both)
    assert bool((rho[S.sum(1) == 0] == 0).all())
    if float(S.max()) == 0:
        return
    assert rel(rho, S @ s.q) <= TOL
    assert rel(j, torch.stack([S @ (s.q * v[d]) for d in range(3)])) <= TOL
    # one output alone
    r1, _ = m.depositor.deposit_densities_device(s, j=False)
    assert torch.equal(r1, rho)


@pytest.mark.parametrize("cubes,order", MESHES)
@pytest.mark.parametrize("n", [1, 127, 1000])
@pytest.mark.parametrize("periodic,radius", [(False, 0.012), (True, 0.00499)])
def test_normalized(cubes, order, n, periodic, radius):
    if periodic and cubes[0] == 1:
        cubes = (2, 2, 2)
    m, s = setup(NormalizedShapeFunctionDepositor(), cubes, order, n, periodic, radius, 2)
    S, within = shape(m, s, radius, 2, periodic)
    mesh = m.discretization.mesh
    w = torch.as_tensor(np.outer(mesh.jacobians, m.depositor.integral_weights).ravel(),
                        device="cuda")
    scale = s.q / (w @ S)
    nn = len(m.discretization)
    rho = torch.empty((nn,), dtype=F64, device="cuda")
    j = torch.empty((3, nn), dtype=F64, device="cuda")
    v = m.velocities_device(s)
    stats = _lib.DepositStats()
    _lib.check(m.lib.prt_deposit_shape(
        m.mesh_data.handle, m.workspace, _lib.DEPOSIT_NORMALIZED, m.depositor._shape_desc(),
        _lib.ptr(m.depositor.integral_weights), n, s.x.data_ptr(), s.q.data_ptr(), v.data_ptr(),
        s.el.data_ptr(), rho.data_ptr(), j.data_ptr(), 0, C.byref(stats), C.c_void_p(0)))
    m.check_status()
    assert rel(rho, S @ scale) <= TOL
    assert rel(j, torch.stack([S @ (scale * v[d]) for d in range(3)])) <= TOL
    assert stats.norm_count == n and stats.el_count == n
    assert stats.norm_sum == pytest.approx(float(scale.sum()), rel=TOL)
    assert stats.node_pair_count == float(within.sum())
    # per particle the positions within the radius: the same pairs in both passes
    assert stats.pair_count == stats.el_sum <= stats.node_pair_count <= within.shape[0] * n


@pytest.mark.parametrize("n", [1, 130, 19001])
@pytest.mark.parametrize("periodic,radius,alpha", [(False, 0.004, 2), (True, 0.003, 2),
                                                   (False, 0.004, 3)])
@pytest.mark.parametrize("ordered", [False, True])
def test_average_forces(n, periodic, radius, alpha, ordered):
    m, s = setup(ShapeFunctionDepositor(), (5, 5, 5), 2, n, periodic, radius, alpha)
    s.el[::9] = -1  # removed particles: forces stay as they were
    if ordered:
        m.sort_by_element(s)
    S, _ = shape(m, s, radius, alpha, periodic)
    mesh = m.discretization.mesh
    iw = np.ascontiguousarray(
        m.discretization.element_groups[0].local_discretization.mass_matrix().sum(axis=1))
    w = torch.as_tensor(np.outer(mesh.jacobians, iw).ravel(), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(n)
    F = torch.randn((6, len(w)), generator=g, dtype=F64, device="cuda")
    v = m.velocities_device(s)
    out = torch.full((3, n), 7.0, dtype=F64, device="cuda")
    vis = torch.full((14, n), 7.0, dtype=F64, device="cuda")
    ptrs = (C.c_void_p * 6)(*[F[k].data_ptr() for k in range(6)])
    live = s.el != -1
    den = (w @ S)[live]
    avg = torch.stack([(w * F[k]) @ S for k in range(6)])[:, live] / den
    want = s.q[live] * (avg[:3] + torch.linalg.cross(v[:, live].T, avg[3:].T).T)
    for k in range(2):
        _lib.check(m.lib.prt_average_forces_ordered(
            m.mesh_data.handle, m.workspace, m.depositor._shape_desc(), _lib.ptr(iw), n,
            s.x.data_ptr(), s.q.data_ptr(), v.data_ptr(), s.el.data_ptr(), ptrs, out.data_ptr(),
            vis.data_ptr() if k else None, None, int(ordered), C.c_void_p(0)))
        if int(live.sum()):
            # (order 2 has negative weights: the denominators cancel up to ~100x)
            assert rel(out[:, live], want) <= 100 * TOL
        assert bool((out[:, ~live] == 7.0).all())
    if int(live.sum()):
        assert rel(vis[:6, live], avg) <= 100 * TOL
        sq = torch.stack([(w * (F[3 * k:3 * k + 3] ** 2).sum(0)) @ S for k in range(2)])[:, live]
        var = sq / den - torch.stack([(avg[:3] ** 2).sum(0), (avg[3:] ** 2).sum(0)])
        big = var > 1e-3 * sq.abs() / den.abs()
        assert torch.allclose(vis[6:8, live][big] ** 2, var[big], rtol=1e-8, atol=0)


@pytest.mark.parametrize("n", [1, 130, 19001])
@pytest.mark.parametrize("periodic,radius,alpha", [(False, 0.004, 2), (True, 0.003, 2),
                                                   (False, 0.004, 3)])
def test_deposit_adjoint(n, periodic, radius, alpha):
    m, s = setup(ShapeFunctionDepositor(), (5, 5, 5), 2, n, periodic, radius, alpha)
    nn = len(m.discretization)
    g = torch.Generator(device="cuda").manual_seed(n)
    grho = torch.randn(nn, generator=g, dtype=F64, device="cuda")
    gj = torch.randn((3, nn), generator=g, dtype=F64, device="cuda") / U.VACUUM_LIGHT_SPEED()
    v = m.velocities_device(s)
    lx = torch.zeros_like(s.x)
    lv = torch.zeros_like(s.x)
    _lib.check(m.lib.prt_deposit_shape_adjoint(
        m.mesh_data.handle, m.workspace, m.depositor._shape_desc(), n, s.x.data_ptr(),
        s.q.data_ptr(), v.data_ptr(), s.el.data_ptr(), grho.data_ptr(), gj.data_ptr(),
        lx.data_ptr(), lv.data_ptr(), C.c_void_p(0)))
    nodes = torch.as_tensor(np.ascontiguousarray(m.discretization.nodes), device="cuda")
    norm = m.depositor.shape_function.normalizer
    h = grho[:, None] + gj.T @ v  # [nodes, particles]
    wx = torch.zeros_like(lx)
    r2 = torch.zeros((nn, n), dtype=F64, device="cuda")
    diffs = []
    for d, ext in enumerate((0.01, 0.012, 0.014)):
        diff = nodes[:, d, None] - s.x[d][None]
        if periodic:
            diff = diff - ext * torch.round(diff / ext)
        diffs.append(diff)
        r2 += diff * diff
    t = torch.clamp(radius - r2 / radius, min=0)
    ds = s.q * norm * alpha * t ** (alpha - 1) * (2 / radius) * h
    for d in range(3):
        wx[d] = (ds * diffs[d]).sum(0)
    wv = s.q * norm * torch.stack([gj[d] @ t ** alpha for d in range(3)])
    assert rel(lx, wx) <= TOL
    assert rel(lv, wv) <= TOL
