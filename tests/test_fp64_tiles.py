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
