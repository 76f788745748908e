"""FP64 depositions with a particle whose charge or velocity is not finite: it
spoils the points within its radius and no others, whatever else is in its
block of tiles. Against brute-force sums over the periodic images."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import _lib, meshgen  # noqa: E402
from pyrticle_b200.cloud import PicMethod  # noqa: E402
from pyrticle_b200.deposition.shape import ShapeFunctionDepositor  # noqa: E402
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.pusher import MonomialParticlePusher  # noqa: E402
from pyrticle_b200.tools import PolynomialShapeFunction  # noqa: E402
from pyrticle_b200.units import SIUnitsWithNaturalConstants as U  # noqa: E402

pytestmark = pytest.mark.gpu

F64 = torch.float64
PERIOD = 0.01


def _method(radius, alpha):
    mesh = meshgen.box_mesh((3, 3, 3), (0, 0, 0), (PERIOD,) * 3, seed=7,
                            periodic=(True, True, True))
    m = PicMethod(Discretization(mesh, 2), U, ShapeFunctionDepositor(),
                  MonomialParticlePusher(), 3, 3)
    m.depositor.set_shape_function(None, PolynomialShapeFunction(radius, 3, alpha))
    return m


def _check(m, pts, radius, alpha, x, q, v, bad, rho, j):
    """rho and j at the points against brute force: without the bad particles
    where none is within the radius, not finite in what they spoil elsewhere."""
    r2 = torch.zeros((len(pts), x.shape[1]), dtype=F64, device="cuda")
    for a in range(3):
        d = pts[:, a, None] - x[a][None]
        d = d - PERIOD * torch.round(d / PERIOD)
        r2 += d * d
    s = m.depositor.shape_function.normalizer * torch.clamp(radius - r2 / radius, min=0) ** alpha
    good = torch.ones(x.shape[1], dtype=torch.bool, device="cuda")
    good[bad] = False
    near = (r2[:, bad] < (radius * (1 - 1e-9)) ** 2).any(dim=1)
    far = (r2[:, bad] > (radius * (1 + 1e-9)) ** 2).all(dim=1)
    assert int(near.sum()) >= 1 and int(far.sum()) >= len(pts) // 2
    w = q[good]
    want = [s[:, good] @ w] + [s[:, good] @ (w * v[a, good]) for a in range(3)]
    for got, ref in zip([rho, j[0], j[1], j[2]], want):
        assert bool(torch.isfinite(got[far]).all())
        assert float((got - ref)[far].abs().max() / ref.abs().max()) <= 1e-12
    assert not bool(torch.isfinite(j[:, near]).any())


@pytest.mark.parametrize("alpha", [2, 3])
@pytest.mark.parametrize("spoilt", ["charge", "velocity"])
@pytest.mark.parametrize("dims", [(12, 12, 12), (30, 28, 26)])  # one and four tiles a block
def test_grid(dims, spoilt, alpha):
    radius, n = 0.0012, 3000
    m = _method(radius, alpha)
    sw = [PERIOD / k for k in dims]
    d = _lib.GridDesc()
    brick = (_lib.Brick * 1)()
    for a in range(3):
        brick[0].stepwidths[a], brick[0].dims[a] = sw[a], dims[a]
    d.brick_count = 1
    d.nodes_per_element = m.discretization.nodes_per_element
    d.bricks = C.cast(brick, C.POINTER(_lib.Brick))
    grid = C.c_void_p()
    _lib.check(m.lib.prt_grid_create(m.mesh_data.handle, C.byref(d), C.byref(grid)))
    rng = np.random.default_rng(dims[0])
    x = torch.as_tensor(rng.uniform(0, PERIOD, (3, n)), device="cuda")
    q = torch.as_tensor(rng.uniform(0.5, 1.5, n), device="cuda")
    v = torch.as_tensor(rng.uniform(0.5, 1.5, (3, n)), device="cuda")
    bad = [17]
    if spoilt == "charge":
        q[17] = float("inf")
    else:
        v[:, 17] = float("nan")
    count = int(np.prod(dims))
    rho = torch.empty((count,), dtype=F64, device="cuda")
    j = torch.empty((3, count), dtype=F64, device="cuda")
    _lib.check(m.lib.prt_deposit_grid(
        grid, m.workspace, _lib.GRID_SHAPE, m.depositor._shape_desc(), n, x.data_ptr(),
        q.data_ptr(), v.data_ptr(), None, rho.data_ptr(), j.data_ptr(), C.c_void_p(0)))
    m.check_status()
    idx = np.stack(np.meshgrid(*[np.arange(k) for k in dims], indexing="ij"), -1)
    idx = idx.transpose(2, 1, 0, 3).reshape(-1, 3)  # x fastest
    pts = torch.as_tensor((idx + 0.5) * np.array(sw), device="cuda")
    _check(m, pts, radius, alpha, x, q, v, bad, rho, j)
    m.lib.prt_grid_destroy(grid)


def test_mesh():
    radius, n = 0.0015, 2000
    m = _method(radius, 2)
    rng = np.random.default_rng(3)
    x = torch.as_tensor(rng.uniform(0, PERIOD, (3, n)), device="cuda")
    q = torch.as_tensor(rng.uniform(0.5, 1.5, n), device="cuda")
    v = torch.as_tensor(rng.uniform(0.5, 1.5, (3, n)), device="cuda")
    v[:, 5] = float("inf")
    nn = len(m.discretization)
    rho = torch.empty((nn,), dtype=F64, device="cuda")
    j = torch.empty((3, nn), dtype=F64, device="cuda")
    _lib.check(m.lib.prt_deposit_shape(
        m.mesh_data.handle, m.workspace, _lib.DEPOSIT_PLAIN, m.depositor._shape_desc(), None, n,
        x.data_ptr(), q.data_ptr(), v.data_ptr(), None, rho.data_ptr(), j.data_ptr(), 0, None,
        C.c_void_p(0)))
    m.check_status()
    pts = torch.as_tensor(np.asarray(m.discretization.nodes).reshape(-1, 3), device="cuda")
    _check(m, pts, radius, 2, x, q, v, [5], rho, j)
