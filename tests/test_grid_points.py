"""Bricks that the grid depositor makes no use of itself but a caller of
prt_deposit_grid may: points several periods apart in one block of tiles,
numbers that two bricks share and numbers that none has. Against brute-force
sums over the periodic images."""

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
PERIOD, RADIUS = 0.01, 0.002


class Grid:
    """A periodic mesh, some particles and a grid of the given bricks:
    (start_index, stepwidths, origin, dims)."""

    def __init__(self, bricks, n=700):
        mesh = meshgen.box_mesh((3, 3, 3), (0, 0, 0), (PERIOD,) * 3, seed=7,
                                periodic=(True, True, True))
        self.m = m = PicMethod(Discretization(mesh, 2), U, ShapeFunctionDepositor(),
                               MonomialParticlePusher(), 3, 3)
        m.depositor.set_shape_function(None, PolynomialShapeFunction(RADIUS, 3, 2))
        self.bricks = bricks
        d = _lib.GridDesc()
        self.structs = (_lib.Brick * len(bricks))()
        for s, (start, sw, origin, dims) in zip(self.structs, bricks):
            s.start_index = start
            for a in range(3):
                s.stepwidths[a], s.origin[a], s.dims[a] = sw[a], origin[a], dims[a]
        d.brick_count = len(bricks)
        d.nodes_per_element = m.discretization.nodes_per_element
        d.bricks = C.cast(self.structs, C.POINTER(_lib.Brick))
        self.handle = C.c_void_p()
        _lib.check(m.lib.prt_grid_create(m.mesh_data.handle, C.byref(d), C.byref(self.handle)))
        self.count = max(b[0] + int(np.prod(b[3])) for b in bricks)
        rng = np.random.default_rng(n)
        self.x = torch.as_tensor(rng.uniform(0, PERIOD, (3, n)), device="cuda")
        self.q = torch.as_tensor(rng.uniform(0.5, 1.5, n), device="cuda")
        self.rho = torch.full((self.count,), 7.0, dtype=F64, device="cuda")

    def __del__(self):
        self.m.lib.prt_grid_destroy(self.handle)

    def deposit(self, stream=None):
        return self.m.lib.prt_deposit_grid(
            self.handle, self.m.workspace, _lib.GRID_SHAPE, self.m.depositor._shape_desc(),
            self.x.shape[1], self.x.data_ptr(), self.q.data_ptr(), None, None,
            self.rho.data_ptr(), None, C.c_void_p(stream or 0))

    def want(self):
        out = torch.zeros((self.count,), dtype=F64, device="cuda")
        for start, sw, origin, dims in self.bricks:
            idx = np.stack(np.meshgrid(*[np.arange(k) for k in dims], indexing="ij"), -1)
            idx = idx.transpose(2, 1, 0, 3).reshape(-1, 3)  # x fastest
            pt = torch.as_tensor(np.array(origin) + (idx + 0.5) * np.array(sw), device="cuda")
            r2 = torch.zeros((len(pt), self.x.shape[1]), dtype=F64, device="cuda")
            for a in range(3):
                diff = pt[:, a, None] - self.x[a][None]
                diff = diff - PERIOD * torch.round(diff / PERIOD)
                r2 += diff * diff
            t = torch.clamp(RADIUS - r2 / RADIUS, min=0)
            out[start:start + len(pt)] = self.m.depositor.shape_function.normalizer * (t * t @
                                                                                     self.q)
        return out


def test_points_several_periods_apart():
    """16 points 0.7 periods apart along x: a tile of 32 is 5 periods long. The
    expansion's rounding is (H/a)^2 2^-53 = 2e-14 of the largest value, H = 14 a."""
    g = Grid([(0, (0.007, 0.002, 0.002), (-0.02, 0.001, 0.001), (16, 2, 2))])
    _lib.check(g.deposit())
    g.m.check_status()
    want = g.want()
    assert bool((want > 0).all())
    assert float((g.rho - want).abs().max() / want.max()) <= 1e-12


def test_numbers_that_no_point_has_are_zero():
    """Two bricks with the same numbers (and points) and a gap of as many: there
    are as many points as numbers, and yet some numbers have none."""
    sw, dims = (0.001, 0.002, 0.003), (3, 4, 2)
    g = Grid([(0, sw, (0, 0, 0), dims), (0, sw, (0, 0, 0), dims),
              (48, sw, (0.005, 0, 0.001), dims)])
    _lib.check(g.deposit())
    g.m.check_status()
    want = g.want()
    assert bool((g.rho[24:48] == 0).all())
    assert float((g.rho - want).abs().max() / want.max()) <= 1e-13


def test_first_call_of_a_grid_under_capture():
    """A grid's tiles are made in its first FP64 deposition, which may be
    recorded into a CUDA graph as any other where the workspace is warm."""
    bricks = [(0, (0.001, 0.001, 0.001), (0, 0, 0), (10, 10, 10))]
    warm, g = Grid(bricks), Grid(bricks)
    _lib.check(warm.deposit())
    torch.cuda.synchronize()
    g.m.workspace, warm.m.workspace = warm.m.workspace, g.m.workspace
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rc = g.deposit(torch.cuda.current_stream().cuda_stream)
    assert rc == _lib.PRT_OK
    assert bool((g.rho == 7.0).all())  # recorded, not run
    graph.replay()
    torch.cuda.synchronize()
    want = g.want()
    assert float((g.rho - want).abs().max() / want.max()) <= 1e-13
    assert torch.equal(g.rho, warm.rho)
    del graph
