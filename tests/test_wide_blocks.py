"""The FP64 pair sums where the points of a block lie thousands of shape radii
apart (few particles in a long beam line, a mesh that is coarse against the
radius): a particle near every node of a thin box 5,000 radii long, whose nodes
are several radii apart, so that every particle has exactly one position within
the radius."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import _lib, meshgen  # noqa: E402
from pyrticle_b200.cloud import PicMethod  # noqa: E402
from pyrticle_b200.deposition.shape import NormalizedShapeFunctionDepositor  # noqa: E402
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.pusher import MonomialParticlePusher  # noqa: E402
from pyrticle_b200.tools import PolynomialShapeFunction  # noqa: E402
from pyrticle_b200.units import SIUnitsWithNaturalConstants as U  # noqa: E402

pytestmark = pytest.mark.gpu

F64 = torch.float64
RADIUS = 9.9998e-6
BOX = (1e-4, 1.2e-4, 0.47)


def setup(n, lo, hi, alpha=2, seed=0):
    """The method, and n particles at lo to hi radii from nodes of their own:
    positions x [3, n]. Displaced along the box, so that those at the ends of
    a block are out of its box by just that."""
    mesh = meshgen.box_mesh((1, 1, 64), (0, 0, 0), BOX, seed=7)
    m = PicMethod(Discretization(mesh, 2), U, NormalizedShapeFunctionDepositor(),
                  MonomialParticlePusher(), 3, 3)
    m.depositor.set_shape_function(None, PolynomialShapeFunction(RADIUS, 3, alpha))
    nodes = np.ascontiguousarray(m.discretization.nodes)
    # the nodes at one position, an ulp apart (5e-12 radii here), count as the
    # first of them, as in the library
    _, first, which = np.unique(np.round(nodes / 1e-9).astype(np.int64), axis=0,
                                return_index=True, return_inverse=True)
    nodes = nodes[first][which.ravel()]
    rng = np.random.default_rng(seed)
    pick = np.sort(rng.permutation(first)[:n])
    away = np.zeros((len(pick), 3))
    away[:, 2] = rng.uniform(lo, hi, len(pick)) * RADIUS * rng.choice([-1, 1], len(pick))
    x = torch.as_tensor((nodes[pick] + away).T.copy(), device="cuda")
    return m, torch.as_tensor(nodes, device="cuda"), x


def pairs(m, nodes, x):
    """x_u - x_p and r^2 of all (node, particle) pairs, by differences."""
    d = nodes.T[:, :, None] - x[:, None, :]
    return d, (d * d).sum(0)


def deposit(m, mode, x, q, stats=None):
    rho = torch.empty((len(m.discretization),), dtype=F64, device="cuda")
    _lib.check(m.lib.prt_deposit_shape(
        m.mesh_data.handle, m.workspace, mode, m.depositor._shape_desc(),
        _lib.ptr(m.depositor.integral_weights), x.shape[1], x.data_ptr(), q.data_ptr(), None,
        None, rho.data_ptr(), None, 0, C.byref(stats) if stats else None, C.c_void_p(0)))
    m.check_status()
    return rho


def test_deposited_pairs_near_the_rim_count():
    """At 0.99999 to 0.999999 radii a - r^2/a is at least 2e-6 a, beyond the
    rounding of the form (H^2 2^-53 a = 1e-9 a for a block of half extent H =
    2,700 radii), which is 2 x 1e-9 / 2e-6 of the weight."""
    m, nodes, x = setup(10_000, 0.99999, 0.999999)
    q = torch.ones(x.shape[1], dtype=F64, device="cuda")
    _, r2 = pairs(m, nodes, x)
    t = torch.clamp(RADIUS - r2 / RADIUS, min=0)
    want = m.depositor.shape_function.normalizer * (t * t).sum(1)
    assert bool((want > 0).all())
    rho = deposit(m, _lib.DEPOSIT_PLAIN, x, q)
    assert float(((rho - want) / want).abs().max()) <= 1e-2


def average(m, x, fields, ordered):
    """The forces on unit charges at rest, [3, n]."""
    n = x.shape[1]
    q = torch.ones(n, dtype=F64, device="cuda")
    v = torch.zeros_like(x)
    out = torch.full_like(x, 7.0)
    ptrs = (C.c_void_p * 6)(*[fields[k].data_ptr() for k in range(6)])
    _lib.check(m.lib.prt_average_forces_ordered(
        m.mesh_data.handle, m.workspace, m.depositor._shape_desc(),
        _lib.ptr(m.depositor.integral_weights), n, x.data_ptr(), q.data_ptr(), v.data_ptr(), None,
        ptrs, out.data_ptr(), None, None, ordered, C.c_void_p(0)))
    return out


def test_averaged_pairs_near_the_rim_count():
    """32 particles at each of 600 nodes, a warp's worth, in a store without a
    spatial order that is taken in its own: blocks as long as the box. With one
    position within the radius the average is the field there."""
    m, nodes, x = setup(600, 0.99999, 0.999999)
    perm = torch.as_tensor(np.random.default_rng(5).permutation(600), device="cuda")
    x = x[:, perm].repeat_interleave(32, 1).contiguous()
    # E_x = 1 at every node: no position left out, whatever its weight's rounding
    fields = torch.zeros((6, len(nodes)), dtype=F64, device="cuda")
    fields[0] = 1
    out = average(m, x, fields, 1)
    assert float((out[0] - 1).abs().max()) <= 1e-14
    assert bool((out[1:] == 0).all())


@pytest.mark.parametrize("alpha", [2, 3])
@pytest.mark.parametrize("n,copies", [(33, 1), (600, 1), (600, 32)])
def test_rounding_does_not_depend_on_the_block(n, copies, alpha):
    """Particles as targets (normalising integral, average, deposition adjoint)
    at up to half a radius from their node: by differences the weight is off
    by some ten roundings (2^-53 each; a power a few more), 4e-15, in blocks a
    thousand radii long and more. A sum about the block's centre would be off by
    1e-10 there."""
    tol = 4e-15
    m, nodes, x = setup(n, 0.1, 0.5, alpha)
    rng = np.random.default_rng(2)
    perm = torch.as_tensor(rng.permutation(n), device="cuda")
    x = x[:, perm].repeat_interleave(copies, 1).contiguous()
    n = x.shape[1]
    x[0] += 1e-7 * torch.as_tensor(rng.uniform(-1, 1, n), device="cuda")
    q = torch.ones(n, dtype=F64, device="cuda")
    mesh, sf = m.discretization.mesh, m.depositor.shape_function
    w = torch.as_tensor(np.outer(mesh.jacobians, m.depositor.integral_weights).ravel(),
                        device="cuda")
    G = torch.as_tensor(rng.normal(size=len(nodes)), device="cuda")
    # the node adjoints of a position are summed first, in ascending order, as in
    # the library (they may cancel)
    pos, which = np.unique(nodes.cpu().numpy(), axis=0, return_inverse=True)
    at_pos = np.zeros(len(pos))
    np.add.at(at_pos, which.ravel(), G.cpu().numpy())
    pos, at_pos = (torch.as_tensor(a, device="cuda") for a in (pos, at_pos))
    integral = torch.zeros(n, dtype=F64, device="cuda")
    lx_want = torch.zeros((3, n), dtype=F64, device="cuda")
    for c in range(0, n, 2000):
        d, r2 = pairs(m, nodes, x[:, c:c + 2000])
        t = torch.clamp(RADIUS - r2 / RADIUS, min=0)
        integral[c:c + 2000] = w @ (sf.normalizer * t ** alpha)
        d, r2 = pairs(m, pos, x[:, c:c + 2000])
        t = torch.clamp(RADIUS - r2 / RADIUS, min=0)
        lx_want[:, c:c + 2000] = torch.stack(
            [at_pos @ (sf.normalizer * alpha * (2 / RADIUS) * t ** (alpha - 1) * d[k])
             for k in range(3)])
    stats = _lib.DepositStats()
    deposit(m, _lib.DEPOSIT_NORMALIZED, x, q, stats)
    scale = 1 / integral
    assert stats.norm_count == n
    assert abs(stats.norm_sum - float(scale.sum())) <= tol * float(scale.abs().sum())
    assert abs(stats.norm_max / float(scale.max()) - 1) <= 4 * tol
    fields = torch.zeros((6, len(nodes)), dtype=F64, device="cuda")
    for ordered in (0, 1):
        out, sc = torch.zeros_like(x), torch.zeros_like(q)
        ptrs = (C.c_void_p * 6)(*[fields[k].data_ptr() for k in range(6)])
        _lib.check(m.lib.prt_average_forces_ordered(
            m.mesh_data.handle, m.workspace, m.depositor._shape_desc(),
            _lib.ptr(m.depositor.integral_weights), n, x.data_ptr(), q.data_ptr(),
            out.data_ptr(), None, ptrs, out.data_ptr(), None, sc.data_ptr(), ordered,
            C.c_void_p(0)))
        assert float((sc / scale - 1).abs().max()) <= 4 * tol
    lx = torch.zeros_like(x)
    _lib.check(m.lib.prt_deposit_shape_adjoint(
        m.mesh_data.handle, m.workspace, m.depositor._shape_desc(), n, x.data_ptr(),
        q.data_ptr(), None, None, G.data_ptr(), None, lx.data_ptr(), None, C.c_void_p(0)))
    err = torch.linalg.norm(lx - lx_want, dim=0) / torch.linalg.norm(lx_want, dim=0)
    assert float(err.max()) <= 4 * tol


@pytest.mark.parametrize("where", [np.inf, -np.inf, np.nan, 1e30, 5.0])
@pytest.mark.parametrize("copies", [1, 600])
def test_a_particle_out_of_reach_takes_nothing_from_its_block(where, copies):
    """Every fifth particle is far outside of the mesh, or at no finite place:
    it has no position within the radius, and the others, with one each, have
    their values to the last bit."""
    m, nodes, good = setup(33, 0.1, 0.5)
    good = good.repeat(1, copies)
    n = good.shape[1] * 5 // 4
    x = torch.empty((3, n), dtype=F64, device="cuda")
    live = torch.arange(n, device="cuda") % 5 != 4
    x[:, live] = good[:, :int(live.sum())]
    x[:, ~live] = torch.tensor([5e-5, where, 0.2], dtype=F64, device="cuda")[:, None]
    rng = np.random.default_rng(1)
    G = torch.as_tensor(rng.normal(size=len(nodes)), device="cuda")
    fields = torch.as_tensor(rng.normal(size=(6, len(nodes))), device="cuda")

    def results(x, ordered):
        n = x.shape[1]
        q = torch.ones(n, dtype=F64, device="cuda")
        lx, f, sc = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(q)
        v = torch.zeros_like(x)
        ptrs = (C.c_void_p * 6)(*[fields[k].data_ptr() for k in range(6)])
        _lib.check(m.lib.prt_average_forces_ordered(
            m.mesh_data.handle, m.workspace, m.depositor._shape_desc(),
            _lib.ptr(m.depositor.integral_weights), n, x.data_ptr(), q.data_ptr(), v.data_ptr(),
            None, ptrs, f.data_ptr(), None, sc.data_ptr(), ordered, C.c_void_p(0)))
        _lib.check(m.lib.prt_deposit_shape_adjoint(
            m.mesh_data.handle, m.workspace, m.depositor._shape_desc(), n, x.data_ptr(),
            q.data_ptr(), None, None, G.data_ptr(), None, lx.data_ptr(), None, C.c_void_p(0)))
        stats = _lib.DepositStats()
        rho = deposit(m, _lib.DEPOSIT_NORMALIZED, x, q, stats)
        return lx, f, sc, rho, stats

    for ordered in (0, 1):
        want = results(x[:, live].contiguous(), ordered)
        with pytest.warns(UserWarning):  # zero mass, no average
            got = results(x, ordered)
        for a, b in zip(got[:3], want[:3]):
            assert torch.equal(a[..., live], b)
            assert bool((a[..., ~live] == 0).all())
        for name in ("norm_count", "norm_min", "norm_max", "el_sum"):
            assert getattr(got[4], name) == getattr(want[4], name)
        assert float((got[3] - want[3]).abs().max()) <= 1e-14 * float(want[3].abs().max())


@pytest.mark.parametrize("call", ["average", "adjoint"])
def test_scratch_does_not_grow_with_the_bins(call):
    """The order of the particles needs no array over the bins, a billion here
    (a radius of a six-hundredth of the box)."""
    mesh = meshgen.box_mesh((2, 2, 2), (0, 0, 0), (0.01, 0.012, 0.014), seed=7)
    m = PicMethod(Discretization(mesh, 2), U, NormalizedShapeFunctionDepositor(),
                  MonomialParticlePusher(), 3, 3)
    m.depositor.set_shape_function(None, PolynomialShapeFunction(2e-5, 3, 2))
    x = torch.full((3, 100), 0.005, dtype=F64, device="cuda")
    q = torch.ones(100, dtype=F64, device="cuda")
    G = torch.ones(len(m.discretization), dtype=F64, device="cuda")
    fields = torch.zeros((6, len(G)), dtype=F64, device="cuda")
    lx = torch.zeros_like(x)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    if call == "average":
        average(m, x, fields, 0)
    else:
        _lib.check(m.lib.prt_deposit_shape_adjoint(
            m.mesh_data.handle, m.workspace, m.depositor._shape_desc(), 100, x.data_ptr(),
            q.data_ptr(), None, None, G.data_ptr(), None, lx.data_ptr(), None, C.c_void_p(0)))
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 1 << 28
