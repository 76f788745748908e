"""Whole RK steps in one launch (prt_lsrk_steps) against the stage-by-stage
launches (prt_lsrk_stage): from nodal fields, from FP64 and from FP32
per-element coefficients, with the tape, over store sizes around a warp and a
block, on a z-periodic mesh that some particles leave through the sides."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import _lib, meshgen  # noqa: E402
from pyrticle_b200.cloud import LSRK4_A, LSRK4_B, PicMethod  # noqa: E402
from pyrticle_b200.deposition.shape import ShapeFunctionDepositor  # noqa: E402
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.pusher import MonomialParticlePusher  # noqa: E402
from pyrticle_b200.units import SIUnitsWithNaturalConstants as U  # noqa: E402

pytestmark = pytest.mark.gpu

F64 = torch.float64
STAGES = 10
DT = 2e-13  # up to 6e-5 m a step: a fifth of the smallest cube edge


def setup(order, n):
    mesh = meshgen.box_mesh((3, 3, 6), (0, 0, 0), (0.001, 0.001, 0.002), seed=4,
                            periodic=(False, False, True))
    m = PicMethod(Discretization(mesh, order), U, ShapeFunctionDepositor(),
                  MonomialParticlePusher(), 3, 3)
    rng = np.random.default_rng(100 * order + n)
    x = rng.uniform(2e-5, 0.98e-3, (n, 3)) * np.array([1.0, 1.0, 2.0])
    mc = U.EL_MASS * U.VACUUM_LIGHT_SPEED()
    p = mc * rng.normal(0, 1.0, (n, 3))
    p[::5] = 0  # at rest: located in place
    s = m.make_state()
    m.add_particles_from_arrays(s, x, p, np.full(n, -U.EL_CHARGE), np.full(n, U.EL_MASS))
    m.sort_by_element(s)
    s.el[::7] = -1  # removed particles stay untouched
    nodes = np.asarray(m.discretization.nodes)
    k = 2 * np.pi / 0.001
    f = np.stack([1e9 * np.cos(k * nodes[:, 0] + i) + 1e8 for i in range(6)])
    f[3:] /= U.VACUUM_LIGHT_SPEED()
    return m, s, torch.as_tensor(f, device="cuda")


def store(s):
    kx = torch.full_like(s.x, 3.0)
    return [s.x.clone(), s.p.clone(), s.el.clone(), kx, torch.full_like(s.p, 5.0)]


def stage_by_stage(m, s, fptrs):
    x, p, el, kx, kp = store(s)
    for t in range(STAGES):
        _lib.check(m.lib.prt_lsrk_stage(
            m.pusher.handle, m.workspace, len(s), x.data_ptr(), p.data_ptr(), s.q.data_ptr(),
            s.m.data_ptr(), el.data_ptr(), kx.data_ptr(), kp.data_ptr(), fptrs, LSRK4_A[t % 5],
            LSRK4_B[t % 5], DT, U.VACUUM_LIGHT_SPEED(), 0, C.c_void_p(0)))
    return x, p, el, kx, kp


def fused(m, s, fptrs, coef, precision=0, tape=None):
    x, p, el, kx, kp = store(s)
    _lib.check(m.lib.prt_lsrk_steps(
        m.pusher.handle, m.workspace, len(s), x.data_ptr(), p.data_ptr(), s.q.data_ptr(),
        s.m.data_ptr(), el.data_ptr(), kx.data_ptr(), kp.data_ptr(),
        None if coef is None else coef.data_ptr(), fptrs, precision, (C.c_double * 5)(*LSRK4_A),
        (C.c_double * 5)(*LSRK4_B), 5, STAGES, DT, U.VACUUM_LIGHT_SPEED(),
        *([None] * 3 if tape is None else [t.data_ptr() for t in tape]), C.c_void_p(0)))
    return x, p, el, kx, kp


def rel(a, b):
    return float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) if float(b.abs().max()) else 0.0


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 33, 129, 19001])
def test_fused_steps_equal_the_stages(order, n):
    m, s, f = setup(order, n)
    fptrs = m.pusher.field_pointers(f)
    want = stage_by_stage(m, s, fptrs)
    m.check_status()
    m.transfer_find_counters()
    counts = []
    for coef in (None, m.pusher.field_coefficients(fptrs)):
        got = fused(m, s, fptrs, coef)
        m.check_status()
        ctr = m.transfer_find_counters()
        counts.append([ctr.find_same, ctr.find_by_neighbor, ctr.find_by_vertex, ctr.find_global])
        assert torch.equal(got[2], want[2])
        # the parity bound of the FP64 stage
        for a, b in zip((got[0], got[1], got[3], got[4]), (want[0], want[1], want[3], want[4])):
            assert rel(a, b) <= 1e-12
        # the tape's slots are the states after every stage, and it changes nothing
        nn = len(s)
        tape = (torch.full((STAGES + 1, 3, nn), 7.0, dtype=F64, device="cuda"),
                torch.full((STAGES + 1, 3, nn), 7.0, dtype=F64, device="cuda"),
                torch.full((STAGES + 1, nn), 7, dtype=torch.int32, device="cuda"))
        taped = fused(m, s, fptrs, coef, tape=tape)
        m.transfer_find_counters()
        for a, b in zip(taped, got):
            assert torch.equal(a, b)
        for t, a in zip(tape, (got[0], got[1], got[2])):
            assert torch.equal(t[STAGES], a)
            assert bool((t[0] == 7).all())
    assert counts[0] == counts[1]


@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_fused_mixed_steps(order):
    m, s, f = setup(order, 5000)
    fptrs = m.pusher.field_pointers(f)
    want = fused(m, s, fptrs, m.pusher.field_coefficients(fptrs))
    got = fused(m, s, fptrs, m.pusher.field_coefficients(fptrs, 1), precision=1)
    assert torch.equal(got[2], want[2])
    # FP32 fields: within the mixed form's 1e-5 in the momentum changes
    assert rel(got[1] - s.p, want[1] - s.p) <= 1e-5
