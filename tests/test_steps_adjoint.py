"""The adjoint of a taped run of stages in one launch (prt_lsrk_steps_adjoint)
against the adjoint stage by stage, and with a basis field that is infinite
somewhere."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import _lib, meshgen  # noqa: E402
from pyrticle_b200.adjoint import _ptrs, monomial_coefficients  # noqa: E402
from pyrticle_b200.cloud import _RK_A, _RK_B, LSRK4_A, LSRK4_B, PicMethod  # noqa: E402
from pyrticle_b200.deposition.shape import ShapeFunctionDepositor  # noqa: E402
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.pusher import MonomialParticlePusher  # noqa: E402
from pyrticle_b200.tools import PolynomialShapeFunction  # noqa: E402
from pyrticle_b200.units import SIUnitsWithNaturalConstants as U  # noqa: E402

pytestmark = pytest.mark.gpu

F64 = torch.float64
STAGES = 10
DT = 2e-13


class Tape:
    """Ten taped stages of 300 electrons, a few of them removed, in a smooth
    field without E_y; adjoints of the end and two basis fields."""

    def __init__(self, order, n=300):
        mesh = meshgen.box_mesh((3, 3, 3), (0, 0, 0), (0.01,) * 3, seed=7, periodic=(True,) * 3)
        self.m = m = PicMethod(Discretization(mesh, order), U, ShapeFunctionDepositor(),
                               MonomialParticlePusher(), 3, 3)
        m.depositor.set_shape_function(None, PolynomialShapeFunction(0.002, 3, 2))
        rng = np.random.default_rng(order)
        s = m.make_state()
        m.add_particles_from_arrays(
            s, rng.uniform(1e-4, 0.0099, (n, 3)),
            U.EL_MASS * U.VACUUM_LIGHT_SPEED() * rng.normal(0, 1, (n, 3)),
            np.full(n, -U.EL_CHARGE), np.full(n, U.EL_MASS))
        s.el[::11] = -1
        self.n, self.s = n, s
        nodes = np.ascontiguousarray(m.discretization.nodes)
        wave = np.cos(300 * nodes @ rng.normal(size=(3, 6)) + np.arange(6))
        wave *= np.array([1e6, 0, 1e6, 0.1, 0.2, 0.3])
        self.F = torch.as_tensor(wave.T.copy(), device="cuda")
        self.comps = [self.F[k] if k != 1 else None for k in range(6)]
        self.coef = m.pusher.field_coefficients(_ptrs(self.comps))
        self.tx, self.tp = (torch.empty((STAGES + 1, 3, n), dtype=F64, device="cuda")
                            for _ in range(2))
        self.te = torch.empty((STAGES + 1, n), dtype=torch.int32, device="cuda")
        self.tx[0], self.tp[0], self.te[0] = s.x, s.p, s.el
        kx, kp = torch.zeros_like(s.x), torch.zeros_like(s.p)
        _lib.check(m.lib.prt_lsrk_steps(
            m.pusher.handle, m.workspace, n, self.tx.data_ptr(), self.tp.data_ptr(),
            s.q.data_ptr(), s.m.data_ptr(), self.te.data_ptr(), kx.data_ptr(), kp.data_ptr(),
            self.coef.data_ptr(), None, 0, _RK_A, _RK_B, 5, STAGES, DT, m.units.
            VACUUM_LIGHT_SPEED(), self.tx.data_ptr(), self.tp.data_ptr(), self.te.data_ptr(),
            C.c_void_p(0)))
        m.check_status()
        g = torch.Generator(device="cuda").manual_seed(order)
        # adjoints of positions and momenta of comparable effect
        scale = (1.0, 1 / (U.EL_MASS * U.VACUUM_LIGHT_SPEED() * 100))
        self.lam = [torch.randn((3, n), generator=g, dtype=F64, device="cuda") * scale[k % 2]
                    for k in range(4)]
        self.basis = [torch.randn(len(nodes), generator=g, dtype=F64, device="cuda")
                      for _ in range(12)]
        self.basis[3] = self.basis[10] = None
        self.basis_coef = monomial_coefficients(m, self.basis)

    def fused(self, basis):
        m, s = self.m, self.s
        lam = [t.clone() for t in self.lam]
        grad = torch.zeros(2, dtype=F64, device="cuda")
        _lib.check(m.lib.prt_lsrk_steps_adjoint(
            m.pusher.handle, m.workspace, self.n, self.tx.data_ptr(), self.tp.data_ptr(),
            self.te.data_ptr(), s.q.data_ptr(), s.m.data_ptr(), *[t.data_ptr() for t in lam],
            self.coef.data_ptr(), 0b111101, _RK_A, _RK_B, 5, STAGES, DT,
            m.units.VACUUM_LIGHT_SPEED(), 2, _ptrs(basis), grad.data_ptr(), C.c_void_p(0)))
        return lam, grad

    def by_stage(self, basis):
        m, s = self.m, self.s
        lam = [t.clone() for t in self.lam]
        grad = torch.zeros(2, dtype=F64, device="cuda")
        coef = monomial_coefficients(m, self.comps)
        for t in reversed(range(STAGES)):
            _lib.check(m.lib.prt_lsrk_stage_adjoint(
                m.pusher.handle, m.workspace, self.n, self.tx[t].data_ptr(),
                self.tp[t].data_ptr(), self.te[t].data_ptr(), s.q.data_ptr(), s.m.data_ptr(),
                *[u.data_ptr() for u in lam], _ptrs(coef), LSRK4_A[t % 5], LSRK4_B[t % 5], DT,
                m.units.VACUUM_LIGHT_SPEED(), None, 2, _ptrs(basis), grad.data_ptr(),
                C.c_void_p(0)))
        return lam, grad


@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_equal_to_the_adjoint_by_stages(order):
    """To rounding: some hundred operations a stage and the coefficients' own
    contraction (1e-14 at order 4), ten stages: 1e-13, an order for
    cancellation."""
    T = Tape(order)
    lam, grad = T.fused(T.basis_coef)
    want, grad_want = T.by_stage(T.basis_coef)
    for a, b in zip(lam, want):
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) <= 1e-12
        # removed particles' adjoints pass through
        assert torch.equal(a[:, ::11], b[:, ::11])
    assert float(((grad - grad_want) / grad_want).abs().max()) <= 1e-12


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_an_infinite_basis_field_has_its_own_gradient_only(value):
    T = Tape(2)
    lam, grad = T.fused(T.basis_coef)
    bad = list(T.basis_coef)
    bad[2] = torch.full_like(bad[2], value)  # E_z of the first basis field
    lam2, grad2 = T.fused(bad)
    assert not np.isfinite(float(grad2[0]))
    assert float(grad2[1]) == float(grad[1])
    for a, b in zip(lam2, lam):
        assert torch.equal(a, b)
