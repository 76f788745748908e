"""The averaging pusher takes the particles in a compact order whatever the
store's: its sums in a store that was sorted once and has moved on, wrapped and
been advanced since are, bit for bit, those of the spatially binned pass."""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import _lib, meshgen  # noqa: E402
from pyrticle_b200.cloud import PicMethod  # noqa: E402
from pyrticle_b200.deposition.shape import ShapeFunctionDepositor  # noqa: E402
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.pusher import AverageParticlePusher  # noqa: E402
from pyrticle_b200.tools import PolynomialShapeFunction  # noqa: E402
from pyrticle_b200.units import SIUnitsWithNaturalConstants as U  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [500, 30_000])
def test_order_of_a_store_that_moved_on(n):
    mesh = meshgen.box_mesh((3, 3, 6), (0, 0, 0), (0.01, 0.01, 0.02), seed=7,
                            periodic=(True, True, True))
    m = PicMethod(Discretization(mesh, 2), U, ShapeFunctionDepositor(), AverageParticlePusher(),
                  3, 3)
    m.depositor.set_shape_function(None, PolynomialShapeFunction(0.002, 3, 2))
    rng = np.random.default_rng(n)
    s = m.make_state()
    m.add_particles_from_arrays(
        s, rng.uniform(0.01, 0.99, (n, 3)) * np.array([0.01, 0.01, 0.02]),
        U.EL_MASS * U.VACUUM_LIGHT_SPEED() * rng.normal(0, 1, (n, 3)),
        np.full(n, U.EL_CHARGE), np.full(n, U.EL_MASS))
    fields = torch.as_tensor(rng.normal(size=(6, len(m.discretization))), device="cuda")
    dt = 1e-12
    m.sort_by_element(s)
    for _ in range(2):
        # 0.3 mm a step, a beam line of 2 cm: a good many wrap
        m.step(s, fields, dt, steps=20, deposit=False, sort_every=0)
        f = m.pusher.forces(s, m.velocities(s), *fields)
        v = m.velocities_device(s)
        out = torch.empty_like(s.x)
        ptrs = (C.c_void_p * 6)(*[fields[k].data_ptr() for k in range(6)])
        _lib.check(m.lib.prt_average_forces(
            m.mesh_data.handle, m.workspace, m.pusher._shape_desc(),
            _lib.ptr(m.pusher.integral_weights), len(s), s.x.data_ptr(), s.q.data_ptr(),
            v.data_ptr(), s.el.data_ptr(), ptrs, out.data_ptr(), None, None, C.c_void_p(0)))
        want = out[:, s.id_order()].T.cpu().numpy()
        assert np.array_equal(np.asarray(f), want)
        s = m.advance_state(s, torch.zeros_like(s.x), torch.zeros_like(s.p))
