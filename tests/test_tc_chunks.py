"""The tensor-core deposition at the edges of its chunks of 128 candidates.

All particles sit within a thousandth of the radius of one point, so that
every tile within reach stages all of them: none, a part of a chunk, one
chunk but one, exactly one, one more, and the ring of five chunks with its
neighbours. Both passes run (the readouts alternate between two halves of the
warps by the chunk's parity). Bars: the FP64 form within 1e-5 (a weight is an
integer of 23 bits, its score carries 22, and nothing cancels: all particles
have one sign), the normalised charge kept to 1e-14.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import meshgen  # noqa: E402
from pyrticle_b200.cloud import PicMethod  # noqa: E402
from pyrticle_b200.deposition.shape import (NormalizedShapeFunctionDepositor,  # noqa: E402
                                            ShapeFunctionDepositor)
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.pusher import MonomialParticlePusher  # noqa: E402
from pyrticle_b200.tools import PolynomialShapeFunction  # noqa: E402
from pyrticle_b200.units import SIUnitsWithNaturalConstants as U  # noqa: E402

from conftest import rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depositor", [ShapeFunctionDepositor, NormalizedShapeFunctionDepositor])
@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 255, 257, 639, 640, 641, 2049])
def test_chunk_edges(depositor, n):
    mesh = meshgen.box_mesh((6, 6, 6), (0, 0, 0), (0.01, 0.01, 0.01),
                            periodic=(False, False, False))
    m = PicMethod(Discretization(mesh, 3), U, depositor("mixed"), MonomialParticlePusher(), 3, 3)
    radius = 0.003
    m.depositor.set_shape_function(None, PolynomialShapeFunction(radius, 3, 2))
    rng = np.random.default_rng(n)
    x = 0.0051 + 1e-3 * radius * rng.uniform(-1, 1, (n, 3))
    p = np.concatenate([rng.normal(size=(n, 2)) * 1e-25, np.full((n, 1), 1e-22)], 1)
    q = np.full(n, -U.EL_CHARGE)
    s = m.make_state()
    m.add_particles_from_arrays(s, x, p, q, np.full(n, U.EL_MASS))
    r64, j64 = m.depositor.deposit_densities_device(s, precision="fp64")
    r, j = m.depositor.deposit_densities_device(s, precision="mixed")
    r2, j2 = m.depositor.deposit_densities_device(s, precision="mixed")
    assert torch.equal(r, r2) and torch.equal(j, j2)
    r64, j64, r, j = (t.cpu().numpy() for t in (r64, j64, r, j))
    assert rel_l2(r, r64) < 1e-5 and rel_l2(j, j64) < 1e-5
    if depositor is NormalizedShapeFunctionDepositor:
        iw, jac = m.depositor.integral_weights, m.discretization.mesh.jacobians
        total = float((r.reshape(-1, len(iw)) @ iw * jac).sum())
        assert abs(total - q.sum()) <= 1e-14 * abs(q.sum())
