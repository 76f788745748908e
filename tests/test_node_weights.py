"""The normalising depositor's integration weights travel as a kernel argument
up to 64 nodes an element and are copied above: orders 5 (56 nodes) and 6 (84).
The deposited charge is that of the particles (1e-12: sums of some 1e4 FP64
terms), in both precisions, and the two agree within the chosen form's 1e-5.
"""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import _lib, meshgen  # noqa: E402
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.meshdata import MeshData  # noqa: E402
from pyrticle_b200.tools import PolynomialShapeFunction  # noqa: E402

from conftest import rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [5, 6])
def test_normalised_charge(order):
    mesh = meshgen.box_mesh((3, 3, 3), (0, 0, 0), (1, 1, 1), periodic=(False, False, False))
    discr = Discretization(mesh, order)
    data = MeshData()
    data.fill_from_discretization(discr)
    lib, n = _lib.load(), 300
    rng = np.random.default_rng(order)
    x = torch.as_tensor(rng.uniform(0.4, 0.6, (3, n)), device="cuda")
    q = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
    v = torch.as_tensor(rng.normal(size=(3, n)), device="cuda")
    el = torch.zeros(n, dtype=torch.int32, device="cuda")
    sf = PolynomialShapeFunction(0.3, 3, 2)
    desc = _lib.ShapeFunctionDesc(sf.radius, sf.exponent, sf.normalizer)
    ldis = discr.element_groups[0].local_discretization
    iw = np.ascontiguousarray(ldis.mass_matrix().sum(axis=1))
    nn = len(discr.nodes)
    ws = C.c_void_p()
    _lib.check(lib.prt_workspace_create(C.byref(ws)))
    rhos = []
    for precision in (0, 1):
        rho = torch.empty(nn, dtype=torch.float64, device="cuda")
        j = torch.empty((3, nn), dtype=torch.float64, device="cuda")
        _lib.check(lib.prt_deposit_shape(
            data.handle, ws, _lib.DEPOSIT_NORMALIZED, desc, _lib.ptr(iw), n, x.data_ptr(),
            q.data_ptr(), v.data_ptr(), el.data_ptr(), rho.data_ptr(), j.data_ptr(), precision,
            None, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        rhos.append(rho.cpu().numpy())
        total = float((rhos[-1].reshape(-1, len(iw)) @ iw * mesh.jacobians).sum())
        assert abs(total + n) <= 1e-12 * n
    assert rel_l2(rhos[1], rhos[0]) < 1e-5
    _lib.check(lib.prt_workspace_destroy(ws))
