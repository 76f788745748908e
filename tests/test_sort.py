"""prt_sort_by_element and prt_sort_by_element_of against a stable host sort.

Sizes: one particle, a warp and a block with their neighbours, the change
from one to four particles a thread (148 x 2048), and 900,001 particles,
where only nine rows fit a group (so residuals make a second one). Removed
particles (all-ones elements) go last; the order is exact.
"""

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from pyrticle_b200 import _lib, meshgen  # noqa: E402
from pyrticle_b200.discretization import Discretization  # noqa: E402
from pyrticle_b200.meshdata import MeshData  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("of_mesh", [True, False])
@pytest.mark.parametrize("residuals", [True, False])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 1025, 148 * 2048, 148 * 2048 + 1, 900_001])
def test_sort(n, residuals, of_mesh):
    mesh = meshgen.box_mesh((3, 3, 4), (0, 0, 0), (1, 1, 1), periodic=(False, False, False))
    data = MeshData()
    data.fill_from_discretization(Discretization(mesh, 1))
    E = data.element_count
    rng = np.random.default_rng(n)
    el = rng.integers(0, E, n).astype(np.uint32)
    el[rng.random(n) < 0.1] = 0xFFFFFFFF
    host = {k: rng.normal(size=(c, n)) for k, c in dict(x=3, p=3, q=1, m=1, kx=3, kp=3).items()}
    host["ids"] = rng.permutation(n).astype(np.int64)[None]
    dev = {k: torch.as_tensor(v, device="cuda").clone() for k, v in host.items()}
    d_el = torch.as_tensor(el.view(np.int32), device="cuda").clone()
    ws = C.c_void_p()
    lib = _lib.load()
    _lib.check(lib.prt_workspace_create(C.byref(ws)))
    args = [d_el.data_ptr(), *(dev[k].data_ptr() for k in ("x", "p", "q", "m")),
            dev["kx"].data_ptr() if residuals else None,
            dev["kp"].data_ptr() if residuals else None, dev["ids"].data_ptr(),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)]
    if of_mesh:
        _lib.check(lib.prt_sort_by_element_of(data.handle, ws, n, *args))
    else:
        _lib.check(lib.prt_sort_by_element(ws, n, *args))
    torch.cuda.synchronize()
    order = np.argsort(el, kind="stable")
    assert np.array_equal(d_el.cpu().numpy().view(np.uint32), el[order])
    for k, v in host.items():
        moved = residuals or k not in ("kx", "kp")
        assert np.array_equal(dev[k].cpu().numpy(), v[:, order] if moved else v), k
    _lib.check(lib.prt_workspace_destroy(ws))
