"""The sort's groups of arrays where few rows or none fit one (3 and 9 million
particles), and the number of launches that the benchmark counts for them."""

import ctypes as C
import sys
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))

import bench  # noqa: E402
from pyrticle_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("n,groups", [(1, 1), (900_001, 1), (932_068, 2), (2_796_202, 3),
                                      (4_000_000, 4), (9_000_001, 5), (16_000_000, 5)])
def test_launches_of_a_sort(n, groups):
    """64 MB are 9 rows of 932,067 particles (x, p, q, m, ids), 3 of 2,796,202
    (x | p | q, m, ids), 2 of 4,000,000 (x | p | q, m | ids), none of 9,000,001."""
    assert bench.sort_launches(n) == 1 + 2 * groups


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3_000_001, 9_000_001])
def test_sort_of_arrays_in_groups_of_their_own(n):
    rng = np.random.default_rng(n)
    el = rng.integers(0, 1000, n).astype(np.uint32)
    el[rng.random(n) < 0.1] = 0xFFFFFFFF
    x, q = rng.normal(size=(3, n)), rng.normal(size=n)
    ids = rng.permutation(n).astype(np.int64)
    dev = [torch.as_tensor(a, device="cuda").clone() for a in (el.view(np.int32), x, q, ids)]
    ws = C.c_void_p()
    lib = _lib.load()
    _lib.check(lib.prt_workspace_create(C.byref(ws)))
    _lib.check(lib.prt_sort_by_element(
        ws, n, dev[0].data_ptr(), dev[1].data_ptr(), None, dev[2].data_ptr(), None, None, None,
        dev[3].data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    order = np.argsort(el, kind="stable")
    for d, h in zip(dev, (el.view(np.int32), x, q, ids)):
        assert np.array_equal(d.cpu().numpy(), h[..., order])
    _lib.check(lib.prt_workspace_destroy(ws))
