"""Points at a brick's upper faces: none beyond its last layer, and a grid with
a number past its end is refused."""

import ctypes as C

import numpy as np
import pytest

from pyrticle_b200 import meshgen
from pyrticle_b200.deposition import grid as G


def test_no_point_beyond_a_brick():
    """A brick whose upper corner rounds to more than its cells: the elements
    at that face take no layer beyond the last (a number of another row, or one
    past the grid's end)."""
    lengths = np.array([0.006, 0.004, 0.0095])
    checked = 0
    for n in range(5, 60):
        dims = np.array([6, 6, n])
        h = lengths / dims
        brick = G.BrickInfo(0, 0, h, np.zeros(3), dims)
        if not (np.ceil(brick.bounding_box()[1] / h) > dims).any():
            continue
        mesh = meshgen.box_mesh((2, 2, 3), (0, 0, 0), lengths, seed=3)
        starts, gidx, pts, w = G.find_points_in_elements(mesh, [brick], 0.12)
        assert gidx.min() >= 0 and gidx.max() < len(brick)
        idx = np.stack([gidx % 6, gidx // 6 % 6, gidx // 36], axis=1)
        assert np.array_equal(brick.point(idx), pts)
        checked += 1
    assert checked >= 2


@pytest.mark.gpu
@pytest.mark.parametrize("number,accepted", [(7, True), (8, False), (2 ** 32 - 1, False)])
def test_grid_number_past_the_end_is_refused(number, accepted):
    from pyrticle_b200 import _lib
    from pyrticle_b200.cloud import PicMethod
    from pyrticle_b200.deposition.shape import ShapeFunctionDepositor
    from pyrticle_b200.discretization import Discretization
    from pyrticle_b200.pusher import MonomialParticlePusher
    from pyrticle_b200.units import SIUnitsWithNaturalConstants as U

    mesh = meshgen.box_mesh((2, 2, 2), (0, 0, 0), (0.01,) * 3, seed=3)
    m = PicMethod(Discretization(mesh, 1), U, ShapeFunctionDepositor(), MonomialParticlePusher(),
                  3, 3)
    brick = (_lib.Brick * 1)()
    for a in range(3):
        brick[0].stepwidths[a], brick[0].dims[a] = 0.005, 2  # 8 points
    d = _lib.GridDesc()
    d.brick_count, d.nodes_per_element, d.eog_count = 1, 4, 1
    d.bricks = C.cast(brick, C.POINTER(_lib.Brick))
    arrays = [np.array([0], np.uint32), np.array([0, 1], np.uint64),
              np.array([number], np.uint32), np.ones(1), np.array([0, 4], np.uint64), np.ones(4)]
    d.eog_elements = _lib.ptr(arrays[0], C.c_uint32)
    d.eog_starts = _lib.ptr(arrays[1], C.c_uint64)
    d.eog_grid_nodes = _lib.ptr(arrays[2], C.c_uint32)
    d.eog_weights = _lib.ptr(arrays[3])
    d.eog_matrix_starts = _lib.ptr(arrays[4], C.c_uint64)
    d.eog_matrices = _lib.ptr(arrays[5])
    handle = C.c_void_p()
    rc = m.lib.prt_grid_create(m.mesh_data.handle, C.byref(d), C.byref(handle))
    assert rc == (_lib.PRT_OK if accepted else -1)
    if accepted:
        m.lib.prt_grid_destroy(handle)
