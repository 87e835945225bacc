"""Where the order of the tiles is formed: the rule's lines on either side, and
on the octree path the ordered image against grid order for trees large enough
to be ordered (their cost is estimated from part of their cells)."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_schedule import bricks
from yt_gb300 import _lib, testing
from yt_gb300.camera import Camera
from yt_gb300.octree import Octree, OctreeVolume, render_octree
from yt_gb300.volume import ORDER_BRICKS, BrickSet, render, render_tables

pytestmark = pytest.mark.gpu


class Spy:
    """The library with one entry point's third argument recorded."""

    def __init__(self, L, name):
        self._L, self._name, self.bytes = L, name, []

    def __getattr__(self, name):
        f = getattr(self._L, name)
        if name != self._name:
            return f

        def call(*a):
            self.bytes.append(a[-2])
            return f(*a)
        return call


@pytest.mark.parametrize("n,size,ordered", [(ORDER_BRICKS - 1, (1024, 1024), False), (ORDER_BRICKS, (1024, 1024), True),
                                            (512, (312, 500), True), (512, (304, 500), False), (512, (288, 500), False),
                                            (512, (4096, 4096), False)])
@pytest.mark.parametrize("resident", [False, True])
def test_bricks_and_tiles(cuda, n, size, ordered, resident, monkeypatch):
    bs = BrickSet(bricks(512, 1)[:n], device=cuda)
    view = Camera(np.array((0.5, 0.4, -1.2)), (0.5, 0.5, 0.6), 0.9, size, lens_type="perspective").device_view()
    order = np.arange(bs.n, dtype=np.int32)
    tables = render_tables(bs, view, order) if resident else None
    spy = Spy(_lib.lib(), "ytgb_render_scheduled")
    monkeypatch.setattr(_lib, "_lib", spy)
    img = torch.zeros((*size, 4), dtype=torch.float64, device=cuda)
    render(bs, view, order, _lib.INTERPOLATED_PROJECTION, img, tables=tables)
    torch.cuda.synchronize()
    assert [b > 0 for b in spy.bytes] == [ordered]


@pytest.fixture(scope="module")
def tree(cuda):
    depth, ipos, lvl, cells = testing.octree_cells(base_level=4, max_level=7, seed=3)
    assert cells.shape[0] > 1 << 16
    oc = Octree(np.zeros(3), np.ones(3), depth)
    oc.add_nodes(ipos, lvl, np.arange(ipos.shape[0], dtype=np.int32))
    return OctreeVolume(oc, cells, cuda)


def need(view, o):
    n = C.c_int64(-1)
    _lib.check(_lib.lib().ytgb_octree_scratch(C.byref(view), C.byref(o), C.byref(n)), "scratch")
    return n.value


def test_octree_rule(cuda, tree):
    o = tree.args()

    def at(pos, size=(1024, 1024)):
        return Camera(np.array(pos), (0.5, 0.5, 0.6), 0.9, size, lens_type="perspective").device_view()

    out = (0.5, 0.4, -1.2)
    assert need(at(out), o) == 6 * 8192
    assert need(at((0.45, 0.55, 0.5)), o) == 0  # inside
    assert need(at((0.45, 0.55, 1.0 + 1e-9)), o) == 6 * 8192
    assert need(at(out, (16 * 38, 8 * 32)), o) == 0 and need(at(out, (16 * 38, 8 * 32 + 1)), o) == 6 * 38 * 33
    assert need(at(out, (4096, 2041)), o) == 0  # 65,536 tiles
    few = tree.args()
    few.n_cells = (1 << 16) - 1
    assert need(at(out), few) == 0
    few.n_cells = 1 << 16
    assert need(at(out), few) == 6 * 8192
    v = at(out)
    v.lens = _lib.LENS_PER_PIXEL
    assert need(v, o) == 0
    n = C.c_int64()
    assert _lib.lib().ytgb_octree_scratch(C.byref(at(out)), None, C.byref(n)) == _lib.ERR_INVALID


@pytest.mark.parametrize("size", [(501, 402), (1024, 1024), (33, 8000)])
@pytest.mark.parametrize("pos", [(0.5, 0.4, -1.2), (3.0, 2.4, -2.9), (0.5, 0.5, 1.0 + 1e-9)])
def test_octree_ordered_equals_grid_order(cuda, tree, size, pos):
    s = torch.cuda.current_stream(cuda)
    view = Camera(np.array(pos), (0.5, 0.5, 0.6), 0.9, size, lens_type="perspective").device_view()
    assert need(view, tree.args()) > 0
    img = torch.zeros((*size, 4), dtype=torch.float64, device=cuda)
    ref = torch.zeros_like(img)
    counters = torch.zeros((2, 4), dtype=torch.int64, device=cuda)
    render_octree(tree, view, _lib.INTERPOLATED_PROJECTION, img, counters=counters[0])
    a = _lib.RenderArgs()
    a.kind, a.n_samples, a.view = _lib.INTERPOLATED_PROJECTION, 1, view
    a.data, a.image, a.counters = tree.verts.data_ptr(), ref.data_ptr(), counters[1].data_ptr()
    o = tree.args()
    _lib.check(_lib.lib().ytgb_render_octree(C.byref(a), C.byref(o), C.c_void_p(s.cuda_stream)), "render")
    torch.cuda.synchronize()
    assert torch.equal(counters[0], counters[1]) and int(counters[0, 2]) == size[0] * size[1]
    assert torch.equal(img.view(torch.int64), ref.view(torch.int64))
