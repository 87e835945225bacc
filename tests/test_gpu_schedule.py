"""ytgb_render_scheduled and ytgb_render_octree_scheduled (the tiles with most work
first) against ytgb_render and ytgb_render_octree:
the same image bit for bit and the same counts, so every tile rendered once;
for images under and over the sort's runs, ragged, of each tile shape, past the
numbers that are ordered, cameras outside and among the bricks, and scratch
memory that is too small."""
import ctypes as C

import numpy as np
import pytest
import torch

from yt_gb300 import _lib, testing
from yt_gb300.camera import Camera
from yt_gb300.octree import Octree, OctreeVolume, render_octree
from yt_gb300.volume import BrickSet, render_tables

pytestmark = pytest.mark.gpu


def bricks(n, seed):
    rng = np.random.default_rng(seed)
    m = 1 << (n - 1).bit_length()
    at = [(x, y, z) for x in range(8) for y in range(8) for z in range(8)][: min(n, 512)] if m > 1 else [(0, 0, 0)]
    w = 1.0 / 8 if m > 1 else 1.0
    out = []
    for p in at:
        le = np.array(p) * w
        d = rng.integers(1, 5)
        out.append(([rng.random((d + 1,) * 3)], None, le, le + w, np.array([d] * 3)))
    return out


@pytest.mark.parametrize("n", [1, 2, 60, 512])
@pytest.mark.parametrize("size", [(1, 1), (400, 301), (1024, 768), (33, 31999), (2900, 2901), (2912, 2896)])
@pytest.mark.parametrize("shape", [0, 1, 2])
def test_scheduled_equals_grid_order(cuda, n, size, shape):
    bs = BrickSet(bricks(n, n), device=cuda)
    s = torch.cuda.current_stream(cuda)
    for k, pos in enumerate([(0.5, 0.4, -1.2), (0.45, 0.55, 0.5)]):
        cam = Camera(np.array(pos), (0.5, 0.5, 0.6), 0.9, size, lens_type="perspective")
        view = cam.device_view()
        order = np.random.default_rng(k).permutation(bs.n).astype(np.int32)
        tab = render_tables(bs, view, order).table
        need = C.c_int64()
        _lib.check(_lib.lib().ytgb_render_scratch(C.byref(view), order.size, C.byref(need)), "scratch")
        got = []
        for bytes_ in (None, need.value, need.value - 1 if need.value else 0):
            img = torch.zeros((*size, 4), dtype=torch.float64, device=cuda)
            counters = torch.zeros(4, dtype=torch.int64, device=cuda)
            mem = torch.full((max(need.value, 8),), 0xff, dtype=torch.uint8, device=cuda)
            a = _lib.RenderArgs()
            a.kind, a.n_samples, a.n_order = _lib.INTERPOLATED_PROJECTION, 1, order.size
            a.flags = shape << _lib.FLAG_TILE_SHIFT
            a.view = view
            a.bricks, a.rects, a.order = bs.desc.data_ptr(), tab.data_ptr(), tab.data_ptr() + 16 * order.size
            a.data, a.bounds, a.image = bs.data.data_ptr(), bs.bounds.data_ptr(), img.data_ptr()
            a.counters = counters.data_ptr()
            if bytes_ is None:
                _lib.check(_lib.lib().ytgb_render(C.byref(a), C.c_void_p(s.cuda_stream)), "render")
            else:
                _lib.check(_lib.lib().ytgb_render_scheduled(C.byref(a), mem.data_ptr(), bytes_,
                                                            C.c_void_p(s.cuda_stream)), "render")
            torch.cuda.synchronize()
            got.append((img, counters.cpu().tolist()))
            del mem
        assert got[0][1][2] == size[0] * size[1]
        for img, counts in got[1:]:
            assert counts == got[0][1]
            assert torch.equal(img.view(torch.int64), got[0][0].view(torch.int64))


@pytest.mark.parametrize("size", [(1, 1), (64, 50), (501, 402), (2912, 2896)])
def test_octree_scheduled_equals_grid_order(cuda, size):
    depth, ipos, lvl, cells = testing.octree_cells(base_level=3, max_level=6, seed=4)
    oc = Octree(np.zeros(3), np.ones(3), depth)
    oc.add_nodes(ipos, lvl, np.arange(ipos.shape[0], dtype=np.int32))
    vol = OctreeVolume(oc, cells, cuda)
    s = torch.cuda.current_stream(cuda)
    for pos in [(0.5, 0.4, -1.2), (0.45, 0.55, 0.5), (0.5, 0.5, 2.0)]:
        view = Camera(np.array(pos), (0.5, 0.5, 0.6), 0.9, size, lens_type="perspective").device_view()
        got = []
        for scheduled in (True, False):
            img = torch.zeros((*size, 4), dtype=torch.float64, device=cuda)
            counters = torch.zeros(4, dtype=torch.int64, device=cuda)
            if scheduled:
                render_octree(vol, view, _lib.INTERPOLATED_PROJECTION, img, counters=counters)
            else:
                a = _lib.RenderArgs()
                a.kind, a.n_samples, a.view = _lib.INTERPOLATED_PROJECTION, 1, view
                a.data, a.image, a.counters = vol.verts.data_ptr(), img.data_ptr(), counters.data_ptr()
                o = vol.args()
                _lib.check(_lib.lib().ytgb_render_octree(C.byref(a), C.byref(o), C.c_void_p(s.cuda_stream)), "render")
            torch.cuda.synchronize()
            got.append((img, counters.cpu().tolist()))
        assert got[0][1] == got[1][1] and got[0][1][2] == size[0] * size[1]
        assert torch.equal(got[0][0].view(torch.int64), got[1][0].view(torch.int64))  # (NaNs too)


def test_scratch_sizes():
    need = C.c_int64(-1)
    v = _lib.View()
    v.nx = v.ny = 1024
    assert _lib.lib().ytgb_render_scratch(C.byref(v), 1, C.byref(need)) == 0 and need.value == 0
    assert _lib.lib().ytgb_render_scratch(C.byref(v), 2, C.byref(need)) == 0 and need.value == 6 * 8192
    v.ny = 0
    assert _lib.lib().ytgb_render_scratch(C.byref(v), 2, C.byref(need)) != 0
    a = _lib.RenderArgs()
    assert _lib.lib().ytgb_render_scheduled(C.byref(a), None, -1, None) == _lib.ERR_INVALID
    assert _lib.lib().ytgb_render_scheduled(C.byref(a), C.c_void_p(2), 64, None) == _lib.ERR_INVALID
