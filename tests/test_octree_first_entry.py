"""The octree path's first cell, whose entry t has no cell before it: cameras
inside the domain, with first entries at t of both signs, at exactly 0 and at
exactly -1, by the CPU harness.

Eight unit cells of value 1 over [0, 2]^3 and the interpolated projection: the
image is the length of t inside the domain, the last exit less the first entry.
"""
import ctypes as C

import numpy as np
import pytest

from test_kernel_host import emu  # noqa: F401  (the harness library)
from yt_gb300 import _lib
from yt_gb300.octree import Octree

Y = 2.0 / 3.0  # along (1, 2, 2) / 3: the plane y = 0 is at t = -1 exactly
CASES = {  # position: first entry and last exit, in units of the direction's length
    "minus-one": ((0.9, Y, 0.9), -1.0 / 3.0, 0.55),
    "ulp-above": ((0.9, np.nextafter(Y, 1.0), 0.9), -1.0 / 3.0, 0.55),
    "ulp-below": ((0.9, np.nextafter(Y, 0.0), 0.9), -1.0 / 3.0, 0.55),
    "zero": ((0.9, 0.0, 0.9), 0.0, 0.55),
    # (at t = 1 the ray leaves its cell through x and y at once: yt's strict
    # comparisons take neither plane and the traversal ends there)
    "outside": ((0.0, -1.0, -0.25), 0.5, 1.0),
}


@pytest.mark.parametrize("float_edges", [True, False])
@pytest.mark.parametrize("kind", [_lib.INTERPOLATED_PROJECTION, _lib.PROJECTION])
@pytest.mark.parametrize("case", CASES)
def test_first_entry(emu, case, kind, float_edges):  # noqa: F811
    pos, enter, leave = CASES[case]
    oc = Octree(np.zeros(3), np.full(3, 2.0), 1)
    ipos = np.array([(i, j, k) for i in (0, 1) for j in (0, 1) for k in (0, 1)], dtype=np.int32)
    oc.add_nodes(ipos, np.ones(8, dtype=np.int32), np.arange(8, dtype=np.int32))
    nodes = oc.nodes()
    verts = np.ones((8, 8), dtype=np.float32)
    le = ipos.astype(np.float64)
    edges = np.ascontiguousarray(np.concatenate([le, le + 1.0, np.ones((8, 3))], axis=1))
    edges_f = np.zeros((8, 12), dtype=np.float32)
    edges_f[:, 0:3], edges_f[:, 6:9] = le, 1.0
    o = _lib.OctreeArgs()
    o.nodes, o.verts, o.edges = nodes.ctypes.data, verts.ctypes.data, edges.ctypes.data
    if float_edges:
        o.edges_f = edges_f.ctypes.data
    o.n_nodes, o.n_cells, o.depth = nodes.size, 8, 1
    for i in range(3):
        o.dle[i], o.dre[i] = 0.0, 2.0
    p, d = np.array([[pos]], dtype=np.float64), np.array([[(1.0, 2.0, 2.0)]])
    assert case != "minus-one" or (0.0 - pos[1]) / (2.0 / 3.0) == -1.0
    a = _lib.RenderArgs()
    a.kind, a.n_samples = kind, 1
    a.view.nx = a.view.ny = 1
    a.view.lens = _lib.LENS_PER_PIXEL
    a.view.px_pos, a.view.px_dir = p.ctypes.data, d.ctypes.data
    a.data = verts.ctypes.data
    img = np.zeros((1, 1, 4))
    a.image = img.ctypes.data
    cnt = np.zeros(4, dtype=np.uint64)
    emu.emu_octree.argtypes = [C.POINTER(_lib.RenderArgs), C.POINTER(_lib.OctreeArgs), C.c_int, C.c_void_p,
                               C.c_void_p, C.c_void_p]
    assert emu.emu_octree(C.byref(a), C.byref(o), 0, None, None, cnt.ctypes.data) == 0
    # (a few float32 roundings over up to four cells)
    assert abs(img[0, 0, 0] - (leave - enter)) <= 8 * 2.0 ** -24
