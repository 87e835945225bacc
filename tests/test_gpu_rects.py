"""Pixel rectangles formed on the device (ytgb_brick_rects_device) against the
host's (ytgb_brick_rects, which the oracle and the reference check): the same
integers, for every extent function, cameras outside, inside and in the planes
of the bricks, one-pixel to ragged images, and more bricks than one block."""
import ctypes as C

import numpy as np
import pytest
import torch

from yt_gb300 import _lib
from yt_gb300.camera import Camera
from yt_gb300.volume import BrickSet

pytestmark = pytest.mark.gpu


def bricks(n, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        le = rng.integers(0, 14, 3) / 16.0 if rng.random() < 0.5 else rng.uniform(0, 0.9, 3)
        out.append(([np.zeros((2, 2, 2))], None, le, le + rng.integers(1, 3) / 16.0, np.array([1, 1, 1])))
    return out


@pytest.mark.parametrize("n", [1, 15, 17, 400])
@pytest.mark.parametrize("size", [(1, 1), (2, 2), (64, 64), (301, 177), (1024, 768)])
@pytest.mark.parametrize("lens", ["plane-parallel", "perspective", "null"])
def test_device_rects_equal_host(cuda, n, size, lens):
    bs = BrickSet(bricks(n, n + size[0]), device=cuda)
    rng = np.random.default_rng(size[1])
    s = torch.cuda.current_stream(cuda)
    for k in range(12):
        # far, near, inside the volume, and in the planes that bricks share
        pos = (0.5 + rng.standard_normal(3) * (0.2, 0.8, 2.0)[k % 3]) if k % 4 else \
            np.array([(-1.0, 0.5, 0.5), (0.5, 0.25, 0.75), (0.5, 0.5, 3.0)][k // 4])
        focus = np.array([0.5, 0.5, 0.5]) + (k // 4 == 1) * np.array([0.0, 0.25, -0.25])
        cam = Camera(pos, focus, rng.uniform(0.3, 2.0), size, lens_type="perspective" if lens == "null" else lens)
        view = cam.device_view()
        if lens == "null":
            view.extent = _lib.EXTENT_NULL
        order = rng.permutation(n).astype(np.int32)
        tab = bs.device_table(view, order, s).cpu().numpy()
        ref = bs.rects(view, order)
        assert np.array_equal(tab[4 * n:], order)
        assert np.array_equal(tab[:4 * n].reshape(n, 4), ref)


def test_device_rects_unknown_brick_and_bad_arguments(cuda):
    bs = BrickSet(bricks(3, 1), device=cuda)
    view = Camera((0.5, 0.5, -1.0), (0.5, 0.5, 0.5), 1.0, 32).device_view()
    s = torch.cuda.current_stream(cuda)
    tab = bs.device_table(view, np.array([0, 7, -1, 2], dtype=np.int32), s).cpu().numpy()[:16].reshape(4, 4)
    assert (tab[1] == 0).all() and (tab[2] == 0).all()
    assert np.array_equal(tab[[0, 3]], bs.rects(view, np.array([0, 2], dtype=np.int32)))
    L = _lib.lib()
    t = torch.zeros(64, dtype=torch.int32, device=cuda)
    bad = [(None, 3, t.data_ptr(), 1, t.data_ptr()), (bs.desc.data_ptr(), 0, t.data_ptr(), 1, t.data_ptr()),
           (bs.desc.data_ptr(), 3, None, 1, t.data_ptr()), (bs.desc.data_ptr(), 3, t.data_ptr(), 1, t.data_ptr() + 4),
           (bs.desc.data_ptr(), 3, t.data_ptr(), -1, t.data_ptr())]
    for d, n, o, k, r in bad:
        assert L.ytgb_brick_rects_device(C.byref(view), d, n, o, k, r, None) == _lib.ERR_INVALID
    assert L.ytgb_brick_rects_device(C.byref(view), None, 0, None, 0, None, None) == _lib.OK
