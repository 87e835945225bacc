"""Splatting by summed stamps (ytgb_offaxis_cells_sums) pixel by pixel against
the subcell kernel (ytgb_offaxis_cells), one cell to an image: a pixel that a cell
only grazes is as exact as one it fills.

The subcell kernel sums at most some 100 products of one sign a pixel in float64
(a few hundred where the image is much higher than wide): 1e-13 of the pixel's
own value is the bound.  The table's rounding is some 50 units of 2^-126 of the
stamp's sum at most, 1e-30 of the cell's largest pixel where it covers up to 10^6;
1e-24 of it is allowed beside."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_offaxis_sums import subcell_image
from yt_gb300 import _lib
from yt_gb300.camera import orientation
from yt_gb300.offaxis import CellSplat, _device_sums

pytestmark = pytest.mark.gpu


def sums_image(s, rot, nx, ny):
    """The projection by ytgb_offaxis_cells_sums, whatever path project() takes."""
    stamp, shape = s.stamp(rot, nx, ny)
    sums = _device_sums(stamp, shape, nx, ny)
    out = [torch.zeros(nx * ny, dtype=torch.float64, device=s.device) for _ in range(2)]
    a = _lib.OffaxisArgs()
    a.xp, a.dxp, a.qty, a.weight = (t.data_ptr() for t in (s.xp, s.dxp, s.qty, s.weight))
    a.stamp, a.buffer, a.buffer_weight = stamp.data_ptr(), out[0].data_ptr(), out[1].data_ptr()
    for i in range(6):
        a.rot[i] = float(rot[i // 3, i % 3])
    a.n, a.nx, a.ny, a.nsx, a.nsy, a.max_depth = s.n, nx, ny, shape[1], shape[2], shape[0]
    st = torch.cuda.current_stream(s.device).cuda_stream
    _lib.check(_lib.lib().ytgb_offaxis_cells_sums(C.byref(a), sums.data_ptr(), None, C.c_void_p(st)), "sums")
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("size", [(64, 64), (257, 257), (40, 300), (640, 700)])
@pytest.mark.parametrize("dx", [0.004, 0.0123, 1.0 / 60.0, 0.05, 0.15])
def test_grazed_pixels(cuda, size, dx):
    nx, ny = size
    rng = np.random.default_rng(int(1e4 * dx) + nx)
    faint = 0
    for k in range(6):
        x = rng.uniform(-0.45, 0.45, (1, 3))
        if k == 0:
            x[:] = 0.0
        rot = orientation(rng.standard_normal(3), rng.standard_normal(3))[0]
        s = CellSplat(x, [dx], [rng.uniform(0.5, 2.0)], [rng.uniform(0.5, 2.0)], device=cuda)
        for g, r in zip(sums_image(s, rot, nx, ny), subcell_image(s, rot, nx, ny)):
            top = float(r.max())
            faint += int(((r > 0) & (r < 1e-3 * top)).sum())
            assert bool(((g - r).abs() <= 1e-13 * r + 1e-24 * top).all())
    assert faint > 0 or dx * nx < 4  # grazed pixels are among them
