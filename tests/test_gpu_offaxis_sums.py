"""Splatting by summed stamps (ytgb_offaxis_cells_sums) against the subcell
kernel (ytgb_offaxis_cells), which the oracle and the reference check: cells
from far below a pixel to wider than the kernel's table of pixel boundaries
(255), on and across the image's edges, one pixel to ragged images, more cells
than one warp's batch and fewer.

Both form every subcell's pixels and shares by the same float64 operations.
The table's rounding is at most 4 units of 2^-58 pixel shares and each side
adds a pixel's contributions in float64 in its own order, so with up to 2^12
contributions of one sign a pixel they agree to 2^12 * 2^-53 of its value;
1e-12 of the image's largest value is the bound."""
import ctypes as C

import numpy as np
import pytest
import torch

from yt_gb300 import _lib
from yt_gb300.camera import orientation
from yt_gb300.offaxis import CellSplat

pytestmark = pytest.mark.gpu


def subcell_image(s, rot, nx, ny):
    """The same projection by ytgb_offaxis_cells."""
    stamp, (max_depth, nsx, nsy) = s.stamp(rot, nx, ny)
    out = [torch.zeros(nx * ny, dtype=torch.float64, device=s.device) for _ in range(2)]
    a = _lib.OffaxisArgs()
    a.xp, a.dxp, a.qty, a.weight = (t.data_ptr() for t in (s.xp, s.dxp, s.qty, s.weight))
    a.stamp, a.buffer, a.buffer_weight = stamp.data_ptr(), out[0].data_ptr(), out[1].data_ptr()
    for i in range(6):
        a.rot[i] = float(rot[i // 3, i % 3])
    a.n, a.nx, a.ny, a.nsx, a.nsy, a.max_depth = s.n, nx, ny, nsx, nsy, max_depth
    st = torch.cuda.current_stream(s.device).cuda_stream
    _lib.check(_lib.lib().ytgb_offaxis_cells(C.byref(a), None, C.c_void_p(st)), "ytgb_offaxis_cells")
    return out


@pytest.mark.parametrize("size", [(1, 1), (2, 3), (31, 31), (32, 33), (63, 200), (257, 257), (513, 700)])
@pytest.mark.parametrize("width,n", [((2e-4, 5e-3), 1000), ((5e-3, 0.12), 333), ((0.25, 0.6), 5), ((1e-3, 0.3), 31)])
def test_sums_equal_subcells(cuda, size, width, n):
    nx, ny = size
    rng = np.random.default_rng(nx + n)
    dx = np.exp(rng.uniform(np.log(width[0]), np.log(width[1]), n))
    x = rng.uniform(-0.7, 0.7, (n, 3))  # some cells beyond the image's edges
    rot = orientation(rng.standard_normal(3), rng.standard_normal(3))[0]
    s = CellSplat(x, dx, rng.uniform(0.5, 2.0, n), rng.uniform(0.5, 2.0, n), device=cuda)
    got, ref = s.project(rot, nx, ny), subcell_image(s, rot, nx, ny)
    for g, r in zip(got, ref):
        top = float(r.abs().max())
        assert float((g - r).abs().max()) <= 1e-12 * top


def test_sums_signed_and_bad_cells(cuda):
    """Quantities of both signs, one cell of no width (skipped, reported), and
    buffers that hold values already."""
    rng = np.random.default_rng(9)
    n, nx = 200, 96
    dx = rng.uniform(0.01, 0.05, n)
    dx[17] = 0.0
    s = CellSplat(rng.uniform(-0.4, 0.4, (n, 3)), dx, rng.standard_normal(n), device=cuda)
    rot = orientation(np.array([0.3, -0.5, 0.8]))[0]
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    ref = subcell_image(s, rot, nx, nx)
    got = s.project(rot, nx, nx, out=tuple(torch.ones(nx * nx, dtype=torch.float64, device=cuda) for _ in range(2)),
                    error=err)
    for g, r in zip(got, ref):
        assert float((g - 1.0 - r).abs().max()) <= 1e-12 * max(1.0, float(r.abs().max()))
    assert int(err) == 4  # YTGB_DEVERR_BAD_CELL


def test_sums_rejects_bad_arguments(cuda):
    L = _lib.lib()
    t = torch.zeros(64, dtype=torch.int64, device=cuda)
    assert L.ytgb_offaxis_sums(t.data_ptr(), 4, 4, 1, 8, 8, t.data_ptr(), None) == _lib.ERR_INVALID
    assert L.ytgb_offaxis_sums(None, 4, 4, 2, 8, 8, t.data_ptr(), None) == _lib.ERR_INVALID
    a = _lib.OffaxisArgs()
    a.nx = a.ny = a.nsx = a.nsy = 4
    a.max_depth = 2
    assert L.ytgb_offaxis_cells_sums(C.byref(a), None, None, None) == _lib.ERR_INVALID
    assert L.ytgb_offaxis_cells_sums(C.byref(a), t.data_ptr(), None, None) == _lib.OK
