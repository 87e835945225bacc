"""Projections of few cells: from one cell over one and two to a warp up to full
batches, and around the number from which on the summed stamps are used, by
either kernel and by project().

Quantities are of one sign: the kernels' sums agree to a few hundred roundings of
each pixel's own value (up to 700 cells a pixel here), 1e-12 of it."""
import numpy as np
import pytest
import torch

from test_gpu_offaxis_grazed import sums_image
from test_gpu_offaxis_sums import subcell_image
from yt_gb300 import offaxis
from yt_gb300.camera import orientation
from yt_gb300.offaxis import FEW_CELLS, CellSplat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 300, FEW_CELLS - 1, FEW_CELLS, FEW_CELLS + 1, 4255, 4256, 4257, 8513, 34049])
def test_few_cells(cuda, n, monkeypatch):
    nx, ny = 130, 130
    rng = np.random.default_rng(n)
    top = min(0.2, 2.0 / n ** 0.5)
    dx = np.exp(rng.uniform(np.log(1e-3), np.log(max(top, 4e-3)), n))
    s = CellSplat(rng.uniform(-0.55, 0.55, (n, 3)), dx, rng.uniform(0.5, 2.0, n), rng.uniform(0.5, 2.0, n), device=cuda)
    rot = orientation(rng.standard_normal(3), rng.standard_normal(3))[0]
    formed = []
    whole = offaxis._device_sums
    monkeypatch.setattr(offaxis, "_device_sums", lambda *a: formed.append(1) or whole(*a))
    got = s.project(rot, nx, ny)
    assert len(formed) == (n > FEW_CELLS)
    ref = subcell_image(s, rot, nx, ny)
    for image in (got, sums_image(s, rot, nx, ny)):
        for g, r in zip(image, ref):
            assert bool(((g - r).abs() <= 1e-12 * r + 1e-24 * float(r.max())).all())
    assert n < 7 or float(ref[0].sum()) > 0  # (few cells may all lie beyond the image)


@pytest.mark.parametrize("size", [(1, 1), (2, 3), (31, 31), (32, 33), (63, 200), (257, 257), (513, 700)])
@pytest.mark.parametrize("width,n", [((2e-4, 5e-3), 1000), ((5e-3, 0.12), 333), ((0.25, 0.6), 5), ((1e-3, 0.3), 31)])
def test_sums_of_few_cells(cuda, size, width, n):
    """Cells from far below a pixel to wider than a warp's table of pixel
    boundaries (518), on and across the image's edges, by the summed stamps,
    which project() does not take for so few."""
    nx, ny = size
    rng = np.random.default_rng(nx + n)
    dx = np.exp(rng.uniform(np.log(width[0]), np.log(width[1]), n))
    x = rng.uniform(-0.7, 0.7, (n, 3))
    rot = orientation(rng.standard_normal(3), rng.standard_normal(3))[0]
    s = CellSplat(x, dx, rng.uniform(0.5, 2.0, n), rng.uniform(0.5, 2.0, n), device=cuda)
    for g, r in zip(sums_image(s, rot, nx, ny), subcell_image(s, rot, nx, ny)):
        assert bool(((g - r).abs() <= 1e-12 * r + 1e-24 * float(r.max())).all())
