"""Quantities and weights that are not finite, zero, tiny or huge, by the summed
stamps and by the subcell kernel: NaN reaches the same pixels (every pixel of the
cell's rectangle), infinities leave the same pixels without a finite value, and
the others agree as for ordinary cells."""
import numpy as np
import pytest
import torch

from test_gpu_offaxis_grazed import sums_image
from test_gpu_offaxis_sums import subcell_image
from yt_gb300.camera import orientation
from yt_gb300.offaxis import CellSplat

pytestmark = pytest.mark.gpu

VALUES = {"nan": np.nan, "inf": np.inf, "minus-inf": -np.inf, "zero": 0.0, "minus-zero": -0.0, "subnormal": 5e-324,
          "tiny": 1e-290, "huge": 1e300, "negative": -2.5}


@pytest.mark.parametrize("where", ["qty", "weight"])
@pytest.mark.parametrize("value", VALUES)
def test_special_factor(cuda, value, where):
    nx, ny = 90, 111
    rng = np.random.default_rng(len(value))
    rot = orientation(rng.standard_normal(3), rng.standard_normal(3))[0]
    x = np.array([[0.0, 0.0, 0.0], [0.31, -0.22, 0.1], [-0.3, 0.3, 0.0], [0.05, 0.02, 0.0]])
    q, w = rng.uniform(0.5, 2.0, 4), rng.uniform(0.5, 2.0, 4)
    (q if where == "qty" else w)[0] = VALUES[value]
    s = CellSplat(x, [0.09, 0.05, 0.013, 0.02], q, w, device=cuda)
    for g, r in zip(sums_image(s, rot, nx, ny), subcell_image(s, rot, nx, ny)):
        if value == "nan":
            assert torch.equal(torch.isnan(g), torch.isnan(r))
        finite = torch.isfinite(r)
        assert torch.equal(torch.isfinite(g), finite)
        g, r = g[finite], r[finite]
        # (cells of both signs cancel in few pixels: relative to the largest there)
        scale = r.abs() if value != "negative" else r.abs().max()
        assert bool(((g - r).abs() <= 1e-12 * scale + 1e-24 * float(r.abs().max())).all())
