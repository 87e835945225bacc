"""Transfer functions whose tables take the shared memory around 48 KB with
the tile's own (23 to 25.6 KB of tables) and far beyond: the single-view and
the batch kernel launch and give the same image."""
import numpy as np
import pytest
import torch

from yt_gb300 import _lib, workloads
from yt_gb300.batch import Batch, Job
from yt_gb300.camera import Camera
from yt_gb300.render import Renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins", [256, 480, 496, 512, 533, 534, 1024, 4096])
def test_table_sizes_launch(cuda, nbins):
    w = workloads.uniform_vr(n=12, res=24)
    b0, b1 = w.tf.x_bounds
    r = Renderer(w.bricks, workloads.color_tf((float(b0), float(b1)), 3, nbins=nbins), device=cuda, kdtree=w.kdtree)
    cam = Camera((1.3, 0.2, -0.7), (0.5, 0.5, 0.5), 1.0, (24, 17), lens_type="perspective")
    one = r.render(cam, kind=_lib.VOLUME_RENDER)
    r.check()
    b = Batch([Job(r, cam)], device=cuda)
    b.launch()
    torch.cuda.synchronize()
    b.check()
    assert torch.equal(one, b.images[0])
    assert np.isfinite(one.cpu().numpy()).all() and float(one.abs().max()) > 0
