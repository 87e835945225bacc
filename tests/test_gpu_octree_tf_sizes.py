"""Transfer functions on the octree path whose tables take the shared memory
around 48 KB (1,024 bins of a ColorTransferFunction, 3,072 of one table and
768 of four are 48 KB exactly): every one launches and gives the oracle's image."""
import numpy as np
import pytest
import torch

from oracle import cpu as ocpu
from test_gpu_octree import LIGHT, dataset
from yt_gb300 import _lib, testing
from yt_gb300.camera import Camera
from yt_gb300.octree import OctreeVolume, render_octree
from yt_gb300.render import relative_error
from yt_gb300.transfer_functions import ColorTransferFunction, MultiVariateTransferFunction, TransferFunction, pack

pytestmark = pytest.mark.gpu


def colour_tf(bounds, nbins):
    tf = ColorTransferFunction(bounds, nbins=nbins)
    for loc, wd, rgba in testing.ctf_layers(bounds, 4):
        tf.add_gaussian(loc, wd, list(rgba))
    return tf


def one_table_tf(bounds, nbins):
    tf = MultiVariateTransferFunction()
    t = TransferFunction(bounds, nbins)
    t.add_gaussian(0.5 * (bounds[0] + bounds[1]), 0.02 * (bounds[1] - bounds[0]), 0.7)
    tf.add_field_table(t, 0)
    tf.link_channels(0, [0, 1, 2, 3])
    return tf


@pytest.mark.parametrize("make,kind,nbins", [
    *[(colour_tf, _lib.VOLUME_RENDER, n) for n in (1021, 1022, 1023, 1024, 1025, 4096)],
    *[(one_table_tf, _lib.VOLUME_RENDER, n) for n in (3070, 3071, 3072, 3073)],
    *[(colour_tf, _lib.LIGHT_SOURCE, n) for n in (767, 768, 769, 3200)]])
def test_table_sizes_launch(cuda, make, kind, nbins):
    depth, ipos, lvl, cells, oc, _ = dataset(base=2, top=4)
    tf = make((float(cells[:, :8].min()), float(cells[:, :8].max())), nbins)
    cam = Camera((0.3, 1.45, -0.9), (0.5, 0.5, 0.5), (1.3, 1.3, 1.3), (24, 20), lens_type="perspective")
    light = LIGHT if kind == _lib.LIGHT_SOURCE else None
    img = torch.zeros((24, 20, 4), dtype=torch.float64, device=cuda)
    error = torch.zeros(1, dtype=torch.int32, device=cuda)
    render_octree(OctreeVolume(oc, cells, cuda), cam.device_view(), kind, img, tf=pack(tf), error=error, light=light)
    torch.cuda.synchronize()
    assert int(error.item()) == 0
    p = cam.sampler_params()
    ld, rgba = light if light else ((1.0, 1.0, 1.0), (1.0, 1.0, 1.0, 1.0))
    s = ocpu.OracleSampler("light_source" if light else "volume_render", p["vp_pos"], p["vp_dir"], p["center"],
                           p["bounds"], p["image"], p["x_vec"], p["y_vec"], p["width"], lens_type=p["lens_type"],
                           camera_data=p["camera_data"], tf=tf, light_dir=ld, light_rgba=rgba)
    ocpu.render_octree(s, cells, ocpu.OracleOctree(depth, np.zeros(3), np.ones(3), ipos, lvl))
    assert relative_error(img.cpu().numpy(), p["image"], channels=(0, 1, 2))[0] <= 1e-5
    assert float(img.abs().max()) > 0
