"""The device gather of host float64 fields around the sizes where its blocks
and passes change: one value, a pass of 256 x 8 values and its neighbours, and
fields shared by several blocks beside small ones."""
import numpy as np
import pytest

from yt_gb300.volume import BrickSet, device_reads_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2), (255, 256, 257), (2047, 2048, 2049), (4095, 4097, 5), (70001, 3, 8193),
                                   (300007, 1)])
@pytest.mark.parametrize("with_lo", [False, True])
def test_gather_sizes(cuda, sizes, with_lo):
    if not device_reads_host(cuda):
        pytest.skip("the device cannot read pageable host memory")
    rng = np.random.default_rng(sizes[0])
    # one cell each and more values than it needs: the arena takes every value
    bricks = [([rng.standard_normal(n + 7)], None, np.zeros(3), np.ones(3), np.array([1, 1, 1])) for n in sizes]
    bricks[0][0][0][:1] = np.inf
    bs = BrickSet(bricks, device=cuda, with_lo=with_lo, direct=True)
    off = bs.desc_host["data_offset"]
    data = bs.data.cpu().numpy()
    for k, (d, *_) in enumerate(bricks):
        want = d[0].astype(np.float32)
        assert np.array_equal(data[off[k]: off[k] + want.size], want)
        if with_lo:
            lo = np.where(np.isfinite(d[0]), (d[0] - want.astype(np.float64)).astype(np.float32), 0.0)
            assert np.array_equal(bs.data_lo.cpu().numpy()[off[k]: off[k] + want.size], lo)
