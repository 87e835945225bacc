"""The stamps' summed-area tables (ytgb_offaxis_sums) against exact integer sums:
every entry of every level, at the edges of the warps' 32 columns and of the
runs of rows."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest
import torch

from yt_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsx,nsy,max_depth", [(1, 1, 2), (4, 4, 2), (15, 17, 5), (16, 31, 5), (17, 32, 6), (33, 33, 7),
                                               (3, 65, 7), (70, 5, 7)])
def test_tables(cuda, nsx, nsy, max_depth):
    rng = np.random.default_rng(nsx * 100 + nsy)
    stamp = np.zeros((max_depth, nsx, nsy))
    for d in range(max_depth):
        jm, km = min(nsx, 1 << d), min(nsy, 1 << d)
        v = rng.random((jm, km)) * 2.0 ** -rng.integers(0, 40, (jm, km)) * (rng.random((jm, km)) < 0.8)
        v[0, 0] = 1.0
        stamp[d, :jm, :km] = v / v.sum()
    L = _lib.lib()
    size = C.c_int64()
    assert L.ytgb_offaxis_sums_bytes(nsx, nsy, max_depth, C.byref(size)) == _lib.OK
    guard = 4096
    sums = torch.full((size.value + guard,), 0xA5, dtype=torch.uint8, device=cuda)
    dev = torch.from_numpy(stamp).to(cuda)
    st = torch.cuda.current_stream(cuda).cuda_stream
    assert L.ytgb_offaxis_sums(dev.data_ptr(), nsx, nsy, max_depth, 50, 60, sums.data_ptr(), C.c_void_p(st)) == _lib.OK
    torch.cuda.synchronize()
    host = sums.cpu().numpy()
    assert (host[size.value:] == 0xA5).all()
    words = host[:size.value].view("<u8").reshape(-1, 2)
    at = 0
    for d in range(max_depth):
        jm, km = min(nsx, 1 << d), min(nsy, 1 << d)
        n = (jm + 1) * (km + 1)
        got = [int(lo) + (int(hi) << 64) for lo, hi in words[at:at + n]]
        at += n
        fits = False
        for shift in range(8):  # the level's unit is 2^-(126 + shift)
            want = [[0] * (km + 1) for _ in range(jm + 1)]
            for j in range(jm):
                row = 0
                for k in range(km):
                    # (a tie goes up)
                    row += int(Fraction(stamp[d, j, k]) * (1 << (126 + shift)) + Fraction(1, 2))
                    want[j + 1][k + 1] = (want[j][k + 1] + row) % (1 << 128)
            fits = fits or got == [x for r in want for x in r]
        assert fits, d
    assert at == len(words)


def test_sums_bytes_rejects_bad_arguments(cuda):
    L = _lib.lib()
    size = C.c_int64()
    assert L.ytgb_offaxis_sums_bytes(0, 4, 2, C.byref(size)) == _lib.ERR_INVALID
    assert L.ytgb_offaxis_sums_bytes(4, 4, 31, C.byref(size)) == _lib.ERR_INVALID
    assert L.ytgb_offaxis_sums_bytes(4, 4, 2, None) == _lib.ERR_INVALID
