"""Every occurrence of a device map against the recipe written out in numpy
(cvmatch_test.go:324-381): windows of no, one and many neighbours, wider than
the map, plateaus of equal scores, NaN scores, widths about the blocks of 256
and the words of 32, and lists cut at the caller's capacity."""
import ctypes as C

import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu


def _recipe(m, thresh, rx, ry):
    h, w = m.shape
    out = []
    for y in range(h):
        for x in range(w):
            v = m[y, x]
            if v < thresh:
                continue
            win = m[max(0, y - ry):y + ry + 1, max(0, x - rx):x + rx + 1]
            if not (win > v).any():
                out.append((x, y))
    return out


@pytest.mark.parametrize("kind", ["noise", "plateaus", "nan", "smooth"])
@pytest.mark.parametrize("w,h,rx,ry", [(1, 1, 3, 3), (31, 9, 0, 0), (33, 20, 1, 0), (255, 12, 0, 2), (257, 17, 40, 9),
                                       (300, 40, 16, 16), (64, 30, 1000, 1000)])
def test_recipe(kind, w, h, rx, ry):
    import torch
    rng = np.random.default_rng(w * h + rx)
    m = rng.standard_normal((h, w)).astype(np.float32)
    if kind == "plateaus":
        m = np.round(m).astype(np.float32)
    elif kind == "nan":
        m[rng.random((h, w)) < 0.1] = np.nan
    elif kind == "smooth":
        m = np.cumsum(np.cumsum(m, 0), 1).astype(np.float32) / (w + h)
    want = _recipe(m, 0.2, rx, ry)
    d = torch.from_numpy(m).cuda()
    for cap in (len(want) + 5, max(1, len(want) // 2)):
        xy = torch.full((cap, 2), -7, dtype=torch.int32, device="cuda")
        n = torch.zeros(1, dtype=torch.int32, device="cuda")
        rc = cvm.lib().cvm_peaks_device(d.data_ptr(), w, h, C.c_float(0.2), rx, ry, xy.data_ptr(), cap, n.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        got = xy.cpu().numpy()
        assert int(n) == len(want)
        k = min(cap, len(want))
        assert [tuple(int(v) for v in p) for p in got[:k]] == want[:k]
        assert (got[k:] == -7).all()
