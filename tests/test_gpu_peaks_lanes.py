"""Occurrences where a warp's lanes scan their own windows (many candidates,
small windows) and where the warp takes its few candidates one by one: both
sides of the line, against the recipe; and plateaus of equal scores, on which
every result is a candidate, cost no more than a few times what noise does."""
import ctypes as C

import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu


def _peaks(d, w, h, thresh, rx, ry, xy, n):
    import torch
    rc = cvm.lib().cvm_peaks_device(d.data_ptr(), w, h, C.c_float(thresh), rx, ry, xy.data_ptr(), xy.shape[0], n.data_ptr(),
                                    torch.cuda.current_stream().cuda_stream)
    assert rc == 0


@pytest.mark.parametrize("share", [1.0, 0.4, 0.1, 0.01])
@pytest.mark.parametrize("w,h,rx,ry", [(300, 41, 1, 1), (257, 30, 2, 2), (290, 33, 0, 9), (290, 33, 1, 13), (270, 37, 9, 0),
                                       (300, 40, 5, 5), (301, 44, 16, 15), (300, 60, 40, 30)])
def test_recipe(w, h, rx, ry, share):
    import torch
    rng = np.random.default_rng(w + 10 * rx + ry)
    m = np.where(rng.random((h, w)) < share, np.float32(0.75), rng.random((h, w), dtype=np.float32) * np.float32(0.5))
    m[h // 2, w // 3] = 0.875          # one above the plateau, and NaN scores beside it
    m[h // 3, ::37] = np.nan
    want = []
    for y in range(h):
        for x in range(w):
            v = m[y, x]
            if v < 0.6:
                continue
            if not (m[max(0, y - ry):y + ry + 1, max(0, x - rx):x + rx + 1] > v).any():
                want.append((x, y))
    d = torch.from_numpy(m).cuda()
    for cap in (len(want) + 3, max(1, len(want) - 5)):
        xy = torch.full((cap, 2), -7, dtype=torch.int32, device="cuda")
        n = torch.zeros(1, dtype=torch.int32, device="cuda")
        _peaks(d, w, h, 0.6, rx, ry, xy, n)
        got = xy.cpu().numpy()
        k = min(cap, len(want))
        assert int(n) == len(want)
        assert [tuple(int(v) for v in p) for p in got[:k]] == want[:k]
        assert (got[k:] == -7).all()


def test_plateaus_cost_what_noise_does():
    import torch
    h, w = 769, 1249
    xy = torch.zeros((1000, 2), dtype=torch.int32, device="cuda")
    n = torch.zeros(1, dtype=torch.int32, device="cuda")
    t = {}
    for name, m in (("noise", torch.rand((h, w), device="cuda")), ("plateau", torch.zeros((h, w), device="cuda"))):
        for _ in range(5):
            _peaks(m, w, h, -1.0, 1, 1, xy, n)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(20):
            _peaks(m, w, h, -1.0, 1, 1, xy, n)
        b.record()
        torch.cuda.synchronize()
        t[name] = a.elapsed_time(b)
    assert t["plateau"] < 3 * t["noise"], t
