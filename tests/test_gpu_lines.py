"""The inverse rows with a thread group per row pair, every length they take
(2^7 .. 2^11) at ragged widths and odd row counts: the exact form bit for
bit against the oracle, and in both forms the extrema of a match without a
score map (results that cannot be extrema skip their quotient) equal to the
first minimum and maximum of the same match's map.  The frames hold flat and
near-flat patches, the template twice, and its negative."""
import ctypes as C

import numpy as np
import pytest

import cvmatch_gb300 as cvm
import oracle
from oracle import fp64

pytestmark = pytest.mark.gpu

# (log2 row length, template width, height, frame width, height)
SIZES = [(7, 16, 16, 320, 131), (7, 31, 7, 333, 95), (8, 64, 48, 640, 121), (9, 57, 41, 1281, 203),
         (10, 96, 32, 1921, 131), (10, 33, 30, 1021, 99), (11, 256, 40, 3841, 113)]


def _scene(seed, w, h, tw, th, ch):
    rng = np.random.default_rng(seed)
    img = rng.integers(0, 256, (h, w, ch), dtype=np.uint8)
    img[:h // 3, :w // 3] = 77                                     # flat windows: den = 0
    img[h // 3:h // 2, :w // 4] = 90 + rng.integers(0, 2, (h // 2 - h // 3, w // 4, ch))  # near-flat ones
    t = img[h - th - 1:h - 1, w - tw - 1:w - 1].copy()
    img[h - th:h, w // 2:w // 2 + tw] = t                          # a second exact copy
    img[0:th, w - tw:w] = 255 - t
    if ch == 1:
        return np.ascontiguousarray(img[..., 0]), np.ascontiguousarray(t[..., 0])
    return img, t


@pytest.mark.parametrize("cn", [1, 3, 4])
@pytest.mark.parametrize("size", SIZES, ids=["-".join(map(str, s)) for s in SIZES])
def test_extrema_without_a_map(size, cn):
    log2n, tw, th, w, h = size
    plan = (C.c_int32 * 6)()
    cvm.lib().cvm_plan(tw, th, w - tw + 1, h - th + 1, plan)
    assert plan[0] == 1 << log2n
    img, tpl = _scene(7 * log2n + cn, w, h, tw, th, 1 if cn == 1 else 4)
    auto, form = cvm.SetAutotune(False), cvm.SetForm(cvm.FORM_EXACT)
    try:
        got, m = cvm.match_u8(img, tpl, cn)
        want, wm = oracle.match_u8(img, tpl, cn, threads=8)
        assert np.array_equal(m.view(np.uint32), wm.view(np.uint32))
        assert tuple(got) == tuple(want)
        assert tuple(cvm.match_u8(img, tpl, cn, want_map=False)[0]) == tuple(want)
        cvm.SetForm(cvm.FORM_FAST)
        fast, fm = cvm.match_u8(img, tpl, cn)
        lean, _ = cvm.match_u8(img, tpl, cn, want_map=False)
    finally:
        cvm.SetForm(form)
        cvm.SetAutotune(auto)
    lo, hi = np.unravel_index(int(np.argmin(fm)), fm.shape), np.unravel_index(int(np.argmax(fm)), fm.shape)
    first = (float(fm[lo]), int(lo[1]), int(lo[0]), float(fm[hi]), int(hi[1]), int(hi[0]))
    assert tuple(fast) == first
    assert tuple(lean) == first
    assert float(np.abs(fm - fp64.ref_match_f64(img, tpl, cn)).max()) <= 1e-4
