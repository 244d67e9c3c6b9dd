"""The extrema of fleets whose CTAs post them to each other while others read:
many row-pair CTAs per member in flight at once, every row length of the
kernel, den from the statistics kernel and on demand.  The same fleet with a
region of interest over the whole frame keeps every score and cuts by nothing:
the same plan, the same bits."""
import ctypes as C

import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu

# (log2 row length, template width, height, frame width, height)
SIZES = [(7, 16, 16, 320, 700), (8, 64, 48, 640, 701), (9, 57, 41, 1281, 703), (10, 96, 32, 1921, 700),
         (11, 256, 40, 3841, 403)]


@pytest.mark.parametrize("gray", [False, True])
@pytest.mark.parametrize("form,stats", [(cvm.FORM_EXACT, None), (cvm.FORM_FAST, cvm.STATS_KERNEL),
                                        (cvm.FORM_FAST, cvm.STATS_EPILOGUE)])
@pytest.mark.parametrize("size", SIZES, ids=[str(s[0]) for s in SIZES])
def test_extrema_posted_by_ctas_in_flight(size, form, stats, gray):
    log2n, tw, th, w, h = size
    plan = (C.c_int32 * 6)()
    cvm.lib().cvm_plan(tw, th, w - tw + 1, h - th + 1, plan)
    assert plan[0] == 1 << log2n
    rng = np.random.default_rng(log2n)
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[..., 3] = 255
    img[: h // 3] = np.minimum(img[: h // 3] >> 5, 254)
    ms = []
    for k in range(6):
        y, x = int(rng.integers(0, h - th)), int(rng.integers(0, w - tw))
        t = img[y:y + th, x:x + tw].copy()
        img[h - th - 1:h - 1, 5:5 + tw] = t          # a second place with the same score for the last one
        ms.append(cvm.NewGrayMatcher(np.ascontiguousarray(t[..., 0])) if gray else cvm.NewMatcher(t))
    frame = np.ascontiguousarray(img[..., 0]) if gray else img
    auto = cvm.SetAutotune(False)
    try:
        fleet = cvm.NewFleet(ms)
        fleet.SetForm(form)
        if stats is not None:
            fleet.SetStats(stats)
        got = [[tuple(r) for r in fleet.FindAll(frame)] for _ in range(4)]
        for i in range(6):
            fleet.SetROI(i, 0, 0, w, h)
        want = [tuple(r) for r in fleet.FindAll(frame)]
    finally:
        cvm.SetAutotune(auto)
    for g in got:
        assert g == want
