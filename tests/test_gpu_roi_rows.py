"""Regions of interest in the inverse rows, every row length they take: the
extrema of regions that partition a frame's results, at odd boundaries, merge
into the extrema of the whole frame; and regions cost less than the frame."""
import ctypes as C

import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu

# (log2 row length, template width, height, frame width, height)
SIZES = [(7, 16, 16, 320, 131), (8, 64, 48, 640, 121), (9, 57, 41, 1281, 203), (10, 96, 32, 1921, 131),
         (11, 256, 40, 3841, 113)]


def _merge(parts):
    lo = min(parts, key=lambda r: (r[0], r[2], r[1]))
    hi = min(parts, key=lambda r: (-r[3], r[5], r[4]))
    return lo[:3] + hi[3:]


@pytest.mark.parametrize("gray", [False, True])
@pytest.mark.parametrize("form", [cvm.FORM_EXACT, cvm.FORM_FAST, cvm.FORM_MIXED])
@pytest.mark.parametrize("size", SIZES, ids=[str(s[0]) for s in SIZES])
def test_regions_merge_into_the_frame(size, form, gray):
    log2n, tw, th, w, h = size
    plan = (C.c_int32 * 6)()
    cvm.lib().cvm_plan(tw, th, w - tw + 1, h - th + 1, plan)
    assert plan[0] == 1 << log2n
    rng = np.random.default_rng(log2n)
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[..., 3] = 255
    img[: h // 3, : w // 3] = 77
    tpl = img[h - th - 1:h - 1, 7:7 + tw].copy()
    img[3:3 + th, w - tw - 2:w - 2] = tpl  # two places of the same score
    frame = np.ascontiguousarray(img[..., 1]) if gray else img
    m = cvm.NewGrayMatcher(np.ascontiguousarray(tpl[..., 1])) if gray else cvm.NewMatcher(tpl)
    rw, rh = w - tw + 1, h - th + 1
    xs = [0, 1, rw // 3 | 1, rw // 2, rw - 3, rw]
    ys = [0, 3, rh // 2 | 1, rh - 1, rh]
    boxes = [(xs[i], ys[j], xs[i + 1], ys[j + 1]) for j in range(len(ys) - 1) for i in range(len(xs) - 1)]
    auto = cvm.SetAutotune(False)
    try:
        fleet = cvm.NewFleet([m] * len(boxes))
        fleet.SetForm(form)
        fleet.SetStats(cvm.STATS_KERNEL)
        whole = [tuple(r) for r in fleet.FindAll(frame)]
        assert len(set(whole)) == 1
        for i, (x0, y0, x1, y1) in enumerate(boxes):
            fleet.SetROI(i, x0, y0, x1 - x0 + tw - 1, y1 - y0 + th - 1)
        parts = [tuple(r) for r in fleet.FindAll(frame)]
    finally:
        cvm.SetAutotune(auto)
    for (x0, y0, x1, y1), r in zip(boxes, parts):
        assert x0 <= r[1] < x1 and y0 <= r[2] < y1 and x0 <= r[4] < x1 and y0 <= r[5] < y1
    assert _merge(parts) == whole[0]


@pytest.mark.parametrize("form", [cvm.FORM_EXACT, cvm.FORM_FAST])
def test_a_region_costs_less_than_the_frame(form):
    import torch
    rng = np.random.default_rng(2)
    h, w = 720, 1280
    img = rng.integers(0, 256, (h, w), dtype=np.uint8)
    frame = torch.from_numpy(img).cuda()
    ms = []
    for _ in range(40):
        tw, th = int(rng.integers(16, 120)), int(rng.integers(16, 120))
        y, x = int(rng.integers(0, h - th)), int(rng.integers(0, w - tw))
        ms.append(cvm.NewGrayMatcher(img[y:y + th, x:x + tw].copy()))
    fleet = cvm.NewFleet(ms)
    fleet.SetForm(form)
    fleet.SetStats(cvm.STATS_KERNEL)
    out = torch.zeros((len(ms), 6), dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream

    def ms_per_call():
        best = 1e9
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                fleet.find_all_device(frame.data_ptr(), w, w, h, out.data_ptr(), st)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) / 10)
        return best

    whole = ms_per_call()
    for i in range(len(ms)):
        fleet.SetROI(i, w // 4, h // 4, w // 2, h // 2)
    assert ms_per_call() < 0.9 * whole
