"""Fast-form fleets on frames without deviation, or with little of it: black
and blank frames, letterbox bars, one small object.  Den on demand gives the
statistics kernel's results, and costs no more than it there."""
import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu


def _frame(kind, rng, h, w):
    img = np.zeros((h, w, 4), np.uint8)
    img[..., 3] = 255
    if kind == "white":
        img[..., :3] = 255
    elif kind == "bars":
        img[h // 4: 3 * h // 4, :, :3] = rng.integers(0, 256, (3 * h // 4 - h // 4, w, 3))
    elif kind == "object":
        img[..., :3] = 100
        img[h // 2:h // 2 + 14, w // 3:w // 3 + 21, :3] = rng.integers(0, 256, (14, 21, 3))
    elif kind == "pixel":
        img[h - 2, w - 2, 1] = 1
    elif kind == "alpha":
        img[..., 3] = 128
        img[h // 3, w // 3, 3] = 129
    return img


def _fleet(tpls, gray):
    f = cvm.NewFleet([(cvm.NewGrayMatcher(np.ascontiguousarray(t[..., 0])) if gray else cvm.NewMatcher(t)) for t in tpls])
    f.SetForm(cvm.FORM_FAST)
    return f


@pytest.mark.parametrize("gray", [False, True])
@pytest.mark.parametrize("kind", ["black", "white", "bars", "object", "pixel", "alpha"])
@pytest.mark.parametrize("h,w", [(203, 390), (401, 1021)])
def test_results(kind, gray, h, w):
    rng = np.random.default_rng(h)
    tpls = [rng.integers(0, 256, (th, tw, 4), dtype=np.uint8) for tw, th in ((5, 4), (16, 16), (64, 33), (97, 96), (21, 14))]
    img = _frame(kind, rng, h, w)
    tpls[-1] = img[h // 2:h // 2 + 14, w // 3:w // 3 + 21].copy()
    tpls[-1][0, 0, 0] ^= 1  # (flat frames: not a flat template)
    frame = np.ascontiguousarray(img[..., 0]) if gray else img
    got = []
    auto = cvm.SetAutotune(False)
    try:
        for mode in (cvm.STATS_KERNEL, cvm.STATS_EPILOGUE):
            f = _fleet(tpls, gray)
            f.SetStats(mode)
            got.append([tuple(r) for r in f.FindAll(frame)])
    finally:
        cvm.SetAutotune(auto)
    assert got[0] == got[1]
    if kind in ("black", "white"):
        assert got[1][:4] == [(0.0, 0, 0, 0.0, 0, 0)] * 4


def test_a_black_frame_costs_no_more():
    import torch
    rng = np.random.default_rng(1)
    h, w = 720, 1280
    frame = torch.from_numpy(_frame("black", rng, h, w)).cuda()
    tpls = [rng.integers(0, 256, (int(rng.integers(16, 90)), int(rng.integers(16, 120)), 4), dtype=np.uint8) for _ in range(24)]
    out = torch.zeros((24, 6), dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    t = []
    for mode in (cvm.STATS_KERNEL, cvm.STATS_EPILOGUE):
        f = _fleet(tpls, False)
        f.SetStats(mode)
        best = 1e9
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                f.find_all_device(frame.data_ptr(), 4 * w, w, h, out.data_ptr(), st)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        t.append(best)
    assert t[1] < 1.1 * t[0], t
