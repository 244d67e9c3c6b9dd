"""Large templates of colour matches: no step of the template's chain may grow
so that the call takes a multiple of what a fixed channel count takes; results
of the replayed, queued and device-resident calls agree."""
import ctypes as C
import time

import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu


def _scene(h, w, th, tw):
    rng = np.random.default_rng(h + tw)
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[..., 3] = 255
    return img, img[h // 3:h // 3 + th, w // 4:w // 4 + tw].copy()


@pytest.mark.parametrize("form", [cvm.FORM_EXACT, cvm.FORM_FAST])
@pytest.mark.parametrize("h,w,th,tw", [(480, 640, 64, 64), (480, 640, 65, 64), (480, 640, 128, 128), (480, 640, 129, 128),
                                       (480, 640, 256, 256), (720, 1280, 256, 256), (1080, 1920, 181, 181)])
def test_same_results(form, h, w, th, tw):
    import torch
    img, tpl = _scene(h, w, th, tw)
    d, t = torch.from_numpy(img).cuda(), torch.from_numpy(tpl).cuda()
    out = torch.zeros(6, dtype=torch.int32, device="cuda")
    before, auto = cvm.SetForm(form), cvm.SetAutotune(False)
    try:
        got = [tuple(cvm.Match(img, tpl)) for _ in range(5)]  # queued, then replayed
        rc = cvm.lib().cvm_match_device(d.data_ptr(), 4 * w, w, h, t.data_ptr(), 4 * tw, tw, th, None, out.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
    finally:
        cvm.SetForm(before)
        cvm.SetAutotune(auto)
    r = out.cpu().numpy()
    dev = (float(r[0:1].view(np.float32)[0]), int(r[1]), int(r[2]), float(r[3:4].view(np.float32)[0]), int(r[4]), int(r[5]))
    assert set(got) == {dev}
    assert dev[4:] == (w // 4, h // 3)


@pytest.mark.parametrize("h,w,th,tw", [(480, 640, 256, 256), (720, 1280, 256, 256)])
def test_a_colour_match_costs_what_three_channels_cost(h, w, th, tw):
    import torch
    img, tpl = _scene(h, w, th, tw)
    d, t = torch.from_numpy(img).cuda(), torch.from_numpy(tpl).cuda()
    out = torch.zeros(6, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    L = cvm.lib()

    def us(go):
        for _ in range(5):
            assert go() == 0
        best = 1e9
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                go()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 100)
        return best

    before, auto = cvm.SetForm(cvm.FORM_FAST), cvm.SetAutotune(False)
    try:
        three = us(lambda: L.cvm_match_u8_device(d.data_ptr(), 4 * w, w, h, t.data_ptr(), 4 * tw, tw, th, 3, 4, None,
                                                 out.data_ptr(), st))
        colour = us(lambda: L.cvm_match_device(d.data_ptr(), 4 * w, w, h, t.data_ptr(), 4 * tw, tw, th, None,
                                               out.data_ptr(), st))
        t0 = []
        for _ in range(20):
            a = time.perf_counter()
            cvm.Match(img, tpl)
            t0.append((time.perf_counter() - a) * 1e6)
    finally:
        cvm.SetForm(before)
        cvm.SetAutotune(auto)
    assert colour < 1.5 * three
    assert min(t0) < 2 * three + 60
