"""Which source of den a fast-form fleet runs when it is left to itself: the
statistics kernel where blocks of results have no bound (strokes on flat
panels under small templates), where everything scores like an extremum (a
linear gradient) and for a few members on a small frame, on demand otherwise --
whatever the first frame was.  The kernels
that a call launches say which; results are the statistics kernel's."""
import ctypes as C

import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu

H, W = 540, 960


def _strokes(rng):
    img = np.full((H, W, 4), 200, np.uint8)
    img[H // 2:, : W // 2, :3] = 90
    for _ in range(H * W // 700):
        x, y = int(rng.integers(0, W - 9)), int(rng.integers(0, H - 9))
        if rng.random() < 0.5:
            img[y, x:x + 8, :3] = rng.integers(0, 80, 3)
        else:
            img[y:y + 8, x, :3] = rng.integers(0, 80, 3)
    img[..., 3] = 255
    return img


def _noise(rng):
    img = rng.integers(0, 256, (H, W, 4), dtype=np.uint8)
    img[..., 3] = 255
    return img


def _gradient():
    img = np.repeat(((np.arange(W) * 255) // W).astype(np.uint8)[None, :, None], H, 0).repeat(4, 2)
    img[..., 3] = 255
    return img


def _black():
    img = np.zeros((H, W, 4), np.uint8)
    img[..., 3] = 255
    return img


def kernels(call):
    """Names of the kernels that call() launches."""
    L = cvm.lib()
    L.cvm_profile_read.argtypes = [C.c_int, C.c_char_p, C.c_size_t, C.POINTER(C.c_double), C.POINTER(C.c_uint64)]
    name, ms, n = C.create_string_buffer(64), C.c_double(), C.c_uint64()
    L.cvm_profile_enable(1)
    try:
        call()
        out, i = set(), 0
        while L.cvm_profile_read(i, name, 64, C.byref(ms), C.byref(n)) == 0:
            if n.value:
                out.add(name.value.decode())
            i += 1
        return out
    finally:
        L.cvm_profile_enable(0)


def on_demand(fleet, frame):
    return "k_vstats" not in kernels(lambda: fleet.FindAll(frame))


def icons(rng, frame, n=12):
    ms = []
    for _ in range(n):
        tw, th = int(rng.integers(12, 30)), int(rng.integers(12, 30))
        y, x = int(rng.integers(0, H - th)), int(rng.integers(0, W - tw))
        t = frame[y:y + th, x:x + tw].copy()
        t[th // 2, tw // 2, 0] ^= 64
        ms.append(cvm.NewMatcher(t))
    return ms


def _fleet(ms):
    f = cvm.NewFleet(ms)
    f.SetForm(cvm.FORM_FAST)
    return f


@pytest.mark.parametrize("first", ["strokes", "noise", "black", "gradient"])
def test_the_choice_follows_the_frames(first):
    rng = np.random.default_rng(3)
    frames = {"strokes": _strokes(rng), "noise": _noise(rng), "black": _black(), "gradient": _gradient()}
    ms = icons(rng, frames["noise"], 64)
    auto = cvm.SetAutotune(False)
    try:
        f, kernel = _fleet(ms), _fleet(ms)
        kernel.SetStats(cvm.STATS_KERNEL)
        f.FindAll(frames[first])
        for name, demand, calls in (("strokes", False, 12), ("noise", True, 160), ("gradient", False, 160)):
            frame = frames[name]
            want = [tuple(r) for r in kernel.FindAll(frame)]
            for _ in range(calls):
                got = [tuple(r) for r in f.FindAll(frame)]
                assert got == want
            assert on_demand(f, frame) == demand, name
    finally:
        cvm.SetAutotune(auto)


def test_a_small_fleet_takes_the_kernel():
    rng = np.random.default_rng(6)
    frame = _noise(rng)[:240, :320].copy()
    f = _fleet([cvm.NewMatcher(np.ascontiguousarray(frame[20 * k:20 * k + 16, 30:60])) for k in range(3)])
    for _ in range(8):
        f.FindAll(frame)
    assert not on_demand(f, frame)


def test_a_capture_uses_what_the_frames_chose():
    import torch
    rng = np.random.default_rng(4)
    frame = _strokes(rng)
    f = _fleet(icons(rng, frame))
    d = torch.from_numpy(frame).cuda()
    out = torch.zeros((len(f), 6), dtype=torch.int32, device="cuda")

    def find():
        f.find_all_device(d.data_ptr(), 4 * W, W, H, out.data_ptr(), torch.cuda.current_stream().cuda_stream)

    find()
    torch.cuda.synchronize()
    want = out.cpu().numpy().copy()
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        find()
        s.synchronize()
        with torch.cuda.graph(g, stream=s):
            find()
    for _ in range(3):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
    assert not on_demand(f, frame)


@pytest.mark.parametrize("order", [("strokes", "noise"), ("noise", "strokes")])
def test_a_stream_follows_the_frames_pushed(order):
    rng = np.random.default_rng(5)
    frames = {"strokes": _strokes(rng), "noise": _noise(rng)}
    ms = icons(rng, frames["noise"], 64)

    def device_ms(s, frame):
        t = []
        for _ in range(21):
            s.push(frame)
            t.append(s.pull()[2])
        return sorted(t)[10]

    auto = cvm.SetAutotune(False)
    try:
        f, fixed = _fleet(ms), {}
        for mode in (cvm.STATS_KERNEL, cvm.STATS_EPILOGUE):
            g = _fleet(ms)
            g.SetStats(mode)
            fixed[mode] = (g, cvm.NewStream(g, None, W, H))
        s = cvm.NewStream(f, None, W, H)
        assert s.info()[0]
        for name in order:
            frame = frames[name]
            want = [tuple(r) for r in fixed[cvm.STATS_KERNEL][0].FindAll(frame)]
            for k in range(160):
                s.push(frame)
                if k % 3 == 0:  # two frames in flight
                    s.push(frame)
                    assert [tuple(r) for r in s.pull()[0]] == want
                assert [tuple(r) for r in s.pull()[0]] == want
            assert s.info()[0]
            assert on_demand(f, frame) == (name == "noise")
            best = min(device_ms(t, frame) for _, t in fixed.values())
            assert device_ms(s, frame) < 1.2 * best, name
    finally:
        cvm.SetAutotune(auto)
