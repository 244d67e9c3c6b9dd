"""One-shot host calls of one shape over and over: from the third on a thread
replays the shape's launches as a graph.  Every call has other pixels, in other
buffers, at other row strides and alignments; shapes take each other's places
in the thread's few; forms change between calls; threads call at once.  All
results equal the oracle's (exact form) or the first, queued call's (fast)."""
import threading

import numpy as np
import pytest

import cvmatch_gb300 as cvm
import oracle

pytestmark = pytest.mark.gpu


def _image(rng, h, w, ch, offset, pad):
    """h x w (x ch) pixels at a byte offset, rows pad bytes apart."""
    row = w * ch + pad
    buf = rng.integers(0, 256, offset + h * row, dtype=np.uint8)
    a = np.lib.stride_tricks.as_strided(buf[offset:], (h, w, ch), (row, ch, 1))
    if ch == 4:
        a[..., 3] = 255
        return a
    return a[..., 0]


CASES = [("gray", 90, 131, 9, 14), ("gray", 300, 700, 40, 33), ("rgba2gray", 120, 200, 16, 20),
         ("rgba2gray", 260, 301, 31, 27), ("rgba", 97, 160, 12, 17), ("rgba", 300, 500, 24, 40)]
SHIFTS = [(0, 0), (4, 12), (1, 3), (16, 16), (3, 0), (8, 8)]


def _call(kind, img, tpl):
    return cvm.Match(img, tpl) if kind == "rgba" else cvm.MatchGray(img, tpl)


def _want(kind, img, tpl):
    if kind == "rgba2gray":
        img, tpl = oracle.rgba_to_gray(np.ascontiguousarray(img)), oracle.rgba_to_gray(np.ascontiguousarray(tpl))
    img, tpl = np.ascontiguousarray(img), np.ascontiguousarray(tpl)
    return tuple(oracle.match_u8(img, tpl, 3 if kind == "rgba" else 1, threads=8, want_map=False)[0])


def _rounds(kind, h, w, th, tw, seed):
    ch = 1 if kind == "gray" else 4
    rng = np.random.default_rng(seed)
    for offset, pad in SHIFTS:
        img, tpl = _image(rng, h, w, ch, offset, pad), _image(rng, th, tw, ch, pad % 5, offset)
        y, x = int(rng.integers(0, h - th)), int(rng.integers(0, w - tw))
        img[y:y + th, x:x + tw] = tpl
        yield img, tpl


@pytest.mark.parametrize("kind,h,w,th,tw", CASES)
def test_repeated_calls(kind, h, w, th, tw):
    for img, tpl in _rounds(kind, h, w, th, tw, h + w):
        assert tuple(_call(kind, img, tpl)) == _want(kind, img, tpl)


def test_shapes_forms_maps_and_occurrences_in_turn():
    rng = np.random.default_rng(3)
    before = cvm.SetForm(cvm.FORM_EXACT)
    try:
        for _ in range(5):
            for k in range(6):  # more shapes than a thread keeps
                h, w = 60 + 7 * k, 90 + 11 * k
                img, tpl = rng.integers(0, 256, (h, w), dtype=np.uint8), rng.integers(0, 256, (9, 12), dtype=np.uint8)
                img[20:29, 30:42] = tpl
                for form in (cvm.FORM_EXACT, cvm.FORM_FAST):
                    cvm.SetForm(form)
                    got, m = cvm.match_u8(img, tpl, 1)
                    assert got[4:] == (30, 20) and tuple(cvm.match_u8(img, tpl, 1, want_map=False)[0]) == tuple(got)
                    if form == cvm.FORM_EXACT:
                        want, wm = oracle.match_u8(img, tpl, 1)
                        assert tuple(got) == tuple(want) and np.array_equal(m.view(np.uint32), wm.view(np.uint32))
            rgba = rng.integers(0, 256, (80, 120, 4), dtype=np.uint8)
            rgba[..., 3] = 255
            cvm.SetForm(cvm.FORM_EXACT)
            at, n = cvm.MatchMapPeaks(rgba, rgba[10:22, 50:66].copy(), 0.99, 4, 4)
            assert n == 1 and at == [(50, 10)]
    finally:
        cvm.SetForm(before)


def test_alpha_decides_the_channels_of_each_call():
    rng = np.random.default_rng(8)
    for i in range(8):
        img = rng.integers(0, 256, (110, 150, 4), dtype=np.uint8)
        if i % 2 == 0:
            img[..., 3] = 200
        tpl = img[30:50, 60:90].copy()
        want = oracle.match_u8(img, tpl, 3 if i % 2 == 0 else 4, want_map=False)[0]
        assert tuple(cvm.Match(img, tpl)) == tuple(want)


def test_threads():
    errors = []

    def work(seed):
        try:
            for kind, h, w, th, tw in CASES[::2]:
                for img, tpl in _rounds(kind, h, w, th, tw, seed):
                    assert tuple(_call(kind, img, tpl)) == _want(kind, img, tpl)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(100 + i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
