"""The exact form's window statistics on both sides of the template area whose
squared window sums fit 32 bits (area x channels x 255^2), on frames with
saturated, black and random regions: a single match and a fleet, bit for bit
against the oracle."""
import numpy as np
import pytest

import cvmatch_gb300 as cvm
import oracle

pytestmark = pytest.mark.gpu

# (channels compared, template width, height): the last area below the line and the first above it
EDGES = [(3, 179, 123), (3, 202, 109), (1, 179, 369), (1, 337, 196), (4, 127, 130), (4, 172, 96), (3, 16, 16), (1, 3, 2)]


def _scene(cn, tw, th):
    rng = np.random.default_rng(tw * th + cn)
    h, w, ch = th + 67, tw + 163, 1 if cn == 1 else 4
    img = rng.integers(0, 256, (h, w, ch), dtype=np.uint8)
    img[:th + 20, :tw + 40] = 255          # windows at the largest squared sum, and just off it
    img[th // 2, tw // 2] = 254
    img[h - 30:, :w // 2] = 0
    if ch == 4 and cn == 3:
        img[..., 3] = 255
    t = img[h - th - 3:h - 3, w - tw - 5:w - 5].copy()
    t[0, 0] = 3
    return (np.ascontiguousarray(img[..., 0]), np.ascontiguousarray(t[..., 0])) if ch == 1 else (img, t)


@pytest.mark.parametrize("cn,tw,th", EDGES)
def test_areas_around_the_line(cn, tw, th):
    area = tw * th * cn * 65025
    assert tw * th < 1000 or abs(area - 2 ** 32) < 2 ** 32 // 1000
    img, tpl = _scene(cn, tw, th)
    got, m = cvm.match_u8(img, tpl, cn)
    want, wm = oracle.match_u8(img, tpl, cn, threads=8)
    assert np.array_equal(m.view(np.uint32), wm.view(np.uint32))
    assert tuple(got) == tuple(want)
    y, x = img.shape[0] - th // 2 - 4, img.shape[1] - tw // 2 - 6
    tpls = [tpl, img[y:y + th // 2 + 1, x:x + tw // 2 + 1].copy()]
    fleet = cvm.NewFleet(*[(cvm.NewGrayMatcher if cn == 1 else cvm.NewMatcher)(t) for t in tpls])
    for r, want in zip(fleet.FindAll(img), oracle.fleet_find_all(tpls, img, threads=8)):
        assert tuple(r) == tuple(want)
