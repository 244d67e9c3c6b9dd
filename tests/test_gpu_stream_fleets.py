"""A frame stream whose fleets are used for other work between its frames:
other sizes, another form."""
import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu


def _frame(rng, h, w):
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[..., 3] = 255
    return img


@pytest.mark.parametrize("form", [cvm.FORM_EXACT, cvm.FORM_FAST])
def test_frames_between_other_sizes(form):
    rng = np.random.default_rng(11)
    h, w = 240, 427
    frames = [_frame(rng, h, w) for _ in range(3)]
    other = _frame(rng, 131, 300)
    cuts = [(9, 14, 12, 17), (40, 60, 33, 21), (100, 200, 16, 48)]
    ms = [cvm.NewMatcher(frames[0][y:y + th, x:x + tw].copy()) for y, x, th, tw in cuts]
    gs = [cvm.NewGrayMatcher(np.ascontiguousarray(frames[1][y:y + th, x:x + tw, 1])) for y, x, th, tw in cuts]
    auto = cvm.SetAutotune(False)
    try:
        color, gray = cvm.NewFleet(ms), cvm.NewFleet(gs)
        for f in (color, gray):
            f.SetForm(form)
        s = cvm.NewStream(color, gray, w, h)
        assert s.info()[0]

        def run(frame):
            s.push(frame)
            c, g, _ = s.pull()
            return [tuple(r) for r in c], [tuple(r) for r in g]

        want = [run(f) for f in frames]
        assert [r[4:6] for r in want[0][0]] == [(x, y) for y, x, _, _ in cuts]
        for k in range(6):
            color.FindAll(other)
            gray.FindAll(np.ascontiguousarray(other[..., 0]))
            if k == 3:
                for f in (color, gray):
                    f.SetForm(cvm.FORM_FAST if form == cvm.FORM_EXACT else cvm.FORM_EXACT)
            assert run(frames[k % 3]) == want[k % 3]
    finally:
        cvm.SetAutotune(auto)
