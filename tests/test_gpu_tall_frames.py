"""Fast-form fleets on frames of more than 4 * 65,535 rows: the summed-area
table's row blocks outnumber a grid's y dimension."""
import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gray,w,h", [(False, 260, 262_141), (False, 24, 262_205), (True, 301, 270_000)])
def test_fleet(gray, w, h):
    rng = np.random.default_rng(h)
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[..., 3] = 255
    at = [(5, h - 12), (3, 131_000), (7, 40)]
    frame = np.ascontiguousarray(img[..., 0]) if gray else img
    ms = [(cvm.NewGrayMatcher if gray else cvm.NewMatcher)(np.ascontiguousarray(frame[y:y + 9, x:x + 11])) for x, y in at]
    auto = cvm.SetAutotune(False)
    try:
        fleet = cvm.NewFleet(ms)
        fleet.SetForm(cvm.FORM_FAST)
        own = [tuple(r) for r in fleet.FindAll(frame)]
        fleet.SetStats(cvm.STATS_KERNEL)
        assert own == [tuple(r) for r in fleet.FindAll(frame)]
    finally:
        cvm.SetAutotune(auto)
    assert [r[4:6] for r in own] == at
