"""The widest frames whose row prefixes fit a CTA's shared memory, by channel
count (227 KB: 8, 12, 16 and 20 bytes a column), and narrow ones beside them,
bit for bit against the oracle."""
import numpy as np
import pytest

import cvmatch_gb300 as cvm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cn,ch,w", [(1, 1, 28900), (2, 2, 19300), (2, 2, 14600), (2, 4, 16001), (2, 2, 301), (2, 3, 64),
                                     (3, 3, 14400), (3, 4, 14401), (4, 4, 11500)])
def test_exact_scores(cn, ch, w):
    rng = np.random.default_rng(w)
    img = rng.integers(0, 256, (19, w, ch), dtype=np.uint8)
    tpl = img[4:13, w // 2:w // 2 + 11].copy()
    if ch == 1:
        img, tpl = np.ascontiguousarray(img[..., 0]), np.ascontiguousarray(tpl[..., 0])
    got, m = cvm.match_u8(img, tpl, cn)
    want, wm = oracle.match_u8(img, tpl, cn, threads=8)
    assert tuple(got) == tuple(want)
    assert np.array_equal(m.view(np.uint32), wm.view(np.uint32))
