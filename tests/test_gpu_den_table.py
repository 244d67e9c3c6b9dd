"""Den on demand: a fast-form fleet whose inverse rows bound den over blocks
of results and form it from the frame's summed-area table only where an
extremum may be, against the same fleet with the statistics kernel -- the
same bits, at the table's edges (ragged frames, unaligned device frames and
pitches, one, three and four channels), at templates smaller and larger than
the blocks, and on contents whose bounds fail: flat panels with strokes, a
linear gradient (every score is an extremum's), one-bit noise, periodic
tiles."""
import numpy as np
import pytest

import cvmatch_gb300 as cvm

pytestmark = pytest.mark.gpu


def _content(kind, rng, h, w, ch):
    if kind == "noise":
        return rng.integers(0, 256, (h, w, ch), dtype=np.uint8)
    if kind == "onebit":
        return (128 + rng.integers(0, 2, (h, w, ch))).astype(np.uint8)
    if kind == "gradient":
        return np.repeat(((np.arange(w) * 255) // w).astype(np.uint8)[None, :, None], h, 0).repeat(ch, 2)
    if kind == "tiles":
        t = rng.integers(0, 256, (16, 16, ch), dtype=np.uint8)
        return np.tile(t, (h // 16 + 1, w // 16 + 1, 1))[:h, :w].copy()
    img = np.full((h, w, ch), 200, np.uint8)  # strokes on flat panels
    img[h // 2:, : w // 2] = 90
    for _ in range(h * w // 700):
        x, y = int(rng.integers(0, w - 9)), int(rng.integers(0, h - 9))
        if rng.random() < 0.5:
            img[y, x:x + 8] = rng.integers(0, 80, ch)
        else:
            img[y:y + 8, x] = rng.integers(0, 80, ch)
    return img


def _fleet(img, sizes, rng, gray):
    h, w = img.shape[:2]
    ms = []
    for tw, th in sizes:
        x, y = int(rng.integers(0, w - tw + 1)), int(rng.integers(0, h - th + 1))
        t = img[y:y + th, x:x + tw].copy()
        t[th // 2, tw // 2, 0] ^= 64  # not flat, and no exact copy
        ms.append(cvm.NewGrayMatcher(np.ascontiguousarray(t[..., 0])) if gray else cvm.NewMatcher(t))
    return cvm.NewFleet(ms)


def _both(find, fleet):
    got = []
    for mode in (cvm.STATS_KERNEL, cvm.STATS_EPILOGUE):
        fleet.SetStats(mode)
        find()
        got.append(np.array(find()))
    return got


SIZES = [(1, 1), (2, 3), (5, 4), (16, 16), (31, 70), (64, 33), (97, 96), (130, 12)]


@pytest.mark.parametrize("kind", ["noise", "onebit", "gradient", "tiles", "strokes"])
@pytest.mark.parametrize("h,w,cn", [(203, 390, 3), (161, 517, 4), (258, 1021, 1), (131, 2049, 3)])
def test_same_bits_as_the_statistics_kernel(kind, h, w, cn):
    rng = np.random.default_rng(h + w + cn)
    img = _content(kind, rng, h, w, 4)
    img[..., 3] = rng.integers(0, 256, (h, w)) if cn == 4 else 255
    fleet = _fleet(img, [(tw, min(th, h)) for tw, th in SIZES], rng, cn == 1)
    fleet.SetForm(cvm.FORM_FAST)
    frame = np.ascontiguousarray(img[..., 0]) if cn == 1 else img

    def find():
        return np.array([tuple(r) for r in fleet.FindAll(frame)], np.float64)

    kernel, table = _both(find, fleet)
    assert np.array_equal(kernel, table), np.argwhere(kernel != table)[:5]


@pytest.mark.parametrize("offset,pad", [(0, 0), (4, 0), (1, 3), (16, 20)])
def test_device_frames_of_any_alignment(offset, pad):
    import torch
    h, w = 143, 611
    rng = np.random.default_rng(offset + pad)
    img = _content("noise", rng, h, w, 4)
    img[..., 3] = 255
    fleet = _fleet(img, SIZES, rng, False)
    fleet.SetForm(cvm.FORM_FAST)
    pitch = 4 * w + pad
    buf = np.zeros(offset + h * pitch, np.uint8)
    for y in range(h):
        buf[offset + y * pitch: offset + y * pitch + 4 * w] = img[y].reshape(-1)
    d = torch.from_numpy(buf).cuda()
    out = torch.zeros((len(fleet), 6), dtype=torch.int32, device="cuda")

    def find():
        fleet.find_all_device(d.data_ptr() + offset, pitch, w, h, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return out.cpu().numpy().copy()

    kernel, table = _both(find, fleet)
    assert np.array_equal(kernel, table)
    host = np.array([tuple(r) for r in fleet.FindAll(img)], np.float64)
    assert np.array_equal(host[:, [1, 2, 4, 5]], table[:, [1, 2, 4, 5]])


def test_the_first_frame_chooses():
    """A fleet left to itself gives the same results whatever it chose."""
    rng = np.random.default_rng(5)
    for kind in ("noise", "strokes"):
        img = _content(kind, rng, 300, 500, 4)
        img[..., 3] = 255
        fleet = _fleet(img, [(12, 14), (20, 17), (25, 30), (16, 16)], rng, False)
        fleet.SetForm(cvm.FORM_FAST)
        own = [tuple(r) for r in fleet.FindAll(img)]
        fleet.SetStats(cvm.STATS_KERNEL)
        assert own == [tuple(r) for r in fleet.FindAll(img)]
