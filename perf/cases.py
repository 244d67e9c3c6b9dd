"""The calls this package is measured on: what a user's program has it do.

Every case goes through the public entry points -- the Python API
(MatchGray, Match, MatchMapPeaks, Matcher, Fleet, Stream) on host arrays,
and the device-resident entry points (cvm_match_device,
cvm_match_u8_device, find_device, find_all_device) on buffers that are on
the GPU already.  Scenes are camera-like frames (1/f amplitude noise, flat
rectangles, colour and sensor noise) or user-interface frames (flat panels
and thin strokes); templates are crops with a brightness shift, or absent
from the frame, in the shares of the benchmark's fleet.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import cvmatch_gb300 as cvm

FORMS = {"exact": cvm.FORM_EXACT, "fast": cvm.FORM_FAST}


def listed():
    return [
        # a screen reader's small icon on a small gray capture: the smallest
        # call, where launches and host work count
        {"name": "gray_320x200_host", "kind": "gray", "form": "exact", "scene": "camera", "w": 320, "h": 200,
         "tw": 16, "th": 16, "rgba": False},
        # MatchGray of RGBA captures, both converted in the call (the first benchmark configuration)
        {"name": "gray_640x480_host", "kind": "gray", "form": "exact", "scene": "camera", "w": 640, "h": 480,
         "tw": 64, "th": 48, "rgba": True},
        # Match of a button on a full-HD screenshot, the reference's own use (the second configuration)
        {"name": "match_1920x1080_host", "kind": "match", "form": "exact", "scene": "ui", "w": 1920, "h": 1080,
         "tw": 96, "th": 32},
        # the same frame size already on the GPU (a capture or decoder output), in the fast form
        {"name": "match_1920x1080_fast", "kind": "match_device", "form": "fast", "scene": "camera", "w": 1920,
         "h": 1080, "tw": 96, "th": 32, "map": False, "alpha": False},
        # the full score map of a large template on a 4K gray frame (the third configuration)
        {"name": "map_3840x2160_fast", "kind": "u8_device", "form": "fast", "scene": "camera", "w": 3840, "h": 2160,
         "tw": 256, "th": 256, "map": True},
        # a sprite with a varying alpha plane (four channels) on an odd-sized window, score map kept
        {"name": "map_1366x767_alpha", "kind": "match_device", "form": "exact", "scene": "camera", "w": 1366, "h": 767,
         "tw": 133, "th": 71, "map": True, "alpha": True},
        # every occurrence of an icon on a laptop screen
        {"name": "peaks_1280x800_host", "kind": "peaks", "form": "exact", "scene": "camera", "w": 1280, "h": 800,
         "tw": 32, "th": 32},
        # a prepared template looked for in frame after frame
        {"name": "find_1280x720_fast", "kind": "find_device", "form": "fast", "scene": "camera", "w": 1280, "h": 720,
         "tw": 57, "th": 41},
        # hundreds of templates of uneven sizes on one frame (the benchmark's default line)
        {"name": "fleet_256_2560x1440_fast", "kind": "fleet_device", "form": "fast", "scene": "camera", "w": 2560,
         "h": 1440, "members": 256, "tmin": 16, "twmax": 192, "thmax": 128},
        # a fleet in the default form, bit for bit the reference's results
        {"name": "fleet_64_1920x1080_exact", "kind": "fleet_device", "form": "exact", "scene": "camera", "w": 1920,
         "h": 1080, "members": 64, "tmin": 24, "twmax": 128, "thmax": 96},
        # gray glyphs and icons on a host frame, in the default form
        {"name": "fleet_24_gray_1280x720_host", "kind": "fleet_gray", "form": "exact", "scene": "camera", "w": 1280,
         "h": 720, "members": 24, "tmin": 12, "twmax": 80, "thmax": 60},
        # a video feed: two frames in flight against colour and gray fleets (the fifth configuration)
        {"name": "stream_1920x1080_fast", "kind": "stream", "form": "fast", "scene": "camera", "w": 1920, "h": 1080,
         "members": 64, "gray": 8, "tmin": 24, "twmax": 128, "thmax": 96},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["gray", "match", "match_device", "match_device", "u8_device", "peaks", "find_device",
                       "fleet_device", "fleet_device", "fleet_gray", "stream"])
    form = rng.choice(["exact", "fast"])
    many = kind in ("fleet_device", "fleet_gray", "stream")
    w = _log(rng, 480 if many else 200, 2560 if many else 3840)
    h = max(120, min(2160, int(w * rng.uniform(0.5, 0.8))))
    c = {"kind": kind, "form": form, "scene": "camera", "w": w, "h": h}
    if many:
        c["members"] = _log(rng, 4, 192)
        c["tmin"] = _log(rng, 10, 24)
        c["twmax"] = max(32, min(192, w // 4, _log(rng, 40, 192)))
        c["thmax"] = max(28, min(128, h // 4, _log(rng, 32, 128)))
        if kind == "fleet_gray":
            c["members"] = min(c["members"], 64)
        if kind == "stream":
            c["members"], c["gray"] = min(c["members"], 64), rng.choice([0, 3, 8])
        return c
    c["tw"], c["th"] = min(w // 3, _log(rng, 12, 256)), min(h // 3, _log(rng, 12, 256))
    if kind in ("match", "gray", "peaks"):
        c["form"] = "exact"
    if kind == "gray":
        c["rgba"] = rng.random() < 0.5
    if kind in ("match_device", "u8_device"):
        c["map"] = rng.random() < 0.5
    if kind == "match_device":
        c["alpha"] = rng.random() < 0.25
    return c


# ------------------------------------------------------------------ scenes


def _camera(g, h, w, ch):
    """h x w x ch float frame on the GPU: 1/f-amplitude noise, per-channel
    noise, flat rectangles, sensor noise."""
    dev = g.device
    f = torch.fft.rfft2(torch.randn((h, w), generator=g, device=dev))
    fy = torch.fft.fftfreq(h, device=dev)[:, None]
    fx = torch.fft.rfftfreq(w, device=dev)[None, :]
    r = torch.sqrt(fx * fx + fy * fy)
    r[0, 0] = 1.0
    f = f / r
    f[0, 0] = 0
    base = torch.fft.irfft2(f, s=(h, w))
    base = base / base.std() * 40 + 128
    img = base[..., None] + torch.randn((h, w, ch), generator=g, device=dev) * 20
    big = max(9, min(w, h) // 6)
    rects = torch.rand((24, 4 + ch), generator=g, device=dev).cpu().tolist()
    for q in rects:
        rw, rh = 8 + int(q[0] * (big - 8)), 8 + int(q[1] * (big - 8))
        x, y = int(q[2] * (w - rw)), int(q[3] * (h - rh))
        img[y:y + rh, x:x + rw] = torch.tensor(q[4:], device=dev) * 255
    return img + torch.randn(img.shape, generator=g, device=dev) * 2


def _ui(g, h, w, ch):
    """A user-interface frame: flat panels, 1-pixel strokes, no noise."""
    dev = g.device
    img = torch.rand((1, 1, ch), generator=g, device=dev).expand(h, w, ch) * 60 + 180
    img = img.contiguous()
    for q in torch.rand((40, 4 + ch), generator=g, device=dev).cpu().tolist():
        rw, rh = 40 + int(q[0] * w / 4), 30 + int(q[1] * h / 4)
        x, y = int(q[2] * (w - rw)), int(q[3] * (h - rh))
        img[y:y + rh, x:x + rw] = torch.tensor(q[4:], device=dev) * 255
    ys = torch.randint(0, h - 12, (3000,), generator=g, device=dev)
    xs = torch.randint(0, w - 12, (3000,), generator=g, device=dev)
    col = torch.randint(0, 80, (3000, ch), generator=g, device=dev).float()
    for i in range(9):
        img[ys[:1500], xs[:1500] + i] = col[:1500]
        img[ys[1500:] + i, xs[1500:]] = col[1500:]
    return img


def _u8(a):
    return a.round().clamp(0, 255).to(torch.uint8)


def _frame(case, g, ch):
    """The frame on the GPU: h x w (ch 1) or h x w x 4 uint8."""
    h, w = case["h"], case["w"]
    if ch == 1:
        return _u8(_camera(g, h, w, 1)[..., 0]).contiguous()
    img = _ui(g, h, w, 3) if case["scene"] == "ui" else _camera(g, h, w, 3)
    out = torch.full((h, w, 4), 255, dtype=torch.uint8, device=g.device)
    out[..., :3] = _u8(img)
    if case.get("alpha"):
        out[..., 3] = _u8(_camera(g, h, w, 1)[..., 0])
    return out


def _crop(frame, g, tw, th):
    """A crop of the frame with a brightness shift a * x + b (alpha kept)."""
    h, w = frame.shape[:2]
    q = torch.rand((4,), generator=g, device=g.device).cpu().tolist()
    x, y = int(q[0] * (w - tw)), int(q[1] * (h - th))
    t = frame[y:y + th, x:x + tw].clone()
    a, b = 0.9 + 0.2 * q[2], 20 * q[3] - 10
    if t.dim() == 3:
        t[..., :3] = _u8(t[..., :3].float() * a + b)
    else:
        t = _u8(t.float() * a + b)
    return t.contiguous()


def _templates(case, frame, g, count):
    """count templates with sizes uniform in tmin..twmax x tmin..thmax, 70 %
    crops and 30 % absent."""
    q = torch.rand((count, 3), generator=g, device=g.device).cpu().tolist()
    out = []
    for a, b, present in q:
        tw = case["tmin"] + int(a * (case["twmax"] - case["tmin"] + 1))
        th = case["tmin"] + int(b * (case["thmax"] - case["tmin"] + 1))
        if present < 0.7:
            out.append(_crop(frame, g, tw, th))
        else:
            t = torch.randint(0, 256, (th, tw) + tuple(frame.shape[2:]), generator=g, device=g.device,
                              dtype=torch.uint8)
            if t.dim() == 3:
                t[..., 3] = 255
            out.append(t)
    return out


def _gray(t):
    v = t.to(torch.int64)
    return ((4899 * v[..., 0] + 9617 * v[..., 1] + 1868 * v[..., 2] + 8192) >> 14).to(torch.uint8).contiguous()


def _inputs(case, seed):
    """The case's frames and templates, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    gray = kind in ("u8_device", "fleet_gray") or (kind == "gray" and not case["rgba"])
    frame = _frame(case, g, 1 if gray else 4)
    d = {"frame": frame}
    if kind in ("fleet_device", "fleet_gray", "stream"):
        d["tpls"] = _templates(case, frame, g, case["members"])
        if kind == "stream":
            nxt = frame.clone()
            nxt[..., :3] = _u8(frame[..., :3].float() + torch.randn(frame.shape[:2] + (3,), generator=g,
                                                                      device=g.device) * 2)
            d["next"] = nxt
            d["gtpls"] = _templates(case, _gray(frame), g, case["gray"])
    else:
        d["tpl"] = _crop(frame, g, case["tw"], case["th"])
    return d


# ------------------------------------------------------------- preparation


def _views(buf):
    """(scores, positions) of a result buffer: n x (min, max) float32 and two
    n x (x, y) int32, all views."""
    return {"scores": buf.view(torch.float32)[:, 0::3], "min_at": buf[:, 1:3], "max_at": buf[:, 4:6]}


def prepare(case, seed):
    cvm.lib()
    d = _inputs(case, seed)
    kind, s = case["kind"], {"case": case, "form": FORMS[case["form"]]}
    if kind in ("gray", "match", "peaks"):
        s["frame"], s["tpl"] = d["frame"].cpu().numpy(), d["tpl"].cpu().numpy()
        return s
    if kind == "stream":
        color = cvm.NewFleet([cvm.NewMatcher(t.cpu().numpy()) for t in d["tpls"]])
        color.SetForm(s["form"])
        gray = None
        if d["gtpls"]:
            gray = cvm.NewFleet([cvm.NewGrayMatcher(t.cpu().numpy()) for t in d["gtpls"]])
            gray.SetForm(s["form"])
        s["stream"] = cvm.NewStream(color, gray, case["w"], case["h"])
        s["frames"] = [d["frame"].cpu().numpy(), d["next"].cpu().numpy()]
        return s
    if kind == "fleet_gray":
        s["fleet"] = cvm.NewFleet([cvm.NewGrayMatcher(t.cpu().numpy()) for t in d["tpls"]])
        s["fleet"].SetForm(s["form"])
        s["frame"] = d["frame"].cpu().numpy()
        return s
    s["frame"] = d["frame"]
    n = case.get("members", 1)
    s["buf"] = torch.zeros((n, 6), dtype=torch.int32, device="cuda")
    s["out"] = _views(s["buf"])
    if kind == "fleet_device":
        s["fleet"] = cvm.NewFleet([cvm.NewMatcher(t.cpu().numpy()) for t in d["tpls"]])
        s["fleet"].SetForm(s["form"])
    elif kind == "find_device":
        s["matcher"] = cvm.NewMatcher(d["tpl"].cpu().numpy())
    else:
        s["tpl"] = d["tpl"]
        if case["map"]:
            s["map"] = torch.empty((case["h"] - case["th"] + 1, case["w"] - case["tw"] + 1), device="cuda")
            s["out"]["map"] = s["map"]
    return s


# -------------------------------------------------------------------- run


def _numbers(results):
    """Host results as arrays: scores n x 2, positions n x 4."""
    a = np.array(results, np.float64)
    return {"scores": a[:, 0::3].astype(np.float32), "at": a[:, [1, 2, 4, 5]].astype(np.int32)}


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "gray":
        return cvm.MatchGray(s["frame"], s["tpl"])
    if kind == "match":
        return cvm.Match(s["frame"], s["tpl"])
    if kind == "peaks":
        got, count = cvm.MatchMapPeaks(s["frame"], s["tpl"], 0.3, case["tw"] // 2, case["th"] // 2, 256)
        at = np.full((256, 2), -1, np.int32)
        if got:
            at[:len(got)] = got
        return {"at": at, "count": count}
    if kind == "stream":
        st = s["stream"]
        for f in s["frames"]:
            st.push(f)
        got = [st.pull() for _ in s["frames"]]
        return [_numbers(r) for c, g, _ in got for r in ((c, g) if g else (c,))]
    if kind == "fleet_gray":
        return _numbers(s["fleet"].FindAll(s["frame"]))
    f, stream = s["frame"], torch.cuda.current_stream().cuda_stream
    w, h = case["w"], case["h"]
    if kind == "fleet_device":
        s["fleet"].find_all_device(f.data_ptr(), 4 * w, w, h, s["buf"].data_ptr(), stream)
        return s["out"]
    before = cvm.SetForm(s["form"])
    try:
        if kind == "find_device":
            s["matcher"].find_device(f.data_ptr(), 4 * w, w, h, s["buf"].data_ptr(), stream)
            return s["out"]
        t, tw, th = s["tpl"], case["tw"], case["th"]
        dmap = s["map"].data_ptr() if case["map"] else None
        if kind == "match_device":
            rc = cvm.lib().cvm_match_device(f.data_ptr(), 4 * w, w, h, t.data_ptr(), 4 * tw, tw, th, dmap,
                                            s["buf"].data_ptr(), stream)
        else:
            rc = cvm.lib().cvm_match_u8_device(f.data_ptr(), w, w, h, t.data_ptr(), tw, tw, th, 1, 1, dmap,
                                               s["buf"].data_ptr(), stream)
    finally:
        cvm.SetForm(before)
    if rc:
        b = ctypes.create_string_buffer(256)
        cvm.lib().cvm_last_error(b, len(b))
        raise cvm.CvmatchError(rc, b.value.decode(errors="replace"))
    return s["out"]


# ------------------------------------------------------------------- work


def work(case):
    """Bytes: the images and templates in, results out.  Flops: real
    transforms of the frame's size (2.5 N log2 N each) -- the frame's
    channels once per frame, one inverse per template, a one-shot's template
    channels too -- the spectral products, and the window sums and score of
    every result."""
    w, h, kind = case["w"], case["h"], case["kind"]
    n = w * h
    fft = 2.5 * n * math.log2(n)
    gray = kind in ("gray", "u8_device", "fleet_gray")
    cn, px = (1, 1) if gray else (4 if case.get("alpha") else 3, 4)
    if kind == "gray" and case["rgba"]:
        px = 4
    if kind in ("fleet_device", "fleet_gray", "stream"):
        m = case["members"]
        tw, th = (case["tmin"] + case["twmax"]) / 2, (case["tmin"] + case["thmax"]) / 2
        res = (w - tw + 1) * (h - th + 1)
        per = fft + 3.0 * n * cn + res * (2 * cn + 12)
        b, f = n * px + 24 * m, cn * fft + m * per
        if kind == "stream":
            b, f = b + 24 * case["gray"], f + (fft if case["gray"] else 0) + case["gray"] * (
                fft + 3.0 * n + res * 14)
            b, f = 2 * b, 2 * f
        return {"bytes": b, "flops": f}
    tw, th = case["tw"], case["th"]
    res = (w - tw + 1) * (h - th + 1)
    templates = 0 if kind == "find_device" else cn
    b = n * px + 24 + (0 if kind == "find_device" else tw * th * px) + (4 * res if case.get("map") else 0)
    return {"bytes": b, "flops": (cn + templates + 1) * fft + 3.0 * n * cn + res * (2 * cn + 12)}


# ------------------------------------------------------------------ exact


class _Exact:
    """TM_CCOEFF_NORMED in 64 bits: the frame's transforms and exact window
    sums, shared by the templates matched against it."""

    def __init__(self, planes):
        self.p = [x.to(torch.int64) for x in planes]
        self.h, self.w = self.p[0].shape
        self.f = [torch.fft.rfft2((x - 128).double()) for x in self.p]
        self.s = [self._table(x) for x in self.p]
        self.q = self._table(sum(x * x for x in self.p))

    @staticmethod
    def _table(x):
        t = torch.zeros((x.shape[0] + 1, x.shape[1] + 1), dtype=torch.int64, device=x.device)
        t[1:, 1:] = x.cumsum(0).cumsum(1)
        return t

    def match(self, planes):
        t = [x.to(torch.int64) for x in planes]
        th, tw = t[0].shape
        rh, rw, area = self.h - th + 1, self.w - tw + 1, float(th * tw)

        def window(s):
            return (s[th:th + rh, tw:tw + rw] - s[:rh, tw:tw + rw] - s[th:th + rh, :rw] + s[:rh, :rw]).double()

        sums = [int(x.sum()) for x in t]
        norm = sum(float((x * x).sum()) / area - (v / area) ** 2 for x, v in zip(t, sums))
        if norm < 2.220446049250313e-16:
            return torch.ones((rh, rw), dtype=torch.float64, device=t[0].device)
        acc = 0
        for x, v, f in zip(t, sums, self.f):
            z = torch.zeros((self.h, self.w), dtype=torch.float64, device=x.device)
            z[:th, :tw] = (x.double() * area - v)
            acc = acc + f * torch.fft.rfft2(z).conj()
        num = torch.fft.irfft2(acc, s=(self.h, self.w))[:rh, :rw] / area
        q = window(self.q)
        d = (q - sum(window(s) ** 2 for s in self.s) / area).clamp_min(0)
        lim = (q * 1.1920929e-06).clamp_max(0.5)
        den = torch.where(d > lim, d.sqrt() * math.sqrt(norm * area), torch.zeros_like(d))
        a = num.abs()
        return torch.where(a < den, num / den, torch.where(a < den * 1.125, num.sign(), torch.zeros_like(num)))


def _planes(t, cn):
    return [t] if t.dim() == 2 else [t[..., k] for k in range(cn)]


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "peaks":
        return None
    if kind == "stream":
        got = []
        for f in (d["frame"], d["next"]):
            for frame, tpls in ((f, d["tpls"]), (_gray(f), d["gtpls"])):
                if not tpls:
                    continue
                e = _Exact(_planes(frame, 3))
                m = [(lambda x: (float(x.min()), float(x.max())))(e.match(_planes(t, 3))) for t in tpls]
                got.append({"scores": np.array(m), "at": None})
        return got
    frame, tpls = d["frame"], d["tpls"] if "tpls" in d else [d["tpl"]]
    if kind == "gray" and case["rgba"]:
        frame, tpls = _gray(frame), [_gray(t) for t in tpls]
    cn = 4 if case.get("alpha") else 3
    e = _Exact(_planes(frame, cn))
    scores, res = [], None
    for t in tpls:
        res = e.match(_planes(t, cn))
        scores.append((float(res.min()), float(res.max())))
    if kind in ("gray", "match"):
        return (scores[0][0], None, None, scores[0][1], None, None)
    if kind == "fleet_gray":
        return {"scores": np.array(scores), "at": None}
    out = {"scores": torch.tensor(scores, dtype=torch.float64), "min_at": None, "max_at": None}
    if case.get("map"):
        out["map"] = res
    return out
