"""Replayed host calls from many threads: they share the graphs the process
keeps.  Exact results against the oracle while shapes change; fast-form results
while another thread switches the autotuner on and off; and the device memory
held stays bounded."""
import threading

import numpy as np
import pytest

import cvmatch_gb300 as cvm
import oracle

pytestmark = pytest.mark.gpu


def _scene(seed, h, w, th, tw):
    rng = np.random.default_rng(seed)
    img = rng.integers(0, 256, (h, w), dtype=np.uint8)
    y, x = int(rng.integers(0, h - th)), int(rng.integers(0, w - tw))
    return img, img[y:y + th, x:x + tw].copy(), (x, y)


def _run(n, work):
    errors, gate = [], threading.Barrier(n)

    def body(i):
        try:
            gate.wait()
            work(i)
            gate.wait(60)  # none ends before all are done
        except Exception as e:  # noqa: BLE001
            errors.append(e)
            gate.abort()

    ts = [threading.Thread(target=body, args=(i,)) for i in range(n)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors[0]


def test_one_shape_from_many_threads_holds_bounded_memory():
    import torch
    h, w = 900, 1400
    img, tpl, at = _scene(1, h, w, 31, 40)
    want = tuple(oracle.match_u8(img, tpl, 1, threads=8, want_map=False)[0])
    for _ in range(4):
        assert tuple(cvm.MatchGray(img, tpl)) == want
    free0 = torch.cuda.mem_get_info()[0]

    def work(i):
        mine = img.copy()
        mine[0, i] ^= 1
        for _ in range(6):
            r = cvm.MatchGray(mine, tpl)
            assert r[4:] == at and r[3] >= 0.999

    _run(32, work)
    assert free0 - torch.cuda.mem_get_info()[0] < 3 << 30  # the graphs' limit, and the pool's for queued calls


def test_shapes_in_turn_from_many_threads():
    shapes = [(90 + 7 * k, 131 + 5 * k, 9 + k % 4, 14) for k in range(40)]
    scenes = [_scene(k, *s) for k, s in enumerate(shapes)]
    want = [tuple(oracle.match_u8(i, t, 1, threads=8, want_map=False)[0]) for i, t, _ in scenes]

    def work(i):
        rng = np.random.default_rng(i)
        for k in rng.integers(0, len(shapes), 150):
            assert tuple(cvm.MatchGray(scenes[k][0], scenes[k][1])) == want[k]

    _run(8, work)


def test_the_autotuner_switched_meanwhile():
    shapes = [(300 + 40 * k, 500 + 60 * k, 20 + k, 30) for k in range(6)]
    scenes = [_scene(k, *s) for k, s in enumerate(shapes)]
    form, auto = cvm.SetForm(cvm.FORM_FAST), cvm.SetAutotune(True)
    stop = threading.Event()

    def toggle():
        on = False
        while not stop.is_set():
            cvm.SetAutotune(on)
            on = not on

    t = threading.Thread(target=toggle)
    t.start()
    try:
        def work(i):
            rng = np.random.default_rng(i)
            for k in rng.integers(0, len(shapes), 60):
                img, tpl, at = scenes[k]
                r = cvm.MatchGray(img, tpl)
                assert r[4:] == at and abs(r[3] - 1) < 1e-5
        _run(6, work)
    finally:
        stop.set()
        t.join()
        cvm.SetForm(form)
        cvm.SetAutotune(auto)
