"""The windowed hybrid iteration's plan: which event lists take the windows
(test hook hybrid_debug_windows), and lists that its items and tasks are cut
from in unusual ways, against the FP64 oracle."""
import ctypes

import numpy as np
import pytest

from test_gpu_hybrid import f32_live, rel_l2
from test_gpu_hybrid_windows import TOL
from test_hybrid_oracle import oracle_setup

pytestmark = pytest.mark.gpu

LENGTH, S_Z, S_DL = 0.45, 0.01, 0.04


def frames(n, p, n_planes, events):
    from oracle import hybrid as oh
    from stripmlem import hybrid as hy
    b = hy.Barrel(radius=(0.16,), n_detectors=(20,), rotation=(0,), w_detector=0.009,
                  h_detector=0.015)
    cfg = (n, n_planes, p, -n_planes * p / 2, LENGTH, S_Z, S_DL)
    r = 0.3 * n * p
    ph = [(0.2 * r, 0.1 * r, 0, 0.4 * r, 0.05, 2.0), (0, 0, 0, r, 0.4 * n_planes * p, 1.0)]
    resp = hy.generate_responses(b, ph, events, LENGTH, S_Z, S_DL, seed=3)
    s = oracle_setup(cfg)
    return cfg, s, b, oh.reconstruct(s, b.centers, hy.synthetic_matrix(b, n, p, n * p / 2), resp, 0)


def iterate(cfg, b, ora, fr, n_iterations=2):
    """Iterations over the frames: the image, and the windowed events, their
    items and their tasks."""
    from stripmlem import hybrid as hy
    n, n_planes, p, z_left = cfg[:4]
    geo = ora["geo"]
    with hy.HybridReconstruction(n, n, n_planes, p, z_left, LENGTH, S_Z, S_DL) as rec:
        rec.set_geometry_soa(len(b.centers), geo["seg"][:, :4], geo["pix"], geo["pos"], ora["w"],
                             geo["lbeg"], geo["lend"])
        rec.set_sensitivity(ora["sens"], given=True)
        rec.set_frames(fr["lor_index"], fr["info_begin"], fr["info_end"], fr["plane_begin"],
                       fr["plane_end"], fr["up"], fr["right"], fr["tan"], fr["sec"])
        w = [ctypes.c_int64() for _ in range(3)]
        rec._check(rec.lib.hybrid_debug_windows(rec._ctx, *(ctypes.byref(v) for v in w)))
        rec(n_iterations)
        return rec.rho, *(v.value for v in w)


def check(cfg, s, ora, fr, img):
    from oracle import hybrid as oh
    live = f32_live(s, ora["geo"], ora["w"], ora["sens"], fr)
    assert len(live) > 0.9 * len(fr)
    f64, _ = oh.mlem(s, ora["geo"], ora["w"], ora["sens"], live, 2, f64=True)
    assert rel_l2(img, f64) < TOL


@pytest.mark.parametrize("n,p,n_planes,events", [
    (24, 0.01, 24, 12_000),
    (40, 0.003, 97, 6_000),
    (64, 0.004, 60, 8_000),
    (24, 0.01, 1, 24_000),  # a window's planes go by 32, so one plane needs more events
])
def test_dense_lists_take_the_windows(n, p, n_planes, events):
    cfg, s, b, ora = frames(n, p, n_planes, events)
    fr = ora["frames"]
    img, windowed, items, tasks = iterate(cfg, b, ora, fr)
    assert windowed > 0.9 * len(fr) and 0 < items <= tasks
    check(cfg, s, ora, fr, img)


def test_more_events_of_a_lor_than_an_item_holds():
    cfg, s, b, ora = frames(24, 0.01, 24, 6_000)
    fr = ora["frames"]
    lors, counts = np.unique(fr["lor_index"], return_counts=True)
    one = fr[fr["lor_index"] == lors[counts.argmax()]]
    copies = np.tile(one, 1_100 // len(one) + 1)[:1_100]
    copies["right"] += np.linspace(-0.1 * S_Z, 0.1 * S_Z, len(copies)).astype(np.float32)
    fr = np.concatenate([fr, copies])
    img, windowed, items, _ = iterate(cfg, b, ora, fr)
    assert windowed == len(fr)  # 24 planes: one slab, so a key per LOR
    assert items >= len(lors) + 2
    check(cfg, s, ora, fr, img)


def test_frames_on_other_lors_infos():
    """Frames far from their LOR's infos go to the per-event kernel, so an item
    spans one LOR and not the whole geometry.  Against the sum of short lists,
    which that kernel takes whole."""
    cfg, s, b, ora = frames(64, 0.004, 60, 8_000)
    geo, fr = ora["geo"], ora["frames"].copy()
    n_infos = len(geo["pos"])
    far = slice(17, None, 200)
    rows = fr["info_end"][far] - fr["info_begin"][far]
    fr["info_begin"][far] = np.where(fr["info_begin"][far] < n_infos // 2, n_infos - rows, 0)
    fr["info_end"][far] = fr["info_begin"][far] + rows
    img, windowed, items, tasks = iterate(cfg, b, ora, fr, 1)
    longest = (geo["lend"] - geo["lbeg"]).max()
    assert 0.9 * len(fr) < windowed <= len(fr) - len(rows) + 1
    assert tasks <= items * ((longest + 1 + 63) // 64)
    total = np.zeros(img.shape)
    for k in range(16):
        one, windowed, _, _ = iterate(cfg, b, ora, fr[k::16], 1)
        assert windowed == 0
        total += one
    assert rel_l2(img, total) < TOL
