"""Strip launches whose windows or constants decide between the tile kernels,
against the FP64 oracle with binary32 pixel sets."""
import numpy as np
import pytest

from oracle import oracle as orc
from test_gpu_row_pairs import CASES, EVENT_TOL, IMAGE_TOL, events, rel

pytestmark = pytest.mark.gpu

# sigma_z of 25 pixels: the closed-form run ends do not settle every row
BROAD = (150.0, 300.0, 200, 300, 1.0, 25.0, 25.0)


def scanner(case):
    import stripmlem as sm
    R, L, n_y, n_z, p, s_z, s_dl = case
    return sm.Scanner(R, L, n_y, n_z, p, p, s_z, s_dl)


def geometry(case):
    R, L, n_y, n_z, p, s_z, s_dl = case
    return orc.geometry(R, L, n_y, n_z, p, p, s_z, s_dl)


def test_column_windows_without_the_closed_form():
    import stripmlem as sm
    g, ev = geometry(BROAD), events(BROAD, 3_001, 5)
    s_z, s_dl = BROAD[5:]
    r = np.random.default_rng(8)
    rho = r.lognormal(0.0, 0.5, (BROAD[2], BROAD[3])).astype(np.float32)
    w = r.uniform(0.5, 2.0, len(ev[0]))
    with sm.Reconstruction(scanner(BROAD)) as rec:
        rec.set_events(*ev)
        # two windows of 128-word columns; the row-major form is no multiple
        assert rec.stats()["smem_bytes"] % 1024 == 0
        y = rec.forward(rho, s_z, s_dl)
        o = orc.forward_f64(g, *ev, rho, s_z, s_dl)
        assert np.array_equal(y > 0, o > 0) and rel(y, o) < IMAGE_TOL
        assert rel(rec.adjoint(w, s_z, s_dl), orc.adjoint_f64(g, *ev, w, s_z, s_dl)) < IMAGE_TOL
        d = np.array(rec.grad_sigma(rho, w, s_z, s_dl))
        d -= orc.grad_sigma_f64(g, *ev, rho, w, s_z, s_dl)
        assert (np.abs(d) < IMAGE_TOL * np.dot(w, o) / np.array([s_z, s_dl])).all()
        rec(None, 3)
        assert rel(rec.rho, orc.mlem_f64(g, *ev, 3)) < IMAGE_TOL


def test_batch_of_every_kind_of_window():
    """Members of each window kind: column-major without and with the row-pair
    kernels, their tall form, row-major (boxes above 128 rows)."""
    import stripmlem as sm
    recs, refs = [], []
    try:
        for case in (BROAD, CASES[0], CASES[4], (150.0, 300.0, 190, 211, 1.0, 6.0, 44.0)):
            ev = events(case, 2_001, 7)
            rec = sm.Reconstruction(scanner(case))
            recs.append(rec)
            rec.set_events(*ev)
            refs.append(orc.mlem_f64(geometry(case), *ev, 2))
        assert recs[-1].stats()["max_box_h"] > 128
        with sm.Batch(recs) as batch:
            batch(2)
        for rec, ref in zip(recs, refs):
            assert rel(rec.rho, ref) < IMAGE_TOL
    finally:
        for rec in recs:
            rec.close()


@pytest.mark.parametrize("sigma", [0.5, 0.6, 1.0, 2.0])
def test_model_sigma_of_a_pixel_and_less(sigma):
    """Projections with a model sigma_z below the geometry's 2 pixels.  All
    coordinates are exact in binary32, so an event's error is that of the
    run's first value, 2^-x at 2.12 geometry sigmas, and of the up to five
    ratios to the row's largest pixel, each 2^r: two roundings of the exponent
    each."""
    import stripmlem as sm
    case = (200.0, 500.0, 128, 128, 1.0, 2.0, 20.0)
    g, n = geometry(case), 4_000
    r = np.random.default_rng(0)
    z = (r.integers(-40 * 64, 40 * 64, n) / 64.0).astype(np.float32)
    dl = (r.integers(-60 * 32, 60 * 32, n) / 32.0).astype(np.float32)
    rho = r.lognormal(0.0, 0.5, (128, 128)).astype(np.float32)
    w = r.uniform(0.5, 2.0, n)
    log2e, t = 1.4427, 2.12 * 2.0
    x, ratio = log2e * t * t / sigma ** 2, log2e * (2 * t + 1) / sigma ** 2
    tol = EVENT_TOL + 0.6931 * 2.0 ** -23 * (x + min(5.0, t) * ratio / 2)
    with sm.Reconstruction(scanner(case)) as rec:
        rec.set_events(z, z, dl)
        y = rec.forward(rho, sigma, 20.0)
        o = orc.forward_f64(g, z, z, dl, rho, sigma, 20.0)
        assert np.abs(y / o - 1).max() < tol
        assert rel(rec.adjoint(w, sigma, 20.0), orc.adjoint_f64(g, z, z, dl, w, sigma, 20.0)) < tol


@pytest.mark.parametrize("mode", [0, 1])
def test_overflow_events_of_column_major_tilings(mode):
    """Boxes too wide for any tile's halo beside an image of few rows: those
    events take the global path, the others column-major windows."""
    import stripmlem as sm
    case = (300.0, 900.0, 120, 400, 1.0, 20.0, 110.0)
    g, s_z, s_dl = geometry(case), case[5], case[6]
    r = np.random.default_rng(3)
    n = 900
    z, y = r.uniform(-190.0, 190.0, n), r.uniform(-58.0, 58.0, n)
    t = np.where(np.arange(n) % 3 == 0, r.uniform(0.9, 1.2, n), r.uniform(-0.2, 0.2, n))
    ev = [v.astype(np.float32) for v in (z + (300.0 - y) * t, z - (300.0 + y) * t,
                                         -2 * y * np.sqrt(1 + t * t))]
    rho = r.lognormal(0.0, 0.5, (120, 400)).astype(np.float32)
    w = r.uniform(0.5, 2.0, n)
    with sm.Reconstruction(scanner(case), mode=mode) as rec:
        for n_subsets in (1, 3):
            rec.set_events(*ev, n_subsets=n_subsets)
            st = rec.stats()
            assert 0 < st["n_overflow"] < n and st["smem_bytes"] % 1024 == 0
            y = rec.forward(rho, s_z, s_dl)
            assert rel(y, orc.forward_f64(g, *ev, rho, s_z, s_dl, mode=mode)) < IMAGE_TOL
            a = rec.adjoint(w, s_z, s_dl)
            assert rel(a, orc.adjoint_f64(g, *ev, w, s_z, s_dl, mode=mode)) < IMAGE_TOL
            rec.rho = np.ones((120, 400), np.float32)
            rec(None, 2)
            assert rel(rec.rho, orc.mlem_f64(g, *ev, 2, mode=mode, n_subsets=n_subsets)) < IMAGE_TOL


@pytest.mark.parametrize("mode", [0, 1])
def test_memory_of_replaced_events(mode):
    """Device memory a context holds once its events were replaced.  The peak of
    a binning is 72 bytes an event; the row-pair kernels' packs (24) are made
    after it, of memory that it gave back or of their own."""
    import torch
    import stripmlem as sm
    case = CASES[0]
    n = 12_000_000
    r = np.random.default_rng(4)
    z, t, dl = (r.uniform(-b, b, n).astype(np.float32) for b in (200.0, 0.3, 300.0))
    zu, zd = z + 200 * t, z - 200 * t
    with sm.Reconstruction(scanner(case), mode=mode) as rec:
        rec.set_events(zu[:9_000], zd[:9_000], dl[:9_000])
        rec(None, 2)  # the kernels are loaded
        free = torch.cuda.mem_get_info()[0]
        for _ in range(2):
            rec.set_events(zu, zd, dl)
            rec(None, 1)
        held = free - torch.cuda.mem_get_info()[0]
    assert held < (72 + 24 + 4) * n


def test_events_replaced_and_subsets_changed_between_kernels():
    """The packs follow the binning: passes of both kernels, projections and
    re-binnings in turn equal fresh contexts'."""
    import stripmlem as sm
    case = CASES[0]
    s_z, s_dl = case[5:]
    rho = np.random.default_rng(8).lognormal(0.0, 0.5, (case[2], case[3])).astype(np.float32)
    with sm.Reconstruction(scanner(case)) as rec:
        for seed, n, n_subsets in ((1, 5_000, 1), (2, 9_000, 2), (3, 700, 1)):
            ev = events(case, n, seed)
            g = geometry(case)
            rec.set_events(*ev)
            rec.rho = np.ones_like(rho)
            rec(None, 1, mode=sm.MODE_GPU)
            assert rel(rec.rho, orc.mlem_f64(g, *ev, 1, mode=1)) < IMAGE_TOL
            rec.rho = np.ones_like(rho)
            rec(None, 2, n_subsets=n_subsets)
            assert rel(rec.rho, orc.mlem_f64(g, *ev, 2, n_subsets=n_subsets)) < IMAGE_TOL
            y = rec.forward(rho, s_z, s_dl)
            assert rel(y, orc.forward_f64(g, *ev, rho, s_z, s_dl)) < IMAGE_TOL
