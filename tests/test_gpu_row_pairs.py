"""The row-pair tile kernels (GaussianKernel over column-major windows) at the
edges of their layout, against the FP64 oracle with binary32 pixel sets:
boxes of a few rows and of the most rows one lane layout holds (80: five
blocks of eight pairs; 81 and more: sixteen lanes an event), boxes clipped at
every image border (rows of a pair of unequal length, or missing), odd window
sizes, items of one event, weights of either sign and zero, and single-row
and single-column images."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

# Per event: binary32 row sums of at most a few hundred recurrence steps and
# values good to a few 1e-7 each, so 3e-6 of the sum; a pixel missing from (or
# added to) a set of n pixels changes it by about 0.05 / n (the kernel at three
# sigma), 5e-5 for the largest sets here, so nine events in ten must meet that.
# An event that shows the field only its ellipse's rim (t = 2.1 sigma_z) also
# feels its coordinates' binary32 rounding, d log K = 2 t / sigma_z^2 times
# three roundings of a length of the field's size.
EVENT_TOL = 3e-6
IMAGE_TOL = 1e-5


def rim_tol(case):
    size = 0.55 * max(case[2], case[3]) * case[4] + case[0]
    return EVENT_TOL + 2 * 2.13 / case[5] * 3 * 2.0 ** -24 * size


# radius, length, n_y, n_z, pixel, sigma_z, sigma_dl
CASES = [
    (200.0, 500.0, 200, 250, 2.0, 10.0, 42.0),   # 64 rows
    (400.0, 800.0, 400, 800, 1.0, 5.0, 25.0),    # 76 rows, five blocks
    (100.0, 200.0, 211, 203, 1.0, 4.0, 26.5),    # 80 rows
    (100.0, 200.0, 211, 203, 1.0, 4.0, 27.2),    # 82 rows: 16 lanes an event
    (150.0, 300.0, 190, 211, 1.0, 6.0, 42.0),    # 126 rows: the tall column stride
    (60.0, 100.0, 111, 97, 1.0, 4.0, 30.0),      # whole image in one window
    (300.0, 500.0, 37, 53, 10.0, 12.0, 30.0),    # boxes of 4 to 10 rows
    (300.0, 500.0, 5, 300, 2.0, 10.0, 42.0),     # a few rows, clipped boxes
    (300.0, 500.0, 300, 4, 2.0, 10.0, 42.0),     # a few columns
]


def rel(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def events(case, n, seed):
    """Events over the whole field and past its borders."""
    R, L, n_y, n_z, p, s_z, s_dl = case
    r = np.random.default_rng(seed)
    z = r.uniform(-0.55, 0.55, n) * n_z * p
    y = r.uniform(-0.55, 0.55, n) * n_y * p
    t = r.uniform(-0.5, 0.5, n) * L / R
    dl = -2 * y * np.sqrt(1 + t * t)
    ev = [z + (R - y) * t, z - (R + y) * t, dl]
    ev = [v.astype(np.float32) for v in ev]
    if n > 100:
        for v in ev:  # events without a pixel set
            v[r.integers(0, n, 5)] = np.nan
            v[r.integers(0, n, 5)] = np.inf
            v[r.integers(0, n, 5)] = -3e38
    return ev


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("n", [1, 6_001])
def test_projections(case, n):
    import stripmlem as sm
    R, L, n_y, n_z, p, s_z, s_dl = case
    g = orc.geometry(R, L, n_y, n_z, p, p, s_z, s_dl)
    ev = events(case, n, 5)
    if n == 1:
        ev = [np.float32([v]) for v in (0.1 * p, -0.2 * p, 0.3 * p)]
    r = np.random.default_rng(8)
    rho = r.lognormal(0.0, 0.5, (n_y, n_z)).astype(np.float32)
    with sm.Reconstruction(sm.Scanner(R, L, n_y, n_z, p, p, s_z, s_dl)) as rec:
        rec.set_events(*ev)
        assert rec.stats()["n_overflow"] == 0
        for k in (1.0, 0.9):  # the model's sigmas may differ from the geometry's
            y = rec.forward(rho, k * s_z, k * s_dl)
            o = orc.forward_f64(g, *ev, rho, k * s_z, k * s_dl)
            live = o > 0
            assert np.array_equal(y > 0, live)
            err = np.abs(y[live] / o[live] - 1)
            assert np.quantile(err, 0.9) < EVENT_TOL
            assert err.max() < rim_tol(case)
        for w in (r.uniform(0.5, 2.0, n), r.uniform(-1.0, 1.0, n), np.arange(n) % 3 == 1.0):
            w = np.where(live, w, 0.0)
            if not w.any():
                continue
            # signed sums cancel: their error is that of the sum of magnitudes
            scale = np.linalg.norm(orc.adjoint_f64(g, *ev, np.abs(w), s_z, s_dl))
            d = rec.adjoint(w, s_z, s_dl) - orc.adjoint_f64(g, *ev, w, s_z, s_dl)
            assert np.linalg.norm(d) < IMAGE_TOL * scale


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("n,item", [(3, 0), (6_001, 0), (6_001, 1), (6_001, 40), (6_001, 8000)])
def test_mlem(case, n, item):
    import stripmlem as sm
    R, L, n_y, n_z, p, s_z, s_dl = case
    g = orc.geometry(R, L, n_y, n_z, p, p, s_z, s_dl)
    ev = events(case, n, 6)
    if n == 3:
        ev = [np.float32([v, 2 * v, -v]) for v in (0.4 * p, -0.6 * p, 0.3 * p)]
    with sm.Reconstruction(sm.Scanner(R, L, n_y, n_z, p, p, s_z, s_dl)) as rec:
        rec.set_item_events(item)
        rec.set_events(*ev)
        rec(None, 3)
        img = rec.rho
    assert rel(img, orc.mlem_f64(g, *ev, 3)) < IMAGE_TOL


def test_batch_of_both_lane_layouts():
    import stripmlem as sm
    recs, refs = [], []
    try:
        for case in (CASES[0], CASES[3], CASES[5], CASES[7]):
            R, L, n_y, n_z, p, s_z, s_dl = case
            ev = events(case, 4_001, 7)
            rec = sm.Reconstruction(sm.Scanner(R, L, n_y, n_z, p, p, s_z, s_dl))
            recs.append(rec)
            rec.set_events(*ev)
            refs.append(orc.mlem_f64(orc.geometry(R, L, n_y, n_z, p, p, s_z, s_dl), *ev, 2))
        with sm.Batch(recs) as batch:
            batch(2)
        for rec, ref in zip(recs, refs):
            assert rel(rec.rho, ref) < IMAGE_TOL
    finally:
        for rec in recs:
            rec.close()


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("n", [1, 6_001])
def test_sigma_gradient(case, n):
    import stripmlem as sm
    R, L, n_y, n_z, p, s_z, s_dl = case
    g = orc.geometry(R, L, n_y, n_z, p, p, s_z, s_dl)
    ev = events(case, n, 9)
    if n == 1:
        ev = [np.float32([v]) for v in (0.1 * p, -0.2 * p, 0.3 * p)]
    r = np.random.default_rng(10)
    rho = r.lognormal(0.0, 0.5, (n_y, n_z)).astype(np.float32)
    w = np.where(r.random(n) < 0.1, 0.0, r.uniform(-0.5, 2.0, n)) if n > 1 else np.ones(1)
    with sm.Reconstruction(sm.Scanner(R, L, n_y, n_z, p, p, s_z, s_dl)) as rec:
        rec.set_events(*ev)
        got = rec.grad_sigma(rho, w, 0.9 * s_z, 0.95 * s_dl)
    o = orc.grad_sigma_f64(g, *ev, rho, w, 0.9 * s_z, 0.95 * s_dl)
    # a row's derivative is a difference of terms of a few times its value, and
    # the events' cancel in the sum: bounded by the sum of y |w| / sigma
    y = orc.forward_f64(g, *ev, rho, 0.9 * s_z, 0.95 * s_dl)
    scale = np.dot(np.abs(w), y)
    assert abs(got[0] - o[0]) < IMAGE_TOL * scale / s_z
    assert abs(got[1] - o[1]) < IMAGE_TOL * scale / s_dl
