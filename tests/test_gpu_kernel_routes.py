"""Strip launches whose windows or constants decide between the tile kernels,
against the FP64 oracle with binary32 pixel sets."""
import numpy as np
import pytest

from oracle import oracle as orc
from test_gpu_row_pairs import CASES, IMAGE_TOL, events, rel

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
