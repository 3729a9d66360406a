"""AnalyticKernel tile launches over small work items (fewer events than a warp
takes per step, fewer than a CTA has warps) and over windows whose sides are no
multiple of the staging patches, against the FP64 oracle."""
import numpy as np
import pytest

import stripmlem as sm
from oracle import oracle as orc
from test_gpu_row_pairs import CASES, events, rel

pytestmark = pytest.mark.gpu

# cases whose field reaches neither past the strips nor into the detectors, where
# the five-point sensitivity and so the images have no binary32 accuracy;
# values good to a few 1e-7, binary32 sums of some hundred terms in the windows
TOL = 1e-5


@pytest.mark.parametrize("case", [CASES[i] for i in (0, 4, 5, 6, 8)])
@pytest.mark.parametrize("n,item", [(1, 0), (1_501, 0), (1_501, 1), (1_501, 17), (1_501, 8000)])
def test_small_items(case, n, item):
    R, L, n_y, n_z, p, s_z, s_dl = case
    g = orc.geometry(R, L, n_y, n_z, p, p, s_z, s_dl)
    ev = events(case, n, 11)
    if n == 1:
        ev = [np.float32([v]) for v in (0.1 * p, -0.2 * p, 0.3 * p)]
    rho = np.random.default_rng(12).lognormal(0.0, 0.5, (n_y, n_z)).astype(np.float32)
    with sm.Reconstruction(sm.Scanner(R, L, n_y, n_z, p, p, s_z, s_dl), mode=sm.MODE_GPU) as rec:
        rec.set_item_events(item)
        rec.set_events(*ev)
        y = rec.forward(rho, s_z, s_dl)
        rec(None, 2)
        img = rec.rho
        assert rec.stats()["n_overflow"] == 0
    assert rel(img, orc.mlem_f64(g, *ev, 2, mode=1)) < TOL
    assert rel(y, orc.forward_f64(g, *ev, rho, s_z, s_dl, mode=1)) < TOL


def test_batch_of_tall_and_short_boxes():
    """Boxes of 81 to 128 rows have tilings of the row-pair kernels' tall columns,
    which the AnalyticKernel reads row-major: beside column-major and row-major
    members, in one batch."""
    recs, refs = [], []
    try:
        for case in (CASES[4], CASES[0], CASES[5], (150.0, 300.0, 190, 211, 1.0, 6.0, 44.0)):
            R, L, n_y, n_z, p, s_z, s_dl = case
            ev = events(case, 1_201, 13)
            rec = sm.Reconstruction(sm.Scanner(R, L, n_y, n_z, p, p, s_z, s_dl),
                                    mode=sm.MODE_GPU)
            recs.append(rec)
            rec.set_events(*ev)
            g = orc.geometry(R, L, n_y, n_z, p, p, s_z, s_dl)
            refs.append(orc.mlem_f64(g, *ev, 2, mode=1))
        with sm.Batch(recs, mode=sm.MODE_GPU) as batch:
            batch(2)
        for rec, ref in zip(recs, refs):
            assert rel(rec.rho, ref) < TOL
    finally:
        for rec in recs:
            rec.close()
