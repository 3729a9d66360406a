"""What the row-pair kernels add up, where a sum's form shows."""
import numpy as np
import pytest

import stripmlem as sm
from oracle import oracle as orc
from test_gpu_row_pairs import CASES, IMAGE_TOL, events, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accum", [sm.ACCUM_FP32, sm.ACCUM_KAHAN, sm.ACCUM_FP64])
def test_pixels_that_an_update_made_infinite(accum):
    """Events that see an infinite pixel have an infinite denominator and add
    nothing, to that pixel either; the others are what they are without it."""
    R, L, n_y, n_z, p, s_z, s_dl = case = CASES[5]
    g, ev = orc.geometry(R, L, n_y, n_z, p, p, s_z, s_dl), events(CASES[5], 6_001, 6)
    with sm.Reconstruction(sm.Scanner(R, L, n_y, n_z, p, p, s_z, s_dl),
                           accumulation=accum) as rec:
        rec.set_item_events(8000)  # one item: the conversion by subnormal products
        rec.set_events(*ev)
        rec(None, 2)
        scale = 3.4e38 / np.quantile(rec.rho, 0.999)
        rec.rho = np.ones((n_y, n_z), np.float32)
        rec(None, 1)
        rec.accumulate()
        rec.update(scale)
        rho = rec.rho
        infinite = np.isinf(rho)
        assert 0 < infinite.sum() < 20 and not np.isnan(rho).any()
        rec(None, 1)
        img = rec.rho
    seen = orc.forward_f64(g, *ev, infinite.astype(np.float32), s_z, s_dl) > 0
    assert 0 < seen.sum() < 3_000
    kept = [v[~seen] for v in ev]
    ref = orc.mlem_f64(g, *kept, 1, rho=np.where(infinite, 0.0, rho))
    assert np.all(img[infinite] == 0.0)
    assert rel(img, ref) < IMAGE_TOL


def test_sigma_gradient_of_rows_whose_values_cancel():
    """A signed image whose sum over every full row is exactly zero: the rows
    still have a derivative.  The sigma_z makes neighbouring kernel values
    powers of two apart, so the binary32 sums cancel without a rounding."""
    s_z, s_dl = 1.6986435651779175, 10.0
    g = orc.geometry(100.0, 200.0, 64, 64, 1.0, 1.0, s_z, s_dl)
    ev = [np.zeros(1, np.float32)] * 3
    rho = np.zeros((64, 64), np.float32)
    rho[:, [30, 33]], rho[:, [31, 32]] = 2.0, -1.0
    with sm.Reconstruction(sm.Scanner(100.0, 200.0, 64, 64, 1.0, 1.0, s_z, s_dl)) as rec:
        rec.set_events(*ev)
        got = rec.grad_sigma(rho, np.ones(1), s_z, s_dl)
    want = orc.grad_sigma_f64(g, *ev, rho, np.ones(1), s_z, s_dl)
    assert abs(got[0] / want[0] - 1) < IMAGE_TOL


def test_binary64_sums_take_the_rows_one_by_one():
    """Three pixels of one column, the first two in rows of one pair: the third
    cancels the first and leaves the second, which a binary32 sum of the first
    two would have rounded."""
    n, s_z, s_dl = 64, 5.0, 10.0
    ev = [np.zeros(1, np.float32)] * 3
    with sm.Reconstruction(sm.Scanner(100.0, 200.0, n, n, 1.0, 1.0, s_z, s_dl),
                           accumulation=sm.ACCUM_FP64) as rec:
        rec.set_events(*ev)

        def forward(values):  # rows 32 and 31: the event's middle pair
            rho = np.zeros((n, n), np.float32)
            for row, v in values:
                rho[row, 30] = v
            return rec.forward(rho, s_z, s_dl)[0]

        k = {row: forward([(row, 1.0)]) for row in (32, 31, 33)}
        small = np.float32(1.1e-6)
        third = np.float32(-k[32] / k[33])
        rows = [(32, np.float32(1.0)), (31, small), (33, third)]
        want = sum(float(np.float32(k[r]) * v) for r, v in rows)
        assert abs(forward(rows) - want) < 1e-12 * k[32]
