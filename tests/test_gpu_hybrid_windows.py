"""The windowed hybrid iteration (dense event lists: many events per LOR)
against the FP64 oracle, at the edges of its windows: one slab of planes and
several, odd and even plane counts, LORs shorter and longer than a task's 64
pixel infos, and events it leaves to the per-event kernel (far outside the
recurrence's range, empty, or walking another LOR's pixel infos)."""
import numpy as np
import pytest

from test_gpu_hybrid import f32_live, rel_l2
from test_hybrid_oracle import oracle_setup

pytestmark = pytest.mark.gpu

# binary32 values and recurrences of at most ~20 steps (a few 1e-7 each),
# two iterations: well inside 1e-5 of the FP64 image
TOL = 1e-5


@pytest.mark.parametrize("n,p,n_planes,events", [
    (24, 0.01, 24, 12_000),    # every plane in one window
    (40, 0.003, 97, 6_000),    # several slabs, odd plane count
    (64, 0.004, 60, 8_000),    # long LORs: tasks of 64 infos and a remainder
    (24, 0.01, 1, 9_000),      # a single plane
])
def test_dense_lists_against_fp64_oracle(n, p, n_planes, events):
    from oracle import hybrid as oh
    from stripmlem import hybrid as hy
    b = hy.Barrel(radius=(0.16,), n_detectors=(20,), rotation=(0,), w_detector=0.009,
                  h_detector=0.015)
    length, s_z, s_dl = 0.45, 0.01, 0.04
    z_left = -n_planes * p / 2
    m = hy.synthetic_matrix(b, n, p, n * p / 2)
    r = 0.3 * n * p
    ph = [(0.2 * r, 0.1 * r, 0, 0.4 * r, 0.05, 2.0), (0, 0, 0, r, 0.4 * n_planes * p, 1.0)]
    resp = hy.generate_responses(b, ph, events, length, s_z, s_dl, seed=3)
    cfg = (n, n_planes, p, z_left, length, s_z, s_dl)
    s = oracle_setup(cfg)
    ora = oh.reconstruct(s, b.centers, m, resp, 0)
    geo, fr = ora["geo"], ora["frames"].copy()
    assert len(fr) > 4_000
    # events for the per-event kernel, among the others
    if n_planes > 1:  # on one plane their binary32 denominators are subnormal
        fr["right"][::50] += 8.6 * s_z  # (1 / D = inf in the reference too)
    fr["info_end"][7::60] += 3
    fr["info_end"] = np.minimum(fr["info_end"], len(geo["pos"]))
    fr["plane_end"][11::300] = fr["plane_begin"][11::300]
    fr["info_end"][13::300] = fr["info_begin"][13::300]
    fr["lor_index"][17::300] = fr["lor_index"][16::300][:len(fr["lor_index"][17::300])]
    with hy.HybridReconstruction(n, n, n_planes, p, z_left, length, s_z, s_dl) as rec:
        rec.set_geometry_soa(len(b.centers), geo["seg"][:, :4], geo["pix"], geo["pos"], ora["w"],
                             geo["lbeg"], geo["lend"])
        rec.set_sensitivity(ora["sens"], given=True)
        rec.set_frames(fr["lor_index"], fr["info_begin"], fr["info_end"], fr["plane_begin"],
                       fr["plane_end"], fr["up"], fr["right"], fr["tan"], fr["sec"])
        rec(2)
        img = rec.rho
        rec.rho = np.ones(rec.shape, np.float32)
        rec(1)
        one = rec.rho
        total = rec.stats()["n_events"]
    live = f32_live(s, geo, ora["w"], ora["sens"], fr)
    assert len(live) > 0.9 * total
    # one iteration from a uniform image: every live event adds sum = 1 / s
    f64, _ = oh.mlem(s, geo, ora["w"], ora["sens"], live, 1, f64=True)
    assert rel_l2(one, f64) < TOL
    f64, _ = oh.mlem(s, geo, ora["w"], ora["sens"], live, 2, f64=True)
    assert rel_l2(img, f64) < TOL
