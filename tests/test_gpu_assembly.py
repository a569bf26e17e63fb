"""GPU: assembly of the plain form's reduced camera system where its blocks change path:
blocks of at most Solver::kShortPairs pairs (one thread per row), longer ones in
chunks (few cameras: every block long; one pair per chunk remainder), and a point
seen twice by a camera.

The FP64 step against the oracle's at the tolerance of the other stage tests (1e-9).
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


# (cameras, points, tracks): 2 cameras: 3 blocks of thousands of pairs; 3: blocks around
# the chunk size; 40: short blocks and long diagonal ones; pairs per block near 48 and 256
@pytest.mark.parametrize("C,P,kmin,kmax", [(2, 3000, 2, 2), (3, 257, 2, 3), (5, 49, 3, 5), (40, 3000, 2, 8)])
def test_step_matches_oracle(gba, oracle, C, P, kmin, kmax):
    prob = gba.synthetic_custom(C, P, kmin, kmax, 1.5, seed=C + P)
    lam = 1e-2
    ref = oracle.schur_step(prob, lam, threads=2)
    with gba.Solver(prob, "plain") as s:
        s.set_schur_layout("dense")
        s.accumulate()
        assert s.damp_invert_v(lam) == 0
        assert s.schur_dense(lam) == 0
        dc = s.download("dc")
        s.back_substitute(lam)
        dp = s.download("dp")
    assert ref["status"] == 0
    assert rel_err(dc, ref["dc"]) < 1e-9
    assert rel_err(dp, ref["dp"]) < 1e-9


def test_point_seen_twice_by_a_camera(gba, oracle):
    prob = gba.synthetic_custom(4, 400, 2, 4, 1.5, seed=9)
    prob.obs_camera = np.concatenate([prob.obs_camera, prob.obs_camera[:300]])
    prob.obs_point = np.concatenate([prob.obs_point, prob.obs_point[:300]])
    prob.obs_pixel = np.concatenate([prob.obs_pixel, prob.obs_pixel[:600] + 0.5])
    lam = 1e-2
    ref = oracle.schur_step(prob, lam, threads=2)
    with gba.Solver(prob, "plain") as s:
        s.accumulate()
        assert s.damp_invert_v(lam) == 0 and s.schur_dense(lam) == 0
        assert rel_err(s.download("dc"), ref["dc"]) < 1e-9
