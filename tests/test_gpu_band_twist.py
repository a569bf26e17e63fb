"""GPU: the band that the automatic layout chooses, factored and solved from both
ends, against the explicit dense layout (FP64 kernels): the narrowest band that is
chosen, odd and even tile counts, wide bands, a shuffled camera order, and a system
that is not positive definite.

Tolerance: both solve the same 1e-3-damped system with backward errors of a few
n u; the band tests hold the same pair to 1e-10.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step(gba, prob, layout, lam):
    with gba.Solver(prob, "plain") as s:
        s.set_schur_layout(layout)
        s.accumulate()
        assert s.damp_invert_v(lam) == 0
        assert s.schur_dense(lam) == 0
        rows = s.schur_band()[0] if layout == "auto" else 0
        first = s.download("dc")
        assert s.schur_dense(lam) == 0  # again, over what the first left
        assert np.array_equal(first, s.download("dc"))
        return first, rows


@pytest.mark.parametrize("C,window", [(90, 4), (97, 4), (104, 4), (200, 9), (201, 20), (611, 10)])
def test_both_ends_match_dense(gba, C, window):
    prob = gba.synthetic_local(C, 100 * C, 2, min(8, window), 1.5, window, seed=C)
    band, rows = _step(gba, prob, "auto", 1e-3)
    assert rows > 0  # the band layout was chosen
    dense, _ = _step(gba, prob, "dense", 1e-3)
    assert np.linalg.norm(band - dense) <= 1e-10 * np.linalg.norm(dense)


def test_not_positive_definite(gba):
    prob = gba.synthetic_local(200, 20000, 2, 8, 1.5, 10, seed=1)
    with gba.Solver(prob, "plain") as s:
        s.accumulate()
        assert s.damp_invert_v(1e-3) == 0
        assert 1 <= s.schur_dense(-2.0) <= 9 * 200  # U_lambda with a negative diagonal
        assert s.schur_band()[0] > 0
        assert s.schur_dense(1e-3) == 0
        dc = s.download("dc")
    assert np.isfinite(dc).all()
    want, _ = _step(gba, prob, "dense", 1e-3)
    assert np.linalg.norm(dc - want) <= 1e-10 * np.linalg.norm(want)
