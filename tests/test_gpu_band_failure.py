"""GPU: a band that is factored from both ends and is not positive definite reports the
column that the rows in their order report (the explicitly chosen band), on every call,
also where both ends meet a bad pivot in the same launch.
"""
import pytest

pytestmark = pytest.mark.gpu


def _infos(gba, prob, layout, lam, times):
    with gba.Solver(prob, "plain") as s:
        s.set_schur_layout(layout)
        s.accumulate()
        assert s.damp_invert_v(1e-3) == 0
        out = [s.schur_dense(lam) for _ in range(times)]
        assert s.schur_band()[0] > 0
        assert s.schur_dense(1e-3) == 0  # and recovers
        return out


# every diagonal entry negative; only some pivots bad
@pytest.mark.parametrize("lam", [-2.0, -0.5])
@pytest.mark.parametrize("C,window", [(104, 4), (200, 10)])
def test_failed_column_is_that_of_the_rows_in_order(gba, C, window, lam):
    prob = gba.synthetic_local(C, 100 * C, 2, min(8, window), 1.5, window, seed=C)
    want = _infos(gba, prob, "band", lam, 1)[0]
    assert want > 0
    assert _infos(gba, prob, "auto", lam, 20) == [want] * 20
