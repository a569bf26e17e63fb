"""GPU: the explicitly chosen layouts of S are factored in FP64, the band as the dense
matrix: the same operations on the same numbers, so the factors agree bit for bit where
the band has entries (cameras in their own order, tiles outside the band exactly zero).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factor(gba, prob, layout, lam):
    with gba.Solver(prob, "plain") as s:
        s.set_schur_layout(layout)
        s.accumulate()
        assert s.damp_invert_v(lam) == 0
        assert s.schur_dense(lam) == 0
        n = s.dims()[3]
        ldb, bt, perm = s.schur_band()
        return s.download("S").reshape(n, -1), n, bt, perm, s.download("dc")


@pytest.mark.parametrize("C,window", [(60, 6), (200, 12)])
def test_band_factor_is_the_dense_fp64_factor(gba, C, window):
    prob = gba.synthetic_local(C, 100 * C, 2, 8, 1.5, window, seed=C)
    band, n, bt, perm, dc_band = _factor(gba, prob, "band", 1e-3)
    dense, _, _, _, dc = _factor(gba, prob, "dense", 1e-3)
    assert np.array_equal(perm, np.arange(C))
    for j in range(n):
        m = min(n, (j // 64 + bt + 1) * 64) - j
        assert np.array_equal(band[j, :m], dense[j, j:j + m]), j
        assert not dense[j, j + m:].any()
    assert np.array_equal(dc_band, dc)
