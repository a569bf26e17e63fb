"""GPU: the fixed-point factorisation is no less precise than FP64 arithmetic: its error
against long double beside that of numpy's FP64 factor of the same matrix, up to
condition numbers of 4e5 and with rows scaled apart. (An FP64 factorisation rounds
every entry of every Schur complement at 2^-53 of it; this one at 2^-60 of the diagonal.)
"""
import numpy as np
import pytest

from test_gpu_cholesky import _cholesky_long_double, _factor

pytestmark = pytest.mark.gpu


def _matrix(n, c, seed, spread):
    rng = np.random.default_rng(seed)
    B = rng.normal(size=(n, n))
    d = 2.0 ** rng.uniform(-spread, spread, n)
    return (B @ B.T / n + c * np.eye(n)) * d[:, None] * d[None, :]


def _error(L, want, A):
    return float(np.linalg.norm(((L - want) / np.sqrt(np.diag(A).astype(np.longdouble))[:, None]).astype(float)))


@pytest.mark.parametrize("n,c,spread", [(64, 1e-3, 0), (192, 0.3, 4), (192, 1e-3, 0), (192, 1e-5, 0), (448, 1e-3, 9)])
def test_factor_no_less_precise_than_fp64(gba, torch_cuda, n, c, spread):
    ratios = []
    for seed in range(3):
        A = _matrix(n, c, seed, spread)
        want = _cholesky_long_double(A)
        L, info = _factor(gba, torch_cuda, A)
        assert info == 0
        ratios.append(_error(L, want, A) / _error(np.linalg.cholesky(A), want, A))
    print(n, c, ratios)
    assert max(ratios) <= 1.0
