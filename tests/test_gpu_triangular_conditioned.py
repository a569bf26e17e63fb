"""GPU: the triangular solves with ill-conditioned diagonal tiles are as backward stable as
substitution: the componentwise backward error max |b - L L^T x| / (|L||L^T||x|) of the
solution, in long double, added up over matrices and compared with that of a plain FP64
substitution in numpy on the same factors. Both are a few tenths of a rounding error (the
bound is n of them), so a sum over 24 matrices scatters by a few per cent: a quarter more
is allowed. Inverted tiles without a refinement come to four times as much at 64 rows.
"""
import numpy as np
import pytest

from test_gpu_triangular import _solve

pytestmark = pytest.mark.gpu


def _substitution(L, b):
    x = b.copy()
    for k in range(len(L)):
        x[k] /= L[k, k]
        x[k + 1:] -= L[k + 1:, k] * x[k]
    for k in reversed(range(len(L))):
        x[k] /= L[k, k]
        x[:k] -= L[k, :k] * x[k]
    return x


def _backward_error(L, b, x):
    Ll, xl = L.astype(np.longdouble), x.astype(np.longdouble)
    return float(np.max(np.abs(Ll @ (Ll.T @ xl) - b) / (np.abs(Ll) @ (np.abs(Ll).T @ np.abs(xl)))))


@pytest.mark.parametrize("n", [64, 192])
@pytest.mark.parametrize("low,spread", [(1e-3, 0), (1e-6, 0), (1e-13, 0), (1e-6, 20)])
def test_backward_error_of_substitution(gba, torch_cuda, n, low, spread):
    ours = theirs = 0.0
    for seed in range(24):
        rng = np.random.default_rng(seed)
        Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
        L = np.linalg.cholesky((Q * np.geomspace(1.0, low, n)) @ Q.T) * 2.0 ** rng.uniform(-spread, spread, n)[:, None]
        b = rng.normal(size=n)
        x = _solve(gba, torch_cuda, np.triu(L.T), b, n, n, 0, False)
        ours += _backward_error(L, b, x)
        theirs += _backward_error(L, b, _substitution(L, b))
    print(n, low, spread, ours / 24 / 2.0**-53, theirs / 24 / 2.0**-53)
    assert ours <= 1.25 * theirs


def test_infinite_weight_beside_an_ill_conditioned_tile(gba, torch_cuda):
    """A row of infinite weight: x = 0 there, the others refined as without it."""
    n, k = 128, 30
    rng = np.random.default_rng(1)
    Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
    L = np.linalg.cholesky((Q * np.geomspace(1.0, 1e-8, n)) @ Q.T)
    L[k], L[:, k] = 0.0, 0.0
    b = rng.normal(size=n)
    keep = np.arange(n) != k
    inf = L.copy()
    inf[k, k] = np.inf
    x = _solve(gba, torch_cuda, np.triu(inf.T), b, n, n, 0, False)
    assert x[k] == 0.0
    sub = L[np.ix_(keep, keep)]
    assert _backward_error(sub, b[keep], x[keep]) <= 2 * max(_backward_error(sub, b[keep], _substitution(sub, b[keep])), 2.0**-53)
