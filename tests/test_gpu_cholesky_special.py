"""GPU: the fixed-point factorisation on inputs that FP64 arithmetic refuses: the failed
column is FP64's (a plain column-by-column factorisation in numpy).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(n, seed):
    B = np.random.default_rng(seed).normal(size=(n, n))
    return B @ B.T / n + 0.5 * np.eye(n)


def _fp64_failed_column(A):
    L = np.tril(A)
    with np.errstate(all="ignore"):
        for k in range(len(L)):
            if not L[k, k] > 0.0:
                return k + 1
            L[k, k] = np.sqrt(L[k, k])
            L[k + 1:, k] *= 1.0 / L[k, k]
            L[k + 1:, k + 1:] -= np.tril(np.outer(L[k + 1:, k], L[k + 1:, k]))
    return 0


def _info(gba, torch, A):
    n = len(A)
    d, info = torch.from_numpy(np.ascontiguousarray(A)).cuda(), torch.full((1,), -7, dtype=torch.int32, device="cuda")
    gba.dense_potrf(d.data_ptr(), n, n, info.data_ptr())
    torch.cuda.synchronize()
    return int(info.item())


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e300, 3.0])
@pytest.mark.parametrize("row,col", [(70, 3), (70, 66), (100, 70), (190, 70)])
def test_entry_beside_an_infinite_diagonal(gba, torch_cuda, row, col, value):
    """Row and column 70 have an infinite diagonal entry; finite entries there do not matter
    (unless their squares overflow in the row), others refuse their row."""
    A = _spd(192, 5)
    A[70, 70] = np.inf
    A[row, col] = A[col, row] = value
    assert _info(gba, torch_cuda, A) == _fp64_failed_column(A)
