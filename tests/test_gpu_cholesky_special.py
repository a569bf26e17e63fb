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


def _cholesky_long_double(A):
    A = A.astype(np.longdouble).copy()
    L = np.zeros_like(A)
    for k in range(len(A)):
        L[k:, k] = A[k:, k] / np.sqrt(A[k, k])
        A[k + 1:, k + 1:] -= np.outer(L[k + 1:, k], L[k + 1:, k])
    return L


@pytest.mark.parametrize("coupling", [2.0**-k for k in (3, 10, 20, 40, 60, 80)])
def test_entries_far_below_the_diagonal(gba, torch_cuda, coupling):
    """Blocks of nine coupled weakly: every entry of the factor within 16 units of 2^-60 of
    its row's scale (at most sqrt(8 A_ii)) of the exact one, and an ulp of its own: what
    the call promises of a coupling, however weak. Below 2^-62 the blocks are factored as
    if there were none."""
    torch = torch_cuda
    n = 192
    A = coupling * _spd(n, 7)
    for k in range(0, n, 9):
        m = min(9, n - k)
        A[k:k + m, k:k + m] = _spd(m, k)
    d, info = torch.from_numpy(A).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
    gba.dense_potrf(d.data_ptr(), n, n, info.data_ptr())
    torch.cuda.synchronize()
    assert int(info.item()) == 0
    want = _cholesky_long_double(A)
    err = np.abs(np.tril(d.cpu().numpy().T) - want)
    assert (err <= 16 * 2.0**-60 * np.sqrt(8 * np.diag(A))[:, None] + 2.0**-53 * np.abs(want)).all()
