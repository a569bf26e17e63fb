"""GPU: the fixed-point Cholesky (panel, tensor-core update, dense and band) against
long double / numpy at the sizes where its work splits differently.

Tolerance of the factor: the scaled entries are exact sums rounded at 2^-60 and the
results round to FP64, so the error relative to a row's diagonal root stays within
2^-52 (an ulp of an entry near 1) plus n units of 2^-58 amplified by the condition
number of the leading blocks (well conditioned here, below 8).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factor(gba, torch, A, lda=None):
    n = A.shape[0]
    lda = lda or n
    stored = np.full((n, lda), 7.0)
    stored[:, :n] = np.triu(A) + np.tril(np.full_like(A, np.nan), -1)  # column-major lower; the upper one is not read
    d = torch.from_numpy(stored).cuda()
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    gba.dense_potrf(d.data_ptr(), n, lda, info.data_ptr())
    torch.cuda.synchronize()
    out = d.cpu().numpy()
    assert np.all(out[:, n:] == 7.0)
    return np.tril(out[:, :n].T), int(info.item())


def _cholesky_long_double(A):
    A = A.astype(np.longdouble).copy()
    L = np.zeros_like(A)
    for k in range(len(A)):
        L[k:, k] = A[k:, k] / np.sqrt(A[k, k])
        A[k + 1:, k + 1:] -= np.outer(L[k + 1:, k], L[k + 1:, k])
    return L


def _spd(n, seed, spread=0.0):
    rng = np.random.default_rng(seed)
    B = rng.normal(size=(n, n))
    A = B @ B.T / n + 0.5 * np.eye(n)
    d = 2.0 ** rng.uniform(-spread, spread, n)
    return A * d[:, None] * d[None, :]


# one tile; one and two row tiles below; odd and even numbers of tiles; rows scaled over 2^+-300
@pytest.mark.parametrize("n,lda,spread", [(64, 64, 0), (128, 130, 20), (192, 192, 300), (256, 256, 3), (448, 449, 8)])
def test_factor_matches_long_double(gba, torch_cuda, n, lda, spread):
    A = _spd(n, n, spread)
    L, info = _factor(gba, torch_cuda, A, lda)
    assert info == 0
    want = _cholesky_long_double(A)
    err = np.abs(L - want) / np.sqrt(np.diag(A).astype(np.longdouble))[:, None]
    assert float(err.max()) <= 2.0**-52 + n * 2.0**-58 * 8


# rows per CTA above the fused group (16 x 152 rows), a second pass of 128 rows
@pytest.mark.parametrize("n", [832, 896, 2688, 5120])  # 12 and 13 tiles: either side of the update kernels
def test_large_factor_residual(gba, torch_cuda, n):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(n)
    B = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)
    A = B @ B.T / n
    A.diagonal().add_(0.5)
    d, info = A.clone(), torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    gba.dense_potrf(d.data_ptr(), n, n, info.data_ptr(), stream)
    L = torch.triu(d).T
    want = torch.linalg.cholesky(A)
    assert int(info.item()) == 0
    # FP64's own error is below 4 n u for this conditioning; the difference is held to that
    assert float((L - want).abs().max()) <= 4 * n * 2.0**-53


@pytest.mark.parametrize("n,col", [(64, 0), (64, 63), (128, 64), (320, 200), (320, 319)])
@pytest.mark.parametrize("kind", ["negative", "zero", "nan", "indefinite", "nan below", "large"])
def test_failed_column(gba, torch_cuda, n, col, kind):
    if kind in ("indefinite", "nan below", "large") and col == 0:
        pytest.skip("needs a column before it")
    A = _spd(n, 3)
    if kind in ("negative", "zero", "nan"):
        A[col, col] = {"negative": -1.0, "zero": 0.0, "nan": np.nan}[kind]
    else:
        A[col, 0] = A[0, col] = {"indefinite": 1.5 * np.sqrt(A[col, col] * A[0, 0]), "nan below": np.nan, "large": 1e200}[kind]
    assert _factor(gba, torch_cuda, A)[1] == col + 1


def test_infinite_weight(gba, torch_cuda):
    """An infinite diagonal entry is a pivot of weight infinity, as in FP64 arithmetic: success, and a zero step there."""
    torch = torch_cuda
    n, k = 192, 70
    A = _spd(n, 5)
    B = A.copy()
    A[k, k] = np.inf
    d, info = torch.from_numpy(A).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
    gba.dense_potrf(d.data_ptr(), n, n, info.data_ptr())
    b = np.random.default_rng(1).normal(size=n)
    x = torch.from_numpy(b.copy()).cuda()
    gba.dense_potrs(d.data_ptr(), n, n, x.data_ptr(), info.data_ptr())
    torch.cuda.synchronize()
    assert int(info.item()) == 0
    x = x.cpu().numpy()
    keep = np.arange(n) != k
    want = np.linalg.solve(B[np.ix_(keep, keep)], b[keep])
    assert x[k] == 0.0
    assert np.max(np.abs(x[keep] - want)) <= 1e-12 * np.max(np.abs(want))


def test_reruns_are_identical(gba, torch_cuda):
    A = _spd(704, 9)
    a, b = _factor(gba, torch_cuda, A)[0], _factor(gba, torch_cuda, A)[0]
    assert np.array_equal(a, b)
