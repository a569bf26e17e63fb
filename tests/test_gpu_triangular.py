"""GPU: the tile-by-tile triangular solves (inverted diagonal tiles, one step per
tile) against numpy, at the sizes where the step's grid and the band's edges change.

Tolerance: the computed x of a Cholesky solve satisfies (A + dA) x = b with
|dA| <= c n u |L||L^T|, u = 2^-53; the residual is compared with 8 n u ||L||_F^2 ||x||
(the constant covers the inverted tiles' products: three 64-term sums per tile).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(gba, torch, L, b, n, ld, bt, band):
    dL, db = torch.from_numpy(np.ascontiguousarray(L)).cuda(), torch.from_numpy(b.copy()).cuda()
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    if band:
        gba.band_potrs(dL.data_ptr(), n, ld, bt, db.data_ptr(), info.data_ptr())
    else:
        gba.dense_potrs(dL.data_ptr(), n, ld, db.data_ptr(), info.data_ptr())
    torch.cuda.synchronize()
    return db.cpu().numpy()


# one tile; two; a grid of one block; more rows than two passes of the blocks cover
# (2 x 152 x 16 = 4,864); lda > n
@pytest.mark.parametrize("n,lda", [(64, 64), (128, 128), (320, 331), (1024, 1024), (5056, 5056)])
def test_dense_solve(gba, torch_cuda, n, lda):
    rng = np.random.default_rng(n)
    L = np.tril(rng.normal(size=(n, n)) / np.sqrt(n))
    L[np.diag_indices(n)] = 1.0 + rng.random(n)
    stored = np.full((n, lda), np.nan)  # rows of this array are columns of the matrix
    stored[:, :n] = L.T
    b = rng.normal(size=n)
    x = _solve(gba, torch_cuda, stored, b, n, lda, 0, False)
    r = L @ (L.T @ x) - b
    assert np.linalg.norm(r) <= 8 * n * 2.0**-53 * np.linalg.norm(L) ** 2 * np.linalg.norm(x)


@pytest.mark.parametrize("n,bt", [(64, 0), (256, 0), (448, 1), (704, 4), (320, 4)])
def test_band_solve(gba, torch_cuda, n, bt):
    rng = np.random.default_rng(10 * n + bt)
    t = np.arange(n) // 64
    L = np.tril(rng.normal(size=(n, n)) * (t[:, None] - t[None, :] <= bt) / 16)
    L[np.diag_indices(n)] = 1.0 + rng.random(n)
    ldb = (bt + 2) * 64
    stored = np.full((n, ldb), np.nan)
    for j in range(n):
        m = min(n, (j // 64 + bt + 1) * 64) - j
        stored[j, :m] = L[j:j + m, j]
    b = rng.normal(size=n)
    x = _solve(gba, torch_cuda, stored, b, n, ldb, bt, True)
    r = L @ (L.T @ x) - b
    assert np.linalg.norm(r) <= 8 * n * 2.0**-53 * np.linalg.norm(L) ** 2 * np.linalg.norm(x)


def test_failed_factorisation_leaves_b(gba, torch_cuda):
    torch = torch_cuda
    L, b = torch.eye(128, dtype=torch.float64, device="cuda"), torch.ones(128, dtype=torch.float64, device="cuda")
    info = torch.full((1,), 5, dtype=torch.int32, device="cuda")
    gba.dense_potrs(L.data_ptr(), 128, 128, b.data_ptr(), info.data_ptr())
    torch.cuda.synchronize()
    assert bool((b == 1).all())
