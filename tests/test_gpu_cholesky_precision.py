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


@pytest.mark.parametrize("n", [832, 2048, 4096])  # integer updates only; mostly and nearly all tensor-core updates
def test_residual_of_large_factors(gba, torch_cuda, n):
    """Root mean square of (A - L L^T)_ij / sqrt(A_ii A_jj) over sampled entries, in long
    double. An entry of A is rounded once per panel at 2^-62 of a scale that makes its
    diagonal at least 1/8, so at most sqrt(n / 64) 8 2^-62 / sqrt(12); the factor's own
    rounding to FP64, here with entries near 2 / sqrt(n), adds up to 2^-53 of those (FP64
    arithmetic on such a matrix: 2^-53 of an entry for each of n sums, 1e-17 at 4,096)."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(n)
    B = torch.randn(n, n // 2, generator=g, device="cuda", dtype=torch.float64)
    A = B @ B.T / (n // 2)
    A.diagonal().add_(0.3)
    d, info = A.clone(), torch.zeros(1, dtype=torch.int32, device="cuda")
    gba.dense_potrf(d.data_ptr(), n, n, info.data_ptr(), torch.cuda.current_stream().cuda_stream)
    L, A = torch.triu(d).T.cpu().numpy(), A.cpu().numpy()
    assert int(info.item()) == 0
    rng = np.random.default_rng(n)
    pairs = np.sort(rng.integers(0, n, (2000, 2)), axis=1)
    r = [float(A[i, j] - np.dot(L[i, :i + 1].astype(np.longdouble), L[j, :i + 1].astype(np.longdouble)))
         / np.sqrt(A[i, i] * A[j, j]) for i, j in pairs]
    rms = float(np.sqrt(np.mean(np.square(r))))
    print(n, rms)
    assert rms <= np.sqrt(n / 64) * 8 * 2.0**-62 / np.sqrt(12) + 2.0**-53 * 2 / np.sqrt(n)
