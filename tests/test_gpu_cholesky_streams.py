"""GPU: the fixed-point factorisation beside other work on the GPU. Its kernels then
get their SMs a few at a time, so blocks of one launch start when others of it have
ended; sums of integers do not depend on the order, so every result is, bit for bit,
what the call gives alone.
"""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(torch, n, bt, seed):
    """SPD, its nonzeros within bt 64-row tiles below each diagonal tile, and a right-hand side."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.arange(n, device="cuda") // 64
    M = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64) * ((t[:, None] - t[None, :]).abs() <= bt)
    A = M + M.T
    A.diagonal().add_(A.abs().sum(dim=1).max())
    return A, torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


def _band(A, n, ldb):
    out = A.new_zeros(n, ldb)
    for j in range(n):
        m = min(n - j, ldb - 64)
        out[j, :m] = A[j:j + m, j]
    return out


def _factor_and_solve(gba, torch, stored, b, n, ld, bt, stream):
    L, x, info = stored.clone(), b.clone(), torch.zeros(1, dtype=torch.int32, device="cuda")
    st = stream.cuda_stream
    if bt is None:
        gba.dense_potrf(L.data_ptr(), n, ld, info.data_ptr(), st)
        gba.dense_potrs(L.data_ptr(), n, ld, x.data_ptr(), info.data_ptr(), st)
    else:
        gba.band_potrf(L.data_ptr(), n, ld, bt, info.data_ptr(), st)
        gba.band_potrs(L.data_ptr(), n, ld, bt, x.data_ptr(), info.data_ptr(), st)
    return L, x, info


# 64 tiles (tensor-core update, panels over all SMs), 12 (integer update), a band
@pytest.mark.parametrize("n,bt", [(4096, None), (832, None), (5504, 3)])
def test_two_streams_and_a_busy_gpu(gba, torch_cuda, n, bt):
    torch = torch_cuda
    ld = n if bt is None else 64 * (bt + 2)
    inputs = []
    for seed in (1, 2):
        A, b = _spd(torch, n, n if bt is None else bt, seed)
        inputs.append((A if bt is None else _band(A, n, ld), b))
    main = torch.cuda.current_stream()
    want = [_factor_and_solve(gba, torch, s, b, n, ld, bt, main) for s, b in inputs]
    torch.cuda.synchronize()
    assert all(int(info.item()) == 0 for _, _, info in want)
    load = torch.randn(2048, 2048, device="cuda")

    def run(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            out = [_factor_and_solve(gba, torch, *inputs[k], n, ld, bt, stream) for _ in range(8)]
            stream.synchronize()
        return all(torch.equal(g, w) for o in out for g, w in zip(o, want[k]))

    def busy(_):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(200):
                load @ load
            stream.synchronize()
        return True

    torch.cuda.synchronize()
    with ThreadPoolExecutor(3) as pool:
        jobs = [pool.submit(run, 0), pool.submit(run, 1), pool.submit(busy, 0)]
        assert all(j.result() for j in jobs)


@pytest.mark.parametrize("n", [64, 1024])
def test_solves_with_factors_in_turn(gba, torch_cuda, n):
    """Two factors in turn: each solve's workspace holds the inverted tiles of the other's."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(n)
    factors = []
    for _ in range(2):
        U = torch.triu(torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64) / n**0.5)  # row j: column j
        U.diagonal().copy_(1.0 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
        factors.append(U)
    b = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    got = []
    for k in range(100):
        x = b.clone()
        gba.dense_potrs(factors[k % 2].data_ptr(), n, n, x.data_ptr(), info.data_ptr(), stream)
        got.append(x)
    torch.cuda.synchronize()
    assert all(torch.equal(x, got[k % 2]) for k, x in enumerate(got))
    for U, x in zip(factors, got):
        r = U.T @ (U @ x) - b
        assert float(r.norm()) <= 8 * n * 2.0**-53 * float(U.norm()) ** 2 * float(x.norm())


def test_two_solvers_in_two_threads(gba):
    """One with the dense layout, one with the band that is factored from both ends."""
    probs = [gba.synthetic_custom(200, 20000, 2, 8, 1.6, seed=4), gba.synthetic_local(400, 40000, 2, 8, 1.5, 10, seed=5)]

    def steps(prob):
        with gba.Solver(prob, "plain") as s:
            s.accumulate()
            assert s.damp_invert_v(1e-3) == 0
            out = []
            for _ in range(12):
                assert s.schur_dense(1e-3) == 0
                out.append(s.download("dc"))
            return out

    want = [steps(p)[0] for p in probs]
    with ThreadPoolExecutor(2) as pool:
        for got, w in zip(pool.map(steps, probs), want):
            assert all(np.array_equal(g, w) for g in got)
