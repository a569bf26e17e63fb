"""GPU: the one-kernel end of a PCG iteration and the persistent one-pass product
at the edges of their ranges: fewer cameras than CTAs of the cluster, the last
camera count with one thread per row (1,808) and the first beyond, the last count
the cluster takes (24,000) and the first that the separate kernels do, points in
warp runs, CTA lists and single ranges in one problem.

The refinement residual is computed by float-float products that share nothing
with these kernels: reaching 1e-10 means that the steps solved the system. A
preconditioner or a sum that leaves something out still converges, but later, so
the iterations are bounded too: against a block-Jacobi PCG in FP64 on the
assembled matrix (the FP32 recurrences may take two iterations more or less per
inner solve), and at the range's edges against the neighbouring count (a problem
of the same distribution: a quarter and three iterations).
"""
import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu
MODEL = PKG / "models" / "coarse_mlp.bin"
LAM = 1e-2
OPTS = dict(refine_tol=1e-10, refine_max_steps=12, pcg_tol=1e-4, pcg_max_iters=400)


def _solve(gba, prob, mode):
    with gba.Solver(prob, "learned") as s:
        s.load_model(MODEL)
        s.set_preconditioner(mode)
        s.accumulate()
        assert s.damp_invert_v(LAM) == 0
        return s.schur_pcg(LAM, learned=True, **OPTS)


def _reference_iterations(S, rhs, C):
    blocks = np.stack([np.linalg.inv(S[9 * c:9 * c + 9, 9 * c:9 * c + 9]) for c in range(C)])
    prec = lambda v: np.einsum("cij,cj->ci", blocks, v.reshape(C, 9)).ravel()  # noqa: E731
    x, r, its, steps = np.zeros_like(rhs), rhs.copy(), 0, 0
    while np.linalg.norm(r) > OPTS["refine_tol"] * np.linalg.norm(rhs):
        e, q, z = np.zeros_like(r), r.copy(), prec(r)
        p, rz, stop = z.copy(), r @ z, OPTS["pcg_tol"] * np.linalg.norm(r)
        while np.linalg.norm(q) > stop:
            Sp = S @ p
            a = rz / (p @ Sp)
            e, q = e + a * p, q - a * Sp
            z = prec(q)
            rz, old = q @ z, rz
            p = z + rz / old * p
            its += 1
        x, steps = x + e, steps + 1
        r = rhs - S @ x
    return its, steps


@pytest.mark.parametrize("C,P,track", [(3, 40, 3), (17, 300, 6), (150, 400, 140), (300, 500, 290)])
def test_iterations_match_fp64_pcg(gba, C, P, track):
    prob = gba.synthetic_custom(C, P, 2, track, 1.1, seed=C)
    with gba.Solver(prob, "plain") as s:
        s.set_schur_layout("dense")
        s.accumulate()
        assert s.damp_invert_v(LAM) == 0
        assert s.schur_dense(LAM) == 0
        n_pad = s.dims()[3]
        L = np.tril(s.download("S").reshape(n_pad, n_pad).T[:9 * C, :9 * C])
        dc = s.download("dc")
    S = L @ L.T
    ref_it, ref_steps = _reference_iterations(S, S @ dc, C)
    it, steps, rr = _solve(gba, prob, "block-jacobi")
    assert rr <= OPTS["refine_tol"]
    assert abs(it - ref_it) <= 2 * max(steps, ref_steps) + 2
    it_l, steps_l, rr_l = _solve(gba, prob, "learned")
    assert rr_l <= OPTS["refine_tol"]
    assert it_l <= 2 * ref_it + 2 * steps_l  # the correction is not worse than this on any basis of these sizes


@pytest.mark.parametrize("mode", ["block-jacobi", "learned"])
@pytest.mark.parametrize("C", [1808, 24000])
def test_edges_of_the_range(gba, C, mode):
    its = []
    for c in (C, C + 1):
        it, steps, rr = _solve(gba, gba.synthetic_custom(c, 12 * c, 2, 8, 1.3, seed=5), mode)
        assert rr <= OPTS["refine_tol"]
        its.append(it)
    assert abs(its[0] - its[1]) <= max(its) / 4 + 3


def test_two_sizes_in_two_threads(gba):
    """Solvers of different sizes share the kernels (and their launch attributes)."""
    from concurrent.futures import ThreadPoolExecutor

    probs = [gba.synthetic_custom(C, 10 * C, 2, 8, 1.3, seed=C) for C in (100, 12000)]
    with ThreadPoolExecutor(2) as pool:
        runs = list(pool.map(lambda p: [_solve(gba, p, "learned") for _ in range(6)], probs))
    for run in runs:
        for it, steps, rr in run:
            assert rr <= OPTS["refine_tol"]
