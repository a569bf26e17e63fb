"""GPU: residuals and Jacobians of single observations over all rotation angles and
the edges of a warp, and the batched blocks' root-free path beside the Cholesky
path that decides for pivots that are not clearly positive.

The reference residual is evaluated in extended precision with the rotation's sine
and cosine, its derivatives by complex steps. Tolerances: about 165 roundings of
1.1e-16 (6e-8 in FP32), amplified at most tenfold by the depth of 2 to 6 under
focal length and distortion, relative to the largest entry: 1e-12 and 1e-4. Blocks:
the inverse of a matrix of condition 1e3 loses three of 16 digits, in about 100
roundings: 1e-11.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _residual(cam, X, obs):
    a, t = cam[:3], cam[3:6]
    th2 = (a * a).sum()
    cross = np.array([a[1] * X[2] - a[2] * X[1], a[2] * X[0] - a[0] * X[2], a[0] * X[1] - a[1] * X[0]])
    if th2.real > 1e-24:
        th = np.sqrt(th2)
        P = np.cos(th) * X + np.sin(th) / th * cross + (2 * np.sin(th / 2) ** 2 / th2) * (a * X).sum() * a + t
    else:
        P = X + cross + t
    u, v = -P[0] / P[2], -P[1] / P[2]
    r2 = u * u + v * v
    d = 1 + r2 * (cam[7] + cam[8] * r2)
    return np.array([cam[6] * d * u, cam[6] * d * v]) - obs


def _reference(cam, X, obs):
    z = np.concatenate([cam, X]).astype(np.clongdouble)
    r = _residual(z[:9], z[9:], obs).real
    J, h = np.empty((2, 12)), np.longdouble(1e-30)
    for k in range(12):
        s = z.copy()
        s[k] += 1j * h
        J[:, k] = (_residual(s[:9], s[9:], obs).imag / h).astype(np.float64)
    return r.astype(np.float64), J[:, :9], J[:, 9:]


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 1e-4)])
@pytest.mark.parametrize("E", [1, 31, 33, 129])
def test_edges_at_all_angles(gba, torch_cuda, E, precision, tol):
    torch = torch_cuda
    rng = np.random.default_rng(E)
    angles = np.array([1e-6, 1e-3, 0.3, 1.0, 2.5, 3.1, 3.162, 3.163, 3.5, 6.0, 40.0])
    C, P = len(angles), 7
    axes = rng.normal(size=(C, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    cams = np.concatenate([axes * angles[:, None], rng.normal(0, 0.1, (C, 2)), np.full((C, 1), -4.0),
                           rng.uniform(400, 600, (C, 1)), rng.normal(0, 0.02, (C, 2))], 1)
    pts = rng.uniform(-1, 1, (P, 3))
    oc, op = rng.integers(0, C, E).astype(np.int32), rng.integers(0, P, E).astype(np.int32)
    px = rng.normal(0, 100, (E, 2))
    dt = torch.float64 if precision == 64 else torch.float32
    dev = [torch.from_numpy(v).cuda() for v in (cams, pts, oc, op, px)]
    outs = [torch.full((E + 1, n), 7.0, dtype=dt, device="cuda") for n in (2, 18, 6)]
    gba.eval_edges(precision, *[t.data_ptr() for t in dev], E, *[t.data_ptr() for t in outs])
    torch.cuda.synchronize()
    got = [t.cpu().numpy().astype(np.float64) for t in outs]
    for g in got:
        assert (g[E] == 7.0).all()  # nothing behind the last row
    for e in range(E):
        c = cams[oc[e]]
        if precision == 32:
            c = c.astype(np.float32).astype(np.float64)
        ref = _reference(c, pts[op[e]], px[e])
        for g, r in zip(got, ref):
            assert np.abs(g[e] - r.ravel()).max() <= tol * max(np.abs(r).max(), 500.0 if r.shape == (2,) else 0.0)


@pytest.mark.parametrize("n", [1, 31, 33, 131, 9999])  # 9,999: more than 64 per SM
def test_blocks_on_both_paths(gba, torch_cuda, n):
    torch = torch_cuda
    rng = np.random.default_rng(n)
    for k in (9, 3):
        Q = np.linalg.qr(rng.normal(size=(n, k, k)))[0]
        A = np.einsum("nij,nj,nkj->nik", Q, 10.0 ** rng.uniform(0, 3, (n, k)), Q)
        A = 0.5 * (A + A.transpose(0, 2, 1))
        kind = np.arange(n) % 5
        for i in range(n):
            if kind[i] == 1:  # diagonal, pivots whose reciprocal is not a normal number
                A[i] = np.diag(np.full(k, 1e-300))
            elif kind[i] == 2:
                A[i] = np.ones((k, k))  # singular
            elif kind[i] == 3:
                A[i, k - 1, k - 1] = -1.0
            elif kind[i] == 4:
                A[i, 0, 0] = np.nan
        spd = kind < 2
        b = rng.normal(size=(n, k)) * np.where(kind == 1, 1e-300, 1.0)[:, None]
        dA, db = torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda()
        ok = torch.full((n + 1,), 7, dtype=torch.int32, device="cuda")
        out = torch.full((n + 1, k if k == 9 else k * k), 7.0, dtype=torch.float64, device="cuda")
        if k == 9:
            gba.batch_chol9_factor_solve(dA.data_ptr(), db.data_ptr(), out.data_ptr(), ok.data_ptr(), n)
        else:
            gba.batch_inverse3_spd(dA.data_ptr(), out.data_ptr(), ok.data_ptr(), n)
        torch.cuda.synchronize()
        o, flags = out.cpu().numpy(), ok.cpu().numpy()
        assert flags[n] == 7 and (o[n] == 7.0).all()
        assert (flags[:n] == spd).all()
        assert (o[:n][~spd] == 7.0).all()  # left as it was
        for i in np.flatnonzero(spd):
            ref = (np.linalg.solve(A[i] / A[i, 0, 0], b[i] / A[i, 0, 0]) if k == 9 else np.linalg.inv(A[i]).ravel())
            assert np.abs(o[i] - ref).max() <= 1e-11 * np.abs(ref).max()
