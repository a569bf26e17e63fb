"""GPU: the buffer of S holds the factor after schur_dense, also of a band that the
automatic layout solves from both ends: read after the step, and through a device
pointer taken before further steps. It is compared with the explicitly chosen band's
(FP64): both factor the same matrix, condition number below 1e8, to FP64's precision.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LAM = 1e-3


def _lower(S, n, bt):
    S = S.reshape(n, -1)
    out = np.zeros_like(S)
    for j in range(n):
        m = min(n, (j // 64 + bt + 1) * 64) - j
        out[j, :m] = S[j, :m]
    return out


def _start(s):
    s.accumulate()
    assert s.damp_invert_v(LAM) == 0
    assert s.schur_dense(LAM) == 0


@pytest.fixture(scope="module")
def prob(gba):
    return gba.synthetic_local(200, 20000, 2, 8, 1.5, 10, seed=3)


@pytest.fixture(scope="module")
def factor(gba, prob):
    with gba.Solver(prob, "plain") as s:
        s.set_schur_layout("band")
        _start(s)
        ldb, bt, _ = s.schur_band()
        n = s.dims()[3]
        return _lower(s.download("S"), n, bt), n, bt


def _check(S, factor):
    want, n, bt = factor
    got = _lower(S, n, bt)
    scale = np.sqrt((want**2).sum())
    assert np.sqrt(((got - want) ** 2).sum()) <= 1e-9 * scale


def test_download_after_the_step(gba, prob, factor):
    with gba.Solver(prob, "plain") as s:
        _start(s)
        first = s.download("dc")
        _check(s.download("S"), factor)
        assert s.schur_dense(LAM) == 0
        _check(s.download("S"), factor)
        assert np.array_equal(first, s.download("dc"))  # reading S does not change the step


def test_device_pointer_through_later_steps(gba, torch_cuda, prob, factor):
    torch = torch_cuda
    with gba.Solver(prob, "plain") as s:
        _start(s)
        ptr, count = s.device_ptr("S"), s.download("S").size

        class View:
            __cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (ptr, False), "version": 2}

        view = torch.as_tensor(View(), device="cuda")
        for _ in range(2):
            assert s.schur_dense(LAM) == 0
            _check(view.cpu().numpy(), factor)
