"""GPU: the MLP's forward and backward kernels at the edges of their row groups
(32 rows per CTA; more rows than one group per SM) against the CPU oracle.

Tolerances: kernel and oracle round the same operands to BF16, but an activation
that FP32 summation moves across a rounding boundary differs by one BF16 ulp
(2^-8 of it) afterwards. One such operand per output bounds the forward pass
(2^-8 of the largest output), two the gradients (2^-7 of the largest entry). The
group's last rows weigh 50 times the others, so that a row left out or counted
twice shows.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,offset", [(1, 0), (31, 0), (33, 1), (1000, 0), (9731, 3)])
def test_batches_match_oracle(gba, torch_cuda, B, offset):
    import mlp_oracle as mo

    torch = torch_cuda
    rng = np.random.default_rng(B)
    params = np.concatenate([rng.normal(0, s, n) for s, n in ((0.2, 128 * 64), (0.1, 128), (0.12, 128 * 128),
                                                              (0.1, 128), (0.1, 96 * 128), (0.1, 96))])
    params = params.astype(np.float32)
    x = rng.normal(0, 1, (B, 64)).astype(np.float32)
    dO = rng.normal(0, 1, (B, 96)).astype(np.float32)
    dO[np.unique(np.minimum(np.array([0, 31, 32, 4863, 4864, B - 1]), B - 1))] *= 50.0
    # matrices that start `offset` floats into their allocation
    xd = torch.zeros(B * 64 + offset, dtype=torch.float32, device="cuda")
    dd = torch.zeros(B * 96 + offset, dtype=torch.float32, device="cuda")
    xd[offset:] = torch.from_numpy(x).cuda().ravel()
    dd[offset:] = torch.from_numpy(dO).cuda().ravel()
    out = torch.full((B + 1, 96), 7.0, dtype=torch.float32, device="cuda")
    m = gba.Mlp(capacity=B)
    m.set_params(params)
    torch.cuda.synchronize()
    m.forward(xd[offset:].data_ptr(), B, out.data_ptr())
    m.backward(xd[offset:].data_ptr(), dd[offset:].data_ptr(), B)
    g = mo.unpack(m.grads().astype(np.float64))
    o = out.cpu().numpy()
    assert (o[B] == 7.0).all()  # nothing behind the last row
    ref, _ = mo.forward(params, x)
    assert np.abs(o[:B] - ref).max() <= 2.0 ** -8 * np.abs(ref).max()
    ref_g = mo.unpack(mo.backward(params, x, dO))
    for name in ref_g:
        assert np.abs(g[name] - ref_g[name]).max() <= 2.0 ** -7 * np.abs(ref_g[name]).max(), name
