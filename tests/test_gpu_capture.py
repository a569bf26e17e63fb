"""GPU: the standalone Cholesky and solve under stream capture: captured calls replay on
new inputs and give what the direct calls give, bit for bit (their workspaces become
nodes of the graph).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _replay(torch, call, inputs, outputs, other):
    """call(stream) on a side stream, captured with the inputs as they are, replayed with `other`."""
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        for i, v in zip(inputs, other):
            i.copy_(v)
        call(s.cuda_stream)
        s.synchronize()
        want = [o.clone() for o in outputs]
        for o in outputs:
            o.zero_()
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            call(s.cuda_stream)
        for i, v in zip(inputs, other):
            i.copy_(v)
        g.replay()
        s.synchronize()
    for w, o in zip(want, outputs):
        assert torch.equal(w, o)


@pytest.mark.parametrize("n", [192, 1024])
def test_cholesky_and_solve(gba, torch_cuda, n):
    torch = torch_cuda
    rng = np.random.default_rng(n)
    B = rng.normal(size=(n, n))
    other = [torch.from_numpy(B @ B.T / n + np.eye(n)).cuda(), torch.from_numpy(rng.normal(size=n)).cuda()]
    A, b = torch.eye(n, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda")
    L, x, info = torch.zeros_like(A), torch.zeros_like(b), torch.zeros(1, dtype=torch.int32, device="cuda")

    def call(stream):
        L.copy_(A)
        x.copy_(b)
        gba.dense_potrf(L.data_ptr(), n, n, info.data_ptr(), stream)
        gba.dense_potrs(L.data_ptr(), n, n, x.data_ptr(), info.data_ptr(), stream)

    _replay(torch, call, [A, b], [L, x], other)
    assert int(info.item()) == 0
