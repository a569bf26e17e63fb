"""GPU: the cluster-wide sums of a PCG iteration (csrc/cluster_sums.cuh) against FP64, with
as many rows per thread as the kernel takes at 24,000 cameras (16 CTAs of 1,500 cameras,
14 rows of nine threads a camera), at 5,000 (three rows) and with one row per thread.

Bounds. A scalar of several rows per thread is kept in float-float throughout: 2^-40 of
the sum of magnitudes (48 bits, some 30 additions). With one row per thread, and for the
coarse sums, a warp's 32 values, and 256 values of a coarse sum, are added in FP32: 2^-24
per addition, at most 8 + 5 + 8 in a chain.
"""
import ctypes
import subprocess
import sys

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "cluster_sums.cuh"
using namespace gba;
using csum::ff;
namespace gba { [[noreturn]] void cuda_fail(cudaError_t, const char*, const char*, int) { abort(); } }
// rows per CTA as pcg_tail's; values (11, n): two scalars' terms and the nine sums'
template <bool kPairs>
__global__ void __launch_bounds__(1024) sums_kernel(const float* __restrict__ val, int n, int per, double* __restrict__ out) {
    __shared__ csum::Shared sm;
    __shared__ double got[2];
    csum::cluster_arrive();
    const int tid = threadIdx.x, rank = blockIdx.x, nctas = gridDim.x;
    const int i0 = min(rank * per, n), rows = min(per, n - i0), step = kPairs ? 9 * (blockDim.x / 9) : blockDim.x;
    const int first = tid < step ? tid : rows, rounds = kPairs ? (rows + step - 1) / step : 1;
    csum::cluster_wait();
    ff s[2] = {{0.f, 0.f}, {0.f, 0.f}}, nine = {0.f, 0.f};
    for (int k0 = 0; k0 < rounds; k0 += csum::kFoldRows) {
        float v[csum::kNine];
        for (int j = 0; j < csum::kNine; ++j) v[j] = 0.f;
        for (int k = k0; k < min(k0 + csum::kFoldRows, rounds); ++k) {
            const int i = first + k * step;
            if (i >= rows) break;
            for (int j = 0; j < 2; ++j) csum::add_term<kPairs>(s[j], val[1ll * j * n + i0 + i]);
            for (int j = 0; j < csum::kNine; ++j) v[j] += val[(2ll + j) * n + i0 + i];
        }
        csum::fold_nine<kPairs>(v, nine);
    }
    csum::totals<2, true, kPairs>(s, nine, sm, 1, rank, nctas, [&](double a, double b) {
        got[0] = a;
        got[1] = b;
    });
    if (tid < 11) out[11 * rank + tid] = tid < 2 ? got[tid] : sm.tot[tid - 2];
}
extern "C" int run(const float* val, int n, int per, int threads, int pairs, double* out) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 16;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(threads);
    cfg.attrs = at;
    cfg.numAttrs = 1;
    auto k = pairs ? sums_kernel<true> : sums_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k, val, n, per, out);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    return e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    sys.path.insert(0, str(PKG))
    import build

    d = tmp_path_factory.mktemp("sums")
    (d / "sums.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), *build._flags(), "-shared", str(d / "sums.cu"), "-o", str(d / "sums.so")], check=True)
    return ctypes.CDLL(str(d / "sums.so"))


@pytest.mark.parametrize("cameras,threads,pairs", [(24000, 1024, 1), (5000, 1024, 1), (1808, 1024, 0), (40, 128, 0)])
def test_totals(torch_cuda, lib, cameras, threads, pairs):
    torch = torch_cuda
    n, per = 9 * cameras, 9 * -(-cameras // 16)
    rng = np.random.default_rng(cameras)
    val = (rng.random((11, n)) * 2.0 ** rng.uniform(-6, 6, (11, n))).astype(np.float32)
    val[1::2] *= rng.choice([-1, 1], val[1::2].shape)  # some with cancellation
    d, out = torch.from_numpy(val).cuda(), torch.zeros(16, 11, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.run(ctypes.c_void_p(d.data_ptr()), n, per, threads, pairs, ctypes.c_void_p(out.data_ptr())) == 0
    out = out.cpu().numpy()
    assert (out == out[0]).all()  # every CTA has the same totals
    v = val.astype(np.float64)
    err = np.abs(out[0] - v.sum(axis=1)) / np.abs(v).sum(axis=1)
    print(cameras, err * 2.0**24)
    assert err[:2].max() <= (2.0**-40 if pairs else 5 * 2.0**-24)
    assert err[2:].max() <= 21 * 2.0**-24
