"""The FP64 reciprocal and reciprocal square root of the hardening and strain kernels against extended
precision, over mantissas (low words of zeros and of ones among them) and every exponent they admit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "hgb_common.cuh"
__global__ void k(const double *y, long n, double *rcp, double *rsq, int *in) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    in[i] = hgb::fast_range(y[i]);
    rcp[i] = in[i] ? hgb::fast_rcp(y[i]) : 0.0;
    rsq[i] = in[i] ? hgb::fast_rsqrt(y[i]) : 0.0;
}
extern "C" int run(const double *y, long n, double *rcp, double *rsq, int *in) {
    k<<<(unsigned)((n + 255) / 256), 256>>>(y, n, rcp, rsq, in);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def helper(tmp_path_factory):
    from holodeck_gb300 import build
    where = tmp_path_factory.mktemp("fast")
    src, lib = where / "fast.cu", where / "fast.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-shared", "-Xcompiler", "-fPIC", "-I",
                    os.path.join(build.ROOT, "include"), "-I", build.CSRC, str(src), "-o", str(lib)], check=True)
    return ctypes.CDLL(str(lib))


def _run(helper, y):
    import torch
    dev = torch.as_tensor(y, device="cuda")
    rcp, rsq = torch.empty_like(dev), torch.empty_like(dev)
    ok = torch.empty(dev.numel(), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert helper.run(p(dev), ctypes.c_long(dev.numel()), p(rcp), p(rsq), p(ok)) == 0
    return rcp.cpu().numpy(), rsq.cpu().numpy(), ok.cpu().numpy()


def test_against_extended_precision(helper):
    rng = np.random.default_rng(0)
    frac = rng.integers(0, 1 << 52, size=1 << 20, dtype=np.uint64)
    frac[0::8] |= np.uint64(0xFFFFFFFF)
    frac[1::8] &= np.uint64(0xFFFFF00000000)
    frac[2::64], frac[3::64], frac[4::64] = 0, (1 << 52) - 1, 0xFFFFFFFF
    field = rng.integers(123, 1923, size=frac.size).astype(np.uint64)
    field[:1800], field[1800:3600] = np.arange(123, 1923), 1922
    field[3600:5400] = 123
    y = (field << np.uint64(52) | frac).view(np.float64)
    rcp, rsq, ok = _run(helper, y)
    assert ok.all()
    big = y.astype(np.longdouble)
    one = np.longdouble(1.0)
    err_rcp = np.abs(rcp.astype(np.longdouble) * big - one).max()
    # r^2 y = (1 + err)^2; r^2 leaves the range of a double, not that of its exponents here
    err_rsq = (np.abs((rsq.astype(np.longdouble) * big) * rsq.astype(np.longdouble) - one) / 2).max()
    print("largest errors", float(err_rcp), float(err_rsq))
    assert err_rcp <= 2.0 ** -53 + 2.0 ** -55
    assert err_rsq <= 1.5 * 2.0 ** -53 + 2.0 ** -55


def test_range(helper):
    outside = np.array([0.0, -0.0, 5e-324, 2.0 ** -901, 2.0 ** 900, np.inf, np.nan, -1.0, -np.inf, -2.0 ** -1000])
    inside = np.array([2.0 ** -900, np.nextafter(2.0 ** 900, 0.0), 1.0])
    assert not _run(helper, outside)[2].any() and _run(helper, inside)[2].all()
