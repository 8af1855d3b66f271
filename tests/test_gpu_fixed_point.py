"""The FP64 reciprocal and reciprocal root that the kernels form in integers, against
CUDA's operators on the same values: 1 / x to one unit in the last place (it is rounded
from 0.5001 units), 1 / sqrt(x) exactly, and both exactly where they fall back to the
operators (zeros, subnormals, infinities, NaN, negative values, the ends of the range)."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = """
#include "hx_common.cuh"
__global__ void k(const double* x, long long n, double* out) {
    const long long t = blockIdx.x * 256ll + threadIdx.x;
    if (t >= n) return;
    out[t] = hx::rcp64(x[t]);
    out[n + t] = 1.0 / x[t];
    out[2 * n + t] = hx::inv_root(x[t]);
    out[3 * n + t] = 1.0 / sqrt(x[t]);
}
extern "C" int run(const double* x, long long n, double* out) {
    double *dx = nullptr, *dout = nullptr;
    int e = cudaMalloc(&dx, n * 8);
    if (!e) e = cudaMalloc(&dout, 4 * n * 8);
    if (!e) e = cudaMemcpy(dx, x, n * 8, cudaMemcpyHostToDevice);
    if (!e) { k<<<(unsigned)((n + 255) / 256), 256>>>(dx, n, dout); e = cudaGetLastError(); }
    if (!e) e = cudaMemcpy(out, dout, 4 * n * 8, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dout);
    return e;
}
"""


def bits(x):
    return x.view(np.int64)


def test_reciprocal_and_root(tmp_path):
    import build_ext
    src, so = tmp_path / "t.cu", tmp_path / "t.so"
    src.write_text(SOURCE)
    subprocess.run([build_ext.nvcc()] + build_ext.NVCC_FLAGS + ["-shared", "-o", str(so), str(src), "-cudart", "static"],
                   check=True)
    rng = np.random.default_rng(1)
    m = rng.integers(0, 1 << 52, size=4_000_000, dtype=np.int64)
    m[:100000] = rng.integers(0, 1 << 10, size=100000)                    # just above a power of two
    m[100000:200000] = (1 << 52) - 1 - rng.integers(0, 1 << 10, size=100000)
    x = ((rng.integers(1, 2047, size=m.size) << 52) | m).view(np.float64)
    x = np.concatenate([x, -x[:1000], [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310],
                        2.0 ** np.arange(-1074, 1024), np.nextafter(2.0 ** np.arange(-1022, 1024), 0.0)])
    lib = ctypes.CDLL(str(so))
    out = np.empty((4, x.size))
    assert lib.run(x.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(x.size), out.ctypes.data_as(ctypes.c_void_p)) == 0
    r, want, s, root = out
    assert np.array_equal(s, root, equal_nan=True)
    inside = (x >= 2.0 ** -1000) & (x <= 2.0 ** 1000)
    assert np.array_equal(r[~inside], want[~inside], equal_nan=True)
    d = np.abs(bits(r)[inside] - bits(want)[inside])
    assert d.max() <= 1 and (d != 0).mean() < 1e-4
