"""silu.cuh by itself against 64 bits: ordinary values, the ends of its reciprocal's range, infinities and NaN, and its error beside that of
the formula written out. The kernels are built here, from the header alone."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "silu.cuh"
__global__ void silu_kernel(const float *x, float *y, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = wb::silu(x[i]);
}
extern "C" int run(const float *x, float *y, int n)
{
    float *d;
    if (cudaMalloc(&d, 8 * (size_t)n) != cudaSuccess) return 1;
    cudaMemcpy(d, x, 4 * (size_t)n, cudaMemcpyHostToDevice);
    silu_kernel<<<(n + 255) / 256, 256>>>(d, d + n, n);
    cudaMemcpy(y, d + n, 4 * (size_t)n, cudaMemcpyDeviceToHost);
    return cudaFree(d) != cudaSuccess;
}
"""


def test_silu(tmp_path):
    (tmp_path / "silu.cu").write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                    str(Path(__file__).resolve().parent.parent / "webllm_b200/csrc"), str(tmp_path / "silu.cu"), "-o", str(tmp_path / "silu.so")],
                   check=True)
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.normal(0, 4, 100000), rng.uniform(-90, 90, 100000), -np.logspace(-30, 30, 1000), np.logspace(-30, 30, 1000),
                        [0., -0., -79.9, -80.1, -87.2, -87.4, -88.8, -3e38, 3e38, np.inf, -np.inf, np.nan]]).astype(np.float32)
    y = np.empty_like(x)
    lib = C.CDLL(str(tmp_path / "silu.so"))
    assert lib.run(x.ctypes.data_as(C.c_void_p), y.ctypes.data_as(C.c_void_p), x.size) == 0
    with np.errstate(all="ignore"):
        want = x.astype(np.float64) / (1 + np.exp(-x.astype(np.float64)))
        f32 = x / (1 + np.exp(-x))  # the formula in f32: what it makes of the ends (NaN at -inf, where the quotient is -inf / inf)
    assert np.array_equal(np.isnan(y), np.isnan(f32)) and np.array_equal(np.isinf(y), np.isinf(f32))
    ok = np.isfinite(want) & ~np.isnan(y)
    # expf is within 2 ulp, its sum with 1 and the quotient after its residual within half an ulp and one: 4 ulp are 2^-21. Under 1e-32 the
    # result may be 0.
    assert (np.abs(y[ok] - want[ok]) <= 2.0 ** -21 * np.abs(want[ok]) + 1e-32).all()


FORMULA = SOURCE.replace("wb::silu(x[i])", "x[i] / (1.f + expf(-x[i]))")


@pytest.mark.parametrize("lo,hi", [(-1e-3, 1e-3), (-1, 1), (-4, 4), (-12, 12), (-30, -10), (-86, -30), (10, 88)])
def test_no_less_exact_than_the_formula(tmp_path, lo, hi):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    x = np.random.default_rng(2).uniform(lo, hi, 1 << 20).astype(np.float32)
    x = x[x != 0]
    want = x.astype(np.float64) / (1 + np.exp(-x.astype(np.float64)))
    err = []
    for name, source in (("formula", FORMULA), ("silu", SOURCE)):
        (tmp_path / f"{name}.cu").write_text(source)
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                        str(Path(__file__).resolve().parent.parent / "webllm_b200/csrc"), str(tmp_path / f"{name}.cu"), "-o",
                        str(tmp_path / f"{name}.so")], check=True)
        y = np.empty_like(x)
        assert C.CDLL(str(tmp_path / f"{name}.so")).run(x.ctypes.data_as(C.c_void_p), y.ctypes.data_as(C.c_void_p), x.size) == 0
        e = np.abs(y - want) / np.abs(want) * 2.0 ** 24
        err.append((np.sqrt(np.mean(e ** 2)), e.max()))
    # (both round the same quotient: what differs is the one in a great many that its last residual leaves on the other side)
    assert err[1][0] <= 1.01 * err[0][0] and err[1][1] <= err[0][1] + 0.1, err
