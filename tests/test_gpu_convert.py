"""cvt64.cuh's integer conversions between FP64 and FP32 against the hardware's
(numpy's) conversions, bit for bit: random bit patterns, the edges of FP32's
normal range, ties and near-ties of the rounding, zeros, subnormals,
infinities and NaN."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "diomedes_gb300", "csrc")
SOURCE = r"""
#include "cvt64.cuh"
__global__ void k_to(const double* x, float* y, unsigned n) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = dio::to_float(x[i]);
}
__global__ void k_widen(const float* x, double* y, unsigned n) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = dio::widen(x[i]);
}
extern "C" int convert(const double* x, float* y, const float* v, double* z, unsigned n) {
    double *dx, *dz;
    float *dy, *dv;
    if (cudaMalloc(&dx, n * 8ull) || cudaMalloc(&dz, n * 8ull) || cudaMalloc(&dy, n * 4ull) || cudaMalloc(&dv, n * 4ull))
        return 1;
    cudaMemcpy(dx, x, n * 8ull, cudaMemcpyHostToDevice);
    cudaMemcpy(dv, v, n * 4ull, cudaMemcpyHostToDevice);
    k_to<<<256, 256>>>(dx, dy, n);
    k_widen<<<256, 256>>>(dv, dz, n);
    cudaMemcpy(y, dy, n * 4ull, cudaMemcpyDeviceToHost);
    cudaMemcpy(z, dz, n * 8ull, cudaMemcpyDeviceToHost);
    cudaFree(dx), cudaFree(dz), cudaFree(dy), cudaFree(dv);
    return cudaGetLastError() != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def convert(tmp_path_factory):
    d = tmp_path_factory.mktemp("convert")
    (d / "c.cu").write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                           "-shared", "-Xcompiler", "-fPIC", "-I", CSRC, str(d / "c.cu"), "-o", str(d / "c.so")])
    return ctypes.CDLL(str(d / "c.so")).convert


@pytest.mark.parametrize("kind", ["any bits", "float range", "ties", "edges"])
def test_conversions_match(convert, kind):
    rng = np.random.default_rng(len(kind))
    n = 1 << 20
    f = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32).view(np.float32)
    if kind == "any bits":
        d = rng.integers(0, 1 << 64, n, dtype=np.uint64).view(np.float64)
    elif kind == "float range":
        d = rng.uniform(-2, 2, n) * np.exp2(rng.integers(-130, 130, n).astype(np.float64))
    elif kind == "ties":
        with np.errstate(all="ignore"):
            d = f.astype(np.float64)  # halfway between two floats, and one ulp to either side
            d = (d.view(np.uint64) + (1 << 28) + rng.integers(-1, 2, n).astype(np.uint64)).view(np.float64)
    else:
        e = np.array([-150, -149, -127, -126, -125, 126, 127, 128, 0, -1022, -1074, 1023], np.float64)
        d = np.concatenate([np.exp2(e), np.nextafter(np.exp2(e), 0), np.nextafter(np.exp2(e), np.inf),
                            [0.0, np.inf, np.nan, np.finfo(np.float32).max, 3.4028235677973366e38]])
        d = np.tile(np.concatenate([d, -d]), 64)
        f = np.tile(np.concatenate([d.astype(np.float32)[:64], f[:64]]), (len(d) + 127) // 128)[: len(d)]
    d, f = np.ascontiguousarray(d, np.float64), np.ascontiguousarray(f, np.float32)
    y, z = np.zeros(len(d), np.float32), np.zeros(len(d), np.float64)
    assert convert(d.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p),
                   f.ctypes.data_as(ctypes.c_void_p), z.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint(len(d))) == 0
    with np.errstate(all="ignore"):
        wy, wz = d.astype(np.float32), f.astype(np.float64)
    assert ((y.view(np.uint32) == wy.view(np.uint32)) | (np.isnan(y) & np.isnan(wy))).all()
    assert ((z.view(np.uint64) == wz.view(np.uint64)) | (np.isnan(z) & np.isnan(wz))).all()
