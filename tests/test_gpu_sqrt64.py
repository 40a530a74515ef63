"""The integer-pipe FP64 square root (csrc/gw_div64.cuh) against the host's IEEE square root, bit for bit: random
arguments, squares and their neighbours, midpoints between two roots' squares, and every exponent."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from gwgb300 import _build

pytestmark = pytest.mark.gpu

SRC = """
#include <cuda_runtime.h>
#include "gw_div64.cuh"
__global__ void k(const double *x, double *r, int n) {
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i < n) r[i] = gw::sqrt_rn(x[i]);
}
extern "C" int sqrt_check(const double *x, double *r, int n) {
    double *d = nullptr;
    const size_t s = sizeof(double) * (size_t)n;
    int e = (int)cudaMalloc(&d, 2 * s);
    if (!e) e = (int)cudaMemcpy(d, x, s, cudaMemcpyHostToDevice);
    if (!e) k<<<(n + 255) / 256, 256>>>(d, d + n, n);
    if (!e) e = (int)cudaMemcpy(r, d + n, s, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sqrt64")
    (d / "sqrt.cu").write_text(SRC)
    subprocess.run([_build.nvcc(), *_build.ARCH, "-O3", "-std=c++17", "-I" + _build.CSRC, "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(d / "sqrt.so"), str(d / "sqrt.cu")], check=True)
    return C.CDLL(str(d / "sqrt.so"))


def _arguments(kind, n, rng):
    if kind == "any":      # every bit pattern: negative, subnormal, infinite and NaN among them
        return rng.integers(0, 1 << 64, n, dtype=np.uint64).view(np.float64)
    if kind == "range":    # concentrations and powers of them
        return np.exp(rng.uniform(-30, 30, n))
    if kind == "squares":  # perfect squares of up to 26 bits, and one and two units in the last place beside them
        m = rng.integers(1, 1 << 26, n).astype(np.float64)
        x = m * m * np.ldexp(1.0, 2 * rng.integers(-300, 300, n).astype(np.int32))
        return (x.view(np.int64) + rng.integers(-2, 3, n)).view(np.float64)
    # "halfway": next to the square of a number halfway between two doubles, where the root's rounding is decided
    r = 1.0 + rng.integers(0, 1 << 52, n).astype(np.float64) * 2.0 ** -52
    hi = (r.astype(np.longdouble) + np.longdouble(2.0) ** -53) ** 2
    x = hi.astype(np.float64) * np.ldexp(1.0, 2 * rng.integers(-500, 500, n).astype(np.int32))
    return (x.view(np.int64) + rng.integers(-1, 2, n)).view(np.float64)


@pytest.mark.parametrize("kind", ["any", "range", "squares", "halfway"])
def test_square_root_is_ieee(lib, kind):
    x = np.ascontiguousarray(_arguments(kind, 1 << 20, np.random.default_rng(len(kind))))
    special = np.array([0.0, -0.0, 5e-324, 2.2250738585072014e-308, 1.0, np.nextafter(1.0, 2), np.nextafter(1.0, 0), 2.0, 4.0,
                        np.finfo(float).max, np.inf, -np.inf, np.nan, -1.0])
    x[:special.size] = special
    r = np.empty_like(x)
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    assert lib.sqrt_check(p(x), p(r), x.size) == 0
    with np.errstate(all="ignore"):
        want = np.sqrt(x)
    same = (r.view(np.uint64) == want.view(np.uint64)) | (np.isnan(r) & np.isnan(want))
    assert same.all(), (x[~same][:3], r[~same][:3], want[~same][:3])
