"""The integer-pipe FP64 division (csrc/gw_div64.cuh) against the host's IEEE division, bit for bit:
random significands, quotients next to a rounding boundary, and operands outside the normal range."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from gwgb300 import _build

pytestmark = pytest.mark.gpu

SRC = """
#include <cuda_runtime.h>
#include "gw_div64.cuh"
__global__ void k(const double *a, const double *b, double *q, int n) {
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i < n) q[i] = gw::div_rn(a[i], b[i]);
}
extern "C" int div_check(const double *a, const double *b, double *q, int n) {
    double *d = nullptr;
    const size_t s = sizeof(double) * (size_t)n;
    int e = (int)cudaMalloc(&d, 3 * s);
    if (!e) e = (int)cudaMemcpy(d, a, s, cudaMemcpyHostToDevice);
    if (!e) e = (int)cudaMemcpy(d + n, b, s, cudaMemcpyHostToDevice);
    if (!e) k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, n);
    if (!e) e = (int)cudaMemcpy(q, d + 2 * (size_t)n, s, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("div64")
    (d / "div.cu").write_text(SRC)
    subprocess.run([_build.nvcc(), *_build.ARCH, "-O3", "-std=c++17", "-I" + _build.CSRC, "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(d / "div.so"), str(d / "div.cu")], check=True)
    return C.CDLL(str(d / "div.so"))


def _bits(sign, exponent, mantissa):
    return ((sign.astype(np.uint64) << np.uint64(63)) | (exponent.astype(np.uint64) << np.uint64(52)) |
            (mantissa & np.uint64((1 << 52) - 1))).view(np.float64)


def _operands(kind, n, rng):
    m = rng.integers(0, 1 << 52, (2, n), dtype=np.uint64)
    s = rng.integers(0, 2, (2, n))
    if kind == "any":      # every bit pattern: subnormals, infinities and NaN among them
        return tuple(rng.integers(0, 1 << 64, n, dtype=np.uint64).view(np.float64) for _ in range(2))
    if kind == "edge":     # exponents at both ends, zeros, powers of two
        e = rng.choice(np.array([0, 1, 2, 3, 1022, 1023, 1024, 2044, 2045, 2046, 2047]), (2, n))
        m *= rng.integers(0, 2, (2, n), dtype=np.uint64)
    elif kind == "near":   # a / b next to 1, and significands of few or nearly all bits
        e = np.full((2, n), 1023)
        few = (np.uint64(0xFFFFFFFFFFFFF) << rng.integers(0, 52, (2, n), dtype=np.uint64)) & np.uint64(0xFFFFFFFFFFFFF)
        m = np.where(rng.random((2, n)) < 0.5, m & few, m | few)
        m[0] = np.where(rng.random(n) < 0.4, m[1] + rng.integers(0, 9, n, dtype=np.uint64), m[0])
    else:                  # "normal"
        e = rng.integers(700, 1400, (2, n))
    return _bits(s[0], e[0], m[0]), _bits(s[1], e[1], m[1])


@pytest.mark.parametrize("kind", ["normal", "near", "edge", "any"])
def test_division_is_ieee(lib, kind):
    a, b = _operands(kind, 1 << 20, np.random.default_rng(len(kind)))
    q = np.empty_like(a)
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    assert lib.div_check(p(a), p(b), p(q), a.size) == 0
    with np.errstate(all="ignore"):
        r = a / b
    same = (q.view(np.uint64) == r.view(np.uint64)) | (np.isnan(q) & np.isnan(r))
    assert same.all(), (a[~same][:3], b[~same][:3], q[~same][:3], r[~same][:3])
