"""The FP32 engine's flux sums (FluxAcc, reduce_partials of csrc/gw_engine.cuh) against exact sums of the same terms,
over the ranges of the fluxes and of the parameters that scale them: order-free, and no further off than the
rounding of each term to 2^-46 units, of the sum to FP64, and of large sums to 2^-40 (derived bounds below).
An FP32 tree over the same terms may be off by 2^-24 of the sum of their magnitudes per addition."""
import ctypes as C
import math
import subprocess

import numpy as np
import pytest

from gwgb300 import _build

pytestmark = pytest.mark.gpu

SRC = """
#include "gw_engine.cuh"
using namespace gw;
using namespace gw::dev;
__global__ void k(const float *v, const int *cl, int n_slots, int per, const double *bound, double *out, int *exps) {
    __shared__ SsaConsts<float> cc;
    __shared__ Partial<false> slots[256];
    __shared__ PartialTail tails[256];
    __shared__ double X[64];
    const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
    const size_t n = (size_t)n_slots * 32 * per;
    if (threadIdx.x < 3) {
        cc.flux_exp[threadIdx.x] = exps[threadIdx.x] = flux_exp_of(bound[threadIdx.x]);
        cc.flux_scale[threadIdx.x] = __int_as_float((127 - cc.flux_exp[threadIdx.x]) << 23);
    }
    __syncthreads();
    for (int s = warp; s < n_slots; s += (int)blockDim.x >> 5) {
        FluxAcc<false> acc(cc);
        for (int q = 0; q < per; ++q) {
            const size_t i = ((size_t)s * per + q) * 32 + lane;
            acc.add(v[i], v[n + i], v[2 * n + i], cl[i]);
        }
        PartialTail t;
        const Partial<false> p = acc.warp_total(t);
        if (lane == 0) {
            slots[s] = p;
            tails[s] = t;
        }
    }
    __syncthreads();
    if (warp < 4) reduce_partials<double>(slots, tails, cc.flux_exp, n_slots, warp, lane, out, X);
}
extern "C" int sums(const float *v, const int *cl, int n_slots, int per, const double *bound, double *out, int *exps) {
    const size_t n = (size_t)n_slots * 32 * per;
    unsigned char *d = nullptr;
    const size_t ov = 64, oc = ov + 12 * n, end = oc + 4 * n;
    if (n_slots > 256) return -1;
    int e = (int)cudaMalloc(&d, end);
    if (!e) e = (int)cudaMemcpy(d, bound, 24, cudaMemcpyHostToDevice);
    if (!e) e = (int)cudaMemcpy(d + ov, v, 12 * n, cudaMemcpyHostToDevice);
    if (!e) e = (int)cudaMemcpy(d + oc, cl, 4 * n, cudaMemcpyHostToDevice);
    double *o = nullptr;
    if (!e) e = (int)cudaMalloc(&o, 48);
    if (!e) k<<<1, 512>>>((float *)(d + ov), (int *)(d + oc), n_slots, per, (double *)d, o, (int *)(o + 4));
    if (!e) e = (int)cudaMemcpy(out, o, 32, cudaMemcpyDeviceToHost);
    if (!e) e = (int)cudaMemcpy(exps, o + 4, 12, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(o);
    return e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("flux")
    (d / "flux.cu").write_text(SRC)
    subprocess.run([_build.nvcc(), *_build.ARCH, "-O3", "-std=c++17", "-I" + _build.CSRC, "-I" + _build.INCLUDE, "-shared",
                    "-Xcompiler", "-fPIC", "-o", str(d / "flux.so"), str(d / "flux.cu")], check=True)
    return C.CDLL(str(d / "flux.so"))


def device_sums(lib, v, cl, slots, per, bound):
    out, exps = np.zeros(4), np.zeros(3, np.int32)
    v, cl, bound = np.ascontiguousarray(v, np.float32), np.ascontiguousarray(cl, np.int32), np.asarray(bound, float)
    p = lambda x: x.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert v.shape == (3, slots * per * 32) and cl.shape == (slots * per * 32,)
    assert lib.sums(p(v), p(cl), slots, per, p(bound), p(out), p(exps)) == 0
    return out[[0, 3, 2]], int(out[1]), exps  # (the engine's order: JLCC, ClCh, Jtr, Jxfer)


BOUND = [64 * 2 * 9.13e-13 * 1e6 / 0.2303e-6 * (1 + 0.682), 64 * 200.0, 64 * 0.333]


@pytest.mark.parametrize("slots,per", [(1, 1), (5, 2), (33, 3), (256, 2)])
@pytest.mark.parametrize("scale", [1.0, 1e-1, 1e-3, 1e-6, 30.0, 0.0])  # of the parameters, and with them of the terms
@pytest.mark.parametrize("size", ["mixed", "rest", "large"])
def test_sums_are_exact(lib, slots, per, scale, size):
    rng = np.random.default_rng(slots * 100 + per)
    n = slots * per * 32
    typical = np.array([[10.0], [50.0], [0.3]])  # amid the release
    if size == "mixed":
        v = typical * np.exp(rng.uniform(-25, 0, (3, n))) * rng.choice([-1.0, 1.0], (3, n))
    elif size == "rest":   # nearly equal, and small
        v = typical * 2e-6 * (1 + 1e-3 * rng.standard_normal((3, n)))
    else:
        v = typical * rng.uniform(0.5, 1.9, (3, n))
    v = (v * scale).astype(np.float32)
    cl = rng.integers(0, 5, n)
    got, gcl, exps = device_sums(lib, v, cl, slots, per, np.array(BOUND) * scale)
    perm = rng.permutation(n)
    again, _, _ = device_sums(lib, v[:, perm], cl[perm], slots, per, np.array(BOUND) * scale)
    assert np.array_equal(got, again)  # whatever lane or warp a term went to
    assert gcl == cl.sum()
    for q in range(3):
        want = math.fsum(v[q].astype(float))
        mag = math.fsum(np.abs(v[q].astype(float)))
        tol = n * 2.0 ** (int(exps[q]) - 47) + (2.0 ** -52 + (2.0 ** -40 if abs(want) > 2.0 ** (int(exps[q]) + 16) else 0.0)) * abs(want)
        err = abs(got[q] - want)
        assert err <= tol, (q, err, tol)
        assert err <= 2.0 ** -30 * mag


@pytest.mark.parametrize("big", [1e6, -3e30, np.inf, np.nan])
def test_terms_out_of_range(lib, big):
    rng = np.random.default_rng(3)
    n = 40 * 2 * 32
    v = (rng.standard_normal((3, n)) * np.array([[10.0], [50.0], [0.3]])).astype(np.float32)
    v[1, 777] = big
    got, _, _ = device_sums(lib, v, np.zeros(n), 40, 2, BOUND)
    # the warp that has it adds two floats per lane and takes an FP64 tree
    for q in range(3):
        if q == 1 and not np.isfinite(big):
            assert not np.isfinite(got[1])
            continue
        want, mag = math.fsum(v[q].astype(float)), math.fsum(np.abs(v[q].astype(float)))
        assert abs(got[q] - want) <= 2.0 ** -24 * mag, q
