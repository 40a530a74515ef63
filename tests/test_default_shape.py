"""The default launch shape (gw_default_shape): cells are spread over more CTAs than they need only as far as all
clusters of the ensemble are resident at once."""
import ctypes as C
import subprocess

import numpy as np
import pytest

# cudaOccupancyMaxActiveClusters of clusters of 1 .. 16 CTAs, one CTA to an SM, on a GB300
RESIDENT = [152, 76, 46, 36, 28, 23, 15, 15, 15, 13, 8, 8, 7, 7, 7, 7]


def _shape(n_cells, max_n, precision):
    from gwgb300 import engine

    return engine.Ensemble.partition_spec(np.full(n_cells, max_n), 1, 0, precision)[2:]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("max_n", [5, 33, 100, 300, 777, 1200, 2362, 3000, 5000, 12500])
def test_spread_clusters_are_resident(enginelib, precision, max_n):
    if precision == "fp64":
        if max_n > 3000:
            pytest.skip("more than an FP64 cell holds")
        need = min(16, -(-max_n // 96))
    else:
        need = 1
        while need < 16 and -(-max_n // need) > 384:
            need *= 2
    for n_cells in range(1, 200):
        cl, tile = _shape(n_cells, max_n, precision)
        assert need <= cl <= 16 and cl * tile >= max_n
        assert cl == need or n_cells <= RESIDENT[cl - 1], (n_cells, cl)
    assert _shape(1, 12500, "fp32")[0] == 16 and (max_n < 100 or _shape(1, max_n, precision)[0] > 1)


SRC = """
#include <cuda_runtime.h>
__global__ void __launch_bounds__(512, 1) k(int *p) {
    extern __shared__ int s[];
    if (p) p[0] = s[0];
}
extern "C" int resident(int *out) {
    int e = (int)cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (!e) e = (int)cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int c = 1; !e && c <= 16; ++c) {
        cudaLaunchConfig_t f = {};
        cudaLaunchAttribute a[1];
        f.gridDim = dim3(c * 100);
        f.blockDim = dim3(512);
        f.dynamicSmemBytes = 200 * 1024;
        a[0].id = cudaLaunchAttributeClusterDimension;
        a[0].val.clusterDim.x = c;
        a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
        f.attrs = a;
        f.numAttrs = 1;
        e = (int)cudaOccupancyMaxActiveClusters(out + c - 1, k, &f);
    }
    return e;
}
"""


@pytest.mark.gpu
def test_resident_clusters_of_this_device(enginelib, tmp_path):
    from gwgb300 import _build

    (tmp_path / "r.cu").write_text(SRC)
    subprocess.run([_build.nvcc(), *_build.ARCH, "-shared", "-Xcompiler", "-fPIC", "-o", str(tmp_path / "r.so"),
                    str(tmp_path / "r.cu")], check=True)
    got = (C.c_int * 16)()
    assert C.CDLL(str(tmp_path / "r.so")).resident(got) == 0
    for n_cells in range(1, 153):  # (cells of 1,000 CRUs: four CTAs unless spread)
        cl, _ = _shape(n_cells, 1000, "fp32")
        assert cl == 4 or n_cells <= got[cl - 1], (n_cells, cl, list(got))
