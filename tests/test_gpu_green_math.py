"""The reciprocal root and sine/cosine of the FP64 Green-kernel samples
(green_math.cuh) against extended precision. Bounds from the functions'
construction: the reciprocal root's correction step has a residual rounded to
half a unit of one and one final rounding (1.5 units with the argument's
product); the reduced phase carries half a unit of its own size and each
polynomial ends in one rounding next to terms below it (1.5 units of the
result's binade at most 1)."""
import ctypes as C
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = pathlib.Path(__file__).resolve().parent.parent / "hornsculpt_b200" / "csrc"
SOURCE = r"""
#include "green_math.cuh"
__global__ void evaluate(const double *x, int n, double *root, double *sine, double *cosine) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    root[i] = hsb::reciprocalRoot(x[i]);
    hsb::sinCos(x[i], sine[i], cosine[i]);
}
extern "C" int run(const double *x, int n, double *out) {
    double *d = nullptr;
    if (cudaMalloc(&d, 4 * size_t(n) * 8) != cudaSuccess)
        return 1;
    cudaMemcpy(d, x, size_t(n) * 8, cudaMemcpyHostToDevice);
    evaluate<<<(n + 127) / 128, 128>>>(d, n, d + n, d + 2 * size_t(n), d + 3 * size_t(n));
    const cudaError_t e = cudaMemcpy(out, d + n, 3 * size_t(n) * 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return int(e);
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    where = tmp_path_factory.mktemp("green")
    (where / "green.cu").write_text(SOURCE)
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-std=c++20", "-O3", "-shared", "-Xcompiler",
                    "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), str(where / "green.cu"),
                    "-o", str(where / "green.so")], check=True)
    lib = C.CDLL(str(where / "green.so"))

    def run(x):
        x = np.ascontiguousarray(x, np.float64)
        out = np.zeros(3 * len(x))
        assert lib.run(x.ctypes.data_as(C.c_void_p), len(x), out.ctypes.data_as(C.c_void_p)) == 0
        return out.reshape(3, -1)

    return run


# squared distances and phases from a panel's own size to kilometres; quadrant edges included
@pytest.mark.parametrize("low,high", [(1e-12, 1e-3), (1e-3, 1.0), (1.0, 1e3), (1e3, 1e7)])
def test_root_sine_and_cosine_to_the_last_places(evaluate, low, high):
    rng = np.random.default_rng(7)
    x = np.exp(rng.uniform(np.log(low), np.log(high), 200000))
    edges = np.round(x[:2000] / (np.pi / 4)) * (np.pi / 4)
    x = np.concatenate([x, edges[edges > 0]])
    root, sine, cosine = evaluate(x)
    wide = x.astype(np.longdouble)
    exact = 1 / np.sqrt(wide)
    assert np.max(np.abs(root - exact) / np.spacing(exact.astype(float))) <= 1.5
    for got, want in ((sine, np.sin(wide)), (cosine, np.cos(wide))):
        assert np.max(np.abs(got - want)) <= 1.5 * 2.0 ** -53
        inner = np.abs(want) > 1e-3
        units = np.abs(got - want)[inner] / np.spacing(np.abs(want[inner]).astype(float))
        assert np.max(units, initial=0.0) <= 1.5
