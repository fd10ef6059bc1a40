"""The inverse root, root and inverse of the float64 kernels (gf_common.cuh) against CUDA's own square root
and division: random mantissas over the exponent range, at both sides of each limit that selects the short
form, and the values outside it.

The seed's relative error is below 2^-19 (e below 2^-18), so the first term left out, e^3 at most, is below
2^-54 and mostly far below. The last operation rounds by half a unit in the last place; the roots also carry half
of the relative rounding of r2 y, a quarter to half a unit. So a result lies within one unit of the true value,
and as far from the correctly rounded one: within one unit too, as both are float64 numbers (1/r within two,
because the quotient it is compared with has the root's own rounding in it). The mean error is 1/4 unit for one
rounding and at most 1/4 + (1/2)^2 / (6 x 1/2) = 1/3 with the second one.
"""

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "gf_common.cuh"
using namespace gf;
__global__ void k_probe(int n, const double* x, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double r, inv;
    inv_root(x[i], r, inv);
    out[6 * i] = r;
    out[6 * i + 1] = inv;
    out[6 * i + 2] = root(x[i]);
    out[6 * i + 3] = in_inverse_range(x[i]) ? inverse(x[i]) : __drcp_rn(x[i]);
    out[6 * i + 4] = __dsqrt_rn(x[i]);
    out[6 * i + 5] = __drcp_rn(fmax(__dsqrt_rn(x[i]), 1e-30));
}
extern "C" int probe(int n, const double* x, double* out) {
    double *dx, *dout;
    if (cudaMalloc(&dx, sizeof(double) * n) != cudaSuccess || cudaMalloc(&dout, sizeof(double) * 6 * n) != cudaSuccess) return 1;
    cudaMemcpy(dx, x, sizeof(double) * n, cudaMemcpyHostToDevice);
    k_probe<<<(n + 255) / 256, 256>>>(n, dx, dout);
    const cudaError_t e = cudaMemcpy(out, dout, sizeof(double) * 6 * n, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dout);
    return e != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def probe(gpulib, tmp_path_factory):
    from galaxy_formation_gb300 import build

    where = tmp_path_factory.mktemp("roots")
    (where / "probe.cu").write_text(SOURCE)
    subprocess.run([build.NVCC, *build.ARCH, *build.FLAGS, "-I", build.CSRC, "-shared", "-o", str(where / "probe.so"),
                    str(where / "probe.cu"), "-lcudart"], check=True, capture_output=True, text=True)
    fn = ctypes.CDLL(str(where / "probe.so")).probe

    def run(x):
        x = np.ascontiguousarray(x, np.float64)
        out = np.empty((len(x), 6))
        assert fn(len(x), ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(out.ctypes.data)) == 0
        return out
    return run


def _units(a, b):
    """|a - b| in units in the last place of b (0 where both are the same, infinities included)."""
    with np.errstate(all="ignore"):
        return np.where(a == b, 0.0, np.abs(a - b) / np.spacing(np.abs(b)))


def _values():
    rng = np.random.default_rng(0)
    mant = rng.uniform(1, 2, 400)
    mant[:4] = 1.0, np.nextafter(1.0, 2), np.nextafter(2.0, 1), 1.5
    exps = list(range(-1022, 1024, 13))
    for limit in (-198, 962, -900, 900):
        exps += [limit - 1, limit, limit + 1]
    return np.concatenate([np.ldexp(mant, e) for e in exps])


def test_within_one_unit(probe):
    x = _values()
    out = probe(x)
    for col, want, most in ((0, out[:, 4], 1.0), (1, out[:, 5], 2.0), (2, out[:, 4], 1.0)):
        assert _units(out[:, col], want).max() <= most, col
    inv = np.abs(np.frexp(x)[1]) < 1020  # whose inverse is a normal number
    assert _units(out[inv, 3], 1.0 / x[inv]).max() <= 1.0


def test_mean_errors(probe):
    """Against extended precision, in units in the last place."""
    long = np.longdouble
    if np.finfo(long).eps >= np.finfo(np.float64).eps:
        pytest.skip("no extended precision in this NumPy")
    x = np.random.default_rng(1).uniform(1, 4, 200000)
    out, xl = probe(x), x.astype(long)
    for col, want, most in ((0, np.sqrt(xl), 1 / 3), (1, 1 / np.sqrt(xl), 1 / 3), (2, np.sqrt(xl), 1 / 3), (3, 1 / xl, 0.255)):
        unit = np.spacing(np.abs(want.astype(np.float64)))
        assert float(np.mean(np.abs(out[:, col] - want) / unit)) < most, col


def test_values_outside_the_range(probe):
    x = np.array([0.0, 5e-324, 2.2e-308, np.inf, np.nan, -0.0, -1.0, -np.inf])
    out = probe(x)
    assert np.array_equal(out[:, 0], out[:, 4], equal_nan=True)
    assert np.array_equal(out[:, 1], out[:, 5], equal_nan=True)
    assert np.array_equal(out[:, 2], out[:, 4], equal_nan=True)
    with np.errstate(divide="ignore", over="ignore"):
        assert np.array_equal(out[:, 3], 1.0 / x, equal_nan=True)
