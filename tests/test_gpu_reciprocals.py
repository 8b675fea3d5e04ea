"""The kernels' reciprocal, reciprocal square root and square root
(hc_device.cuh) against extended precision, and at 0, tiny, negative, infinite
and NaN arguments.

Bounds, with u = 2^-53 and a hardware seed good to 2^-20 (a seed any worse
fails here): rcpN rounds once and leaves e^3 = 2^-60, 1.01 u; rsqrtN rounds
x y too, which half of reaches the result, and leaves 5/16 (2^-19)^3, 1.53 u;
sqrtN's last correction is exact to second order, 1.001 u."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, gpu_available

pytestmark = pytest.mark.gpu

CSRC = os.path.join(ROOT, "heliocubed_b200", "csrc")
SOURCE = """
#include "hc_device.cuh"
__global__ void apply(int what, const double* x, double* y, long n) {
  const long t = blockIdx.x * 256L + threadIdx.x;
  if (t >= n) return;
  y[t] = what == 0 ? hc::rcpN(x[t]) : what == 1 ? hc::rsqrtN(x[t]) : what == 2 ? hc::sqrtN(x[t]) : hc::rcpDensity(x[t]);
}
extern "C" int run(int what, const double* x, double* y, long n) {
  apply<<<(unsigned)((n + 255) / 256), 256>>>(what, x, y, n);
  return (int)cudaDeviceSynchronize();
}
"""
RCP, RSQRT, SQRT, RCP_DENSITY = range(4)


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    if not gpu_available():
        pytest.skip("no CUDA device")
    import torch

    from heliocubed_b200.build import ARCH, COMMON, NVCC
    where = tmp_path_factory.mktemp("reciprocals")
    src, lib = where / "apply.cu", where / "apply.so"
    src.write_text(SOURCE)
    subprocess.run([NVCC, *ARCH, *COMMON, "-shared", str(src), "-o", str(lib)], check=True)
    run = C.CDLL(str(lib)).run
    run.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_long]

    def call(what, values):
        x = torch.tensor(values, dtype=torch.float64, device="cuda")
        y = torch.empty_like(x)
        torch.cuda.synchronize()
        assert run(what, x.data_ptr(), y.data_ptr(), x.numel()) == 0
        return y.cpu().numpy()

    return call


@pytest.mark.parametrize("what,bound", [(RCP, 1.01), (RSQRT, 1.53), (SQRT, 1.001), (RCP_DENSITY, 1.01)])
def test_error_in_units_of_the_last_place(evaluate, what, bound):
    rng = np.random.default_rng(what)
    x = np.concatenate([(1 + rng.random(1 << 20)) * 2.0 ** rng.integers(-2, 3, 1 << 20),   # every mantissa
                        10.0 ** rng.uniform(-288, 300, 1 << 20),
                        np.nextafter(2.0 ** np.arange(-950, 990), 0), 2.0 ** np.arange(-950, 990)])
    y, z = evaluate(what, x).astype(np.longdouble), x.astype(np.longdouble)
    if what in (RCP, RCP_DENSITY):
        err = y * z - 1
    elif what == RSQRT:
        err = y * np.sqrt(z) - 1
    else:
        err = y / np.sqrt(z) - 1
    assert np.abs(err).max() <= bound * 2.0 ** -53


def test_special_arguments(evaluate):
    inf, nan = np.inf, np.nan
    assert not np.isfinite(evaluate(RCP, [0.0, inf, nan])).any()
    assert not np.isfinite(evaluate(RSQRT, [0.0, inf, nan])).any()
    np.testing.assert_array_equal(evaluate(RCP_DENSITY, [inf, nan]), [0.0, nan])
    np.testing.assert_array_equal(evaluate(SQRT, [0.0, -0.0, 1e-291, 5e-324, -1.0, -inf, inf, nan, -nan]),
                                  [0.0, 0.0, 0.0, 0.0, 0.0, 0.0, inf, nan, nan])
