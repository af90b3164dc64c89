"""The batched sparse-LU kernel's own arithmetic (csrc/kernels_lanes_impl.cuh) against CUDA's and numpy's: the FP64
reciprocal of the pivots, the step-size factor and the powers of two that scale the particles' rows. Bounds: each
Newton-Raphson pass squares the relative error, 2^-20 and 1e-6 at the start, so two passes leave the rounding of the last
one, an ulp for the reciprocal and, with the factors 1/3 and 0.9, four for the step factor."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "tchem-atm_gb300" / "csrc"
SOURCE = r"""
#include "kernels_lanes_impl.cuh"
using K = tchem_gb::lanes::Kernel<double, 1, 8, true>;
template <int WHAT>
__global__ void run(const double* x, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (WHAT == 0) y[i] = tchem_gb::lanes::Num<double>::recip(x[i]);
  if (WHAT == 1) y[i] = K::step_factor(x[i]);
  if (WHAT == 2) y[i] = K::power_of_two_below(x[i]);
  if (WHAT == 3) y[i] = K::inverse_unit(x[i]);
}
extern "C" int lane_arithmetic(int what, const double* x, double* y, int n) {
  const int grid = (n + 255) / 256;
  if (what == 0) run<0><<<grid, 256>>>(x, y, n);
  if (what == 1) run<1><<<grid, 256>>>(x, y, n);
  if (what == 2) run<2><<<grid, 256>>>(x, y, n);
  if (what == 3) run<3><<<grid, 256>>>(x, y, n);
  return static_cast<int>(cudaDeviceSynchronize());
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    d = tmp_path_factory.mktemp("lane_arithmetic")
    (d / "t.cu").write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I",
                    str(CSRC), "-shared", "-o", str(d / "t.so"), str(d / "t.cu")], check=True)
    f = C.CDLL(str(d / "t.so")).lane_arithmetic
    f.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int]

    def call(what, x):
        a = torch.as_tensor(np.ascontiguousarray(x, dtype=np.float64)).cuda()
        b = torch.empty_like(a)
        torch.cuda.synchronize()
        assert f(what, a.data_ptr(), b.data_ptr(), a.numel()) == 0
        return b.cpu().numpy()
    return call


def test_reciprocal(evaluate):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(1.0, 2.0, 400_000), 10.0 ** rng.uniform(-300, 300, 400_000),
                        1.0 + 2.0 ** -np.arange(1.0, 53.0), 2.0 - 2.0 ** -np.arange(1.0, 52.0)])
    x = np.concatenate([x, -x])
    assert (np.abs(evaluate(0, x) * x - 1.0)).max() <= 2.0 ** -52 + 2.0 ** -53  # an ulp, and the product's rounding
    assert np.array_equal(evaluate(0, 2.0 ** np.arange(-300.0, 300.0)), 2.0 ** -np.arange(-300.0, 300.0))
    v = evaluate(0, [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324])  # rejected pivots: NaN or zero
    assert np.all(np.isnan(v) | (v == 0.0))


def test_step_factor(evaluate):
    e = np.concatenate([10.0 ** np.random.default_rng(2).uniform(-30, 30, 400_000), np.linspace(0.04, 210.0, 200_001)])
    ref = np.clip(0.9 * np.cbrt(1.0 / e), 0.2, 2.0)
    assert (np.abs(evaluate(1, e) - ref) / ref).max() <= 4 * 2.0 ** -52
    assert np.array_equal(evaluate(1, [0.0, 5e-324, 1e300]), [2.0, 2.0, 0.2])


def test_units(evaluate):
    x = np.concatenate([10.0 ** np.random.default_rng(3).uniform(-80, 80, 100_000), 2.0 ** np.arange(-250.0, 250.0)])
    u = evaluate(2, x)
    assert np.all((u <= x) & (x < 2 * u))
    assert np.all(np.frexp(u)[0] == 0.5) and np.array_equal(evaluate(3, u) * u, np.ones_like(u))
    assert np.array_equal(evaluate(2, [0.0, np.inf, np.nan, 5e-324, 1e-200, 1e200]), np.ones(6))
