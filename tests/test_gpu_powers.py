"""The powers of the Newton stopping rules against extended precision, called in
a kernel of their own (no entry point returns them)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from goss_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = """
#include "goss_kernels.cuh"
namespace {
__global__ void powers(const double* x, const int* n, double* eta, double* power, int count)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) {
        eta[i] = goss_b200::pow_0_8(x[i]);
        power[i] = goss_b200::pow_int(x[i], n[i]);
    }
}
}
extern "C" __attribute__((visibility("default"))) int run(const void* x, const void* n, void* eta, void* power, int count)
{
    powers<<<(count + 127) / 128, 128>>>((const double*)x, (const int*)n, (double*)eta, (double*)power, count);
    return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    import torch

    d = tmp_path_factory.mktemp("powers")
    (d / "powers.cu").write_text(SOURCE)
    build._run([build.nvcc(), *build.ARCH, *build.COMMON, "--use_fast_math", "-shared", str(d / "powers.cu"), "-o",
                str(d / "powers.so")])
    lib = C.CDLL(str(d / "powers.so"))

    def call(x, n):
        x, n = torch.tensor(x, device="cuda"), torch.tensor(n, dtype=torch.int32, device="cuda")
        eta, power = torch.empty_like(x), torch.empty_like(x)
        torch.cuda.synchronize()
        ptrs = [C.c_void_p(t.data_ptr()) for t in (x, n, eta, power)]
        assert lib.run(*ptrs, x.numel()) == 0
        return eta.cpu().numpy(), power.cpu().numpy()

    return call


def _ulps(got, ref):
    return float((np.abs(got.astype(np.longdouble) - ref) / np.spacing(ref.astype(float))).max())


def test_powers_against_extended_precision(run):
    rng = np.random.default_rng(3)
    x = np.exp(rng.uniform(np.log(2.0 ** -52), np.log(1e16), 100_001))
    eta, _ = run(x, np.zeros(x.size))
    # 2 ulp: the bound that CUDA documents for pow
    assert _ulps(eta, np.power(x.astype(np.longdouble), np.longdouble(0.8))) <= 2
    x = rng.uniform(1e-3, 1, 100_001)
    n = rng.integers(0, 32, x.size)
    _, power = run(x, n)
    assert _ulps(power, np.power(x.astype(np.longdouble), n)) <= 2
    _, power = run(x, -n)
    assert _ulps(power, np.power(x.astype(np.longdouble), -n)) <= 2


def test_powers_of_special_operands(run):
    x = np.array([0.0, np.inf, np.nan, 1e-80, 1e80, 1e-310, 5e-324, 1.7e308, 1.0])
    eta, power = run(x, [1, 0, 1, 0, 1, 0, 0, 0, 30])
    np.testing.assert_allclose(eta, np.power(x, 0.8), rtol=1e-15)
    np.testing.assert_array_equal(power, [0.0, 1.0, np.nan, 1.0, 1e80, 1.0, 1.0, 1.0, 1.0])
