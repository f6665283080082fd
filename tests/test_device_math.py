"""The reciprocals that stand in for divisions, on every float of their range.

The device functions are compiled out of the kernels' own headers.  One step of Newton's iteration leaves the error of its last
rounding (half a unit) and a square of the approximation's, far below a hundredth of a unit: 0.51 * 2^-23 of the value.  A
product adds half a unit.
"""
import ctypes
import importlib
import subprocess

import pytest

from conftest import cg

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdint>
#include "act.cuh"
#include "mma.cuh"

// largest error of the floats from_bits .. to_bits, in 2^-23 of the value (of 2^-126 at least)
template <class F>
__device__ void worst(uint32_t from_bits, uint32_t to_bits, unsigned long long* out, F error) {
  double w = 0;
  for (uint64_t b = from_bits + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b <= to_bits; b += (uint64_t)gridDim.x * blockDim.x) {
    const double e = error(__uint_as_float((uint32_t)b));
    if (!(e <= w)) w = e;   // (a NaN counts)
    if (w != w) w = 1e300;
  }
  atomicMax(out, (unsigned long long)__double_as_longlong(w));  // (no negative number: ordered like its bits)
}
__device__ double units(float got, double want) { return fabs((double)got - want) / (fmax(fabs(want), 0x1p-126) * 0x1p-23); }
__global__ void k_rcp(uint32_t from, uint32_t to, unsigned long long* out) {
  worst(from, to, out, [](float x) { return units(cg::rcp_newton(x), 1.0 / (double)x); });
}
__global__ void k_over(uint32_t from, uint32_t to, float g, unsigned long long* out) {
  worst(from, to, out, [g](float e) { return units(cg::over_one_plus(g, e), (double)g / (double)(1.f + e)); });
}
__global__ void k_one(int which, float a, float b, float* out) { *out = which ? cg::over_one_plus(a, b) : cg::rcp_newton(a); }

static double read(unsigned long long* d) {
  unsigned long long v;
  if (cudaMemcpy(&v, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  cudaFree(d);
  double e;
  __builtin_memcpy(&e, &v, 8);
  return e;
}
static unsigned long long* zero() {
  unsigned long long* d = nullptr;
  cudaMalloc(&d, 8);
  cudaMemset(d, 0, 8);
  return d;
}
extern "C" double rcp_error(uint32_t from, uint32_t to) {
  auto* d = zero();
  k_rcp<<<148 * 8, 256>>>(from, to, d);
  return read(d);
}
extern "C" double over_error(uint32_t from, uint32_t to, float g) {
  auto* d = zero();
  k_over<<<148 * 8, 256>>>(from, to, g, d);
  return read(d);
}
extern "C" float one(int which, float a, float b) {
  float *d = (float*)zero(), v = -1.f;
  k_one<<<1, 1>>>(which, a, b, d);
  cudaMemcpy(&v, d, 4, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return v;
}
"""

INF = 0x7F800000


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not __import__("torch").cuda.is_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("device_math")
    (d / "math.cu").write_text(SOURCE)
    b = importlib.import_module(cg.__name__ + ".build")
    subprocess.check_call([b.NVCC, *b.FLAGS, "-shared", "-I", b.CSRC, "-o", str(d / "math.so"), str(d / "math.cu")])
    lib = ctypes.CDLL(str(d / "math.so"))
    lib.rcp_error.restype = lib.over_error.restype = ctypes.c_double
    lib.rcp_error.argtypes = [ctypes.c_uint32, ctypes.c_uint32]
    lib.over_error.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_float]
    lib.one.restype, lib.one.argtypes = ctypes.c_float, [ctypes.c_int, ctypes.c_float, ctypes.c_float]
    return lib


def bits(x):
    return ctypes.c_uint32.from_buffer(ctypes.c_float(x)).value


def test_reciprocal(lib):
    assert lib.rcp_error(bits(1.0), bits(1e37)) <= 0.51
    inf, nan = float("inf"), float("nan")
    assert lib.one(0, 1.0, 0) == 1.0 and lib.one(0, 2.0, 0) == 0.5
    assert 0 <= lib.one(0, inf, 0) <= 1.01e-37 and 0 <= lib.one(0, 3e38, 0) <= 1.01e-37 and lib.one(0, nan, 0) != lib.one(0, nan, 0)


@pytest.mark.parametrize("g", [1.0, -88.5, -0.3, 7.77e-5, 3e38])
def test_quotient_by_one_plus(lib, g):
    """e from 0 to the largest number: sigmoids down to 2^-128, which a reciprocal of 1 + e would lose."""
    assert lib.over_error(0, INF - 1, g) <= 1.02
    if g == 1.0:
        assert lib.over_error(0, bits(2.0 ** 126), g) <= 0.51
    inf, nan = float("inf"), float("nan")
    assert lib.one(1, g, 0.0) == ctypes.c_float(g).value and lib.one(1, g, inf) == 0.0
    assert lib.one(1, g, nan) != lib.one(1, g, nan) and lib.one(1, -inf, inf) != lib.one(1, -inf, inf)
