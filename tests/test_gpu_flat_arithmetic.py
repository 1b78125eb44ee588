"""The branch-free square root and divisions (common.cuh) against CUDA's, bit
for bit: the square root of every non-negative finite float, the reciprocal of
every significand at every exponent taken, and quotients of random significands
with exponents all over and around each bound of the guards, wherever the guard
holds.  (A kernel of the test's own, compiled with the library's flags.)"""
import ctypes
import subprocess

import pytest

from prtcl_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "common.cuh"
using namespace prtcl_gpu;
using u32 = uint32_t;
using u64 = unsigned long long;

__device__ u32 mix(u64 k) {
  k ^= k >> 33; k *= 0xff51afd7ed558ccdull; k ^= k >> 33; k *= 0xc4ceb9fe1a85ec53ull; k ^= k >> 33;
  return u32(k);
}
// a float of random sign and significand, its exponent in [lo, hi]
__device__ float rnd(u64 k, int lo, int hi, bool sign) {
  u32 a = mix(k), e = u32(lo + int(mix(k + 0x9e3779b97f4a7c15ull) % u32(hi - lo + 1)) + 127);
  u32 m = a & 0x7fffffu;
  if ((a >> 23 & 7u) == 0u) m = (a >> 26 & 1u) ? 0x7fffffu : 0u; // ends of a binade
  return __uint_as_float((sign && (a >> 31) ? 0x80000000u : 0u) | (e > 254u ? 254u : e) << 23 | m);
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// out: [0] compared, [1] different, [2] not covered by the guard
__device__ void note(u64 *out, bool covered, bool equal) {
  if (!covered) atomicAdd(out + 2, 1ull);
  else {
    atomicAdd(out, 1ull);
    if (!equal) atomicAdd(out + 1, 1ull);
  }
}

__global__ void k_sqrt(u64 *out) {
  u64 n = 0, bad = 0;
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < 0x7f800000ull; i += u64(gridDim.x) * blockDim.x) {
    float x = __uint_as_float(u32(i));
    ++n;
    if (!same(sqrt_flat(x), sqrtf(x))) ++bad;
  }
  atomicAdd(out, n);
  atomicAdd(out + 1, bad);
}
__global__ void k_reciprocal(u64 *out) {
  u64 n = 0, bad = 0;
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < 80ull << 23; i += u64(gridDim.x) * blockDim.x) {
    float b = __uint_as_float((u32(i >> 23) + 127u - 40u) << 23 | u32(i & 0x7fffffull)); // 2^-40 ... 2^40
    ++n;
    if (!same(reciprocal_flat(b), 1.0f / b)) ++bad;
  }
  atomicAdd(out, n);
  atomicAdd(out + 1, bad);
}
// exponents of the numerator (or of the quotient) and of the divisor
__global__ void k_divide(u64 *out, u64 samples, int alo, int ahi, int blo, int bhi, int of_quotient, int zero) {
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < samples; i += u64(gridDim.x) * blockDim.x) {
    float b = rnd(i * 4, blo, bhi, false), a = rnd(i * 4 + 2, alo, ahi, true);
    if (of_quotient) a = a * b;
    if (zero) a = copysignf(0.0f, a);
    float q = divide_flat(a, b);
    note(out, divides_flat(a, b, q), same(q, a / b));
  }
}
__global__ void k_quotient(u64 *out, u64 samples, int alo, int ahi, int blo, int bhi, int of_quotient, int zero,
                           int guarded) {
  for (u64 i = blockIdx.x * u64(blockDim.x) + threadIdx.x; i < samples; i += u64(gridDim.x) * blockDim.x) {
    float b = rnd(i * 4, blo, bhi, false), a = rnd(i * 4 + 2, alo, ahi, true);
    if (of_quotient) a = a * b;
    if (zero) a = copysignf(0.0f, a);
    Divisor c = divisor(b);
    note(out, !guarded || quotient_exact(a, c), same(quotient(a, c), a / b));
  }
}

extern "C" int check(int what, u64 samples, int alo, int ahi, int blo, int bhi, int of_quotient, int zero, u64 *host) {
  u64 *d = nullptr;
  if (cudaMalloc(&d, 3 * sizeof(u64)) != cudaSuccess) return 1;
  cudaMemset(d, 0, 3 * sizeof(u64));
  if (what == 0) k_sqrt<<<1216, 256>>>(d);
  if (what == 1) k_reciprocal<<<1216, 256>>>(d);
  if (what == 2) k_divide<<<1216, 256>>>(d, samples, alo, ahi, blo, bhi, of_quotient, zero);
  if (what >= 3) k_quotient<<<1216, 256>>>(d, samples, alo, ahi, blo, bhi, of_quotient, zero, what == 3);
  cudaError_t e = cudaMemcpy(host, d, 3 * sizeof(u64), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("flat")
    src, so = d / "flat.cu", d / "flat.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-I", build.CSRC, "-shared", "-cudart", "static", str(src),
                    "-o", str(so)], check=True)
    f = ctypes.CDLL(str(so)).check
    f.argtypes = [ctypes.c_int, ctypes.c_ulonglong] + [ctypes.c_int] * 6 + [ctypes.POINTER(ctypes.c_ulonglong)]

    def run(what, samples=0, a=(0, 0), b=(0, 0), of_quotient=False, zero=False):
        out = (ctypes.c_ulonglong * 3)()
        assert f(what, samples, *a, *b, int(of_quotient), int(zero), out) == 0
        return tuple(out)

    return run


def test_square_root(check):
    assert check(0)[:2] == (0x7F800000, 0)


def test_reciprocal(check):
    assert check(1)[:2] == (80 << 23, 0)


SAMPLES = 1 << 24

# numerator (or quotient) exponents, divisor exponents, whether the numerator is
# quotient times divisor, share of the samples that the guard covers at least
DIVIDE = [
    ((-126, 127), (-126, 127), False, 0.1), ((-90, 60), (-39, 39), False, 0.9),
    ((-102, -98), (-39, 39), False, 0.2),                                   # the numerator's bound
    ((-122, -118), (-39, 39), True, 0.0), ((98, 102), (-39, 20), True, 0.3),  # the quotient's
    ((-60, 60), (-42, -38), False, 0.2), ((-60, 60), (38, 42), False, 0.2),   # the divisor's
]


@pytest.mark.parametrize("a,b,of_quotient,share", DIVIDE)
def test_division(check, a, b, of_quotient, share):
    n, bad, outside = check(2, SAMPLES, a, b, of_quotient)
    assert n + outside == SAMPLES and n >= share * SAMPLES and bad == 0


QUOTIENT = [
    ((-126, 127), (-126, 127), False, 0.1), ((-59, 59), (-39, 39), False, 0.99),
    ((-62, -58), (-39, 39), False, 0.3), ((58, 62), (-39, 39), False, 0.3),
    ((-59, 59), (-42, -38), False, 0.2), ((-59, 59), (38, 42), False, 0.2),
]


@pytest.mark.parametrize("a,b,of_quotient,share", QUOTIENT)
def test_prepared_division(check, a, b, of_quotient, share):
    n, bad, outside = check(3, SAMPLES, a, b, of_quotient)
    assert n + outside == SAMPLES and n >= share * SAMPLES and bad == 0


@pytest.mark.parametrize("what", [2, 3])
def test_zero_numerators(check, what):
    n, bad, outside = check(what, 1 << 16, (0, 0), (-40, 39), zero=True)
    assert (n, bad, outside) == (1 << 16, 0, 0)


# the kernel's own use (QuickKernel): distances from 2^-75 on and spline values,
# by smoothing scales between 2^-12 and 2^12 and their cubes, without a guard
@pytest.mark.parametrize("b", [(-12, 11), (-36, 35)])
def test_prepared_division_of_distances(check, b):
    n, bad, _ = check(4, SAMPLES, (-75, 13), b)
    assert n == SAMPLES and bad == 0
