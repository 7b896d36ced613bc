"""The reciprocal and quotient of exact_div.cuh against CUDA's correctly rounded
ones, bit for bit: every mantissa at the ends and the middle of the exponents that
the short path takes, and the operands that it does not take (FP64: four million
mantissas each and those at the ends)."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu

CSRC = pathlib.Path(__file__).resolve().parents[1] / "starpolymersmd_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "exact_div.cuh"
__device__ unsigned long long bad[3];
__global__ void rcp(unsigned from, unsigned n) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (unsigned sign = 0; sign < 2; ++sign) {
      const float x = __uint_as_float((from + i) | sign << 31);
      if (__float_as_uint(smpc::rcp_exact(x)) != __float_as_uint(__frcp_rn(x))) atomicAdd(bad, 1ull);
    }
}
__global__ void quot(float b, unsigned from, unsigned n) {
  const float rb = smpc::rcp_exact(b);
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float a = __uint_as_float(from + i);
    if (__float_as_uint(smpc::div_exact(a, b, rb)) != __float_as_uint(__fdiv_rn(a, b))) atomicAdd(bad + 1, 1ull);
  }
}
__global__ void quot64(double b, unsigned e, unsigned n) {
  const double rb = 1.0 / b;
  unsigned long long s = (e * 2654435761ull + blockIdx.x * blockDim.x + threadIdx.x) * 0x9E3779B97F4A7C15ull + 1;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    const unsigned long long mant = i < 64 ? (i & 32 ? ~0ull - (i & 31) : i & 31) : s ^ s >> 29;
    const double a = __longlong_as_double(static_cast<long long>((mant & 0x800FFFFFFFFFFFFFull) | static_cast<unsigned long long>(e) << 52));
    if (__double_as_longlong(smpc::div_exact(a, b, rb)) != __double_as_longlong(__ddiv_rn(a, b))) atomicAdd(bad + 2, 1ull);
  }
}
int main() {
  const unsigned per = 1u << 23;
  for (unsigned e : {0u, 1u, 2u, 60u, 126u, 127u, 128u, 200u, 251u, 252u, 253u, 254u}) rcp<<<1024, 256>>>(e * per, per);
  for (float b : {5.0f, 1.0f, 3.0f, 0.1f, 1.99999988f, 1e-12f, 1.2e-12f, 1e12f, 3e-39f})
    for (unsigned e : {0u, 56u, 57u, 126u, 127u, 197u, 198u, 254u}) quot<<<1024, 256>>>(b, e * per, per);
  for (double b : {5.0, 1.0, 3.0, 0.1, 1.9999999999999998, 1e-60, 1e-61, 1e60, 3e-310})
    for (unsigned e : {0u, 522u, 523u, 1022u, 1023u, 1523u, 1524u, 2046u}) quot64<<<1024, 256>>>(b, e, 1u << 22);
  unsigned long long h[3] = {1, 1, 1};
  const cudaError_t rc = cudaMemcpyFromSymbol(h, bad, sizeof(h));
  std::printf("%d %llu %llu %llu\n", static_cast<int>(rc), h[0], h[1], h[2]);
}
"""


def test_exact_division_has_the_bits_of_the_general_one(tmp_path):
    (tmp_path / "t.cu").write_text(PROGRAM)
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3", "-I", str(CSRC),
                    "-o", str(tmp_path / "t"), str(tmp_path / "t.cu")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0", "0", "0"]
