"""The reciprocal and quotient of exact_div.cuh against CUDA's correctly rounded
ones, bit for bit: every mantissa at the ends and the middle of the exponents that
the short path takes, and the operands that it does not take."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu

CSRC = pathlib.Path(__file__).resolve().parents[1] / "starpolymersmd_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "exact_div.cuh"
__device__ unsigned long long bad[2];
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
int main() {
  const unsigned per = 1u << 23;
  for (unsigned e : {0u, 1u, 2u, 60u, 126u, 127u, 128u, 200u, 251u, 252u, 253u, 254u}) rcp<<<1024, 256>>>(e * per, per);
  for (float b : {5.0f, 1.0f, 3.0f, 0.1f, 1.99999988f, 1e-12f, 1.2e-12f, 1e12f, 3e-39f})
    for (unsigned e : {0u, 56u, 57u, 126u, 127u, 197u, 198u, 254u}) quot<<<1024, 256>>>(b, e * per, per);
  unsigned long long h[2] = {1, 1};
  const cudaError_t rc = cudaMemcpyFromSymbol(h, bad, sizeof(h));
  std::printf("%d %llu %llu\n", static_cast<int>(rc), h[0], h[1]);
}
"""


def test_exact_division_has_the_bits_of_the_general_one(tmp_path):
    (tmp_path / "t.cu").write_text(PROGRAM)
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3", "-I", str(CSRC),
                    "-o", str(tmp_path / "t"), str(tmp_path / "t.cu")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0", "0"]
