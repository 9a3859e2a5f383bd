"""The device half of csrc/quotient.cuh against CUDA's own division: the reciprocal
of every significand, and quotients over the allowed divisors and dividends of
every size, tiny and subnormal ones among them."""
import os
import subprocess

import pytest

import hmclab_gb300 as H
from hmclab_gb300 import build

_SOURCE = r"""
#include <cstdio>
#include "quotient.cuh"
__device__ unsigned long long taken[2], wrong[2];
__device__ unsigned mix(unsigned x) {  // a permutation of the 32-bit words
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x;
}
__device__ void check(int k, float got, float want) {
  atomicAdd(&taken[k], 1ull);
  if (!(got == want)) atomicAdd(&wrong[k], 1ull);  // (up to the sign of a zero)
}
// every significand at 31 exponents (2^-30 .. 2), both signs at one
__global__ void reciprocals() {
  const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
  for (int e = -30; e <= 0; ++e)
    for (unsigned s = 0; s < (e == 0 ? 2u : 1u); ++s) {
      const float b = __uint_as_float(s << 31 | (unsigned)(e + 127) << 23 | m);
      if (hmc::plain_divisor(b)) check(0, hmc::reciprocal(b), 1.f / b);
    }
}
__global__ void quotients() {
  const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
  for (unsigned k = 0; k < 16; ++k) {
    unsigned ia = mix(16 * id + k), ib = mix(ia ^ 0x9e3779b9u);
    ib = (ib & 0x807fffffu) | (97 + (ib >> 23) % 31) << 23;
    if (k % 4 == 1) ia &= 0x83ffffffu;                  // tiny dividends
    if (k % 4 == 2) ia &= 0x80ffffffu;                  // subnormal ones
    if (k % 4 == 3) ib &= k & 4 ? 0xff800000u : 0xfffff000u;  // powers of two, few bits
    const float a = __uint_as_float(ia), b = __uint_as_float(ib);
    bool plain = hmc::plain_divisor(b);
    if (!plain) continue;
    const float q = hmc::quotient(a, b, hmc::reciprocal(b), plain);
    if (plain) check(1, q, a / b);
  }
}
int main() {
  reciprocals<<<(1 << 23) / 256, 256>>>();
  quotients<<<(1 << 22) / 256, 256>>>();
  unsigned long long t[2], w[2];
  if (cudaMemcpyFromSymbol(t, taken, sizeof t) != cudaSuccess || cudaMemcpyFromSymbol(w, wrong, sizeof w) != cudaSuccess) return 1;
  printf("%llu %llu %llu %llu\n", t[0], w[0], t[1], w[1]);
}
"""


@pytest.mark.gpu
def test_reciprocals_and_quotients(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    src, exe = tmp_path / "q.cu", tmp_path / "q"
    src.write_text(_SOURCE)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run([build._nvcc()] + build.ARCH_FLAGS + ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", csrc, str(src),
                                                         "-o", str(exe)], check=True)
    r, r_wrong, q, q_wrong = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert r == 32 * (2**23 - 1) and q > 2**25  # the significand of all ones is not taken
    assert r_wrong == 0 and q_wrong == 0
