"""The integer form of an FP64 product is the rounded product, bit for bit:
compiled here by the host's compiler and compared with its multiplication over
random factors and those whose products are ties, all ones, or at the ends of
the exponents' range."""
import pathlib
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "aerial-3d-model_gb300" / "csrc"
MAIN = r"""
#include "mul_int.cuh"
#include <cstdio>
#include <cstring>
#include <random>
int main() {
  std::mt19937_64 g(%d);
  const uint64_t frac = 0xfffffffffffffull;
  long bad = 0;
  for (long i = 0; i < 4000000; ++i) {
    uint64_t a = g(), b = g(), ea = 512 + g() %% 1021, eb = 512 + g() %% 1021;
    switch (%d) {
      case 1: a &= ~0x3ffffffull, b &= ~0x3ffffffull; break;  // exact products
      case 2: a &= ~0x1ffffffull, b &= ~0x3ffffffull; break;  // up to one bit more
      case 3: a |= frac - 0xf, b |= g() & frac; break;
      case 4: a |= frac, b &= ~frac | 1; break;
      case 5: ea = eb = i & 1 ? 512 : 1532; break;
    }
    a = (a & ~(0x7ffull << 52)) | ea << 52, b = (b & ~(0x7ffull << 52)) | eb << 52;
    double x, y;
    std::memcpy(&x, &a, 8), std::memcpy(&y, &b, 8);
    const double r = x * y;
    uint64_t want;
    std::memcpy(&want, &r, 8);
    bad += want != ba::mul_bits(ba::mul_op_bits(a >> 32, (uint32_t)a),
                                ba::mul_op_bits(b >> 32, (uint32_t)b));
    bad += !ba::mul_safe_hi(a >> 32) + !ba::mul_safe_hi(b >> 32);
  }
  for (uint32_t e : {0u, 511u, 1533u, 2047u})
    bad += ba::mul_safe_hi(e << 20) + ba::mul_safe_hi(0x800fffffu | e << 20);
  std::printf("%%ld\n", bad);
}
"""


@pytest.mark.parametrize("kind", range(6))
def test_products_match(kind, tmp_path):
    src, exe = tmp_path / "m.cpp", tmp_path / "m"
    src.write_text(MAIN % (kind + 1, kind))
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "0\n"
