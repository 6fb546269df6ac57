"""The integer double arithmetic of easier_gb300/csrc/soft64.cuh, compiled for
the host, against the host's own IEEE operations: bit for bit on random
operands, near rounding midpoints, at mantissa extremes and for zeros,
subnormals, infinities and NaN; the FP32 reciprocal approximation is taken up
to two units off, more than the device's is."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "easier_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "soft64.cuh"
using namespace soft64;

static uint64_t state = 88172645463325252ull;
static uint64_t rnd() { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; }
static const uint64_t kMant = 0xfffffffffffffull;
static double around_one(uint64_t m) { return value((m & kMant) | 0x3ff0000000000000ull); }
static double scaled(uint64_t m, int spread) {
  return value((m & 0x800fffffffffffffull) | ((uint64_t)(1023 - spread + (int)(rnd() % (2 * spread + 1))) << 52));
}
static bool same(double a, double b) { return bits(a) == bits(b) || (std::isnan(a) && std::isnan(b)); }

static void operands(int mode, double &a, double &b) {
  const uint64_t x = rnd(), y = rnd();
  const uint64_t pat[8] = {0, 1, 2, kMant, kMant - 1, 1ull << 51, (1ull << 51) - 1, x & kMant};
  const double odd[8] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, 2.2250738585072014e-308, 1.7976931348623157e308};
  switch (mode) {
    case 0: a = scaled(x, 30); b = scaled(y, 30); break;
    case 1: a = value(x); b = value(y); break;                            // any bit pattern
    case 2: b = around_one(y); a = value(bits(b * around_one(x)) + rnd() % 5 - 2); break;  // near a quotient's midpoint
    case 3: a = around_one(pat[rnd() % 8]); b = around_one(pat[rnd() % 8]); break;
    case 4: a = around_one(x << (y % 52)); b = around_one(y << (x % 52)); break;  // few bits
    case 5: a = odd[rnd() % 8]; b = rnd() & 1 ? scaled(y, 30) : odd[rnd() % 8]; break;
    default: a = scaled(x, 1000); b = scaled(y, 1000); break;             // results at the range's ends
  }
  if (rnd() & 1) { const double t = a; a = b; b = t; }
}

int main() {
  long bad = 0;
  for (long i = 0; i < 7000000; ++i) {
    double a, b;
    operands((int)(i % 7), a, b);
    Divisor d(b);
    const uint32_t hi = (uint32_t)(bits(b) >> 32), lo = (uint32_t)bits(b);
    const float bh = fvalue((((hi << 3) | (lo >> 29)) & 0x7fffffu) | 0x3f800000u);
    d.r = reciprocal(hi, lo, fvalue(fbits(1.0f / bh) + (uint32_t)(rnd() % 5) - 2u));
    if (!same(quotient(a, d), a / b) && bad++ < 5) std::printf("%a / %a\n", a, b);
    if (!same(product(a, b), a * b) && bad++ < 5) std::printf("%a * %a\n", a, b);
    if (!same(half(a), a * 0.5) && bad++ < 5) std::printf("%a / 2\n", a);
    if (!same(from_zero(a), 0.0 + a) && bad++ < 5) std::printf("0 + %a\n", a);
  }
  std::printf("bad %ld\n", bad);
  return bad != 0;
}
"""


def test_integer_arithmetic_is_the_machines(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "soft64.cpp", tmp_path / "soft64"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
