"""soft64.cuh where its dispatch tests draw their lines: factors whose exponents
lie at the ends of the window that the integer product takes, products and
quotients whose result falls at the ends of the normal range or beyond it.
Every pair of the exponents in question, all signs, mantissas at random and at
their extremes; bit for bit the host's own operations (no GPU)."""
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

static uint64_t state = 0x9e3779b97f4a7c15ull;
static uint64_t rnd() { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; }
static const uint64_t kMant = 0xfffffffffffffull;
static uint64_t mantissa() {
  const uint64_t pat[8] = {0, 1, kMant, kMant - 1, 1ull << 51, 0x6a09e667f3bcdull, 0x6a09e667f3bccull, rnd() & kMant};
  return rnd() & 1 ? rnd() & kMant : pat[rnd() % 8];
}
static double of(int exponent) { return value(mantissa() | (uint64_t)exponent << 52 | (rnd() & 1) << 63); }
static bool same(double a, double b) { return bits(a) == bits(b) || (std::isnan(a) && std::isnan(b)); }

static long bad = 0, overflows = 0;
static void product_of(int ea, int eb) {
  for (int i = 0; i < 96; ++i) {
    const double a = of(ea), b = of(eb), want = a * b;
    overflows += std::isinf(want) && ea < 2047 && eb < 2047;
    if (!same(product(a, b), want) && bad++ < 8) std::printf("%a * %a = %a, not %a\n", a, b, want, product(a, b));
  }
}
static void quotient_of(int ea, int eb) {
  if (ea < 0 || ea > 2047 || eb < 0 || eb > 2047) return;
  for (int i = 0; i < 96; ++i) {
    const double a = of(ea), b = of(eb), want = a / b;
    if (!same(quotient(a, Divisor(b)), want) && bad++ < 8) std::printf("%a / %a = %a\n", a, b, want);
  }
}

int main() {
  const int ends[] = {0, 1, 2, 510, 511, 512, 513, 514, 1021, 1022, 1023, 1024, 1025,
                      1530, 1531, 1532, 1533, 1534, 1535, 1536, 1537, 1538, 2044, 2045, 2046, 2047};
  for (int ea : ends)
    for (int eb : ends) {
      product_of(ea, eb);
      quotient_of(ea, eb);
    }
  for (int eb = 0; eb < 2048; ++eb)  // results at either end of the range
    for (int d = -2; d <= 2; ++d) {
      const int low = 1023 + d - eb, high = 3069 + d - eb;
      if (low >= 0 && low < 2048) product_of(low, eb);
      if (high >= 0 && high < 2048) product_of(high, eb);
      quotient_of(eb - 1023 + d, eb);
      quotient_of(eb + 1023 + d, eb);
    }
  for (int e = 0; e < 2048; ++e)
    for (int i = 0; i < 16; ++i) {
      const double a = of(e);
      if (!same(half(a), a * 0.5) && bad++ < 8) std::printf("%a / 2\n", a);
    }
  std::printf("bad %ld of them, %ld overflows\n", bad, overflows);
  return bad != 0 || overflows < 1000;
}
"""


def test_results_at_the_ends_of_the_range(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "edges.cpp", tmp_path / "edges"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
def test_the_devices_products_at_the_ends_of_the_range():
    """Linsys.forward forms x * Av with soft64::product: every pair of the ends'
    exponents against torch's product (edges of a row add zeros)."""
    import torch

    import easier_gb300 as esr
    from easier_gb300 import ops
    from easier_gb300.numeric import Linsys

    e = torch.tensor([0, 1, 511, 512, 513, 1022, 1023, 1024, 1532, 1533, 1534, 1535, 1536, 2045, 2046, 2047])
    g = torch.Generator().manual_seed(7)

    def values(exponents):
        m = torch.randint(0, 1 << 52, exponents.shape, generator=g)
        m = torch.where(torch.rand(exponents.shape, generator=g) < 0.3, torch.tensor((1 << 52) - 1), m)
        sign = torch.randint(0, 2, exponents.shape, generator=g)
        return (m | exponents << 52).view(torch.float64) * (1.0 - 2.0 * sign)

    ea, eb = e.repeat_interleave(e.numel()).repeat(64), e.repeat(e.numel()).repeat(64)
    x, av = values(ea), values(eb)
    n = x.numel()

    class M(esr.Module):
        def __init__(self):
            super().__init__()
            empty = torch.zeros(0, dtype=torch.int64)
            self.sel, self.red = esr.Selector(empty), esr.Reducer(empty, n)
            self.Ae = esr.Tensor(torch.zeros(0, dtype=torch.float64), mode="partition")
            self.Av = esr.Tensor(av, mode="partition")
            self.A = Linsys(self.Av, self.Ae, self.sel, self.red)

    mod = M()
    esr.compile([mod], "cuda")
    got = ops.linsys_apply(mod.A, x.cuda())
    assert got is not None
    got, want = got.cpu(), 0.0 + x * av
    assert int(want.isinf().sum()) > 1000
    assert torch.equal(got.isnan(), want.isnan())
    ok = ~want.isnan()
    assert torch.equal(got[ok].view(torch.int64), want[ok].view(torch.int64))
