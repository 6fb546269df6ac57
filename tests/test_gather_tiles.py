"""What every thread of a Selector gather loads and stores, on the CPU: the
kernel's own index arithmetic (easier_gb300/csrc/gather_tile.cuh) over
pointers that check each access, for rows narrower and wider than a tile, one
and many of them, and indices out of range; and on the GPU the launches whose
threads' last vectors lie past the end of a row cut into column blocks."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "easier_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "gather_tile.cuh"

static long bad = 0;
template <class T>
struct Checked {  // p[0, n)
  T *p;
  int64_t at, n;
  Checked operator+(int64_t k) const { return {p, at + k, n}; }
  T &operator[](int64_t k) const {
    const int64_t i = at + k;
    if (i < 0 || i >= n) {
      if (bad++ < 8) std::printf("access %lld of %lld\n", (long long)i, (long long)n);
      return p[0];
    }
    return p[i];
  }
};
static int32_t load_index(const Checked<int32_t> &p) { return p[0]; }

constexpr int kThreads = 256;

template <int D, int U>
static void run(int64_t vpr, int64_t m, int64_t n_in, bool broken) {
  std::vector<uint32_t> x(n_in * vpr), y(m * vpr, 0xdeadbeefu);
  std::vector<int32_t> idx(m);
  for (size_t i = 0; i < x.size(); ++i) x[i] = (uint32_t)i;
  const int32_t out[3] = {-1, (int32_t)n_in, 2147483647};
  for (int64_t k = 0; k < m; ++k) idx[k] = broken && k % 5 == 2 ? out[k % 3] : (int32_t)((k * 7 + 3) % n_in);
  const int width = gather::tile_width(vpr), rows = gather::tile_rows(width, U * kThreads);
  const int64_t gx = (m + rows - 1) / rows, gy = (vpr + gather::kCols - 1) / gather::kCols;
  bool ok = true;
  for (int64_t by = 0; by < gy; ++by)
    for (int64_t bx = 0; bx < gx; ++bx)
      for (int t = 0; t < kThreads; ++t)
        ok = gather::copy_part<uint32_t, D, U, uint32_t, kThreads>(
                 Checked<uint32_t>{x.data(), 0, n_in * vpr}, (uint32_t)n_in, (uint32_t)vpr,
                 Checked<int32_t>{idx.data(), 0, m}, m, Checked<uint32_t>{y.data(), 0, m * vpr}, rows,
                 gather::fast_div(width), 0, (uint32_t)bx, (uint32_t)by, (uint32_t)t) && ok;
  if (ok == (broken && m > 2)) bad++, std::printf("status\n");
  for (int64_t k = 0; k < m; ++k) {
    const bool in = idx[k] >= 0 && idx[k] < n_in;
    for (int64_t c = 0; c < vpr; ++c)
      if (y[k * vpr + c] != (in ? (uint32_t)(idx[k] * vpr + c) : 0xdeadbeefu) && bad++ < 8)
        std::printf("row %lld of %lld, vector %lld of %lld\n", (long long)k, (long long)m, (long long)c, (long long)vpr);
  }
}

int main() {
  const int64_t rows[] = {1, 2, 3, 5, 257, 1025};
  const int64_t widths[] = {2, 4, 5, 7, 255, 256, 257, 511, 512, 513, 1000, 1023, 1024, 1025, 1279, 1281, 2047, 2048, 2049, 4100};
  for (int64_t m : rows)
    for (int64_t n_in : {(int64_t)1, (int64_t)2, (int64_t)19}) {
      for (int broken = 0; broken < 2; ++broken) {
        run<1, 1>(1, m, n_in, broken);
        run<1, 4>(1, m, n_in, broken);
        for (int64_t w : widths) {
          if (m * w > 300000) continue;
          run<0, 1>(w, m, n_in, broken);
          run<0, 4>(w, m, n_in, broken);
        }
      }
    }
  std::printf("bad %ld\n", bad);
  return bad != 0;
}
"""


def test_every_access_of_a_gather_is_in_bounds(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "tiles.cpp", tmp_path / "tiles"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1, 1025), (1, 4100), (3, 1279), (37, 2047), (2, 1024)])
def test_four_vectors_a_thread_of_wide_rows(rows, cols):
    """Enough rows for the form that keeps four vectors in flight (at least
    1,245,184 vectors)."""
    import torch

    import easier_gb300 as esr

    m = 1_245_184 // cols + 3
    g = torch.Generator().manual_seed(cols)
    idx = torch.randint(0, rows, (m,), generator=g)

    class M(esr.Module):
        def __init__(self):
            super().__init__()
            self.sel = esr.Selector(idx)

    mod = M()
    esr.compile([mod], "cuda")
    flat = torch.cat([torch.zeros(1), torch.randn(rows * cols, generator=g)]).cuda()
    x = flat[1:].view(rows, cols)  # (off 8 and 16 bytes: vectors of four)
    assert torch.equal(mod.sel(x), x[idx.cuda()])
