"""The copies of the FP64 tensor-core kernel along K (csrc/dmma_slab.h), run on the host: K of 2^31 and
more, whose slab counter has to outlive 32 bits, beside small and ragged ones."""
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
SRC = r'''
#include "dmma_slab.h"
#include <cstdio>
using namespace ssb;
// counts the valid elements and checks each source against the operand: the copies of one line (row r of an
// operand stored K-contiguous, K line 0 mod LSTEP otherwise) are consecutive, and none is past the end
struct Count {
  mutable long n = 0, last = -1;
  const double* X;
  long size;
  mutable bool ok = true;
  void take(const void* p, int bytes) const {
    if (bytes == 0) return;
    const long at = (const double*)p - X;
    if (at < 0 || at + bytes / 8 > size || at <= last) ok = false;
    last = at + bytes / 8 - 1;
    n += bytes / 8;
  }
  void cp16(uint32_t, const void* p, int bytes) const { take(p, bytes); }
  void cp8(uint32_t, const void* p, int bytes) const { take(p, bytes); }
};
// one row of K elements: each of its threads (2 k of every slab, K-contiguous; one k line in LSTEP otherwise)
// copies its share; ends: the first and the last of them only
template <bool MN>
bool row(long K, const double* X, bool ends) {
  constexpr int BK = 16, NT = 128;
  using S = Slab<64, BK, NT, MN>;
  for (int t = 0; t < NT; ++t) {
    if (MN ? t % S::CPL != 0 : t >= S::CPL) continue;
    if (ends && t != 0 && t != (MN ? NT - S::CPL : S::CPL - 1)) continue;
    S s;
    s.init(X, 1, K, MN ? 1 : K, 0, t);
    if (s.slabs() != (K + BK - 1) / BK) return false;
    Count c;
    c.X = X;
    c.size = K;
    const int all = s.slabs();
    for (int i = 0; i < all; ++i) s.copy(0, c);
    long share = 0;      // k of this thread: a whole slab's, and those of the rest
    for (int k = 0; k < BK; ++k)
      if (MN ? k % S::LSTEP == t / S::CPL : k / 2 == t) share += K / BK + (k < K % BK ? 1 : 0);
    if (!c.ok || c.n != share) return false;
  }
  return true;
}
int main() {
  // never read: a base on the 16-byte grid and one off it
  const double* bases[2] = {(const double*)(uintptr_t)(1ull << 32), (const double*)(uintptr_t)((1ull << 32) + 8)};
  for (const double* X : bases)
    for (long K = 1; K < 100; ++K)
      if (!row<false>(K, X, false) || !row<true>(K, X, false)) return std::printf("K %ld\n", K), 1;
  const long K = KVALUE;
  if (!row<false>(K, bases[0], true) || !row<true>(K, bases[1], true)) return std::printf("K %ld\n", K), 2;
  std::puts("ok");
  return 0;
}
'''


@pytest.mark.parametrize("k", [2 ** 31 + 1607, 2 ** 32 + 5])
def test_long_k(tmp_path, k):
    src = tmp_path / "t.cpp"
    src.write_text(SRC.replace("KVALUE", f"{k}L"))
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O3", "-I", str(ROOT / "ssblasex_b200" / "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout)
