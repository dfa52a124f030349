"""Host check of the two-electron gradient's work tables (no GPU)."""
import pytest

from conftest import REPO

GRAD_TABLE_CHECK = r"""
#include <cstdio>
#include "classes.h"
#include "grad.cuh"
using namespace sf;
// every output once per direction with its own offsets, the outputs of one
// exponent quadruple in a row on one lane, the last of them marked
template <int LA, int LB, int LC, int LD>
int check(int T) {
  using Q = QC<LA, LB, LC, LD>;
  using G = QG<LA, LB, LC, LD>;
  std::vector<uint2> tab;
  int2 hdr[3];
  grad_table<LA, LB, LC, LD>(T, tab, hdr);
  int bad = 0;
  for (int d = 0; d < 3; ++d) {
    std::vector<int> seen(Q::NABCD, 0), closed(G::NX, 0);
    for (int t = 0; t < T; ++t) {
      int open = -1;
      for (int k = 0; k < hdr[d].y; ++k) {
        const uint2 w = tab[hdr[d].x + k * T + t];
        if (w.x == ~0u) { bad += open >= 0; break; }
        const int o = w.x & 2047, e = w.y;
        ++seen[o];
        bad += Q::toff(o, d) != e || (open >= 0 && open != e) || closed[e];
        bad += (int)((w.x >> 11) & 255) != G::eoff(o, (d + 1) % 3) || (int)((w.x >> 19) & 255) != G::eoff(o, (d + 2) % 3);
        open = e;
        if (w.x >> 31) { ++closed[e]; open = -1; }
      }
      bad += open >= 0;
    }
    for (int v : seen) bad += v != 1;
    // a quadruple's derivative entries lie inside the extended table
    for (int e = 0; e < G::NX; ++e)
      bad += G::xoff(e) + G::SA >= G::SZE || (G::ex(e, 0) && G::xoff(e) - G::SA < 0) ||
             (G::ex(e, 2) && G::xoff(e) - G::SC < 0);
  }
  return bad;
}
int main() {
  int bad = 0;
#define SF_C(id, la, lb, lc, ld, t64, t32)                                        \
  for (int T : {2, tgrad(QC<la, lb, lc, ld>::NABCD), 32}) {                       \
    const int b = T > 1 ? check<la, lb, lc, ld>(T) : 0;                           \
    if (b) printf("%d%d%d%d T=%d: %d\\n", la, lb, lc, ld, T, b);                   \
    bad += b;                                                                     \
  }
  SF_CLASS_LIST(SF_C)
  return bad != 0;
}
"""


def test_gradient_work_tables(tmp_path):
    """The two-electron gradient's work tables (grad.cuh) on the host: coverage, offsets and grouping."""
    import os
    import shutil
    import subprocess
    nvcc = shutil.which("nvcc")
    if nvcc is None and os.path.exists("/usr/local/cuda/bin/nvcc"):
        nvcc = "/usr/local/cuda/bin/nvcc"
    if nvcc is None:
        pytest.skip("no nvcc")
    src = tmp_path / "tables.cu"
    src.write_text(GRAD_TABLE_CHECK)
    exe = tmp_path / "tables"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", f"{REPO}/include", "-I", f"{REPO}/segfault_py_gb300/csrc", str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
