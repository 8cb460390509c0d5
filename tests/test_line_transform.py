"""The stream passes' line transforms (csrc/bgp_lfft.cuh), emulated on the CPU thread by
thread and stage by stage from the same index arithmetic: every compiled length and
factorization, forward against the transform's definition in long double, and forward
then inverse against the input, for full lines and for lines whose upper half is zero
(and unused on the way back).

Tolerance (2-norm, relative): eps log2 L per transform, twice that for the pair."""
import math
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LENGTHS = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768)

SRC = r"""
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include <math.h>
#include "bgp_lfft.cuh"
using namespace bgp;
template <int L, int V, bool HALF> void check() {
  typedef std::complex<long double> C;
  std::vector<double2> w(L), tab(lf_tab_len(L, V)), x(L), y;
  std::vector<C> wl(L);
  for (int t = 0; t < L; ++t) {
    const long double a = 2.0L * acosl(-1.0L) * t / L;
    wl[t] = C(cosl(a), -sinl(a));
    w[t] = cmk((double)cosl(a), -(double)sinl(a));
  }
  lf_fill_table<L, V>(w.data(), tab.data());
  srand(7 * L + V);
  for (int n = 0; n < L; ++n)
    x[n] = (HALF && n >= L / 2) ? cmk(0, 0) : cmk(rand() / (double)RAND_MAX - 0.5, rand() / (double)RAND_MAX - 0.5);
  y = x;
  if (HALF) for (int n = L / 2; n < L; ++n) y[n] = cmk(7.0, 7.0);   // must not be read
  lf_host_line<L, V, false, HALF>(y.data(), tab.data());
  long double e = 0, s = 0;
  for (int k = 0; k < L; ++k) {
    C z = 0;
    for (int n = 0; n < L; ++n) z += C(x[n].x, x[n].y) * wl[(long)n * k % L];
    e += std::norm(z - C(y[k].x, y[k].y));
    s += std::norm(z);
  }
  lf_host_line<L, V, true, HALF>(y.data(), tab.data());
  long double g = 0, h = 0;
  for (int n = 0; n < (HALF ? L / 2 : L); ++n) {
    g += std::norm(C(y[n].x / L - x[n].x, y[n].y / L - x[n].y));
    h += std::norm(C(x[n].x, x[n].y));
  }
  printf("%d %d %d %.3Le %.3Le\n", L, V, (int)HALF, sqrtl(e / s), sqrtl(g / h));
}
int main() {
#define CHECK(l) check<l, 0, false>(); check<l, 0, true>(); check<l, 1, false>(); check<l, 1, true>(); \
  check<l, 2, false>(); check<l, 2, true>();
  LENGTHS
}
"""


def test_every_length_and_factorization(tmp_path):
    nvcc = os.environ.get("NVCC", "nvcc")
    if shutil.which(nvcc) is None:
        pytest.skip("nvcc is not on PATH")
    src = tmp_path / "line.cu"
    src.write_text(SRC.replace("  LENGTHS", " ".join(f"CHECK({n})" for n in LENGTHS)))
    exe = tmp_path / "line"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-I",
                    os.path.join(ROOT, "becgpp_b200", "csrc"), str(src), "-o", str(exe)], check=True,
                   capture_output=True)
    rows = [r.split() for r in subprocess.run([str(exe)], check=True, capture_output=True,
                                              text=True).stdout.splitlines()]
    assert len(rows) == 6 * len(LENGTHS)
    for L, v, half, fwd, pair in rows:
        tol = 2.0 ** -52 * math.log2(int(L))
        assert float(fwd) < tol and float(pair) < 2 * tol, (L, v, half, fwd, pair)
