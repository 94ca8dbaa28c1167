"""Rounding of the cell kernels' 1D contraction (contract.cuh), built with the host compiler: the
packed FP32 pairs compute what FP32 does."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "meltpooldg_b200",
                    "csrc")

HEAD = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#define __device__
#define __forceinline__ inline
#include "fe_tables.hpp"
namespace mpdg { using std::fma; using std::fmaf; }
#include "contract.cuh"
using namespace mpdg;
static std::vector<double> tab, w, xl;
namespace mpdg {
template <> inline double ctab<double>(int i) { return tab[i]; }
template <> inline float ctab<float>(int i) { return (float)tab[i]; }
}
"""

PAIRS = HEAD + r"""
namespace mpdg {
struct F2 {
  float a, b;
  F2() = default;
  F2(float s) : a(s), b(s) {}
  F2(float x, float y) : a(x), b(y) {}
};
inline F2 operator+(F2 x, F2 y) { return F2(x.a + y.a, x.b + y.b); }
inline F2 operator-(F2 x, F2 y) { return F2(x.a - y.a, x.b - y.b); }
inline F2 operator*(F2 x, F2 y) { return F2(x.a * y.a, x.b * y.b); }
inline F2 operator-(F2 x) { return F2(-x.a, -x.b); }
inline F2 fma(F2 x, F2 y, F2 z) { return F2(std::fma(x.a, y.a, z.a), std::fma(x.b, y.b, z.b)); }
inline F2 minus_twice(F2 x, F2 y) { return F2(std::fma(-2.f, y.a, x.a), std::fma(-2.f, y.b, x.b)); }
template <> inline F2 ctab<F2>(int i) { return F2((float)tab[i]); }
}
static int differ = 0;
template <int n, int kind, bool add> void check(std::mt19937 &g)
{
  std::uniform_real_distribution<float> u(-1.f, 1.f);
  for (int rep = 0; rep < 200; ++rep) {
    F2 x[n], y[n];
    float xa[n], xb[n], ya[n], yb[n];
    for (int i = 0; i < n; ++i) {
      x[i] = F2(xa[i] = u(g), xb[i] = u(g));
      y[i] = F2(ya[i] = u(g), yb[i] = u(g));
    }
    contract_row<n, kind, add>(x, y);
    contract_row<n, kind, add>(xa, ya);
    contract_row<n, kind, add>(xb, yb);
    for (int i = 0; i < n; ++i) differ += y[i].a != ya[i] || y[i].b != yb[i];
  }
}
template <int n> void kinds(std::mt19937 &g)
{
  check<n, kS, false>(g);
  check<n, kST, false>(g);
  check<n, kD, false>(g);
  check<n, kDT, true>(g);
}
int main()
{
  fill_even_odd(tab, w, xl);
  std::mt19937 g(1);
  kinds<2>(g);
  kinds<3>(g);
  kinds<4>(g);
  std::printf("%d\n", differ);
}
"""


def run(tmp_path, source):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", "-I",
                    CSRC, str(src), "-o", str(exe)], check=True, timeout=300)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True,
                          timeout=300).stdout


def test_packed_pairs_round_as_fp32_does(tmp_path):
    """Every lane of the packed kernel's contractions (n <= 4) has the bits of the FP32 one: the FP64
    forms are chosen by the type, not by its size."""
    assert int(run(tmp_path, PAIRS)) == 0
