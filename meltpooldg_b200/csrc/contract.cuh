// The 1D contraction of the cell kernels: one line of n values with an n x n matrix of fe_tables.hpp.
// No CUDA header is needed, so that a host compiler can build it (with __device__ and
// __forceinline__ defined) and its rounding can be tested on the CPU.
#pragma once

#include <type_traits>

#include "fe_tables.hpp"

namespace mpdg {

// entry i of the matrices' table (fill_even_odd); each arithmetic type defines its own
template <typename T> __device__ __forceinline__ T ctab(int i);

// a - 2 b (one operation)
__device__ __forceinline__ float minus_twice(float a, float b) { return fmaf(-2.f, b, a); }
__device__ __forceinline__ double minus_twice(double a, double b) { return fma(-2.0, b, a); }

// y = A x (or y += A x) for the n x n matrix of `kind`, centro-(anti)symmetric. Even-odd split:
// with E and O the even and odd parts of an output row, y_q accumulates O onto E, all in fused
// operations. The mirrored output E - O (or O - E) is y_q - 2 E or its negative in FP64, one
// operation: 14 instead of the 16 operations a row of E + O and E - O at n = 4, 19 instead of 24
// at n = 5; the plain product is shorter where there is too little to fold, at n = 2 and for
// y += A x up to n = 4. FP32 keeps the roundings of the separate sums: the mirrored output
// accumulates -O onto E, and y += A x adds the finished row (y_q - 2 E and accumulation onto y
// measured 6-12 % more error in the operator).
template <int n, int kind, bool add, typename T>
__device__ __forceinline__ void contract_row(const T (&x)[n], T (&y)[n])
{
  constexpr int h = n / 2;
  constexpr int off = tab_off(n, kind);
  constexpr bool even = kind_sym(kind) > 0, fp64 = std::is_same<T, double>::value;
  if constexpr (n == 2 || (fp64 && add && n <= 4)) {
    constexpr int full = off + tab_full(n);
    constexpr bool onto = add && fp64;
    T r[n];
#pragma unroll
    for (int q = 0; q < n; ++q) {
      r[q] = onto ? fma(ctab<T>(full + q * n), x[0], y[q]) : ctab<T>(full + q * n) * x[0];
#pragma unroll
      for (int l = 1; l < n; ++l) r[q] = fma(ctab<T>(full + q * n + l), x[l], r[q]);
    }
#pragma unroll
    for (int q = 0; q < n; ++q) y[q] = add && !onto ? y[q] + r[q] : r[q];
  } else {
    T e[h], o[h];
    const T mid = x[h];
#pragma unroll
    for (int l = 0; l < h; ++l) {
      e[l] = x[l] + x[n - 1 - l];
      o[l] = x[l] - x[n - 1 - l];
    }
#pragma unroll
    for (int q = 0; q < h; ++q) {
      T E = (n & 1) ? ctab<T>(off + 2 * n * h + q) * mid : ctab<T>(off + q * h) * e[0];
#pragma unroll
      for (int l = (n & 1) ? 0 : 1; l < h; ++l) E = fma(ctab<T>(off + q * h + l), e[l], E);
      T y0 = E, y1 = E;
#pragma unroll
      for (int l = 0; l < h; ++l) y0 = fma(ctab<T>(off + n * h + q * h + l), o[l], y0);
      // the mirrored output, E - O
      if constexpr (h > 1 && fp64) {
        y1 = -minus_twice(y0, E);
      } else {
#pragma unroll
        for (int l = 0; l < h; ++l) y1 = fma(-ctab<T>(off + n * h + q * h + l), o[l], y1);
      }
      y[q] = add ? y[q] + y0 : y0;
      if (even)
        y[n - 1 - q] = add ? y[n - 1 - q] + y1 : y1;
      else
        y[n - 1 - q] = add ? y[n - 1 - q] - y1 : -y1;
    }
    if constexpr (n & 1) {  // the middle row has only its even (or odd) part
      T c = even ? ctab<T>(off + 2 * n * h + h) * mid : ctab<T>(off + n * h + h * h) * o[0];
#pragma unroll
      for (int l = even ? 0 : 1; l < h; ++l)
        c = fma(ctab<T>(off + (even ? 0 : n * h) + h * h + l), even ? e[l] : o[l], c);
      y[h] = add ? y[h] + c : c;
    }
  }
}

}  // namespace mpdg
