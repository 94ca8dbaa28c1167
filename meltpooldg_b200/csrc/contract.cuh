// The 1D contraction of the cell kernels: a line of n values with an n x n matrix of fe_tables.hpp.
// No CUDA header is needed, so that a host compiler can build it (with __device__ and
// __forceinline__ defined) and its rounding can be tested on the CPU.
#pragma once

#include <type_traits>

#include "fe_tables.hpp"

namespace mpdg {

// entry i of the matrices' table (fill_even_odd); each arithmetic type defines its own
template <typename T> __device__ __forceinline__ T ctab(int i);

// y = A x (or y += A x, which adds the finished row) for the n x n matrix of `kind`,
// centro-(anti)symmetric. Even-odd split: with E and O the even and odd parts of an output row, the
// output is E + O and its mirror image E - O (or O - E), h = n / 2 pairs a row.
//
// The forms are the shortest whose error is not above that of separately summed parts. Values that
// vary smoothly over a cell have |E| >> |O|, so it counts how often a sum of E's size is rounded:
// h + 1 times with separate parts (2 h + 2 operations a pair at even n).
//   n = 2: the plain product; for the derivatives, where it would round values that cancel, and at
//     n = 3, O is one product fused onto E.
//   n = 4, 6 in FP64: E accumulates onto O and the mirror image takes 2 O off again, 2 h + 1
//     operations, rounded h and h + 1 times (the operator's error 0.91-1.05 of separate parts').
//   Else separate parts. O accumulated onto E rounds 2 h times at E's size: FP32 in as many
//     operations at n = 4, 5 and more at 6, 7, with 1.10-1.17 (n = 4), 1.04-1.09 (5), 1.14-1.29
//     (6, 7) times the error; FP64 with twice E taken off for the mirror image 1.02-1.19 times.
// (Emulated operator on sine products, a Gaussian of radius 0.05 and a temperature field; on random
// operands, where E and O are alike, all forms are within 8 %.) On a B200 the FP64 forms take
// 1.33 ms for the k(T) tangent on 128^3 cells of FE_Q(3) (with twice E 1.41), 375 us for FE_Q(5) on
// 53 x 49 x 51 (416), 226 us for FE_Q(6) on 33^3 (218), 158 us for FE_Q(1) on 150^3 (155).
template <int n, int kind, bool add, typename T>
__device__ __forceinline__ void contract_row(const T (&x)[n], T (&y)[n])
{
  constexpr int h = n / 2;
  constexpr int off = tab_off(n, kind);
  constexpr bool even = kind_sym(kind) > 0;
  if constexpr (n == 2 && even) {
    constexpr int full = off + tab_full(n);
    const T y0 = fma(ctab<T>(full + 1), x[1], ctab<T>(full) * x[0]);
    const T y1 = fma(ctab<T>(full + 3), x[1], ctab<T>(full + 2) * x[0]);
    y[0] = add ? y[0] + y0 : y0;
    y[1] = add ? y[1] + y1 : y1;
  } else {
    T e[h], o[h];
    const T mid = x[h];
#pragma unroll
    for (int l = 0; l < h; ++l) {
      e[l] = x[l] + x[n - 1 - l];
      o[l] = x[l] - x[n - 1 - l];
    }
    constexpr bool onto_odd = std::is_same<T, double>::value && n % 2 == 0;
#pragma unroll
    for (int q = 0; q < h; ++q) {
      auto ae = [&](int l) { return ctab<T>(off + q * h + l); };
      auto ao = [&](int l) { return ctab<T>(off + n * h + q * h + l); };
      T O = ao(0) * o[0], E, y0, y1;
#pragma unroll
      for (int l = 1; l < h; ++l) O = fma(ao(l), o[l], O);
      if constexpr (onto_odd) {
        y0 = O;
#pragma unroll
        for (int l = 0; l < h; ++l) y0 = fma(ae(l), e[l], y0);
        y1 = even ? fma(T(-2), O, y0) : fma(T(2), O, -y0);
      } else {
        E = (n & 1) ? ctab<T>(off + 2 * n * h + q) * mid : ae(0) * e[0];
#pragma unroll
        for (int l = (n & 1) ? 0 : 1; l < h; ++l) E = fma(ae(l), e[l], E);
        if constexpr (h == 1) {
          y0 = fma(ao(0), o[0], E);
          y1 = even ? fma(-ao(0), o[0], E) : fma(ao(0), o[0], -E);
        } else {
          y0 = E + O;
          y1 = even ? E - O : O - E;
        }
      }
      y[q] = add ? y[q] + y0 : y0;
      y[n - 1 - q] = add ? y[n - 1 - q] + y1 : y1;
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
