// Line kernel of the operator application: one thread per 1D line of a cell (n^2 threads a cell),
// the lines in registers, three shared arrays a cell between the directions.
//
// Evaluation with the nodal value and derivative matrices S and G, one direction at a time:
//   z-lines  a = S u, az = G u                                  (2 arrays written)
//   y-lines  S a, G a, S az                                     (in place, a third array)
//   x-lines  S a, G a, S (G a), S az: the point's value and gradient, in registers
// the quadrature points of an x-line in its thread's registers, and integration in reverse:
//   x-lines  S^T val + G^T f_x, S^T f_y, S^T f_z
//   y-lines  S^T . + G^T ., S^T .
//   z-lines  S^T . + G^T ., scattered
// 18 sweeps and 4 block barriers a batch. The first form swept values and collocation derivatives
// one at a time through 5 to 9 shared arrays, 12 sweeps and 12 barriers (FP64 p = 4 on 64^3 cells:
// k(T) from its fields 0.91 -> 0.50 ms, deformed 0.95 -> 0.66 ms; FP32 p = 6 constant law on 45^3
// cells 0.49 -> 0.28 ms, k(T) deformed 0.74 -> 0.47 ms). Shared memory and the barriers bound it.
// FP32 p = 4 on deformed meshes, against register planes: 48^3 cells constant law 182 -> 162 us,
// k(T) 254 -> 209 us; 30^3 liquid-solid 172 -> 65 us, three-phase fields 120 -> 59 us.
// A thread rewrites only the lines it has read, so a batch needs no barrier before the next one.
// z-lines are gathered and scattered with the lanes along x, so rows of nodes are contiguous.
#pragma once

#include "cell_kernels.cuh"

namespace mpdg {

// shared doubles (floats) per cell: three arrays [k][j][i]; at even n an odd row stride keeps the
// x-lines' stride odd
template <int n> __host__ __device__ constexpr int ln_row() { return (n & 1) ? n : n + 1; }
template <int n> __host__ __device__ constexpr int ln_array() { return n * n * ln_row<n>(); }
template <int n, typename T> __host__ __device__ constexpr size_t ln_smem()
{
  return sizeof(T) * cells_per_block(n) * 3 * ln_array<n>();
}

// the three line directions of a thread: (c0, c1) = (i, j) of its z-line, (i, k) of its y-line,
// (j, k) of its x-line
template <int n> struct Lines {
  int z, y, x;  // first entry; strides n * row, row and 1
  __device__ __forceinline__ Lines(int line)
  {
    const int c0 = line % n, c1 = line / n, R = ln_row<n>();
    z = c0 + R * c1;
    y = c0 + n * R * c1;
    x = R * (c0 + n * c1);
  }
  static constexpr int sz = n * ln_row<n>();
  static constexpr int sy = ln_row<n>();
};

template <int n, typename T> __device__ __forceinline__ void get_line(const T *b, int s, T (&x)[n])
{
#pragma unroll
  for (int q = 0; q < n; ++q) x[q] = b[q * s];
}
template <int n, typename T> __device__ __forceinline__ void put_line(T *b, int s, const T (&x)[n])
{
#pragma unroll
  for (int q = 0; q < n; ++q) b[q * s] = x[q];
}

// value and reference gradient on the x-line from the nodal values of the z-line; b: 3 arrays
template <int n, typename T>
__device__ __forceinline__ void ln_evaluate(const T (&u)[n], T *b, const Lines<n> &l, T (&v)[n],
                                            T (&gx)[n], T (&gy)[n], T (&gz)[n])
{
  constexpr int N = ln_array<n>(), sz = Lines<n>::sz, sy = Lines<n>::sy;
  T r[n], s[n], t[n];
  contract_row<n, kS, false>(u, r);
  put_line<n>(b + l.z, sz, r);
  contract_row<n, kG, false>(u, r);
  put_line<n>(b + N + l.z, sz, r);
  __syncthreads();
  get_line<n>(b + l.y, sy, r);
  get_line<n>(b + N + l.y, sy, s);
  contract_row<n, kS, false>(r, t);
  put_line<n>(b + l.y, sy, t);
  contract_row<n, kS, false>(s, t);
  put_line<n>(b + N + l.y, sy, t);
  contract_row<n, kG, false>(r, t);
  put_line<n>(b + 2 * N + l.y, sy, t);
  __syncthreads();
  get_line<n>(b + l.x, 1, r);
  contract_row<n, kS, false>(r, v);
  contract_row<n, kG, false>(r, gx);
  get_line<n>(b + 2 * N + l.x, 1, r);
  contract_row<n, kS, false>(r, gy);
  get_line<n>(b + N + l.x, 1, r);
  contract_row<n, kS, false>(r, gz);
}

// values only
template <int n, typename T>
__device__ __forceinline__ void ln_values(const T (&u)[n], T *b, const Lines<n> &l, T (&v)[n])
{
  T r[n], t[n];
  contract_row<n, kS, false>(u, r);
  put_line<n>(b + l.z, Lines<n>::sz, r);
  __syncthreads();
  get_line<n>(b + l.y, Lines<n>::sy, r);
  contract_row<n, kS, false>(r, t);
  put_line<n>(b + l.y, Lines<n>::sy, t);
  __syncthreads();
  get_line<n>(b + l.x, 1, r);
  contract_row<n, kS, false>(r, v);
}

// the z-line's integrals of the x-line's value and flux
template <int n, typename T>
__device__ __forceinline__ void ln_integrate(const T (&v)[n], const T (&fx)[n], const T (&fy)[n],
                                             const T (&fz)[n], T *b, const Lines<n> &l, T (&w)[n])
{
  constexpr int N = ln_array<n>(), sz = Lines<n>::sz, sy = Lines<n>::sy;
  T r[n], s[n];
  contract_row<n, kST, false>(v, r);
  contract_row<n, kGT, true>(fx, r);
  put_line<n>(b + l.x, 1, r);
  contract_row<n, kST, false>(fz, r);
  put_line<n>(b + N + l.x, 1, r);
  contract_row<n, kST, false>(fy, r);
  put_line<n>(b + 2 * N + l.x, 1, r);
  __syncthreads();
  get_line<n>(b + l.y, sy, r);
  contract_row<n, kST, false>(r, s);
  get_line<n>(b + 2 * N + l.y, sy, r);
  contract_row<n, kGT, true>(r, s);
  put_line<n>(b + l.y, sy, s);
  get_line<n>(b + N + l.y, sy, r);
  contract_row<n, kST, false>(r, s);
  put_line<n>(b + N + l.y, sy, s);
  __syncthreads();
  get_line<n>(b + l.z, sz, r);
  contract_row<n, kST, false>(r, w);
  get_line<n>(b + N + l.z, sz, r);
  contract_row<n, kGT, true>(r, w);
}

// The trilinear map of a cell along an x-line (eta, zeta fixed): dx/dxi is constant, dx/deta and
// dx/dzeta are linear in xi, and so are the cofactor columns c1 = dx/dzeta x dx/dxi and
// c2 = dx/dxi x dx/deta.
template <typename T> struct LineMap {
  T jx[3], jy0[3], jy1[3], jz0[3], jz1[3];
  LineMap() = default;
  __device__ __forceinline__ LineMap(const MeshDims &d, const double *__restrict__ vert, int cx,
                                     int cy, int cz, T eta, T zeta)
  {
    const int64_t row = 3 * (int64_t)(d.m[0] + 1), layer = row * (d.m[1] + 1);
    const double *v = vert + layer * cz + row * cy + 3 * cx;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const T x0 = __ldg(v + e), x1 = __ldg(v + 3 + e), x2 = __ldg(v + row + e),
              x3 = __ldg(v + row + 3 + e), x4 = __ldg(v + layer + e), x5 = __ldg(v + layer + 3 + e),
              x6 = __ldg(v + layer + row + e), x7 = __ldg(v + layer + row + 3 + e);
      const T ex = x1 - x0, ey = x2 - x0, exy = (x3 - x2) - ex, exz = (x5 - x4) - ex,
              eyz = (x6 - x4) - ey, exyz = ((x7 - x6) - (x5 - x4)) - exy;
      const T mx = fma(exyz, zeta, exy);  // d/dxi d/deta on the line
      jx[e] = fma(mx, eta, fma(exz, zeta, ex));
      jy0[e] = fma(eyz, zeta, ey);
      jy1[e] = mx;
      jz0[e] = fma(eyz, eta, x4 - x0);
      jz1[e] = fma(exyz, eta, exz);
    }
  }
};

// Geometry of a deformed mesh: FP64 evaluates the vertices' map where the coefficients need no
// T_lin (k(T) tangent from its fields p = 4 on 64^3 cells 0.66 against 0.69 ms with the stored
// factors, p = 6 on 45^3 0.80 against 0.83 ms); with T_lin's four values a point in registers as
// well it spills (p = 4 0.80 against 0.74 ms stored). FP32 reads the stored factors.
template <typename T, int GEO, int LAW> constexpr int ln_geometry()
{
  return GEO == 1 && sizeof(T) == 8 && !law_tdep<LAW>() ? 2 : GEO;
}

// Blocks per SM for the register allocator. FP64 holds 4 to 8 lines of n values and wants 128 to
// 168 registers (p = 4 constant law on 64^3 cells 0.42 ms at 3 blocks, 0.50 at 5); the fields' laws on
// a uniform box hold fewer (k(T) 0.52 ms at 3, 0.50 at 5). FP32 p = 5: 0.35 ms at 5, 0.39 at 3.
template <int n, typename T, int GEO, int LAW> constexpr int ln_min_blocks()
{
  constexpr bool tdep = law_tdep<LAW>();
  if (sizeof(T) == 4) return n == 6 ? (GEO == 1 && tdep ? 4 : 5) : (n == 7 ? 5 : 4);
  if (n == 5) return GEO == 0 && !tdep && LAW != 0 ? 5 : (GEO == 1 ? 4 : 3);
  return 3;
}

// dst += J src; GEO 0 uniform box, 1 stored per-point geometry, 2 from the cell's vertices
template <int n, typename T, int GEO, int LAW>
__global__ void __launch_bounds__(block_threads(n), (ln_min_blocks<n, T, GEO, LAW>()))
  k_vmult_lines(CellArgs<T> a)
{
  constexpr int n2 = n * n, n3 = n2 * n, CPB = cells_per_block(n);
  constexpr bool TDEP = law_tdep<LAW>(), TOLD = law_told<LAW>();
  if (a.st && a.st->done) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int cl = threadIdx.x / n2, line = threadIdx.x % n2;
  const int c0 = line % n, c1 = line / n;  // z-line: node (i, j); x-line: point (j, k)
  const Lines<n> l(line);
  T *b = reinterpret_cast<T *>(smem_raw) + cl * 3 * ln_array<n>();
  const MeshDims &d = a.d;
  const int64_t rs = d.nd[0], ps = (int64_t)d.nd[0] * d.nd[1];
  const T wl = cw<T>(w_off(n) + c0) * cw<T>(w_off(n) + c1);  // weights of the x-line's (j, k)
  const T eta = cw<T>(xg_off(n) + c0), zeta = cw<T>(xg_off(n) + c1);
  double dot = 0.0;
  const int64_t n_batches = (a.n_cells + CPB - 1) / CPB;
  CellWalk at(d, (int64_t)blockIdx.x * CPB + cl, (int64_t)gridDim.x * CPB, a.n_cells);
  for (int64_t batch = blockIdx.x; batch < n_batches; batch += gridDim.x) {
    const int64_t cell = batch * CPB + cl;
    const bool active = cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    // (inactive cells read cell 0 and scatter nothing)
    const int cx = active ? at.x : 0, cy = active ? at.y : 0, cz = active ? at.z : 0;
    at.advance(d);
    const int I = d.p * cx + c0, J = d.p * cy + c1, K0 = d.p * cz;
    const int64_t base = I + rs * J + ps * K0;
    const bool con = constrained(d, I, J, -1), lo = (d.dmask & 16) && K0 == 0,
               hi = (d.dmask & 32) && K0 + d.p == d.nd[2] - 1;
    T u[n];
#pragma unroll
    for (int k = 0; k < n; ++k) u[k] = __ldg(a.src + base + ps * k);
    T tl[TDEP ? n : 1], to[TOLD ? n : 1];
    if constexpr (TDEP) {
#pragma unroll
      for (int k = 0; k < n; ++k) tl[k] = __ldg(a.Tl + base + ps * k);
    }
    if constexpr (TOLD) {
      if (a.m.need_told) {
#pragma unroll
        for (int k = 0; k < n; ++k) to[k] = __ldg(a.To + base + ps * k);
      }
    }
    // L2 prefetch of the next batch's nodes and per-point data
    {
      const int64_t next = (batch + gridDim.x) * CPB + cl;
      if (next < a.n_cells) {
        const int64_t nb = rs * (d.p * at.y + c0) + ps * (d.p * at.z + c1) + d.p * at.x;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.src + nb));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.src + nb + n - 1));
        if (TDEP) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.Tl + nb));
        constexpr int nf = LAW == 4 || LAW == 5 ? 5 : (LAW == 6 ? 8 : (LAW == 7 ? 4 : 0));
        if constexpr (nf > 0) {
          const char *f = reinterpret_cast<const char *>(a.cf + next * nf * n3);
          for (int off = line * 128; off < nf * n3 * (int)sizeof(T); off += n2 * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(f + off));
        }
        if constexpr (GEO == 1) {
          const char *g = reinterpret_cast<const char *>(a.g.q + next * 7 * n3);
          for (int off = line * 128; off < 7 * n3 * (int)sizeof(T); off += n2 * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(g + off));
        }
      }
    }
#pragma unroll
    for (int k = 0; k < n; ++k)
      if (con || (k == 0 && lo) || (k == n - 1 && hi)) u[k] = T(0);

    // the linearisation point's values and gradients on the x-line
    T Tq[TDEP ? n : 1], Tx[TDEP ? n : 1], Ty[TDEP ? n : 1], Tz[TDEP ? n : 1], To[TOLD ? n : 1];
    if constexpr (TOLD) {
      if (a.m.need_told) {
        ln_values<n>(to, b, l, To);
        __syncthreads();
      }
    }
    if constexpr (TDEP) {
      ln_evaluate<n>(tl, b, l, Tq, Tx, Ty, Tz);
      __syncthreads();
    }
    T v[n], gx[n], gy[n], gz[n];
    ln_evaluate<n>(u, b, l, v, gx, gy, gz);

    // quadrature points (i, j = c0, k = c1)
    const int64_t q0 = (int64_t)n * line;
    LineMap<T> map = [&]() {
      if constexpr (GEO == 2) return LineMap<T>(d, a.g.vert, cx, cy, cz, eta, zeta);
      else return LineMap<T>();
    }();
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const T w = wl * cw<T>(w_off(n) + i);
      T jxw, G[6], k0v[3], k1v[3], k2v[3], s;
      if constexpr (GEO == 0) {
        jxw = a.g.detJ * w;
        G[0] = a.g.Gd[0] * w;
        G[3] = a.g.Gd[1] * w;
        G[5] = a.g.Gd[2] * w;
        G[1] = G[2] = G[4] = T(0);
      } else if constexpr (GEO == 1) {
        const T *gb = a.g.q + cc * 7 * n3 + q0 + i;
        jxw = __ldg(gb);
#pragma unroll
        for (int f = 0; f < 6; ++f) G[f] = __ldg(gb + (1 + f) * n3);
      } else {
        const T xi = cw<T>(xg_off(n) + i);
        T jy[3], jz[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          jy[e] = fma(map.jy1[e], xi, map.jy0[e]);
          jz[e] = fma(map.jz1[e], xi, map.jz0[e]);
        }
        cross(jy, jz, k0v);
        cross(jz, map.jx, k1v);
        cross(map.jx, jy, k2v);
        const T det = map.jx[0] * k0v[0] + map.jx[1] * k0v[1] + map.jx[2] * k0v[2];
        jxw = w * det;
        s = w / det;
      }
      const T uu = v[i], ux = gx[i], uy = gy[i], uz = gz[i];
      T f0, f1, f2, val;
      if constexpr (LAW == 4) {
        const T *cf = a.cf + cc * 5 * n3 + q0 + i;
        const T kk = __ldg(cf + n3);
        val = a.m.idt * __ldg(cf) * uu + __ldg(cf + 2 * n3) * ux + __ldg(cf + 3 * n3) * uy +
              __ldg(cf + 4 * n3) * uz;
        f0 = kk * ux;
        f1 = kk * uy;
        f2 = kk * uz;
      } else if constexpr (LAW == 6) {  // c u + rho_cp b.grad(u), flux k grad(u) + dk grad(T_lin) u
        const T *cf = a.cf + cc * 8 * n3 + q0 + i;
        const T kk = __ldg(cf + n3);
        val = __ldg(cf) * uu + __ldg(cf + 2 * n3) * ux + __ldg(cf + 3 * n3) * uy +
              __ldg(cf + 4 * n3) * uz;
        f0 = kk * ux + __ldg(cf + 5 * n3) * uu;
        f1 = kk * uy + __ldg(cf + 6 * n3) * uu;
        f2 = kk * uz + __ldg(cf + 7 * n3) * uu;
      } else if constexpr (LAW == 7) {
        const T *cf = a.cf + cc * 4 * n3 + q0 + i;
        const T kk = __ldg(cf);
        f0 = kk * ux + __ldg(cf + n3) * uu;
        f1 = kk * uy + __ldg(cf + 2 * n3) * uu;
        f2 = kk * uz + __ldg(cf + 3 * n3) * uu;
        val = a.m.idt * (a.m.rho_l * a.m.cp_l) * uu * jxw;
      } else {
        T rhocp, kk, drhocp, dk, b0 = T(0), b1 = T(0), b2 = T(0);
        if constexpr (LAW == 5) {
          const T *cf = a.cf + cc * 5 * n3 + q0 + i;
          mat_eval_w(a.m, Tq[i], __ldg(cf), rhocp, kk, drhocp, dk);
          b0 = __ldg(cf + 2 * n3);
          b1 = __ldg(cf + 3 * n3);
          b2 = __ldg(cf + 4 * n3);
        } else {
          mat_eval<LAW>(a.m, TDEP ? Tq[TDEP ? i : 0] : T(0), rhocp, kk, drhocp, dk);
        }
        T cval = a.m.idt * rhocp;
        f0 = kk * ux;
        f1 = kk * uy;
        f2 = kk * uz;
        if constexpr (TDEP) {
          if constexpr (TOLD) {
            if (a.m.need_told) cval += a.m.idt * drhocp * (Tq[i] - To[i]);
          }
          f0 += dk * Tx[i] * uu;
          f1 += dk * Ty[i] * uu;
          f2 += dk * Tz[i] * uu;
        }
        val = cval * uu * jxw;
        if constexpr (LAW == 5)  // rho_cp b.grad(u) + d(rho_cp)/dT (b.grad T) u, b = JxW J^-1 v
          val += rhocp * (b0 * ux + b1 * uy + b2 * uz) +
                 drhocp * (b0 * Tx[i] + b1 * Ty[i] + b2 * Tz[i]) * uu;
      }
      v[i] = val;
      if constexpr (GEO == 2) {
        T m[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) m[e] = s * (k0v[e] * f0 + k1v[e] * f1 + k2v[e] * f2);
        gx[i] = k0v[0] * m[0] + k0v[1] * m[1] + k0v[2] * m[2];
        gy[i] = k1v[0] * m[0] + k1v[1] * m[1] + k1v[2] * m[2];
        gz[i] = k2v[0] * m[0] + k2v[1] * m[1] + k2v[2] * m[2];
      } else {
        apply_G<GEO>(G, f0, f1, f2, gx[i], gy[i], gz[i]);
      }
    }
    T w[n];
    ln_integrate<n>(v, gx, gy, gz, b, l, w);

    // src.dst partial and scatter (constrained rows skipped)
    if (active) {
      if (a.fin != FIN_NONE) {
        T x[n];
#pragma unroll
        for (int k = 0; k < n; ++k) x[k] = __ldg(a.src + base + ps * k);
#pragma unroll
        for (int k = 0; k < n; ++k)
          dot += con || (k == 0 && lo) || (k == n - 1 && hi) ? 0.0 : (double)x[k] * (double)w[k];
      }
#pragma unroll
      for (int k = 0; k < n; ++k)
        if (!(con || (k == 0 && lo) || (k == n - 1 && hi)))
          atomic_add(a.dst + base + ps * k, w[k]);
    }
  }
  if (a.fin != FIN_NONE) {
    double r[1] = {dot}, tot[1];
    if (grid_sum<1>(r, a.partials, a.counter, tot)) {
      if (a.extra_dot) tot[0] += *a.extra_dot;
      if (a.fin == FIN_STORE) {
        *a.out = tot[0];
      } else {
        SolverState *st = a.st;
        st->pAp = tot[0];
        if (!(tot[0] > 0.0) || !isfinite(tot[0])) {
          st->done = 2;
          st->status = 5;  // breakdown
        } else {
          st->alpha = st->rz / tot[0];
        }
      }
    }
  }
}

}  // namespace mpdg
