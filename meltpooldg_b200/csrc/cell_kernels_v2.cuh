// Register-resident cell kernel for the operator application (n = p + 1 <= 4 in FP64, <= 5 in FP32;
// the constant law on a uniform box n <= 6).
//
// Layout: every cell gets n threads of one warp (32/n cells per warp); thread t
// holds one 2D plane of the cell's n^3 tensor in registers:
//   Z-layout  thread t holds P[j][i] = u(i, j, k = t)   (x and y in registers)
//   X-layout  thread t holds Q[k][j] = u(i = t, j, k)   (y and z in registers)
// so x/y contractions run on Z-planes and y/z contractions on X-planes without
// touching shared memory. Switching layouts goes through a per-cell shared
// buffer buf[k][j][i] (plane stride n^2+1, cell stride = 4 mod 16 doubles),
// which keeps both the plane-wise writes and the strided reads free of bank
// conflicts. A cell never spans two warps, so __syncwarp is the only barrier.
//
// Operator application per cell (TDEP = temperature-dependent law):
//   T_lin: gather X, S_y S_z, copy D_z, X->Z (2 planes), S_x (2), D_y, D_x
//          -> per-point coefficients k, dk dT/dxi_d (staged in a thread-private
//             interleaved shared area: the same thread writes and reads them)
//   u:     gather X (masked), S_y S_z, copy D_z, X->Z (2), S_x (2), D_y
//   q-op:  row by row D_x, val = c u JxW, f = G (k grad u + dk u grad T), D_x^T f_x
//   integ: t = val + D_x^T f_x + D_y^T f_y, S_x^T t, S_x^T f_z, Z->X (2),
//          w = t + D_z^T f_z, S_y^T, S_z^T, atomic scatter of column t
// i.e. 21 1D sweeps and 6 layout switches per cell for k(T), 14 and 4 without.
#pragma once

#include "cell_kernels.cuh"
#include "launch.cuh"

namespace mpdg {

template <int n> __host__ __device__ constexpr int v2_cells_per_warp() { return 32 / n; }
template <int n> __host__ __device__ constexpr int v2_plane_stride() { return n * n + 1; }
template <int n> __host__ __device__ constexpr int v2_cell_stride()
{
  int s = n * v2_plane_stride<n>();
  while (s % 16 != 4) ++s;
  return s;
}
template <int LAW> __host__ __device__ constexpr int v2_ncoef()
{
  return (LAW == 1) ? 4 : (LAW == 2 ? 5 : (LAW == 8 ? 1 : 0));
}
constexpr int kV2Warps = 2;  // warps per CTA
// the instances that are launched as dependents (the FP64 iteration's)
template <typename T> __host__ __device__ constexpr bool v2_dependent() { return sizeof(T) == 8; }
// LAW 7's fields per point on register planes: k1 T_lin and k1 dT_lin/dzeta. (The line kernel reads
// four, {k(T_lin), k1 grad_ref T_lin}.) Storing all four took 1.35 ms per application on 128^3 cells
// of FE_Q(3), 5.6 GB; these two and the derivatives along the plane 1.25 ms, 3.4 GB (p = 2 0.59 ->
// 0.51 ms, p = 1 on 160^3 0.30 -> 0.25 ms).
constexpr int kTanFields2 = 2;
template <int n> __host__ __device__ constexpr bool v2_map_shared() { return n >= 4; }
template <int n, typename T, int LAW, int GEO = 0>
__host__ __device__ constexpr size_t v2_smem_per_warp()
{
  return sizeof(T) * ((size_t)2 * (v2_cells_per_warp<n>() + 1) * v2_cell_stride<n>() +
                      (size_t)v2_ncoef<LAW>() * n * n * 32 + (GEO == 2 && v2_map_shared<n>() ? 21 * 32 : 0));
}
template <int n, typename T, int LAW, int GEO = 0> __host__ __device__ constexpr size_t v2_smem()
{
  return kV2Warps * v2_smem_per_warp<n, T, LAW, GEO>();
}

// 1D contraction of matrix `kind` along the second index of A[a][b] for every a
// (B may alias A).
template <int n, int kind, bool add, typename T>
__device__ __forceinline__ void psweep_b(const T (&A)[n][n], T (&B)[n][n])
{
#pragma unroll
  for (int a = 0; a < n; ++a) {
    T x[n];
#pragma unroll
    for (int i = 0; i < n; ++i) x[i] = A[a][i];
    contract_row<n, kind, add>(x, B[a]);
  }
}

// 1D contraction along the first index of A[a][b] for every b (B may alias A).
template <int n, int kind, bool add, typename T>
__device__ __forceinline__ void psweep_a(const T (&A)[n][n], T (&B)[n][n])
{
#pragma unroll
  for (int b = 0; b < n; ++b) {
    T x[n], y[n];
#pragma unroll
    for (int i = 0; i < n; ++i) {
      x[i] = A[i][b];
      if (add) y[i] = B[i][b];
    }
    contract_row<n, kind, add>(x, y);
#pragma unroll
    for (int i = 0; i < n; ++i) B[i][b] = y[i];
  }
}

// Layout switches through the per-cell shared buffer buf[k][j][i].
// Z -> X: thread t writes plane k = t, then reads column i = t.
template <int n, typename T>
__device__ __forceinline__ void z_to_x1(const T (&A)[n][n], T (&QA)[n][n], T *ba, int t)
{
  constexpr int PS = v2_plane_stride<n>();
#pragma unroll
  for (int j = 0; j < n; ++j)
#pragma unroll
    for (int i = 0; i < n; ++i) ba[t * PS + j * n + i] = A[j][i];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < n; ++k)
#pragma unroll
    for (int j = 0; j < n; ++j) QA[k][j] = ba[k * PS + j * n + t];
  __syncwarp();
}

template <int n, typename T>
__device__ __forceinline__ void z_to_x2(const T (&A)[n][n], const T (&B)[n][n], T (&QA)[n][n],
                                        T (&QB)[n][n], T *ba, T *bb, int t)
{
  constexpr int PS = v2_plane_stride<n>();
#pragma unroll
  for (int j = 0; j < n; ++j)
#pragma unroll
    for (int i = 0; i < n; ++i) {
      ba[t * PS + j * n + i] = A[j][i];
      bb[t * PS + j * n + i] = B[j][i];
    }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < n; ++k)
#pragma unroll
    for (int j = 0; j < n; ++j) {
      QA[k][j] = ba[k * PS + j * n + t];
      QB[k][j] = bb[k * PS + j * n + t];
    }
  __syncwarp();
}

// X -> Z: thread t writes column i = t, then reads plane k = t.
template <int n, typename T>
__device__ __forceinline__ void x_to_z2(const T (&QA)[n][n], const T (&QB)[n][n], T (&A)[n][n],
                                        T (&B)[n][n], T *ba, T *bb, int t)
{
  constexpr int PS = v2_plane_stride<n>();
#pragma unroll
  for (int k = 0; k < n; ++k)
#pragma unroll
    for (int j = 0; j < n; ++j) {
      ba[k * PS + j * n + t] = QA[k][j];
      bb[k * PS + j * n + t] = QB[k][j];
    }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < n; ++j)
#pragma unroll
    for (int i = 0; i < n; ++i) {
      A[j][i] = ba[t * PS + j * n + i];
      B[j][i] = bb[t * PS + j * n + i];
    }
  __syncwarp();
}

template <int n, typename T>
__device__ __forceinline__ void x_to_z1(const T (&QA)[n][n], T (&A)[n][n], T *ba, int t)
{
  constexpr int PS = v2_plane_stride<n>();
#pragma unroll
  for (int k = 0; k < n; ++k)
#pragma unroll
    for (int j = 0; j < n; ++j) ba[k * PS + j * n + t] = QA[k][j];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < n; ++j)
#pragma unroll
    for (int i = 0; i < n; ++i) A[j][i] = ba[t * PS + j * n + i];
  __syncwarp();
}

// entry t of a table of n entries at off (the weights or points of the Gauss rule)
template <int n, typename T> __device__ __forceinline__ T cw_at(int off, int t)
{
  T w = cw<T>(off);
#pragma unroll
  for (int q = 1; q < n; ++q)
    if (t == q) w = cw<T>(off + q);
  return w;
}

// Dirichlet test of the DoFs of plane K of cell (I0, J0): face flags per row, the
// x faces only at i = 0 and i = n - 1.
struct PlaneMask {
  bool plane, xlo, xhi, ylo, yhi;
  __device__ __forceinline__ PlaneMask(const MeshDims &d, int I0, int J0, int K, int p)
  {
    plane = ((d.dmask & 16) && K == 0) || ((d.dmask & 32) && K == d.nd[2] - 1);
    xlo = (d.dmask & 1) && I0 == 0;
    xhi = (d.dmask & 2) && I0 + p == d.nd[0] - 1;
    ylo = (d.dmask & 4) && J0 == 0;
    yhi = (d.dmask & 8) && J0 + p == d.nd[1] - 1;
  }
  template <int n>
  __device__ __forceinline__ bool at(int i, int j) const
  {
    return plane || (j == 0 && ylo) || (j == n - 1 && yhi) || (i == 0 && xlo) ||
           (i == n - 1 && xhi);
  }
};

// L2 prefetch of the n rows (n values each) of plane K of a cell
template <int n, typename T>
__device__ __forceinline__ void prefetch_plane(const T *g, int64_t base, int nd0)
{
#pragma unroll
  for (int j = 0; j < n; ++j) {
    const T *row = g + base + (int64_t)nd0 * j;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(row));
    if ((reinterpret_cast<uintptr_t>(row) & 127) + n * sizeof(T) > 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(row + n - 1));
  }
}

// A thread's row of n consecutive per-point values (row j of its quadrature plane): one 16- or
// 32-byte load where n is even (the cells' blocks are then multiples of the load's size).
template <int n, typename T>
__device__ __forceinline__ void load_row(const T *__restrict__ p, T (&r)[n])
{
  if constexpr (n == 4 && sizeof(T) == 8) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(r[0]), "=d"(r[1]), "=d"(r[2]), "=d"(r[3]) : "l"(p));
  } else if constexpr (n == 4) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
    r[0] = v.x;
    r[1] = v.y;
    r[2] = v.z;
    r[3] = v.w;
  } else if constexpr (n == 2 && sizeof(T) == 8) {
    const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
    r[0] = v.x;
    r[1] = v.y;
  } else if constexpr (n == 2) {
    const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
    r[0] = v.x;
    r[1] = v.y;
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) r[i] = __ldg(p + i);
  }
}

// Dirichlet test of the DoFs of an x-column (I fixed, y and z in registers) of a cell
struct ColumnMask {
  bool col, ylo, yhi, zlo, zhi;
  __device__ __forceinline__ ColumnMask(const MeshDims &d, int I, int J0, int K0, int p)
  {
    col = ((d.dmask & 1) && I == 0) || ((d.dmask & 2) && I == d.nd[0] - 1);
    ylo = (d.dmask & 4) && J0 == 0;
    yhi = (d.dmask & 8) && J0 + p == d.nd[1] - 1;
    zlo = (d.dmask & 16) && K0 == 0;
    zhi = (d.dmask & 32) && K0 + p == d.nd[2] - 1;
  }
  template <int n>
  __device__ __forceinline__ bool at(int j, int k) const
  {
    return col || (j == 0 && ylo) || (j == n - 1 && yhi) || (k == 0 && zlo) ||
           (k == n - 1 && zhi);
  }
  __device__ __forceinline__ bool any() const { return col || ylo || yhi || zlo || zhi; }
};

// gather a cell's x-column at base (X-layout Q[k][j]); rs, ps: strides of a row and of a plane
template <int n, typename T>
__device__ __forceinline__ void gather_column(const T *__restrict__ g, int64_t base, int64_t rs,
                                              int64_t ps, T (&Q)[n][n], bool active)
{
  const T *p = g + base;
#pragma unroll
  for (int k = 0; k < n; ++k)
#pragma unroll
    for (int j = 0; j < n; ++j) Q[k][j] = active ? __ldg(p + (rs * j + ps * k)) : T(0);
}
// the same of a vector that the predecessor of a dependent launch writes
template <int n>
__device__ __forceinline__ void gather_live(const double *g, int64_t base, int64_t rs, int64_t ps,
                                            double (&Q)[n][n], bool active)
{
  const double *p = g + base;
#pragma unroll
  for (int k = 0; k < n; ++k)
#pragma unroll
    for (int j = 0; j < n; ++j) Q[k][j] = active ? load_live(p + (rs * j + ps * k)) : 0.0;
}
template <int n, typename T>
__device__ __forceinline__ void mask_column(const ColumnMask &cm, T (&Q)[n][n])
{
  if (cm.any()) {
#pragma unroll
    for (int k = 0; k < n; ++k)
#pragma unroll
      for (int j = 0; j < n; ++j)
        if (cm.template at<n>(j, k)) Q[k][j] = T(0);
  }
}

// Geometry of a deformed mesh in the operator kernel: 1 the stored factors (7 per point), 2 the
// trilinear map of the cell's 8 vertices evaluated at the points. In FP64 from p = 2 on the
// evaluation (~55 operations a point, on FP64 units that the loads leave idle) is shorter than
// reading 56 bytes a point: constant law p = 2 on 96^3 cells 0.36 -> 0.29 ms, p = 3 on 133^3 cells
// 2.40 -> 1.87 ms, k(T) tangent p = 3 on 64^3 cells 0.54 -> 0.31 ms; at p = 1 a cell has as many
// vertices as nodes and it is not (0.36 -> 0.40 ms on 160^3), and the liquid-solid law at p = 3 has
// no registers left for it (40^3 cells 183 us stored, 209 us evaluated). FP32 keeps the stored
// factors, which are rounded from FP64 ones.
template <int n, typename T, int GEO, int LAW> constexpr int v2_geometry()
{
  return GEO == 1 && sizeof(T) == 8 && n >= 3 && !(n == 4 && LAW == 2) ? 2 : GEO;
}

// The trilinear map of a cell on the plane zeta = const of its unit cube,
// dx/dxi = A + B eta, dx/deta = C + B xi, dx/dzeta = (D + F eta) + (E + H eta) xi: 21 values
// (entry e of vector f at (3 f + e) * stride). At n = 4 they are kept in thread-private shared
// columns, where in registers they spill (constant law on 133^3 cells 1.87 against 2.04 ms); at
// n = 3 in registers (0.29 against 0.34 ms on 96^3 cells).
enum { kMapA, kMapB, kMapC, kMapD, kMapE, kMapF, kMapH };
template <typename T>
__device__ __forceinline__ void load_map(const MeshDims &d, const double *__restrict__ vert, int cx,
                                         int cy, int cz, T zeta, T *map, int stride)
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
    map[(3 * kMapA + e) * stride] = fma(exz, zeta, ex);
    map[(3 * kMapB + e) * stride] = fma(exyz, zeta, exy);
    map[(3 * kMapC + e) * stride] = fma(eyz, zeta, ey);
    map[(3 * kMapD + e) * stride] = x4 - x0;
    map[(3 * kMapE + e) * stride] = exz;
    map[(3 * kMapF + e) * stride] = eyz;
    map[(3 * kMapH + e) * stride] = exyz;
  }
}
// Blocks per SM that the register allocator is held to. Without a bound it hoists the row loads
// and the scatter's addresses until half as many warps fit (FP32 Picard p = 3: 195 registers, 8
// warps, 0.96 ms against 0.52 ms with 128 registers, 16 warps, on 128^3 cells); a tighter bound
// spills (0.56 ms at 20 warps; the FP64 k(T) tangent 1.71 ms at 12 warps, 1.36 ms at 8). Laws and
// geometries that load per-point rows want more registers for the loads in flight (FP32 p = 3
// deformed constant law on 96^3 cells: 0.36 ms at 12 warps, 0.40 ms at 16).
template <int n, typename T, int GEO, int LAW> constexpr int v2_min_blocks()
{
  constexpr bool rows = GEO != 0 || (LAW != 0 && LAW != 3);
  if (sizeof(T) == 4)
    return n == 2 ? (GEO == 1 ? 12 : 10) : n == 3 ? 8 : n == 4 ? (rows ? 6 : 8) : (rows ? 4 : 6);
  return n == 2 ? 8 : n == 3 ? (GEO != 0 ? 4 : 6) : 4;
}

// Work split: the gather and the scatter run on x-columns (thread t = x node t of its cell), so a
// warp's 32 lanes read 32 / n neighbouring cells' x-rows as one contiguous run of nodes; the
// quadrature points run on z-planes (thread t = the n^2 points of plane t), so a thread's
// per-point data are contiguous and come in 16- and 32-byte loads. The x-derivative and its
// transpose stay within a row, so they are formed row by row inside the quadrature loop and only
// three planes (value, d/dy, d/dz) are live there.
// ROWS (FP32 Picard operator at p = 3): the operand is in the cell-row layout, in which the n = 4
// nodes of a cell's x-row are one aligned float4 and a node shared by x-neighbours is stored in
// both cells' rows (cell_row_index below): a warp's 8 cells are then one aligned 128-byte line.
// The result is scattered into the lexicographic dst as usual; no src.dst partial (the host
// passes FIN_NONE).
template <int n, typename T, int GEO, int LAW, bool ROWS = false>
__global__ void __launch_bounds__(32 * kV2Warps, (v2_min_blocks<n, T, GEO, LAW>()))
  k_vmult2(CellArgs<T> a)
{
  static_assert(!ROWS || (n == 4 && sizeof(T) == 4 && LAW == 3), "cell rows: FP32 Picard, p = 3");
  constexpr int CW = v2_cells_per_warp<n>();
  constexpr int CS = v2_cell_stride<n>();
  constexpr int npt = n * n * n;
  // LAW 3: conductivity field k(q), no tangent; LAW 4: coefficient fields a.cf; LAW 6: the
  // tangent coefficient fields of LAW 5 built at the linearisation point (8 per point); LAW 8:
  // the Picard operator of the linear-k law with k(T_lin(q)) interpolated from the gathered
  // T_lin (k is affine in T, so this is the conductivity field of LAW 3 without storing it)
  constexpr bool TDEP = LAW == 1 || LAW == 2;
  constexpr bool TLIN = TDEP || LAW == 8;
  dependents_may_start();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = lane / n, t = lane % n;
  const bool lane_ok = cw < CW;
  T *wbuf = reinterpret_cast<T *>(smem_raw) + (size_t)warp * (v2_smem_per_warp<n, T, LAW, GEO>() / sizeof(T));
  T *bufA = wbuf + cw * CS;                     // idle lanes use the spare slot cw == CW
  T *bufB = wbuf + (CW + 1) * CS + cw * CS;
  T *coef = wbuf + 2 * (CW + 1) * CS;           // [NCOEF][n*n][32], thread-private columns
  T *map_s = coef + v2_ncoef<LAW>() * n * n * 32 + lane;  // GEO 2: [21][32]
  T map_r[GEO == 2 && !v2_map_shared<n>() ? 21 : 1];
  auto map = [&](int f, int e) -> T {  // (volatile: read where it is used, not kept in registers)
    if constexpr (v2_map_shared<n>())
      return reinterpret_cast<const volatile T *>(map_s)[(3 * f + e) * 32];
    else
      return map_r[3 * f + e];
  };
  const MeshDims &d = a.d;
  const int64_t rs = d.nd[0], ps = (int64_t)d.nd[0] * d.nd[1];
  const T wt = cw_at<n, T>(w_off(n), t), zt = cw_at<n, T>(xg_off(n), t);
  double dot = 0.0;
  const int64_t stride = (int64_t)gridDim.x * kV2Warps * CW;
  const int64_t first = ((int64_t)blockIdx.x * kV2Warps + warp) * CW;  // the warp's first cell
  CellWalk at(d, first + cw, stride, a.n_cells);
  wait_for_predecessor();
  if (a.st && a.st->done) return;
  for (int64_t head = first; head < a.n_cells; head += stride) {
    const int64_t cell = head + cw;
    const bool active = lane_ok && cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    // inactive lanes' addresses are not read
    const int cx = at.x, cy = at.y, cz = at.z, I = d.p * cx + t, J0 = d.p * cy, K0 = d.p * cz;
    const int64_t base = I + rs * J0 + ps * K0;
    at.advance(d);
    const ColumnMask cm(d, I, J0, K0, d.p);

    // both gathers first so their latencies overlap
    T Q[n][n];
    if constexpr (ROWS) {
      const int64_t crs = 4 * (int64_t)d.m[0];
      gather_column<n>(a.src, 4 * cx + t + crs * (J0 + (int64_t)d.nd[1] * K0), crs,
                       crs * d.nd[1], Q, active);
    } else if constexpr (v2_dependent<T>()) {
      gather_live<n>(a.src, base, rs, ps, Q, active);
    } else {
      gather_column<n>(a.src, base, rs, ps, Q, active);
    }
    T Qt[n][n];
    if (TLIN) gather_column<n>(a.Tl, base, rs, ps, Qt, active);
    if constexpr (GEO == 2)  // (inactive lanes: cell 0)
      load_map(d, a.g.vert, active ? cx : 0, active ? cy : 0, active ? cz : 0, zt,
               v2_map_shared<n>() ? map_s : map_r, v2_map_shared<n>() ? 32 : 1);
    mask_column<n>(cm, Q);

    // L2 prefetch of the next group's rows (and per-point data) while this one computes
    {
      const int64_t ncell = cell + stride;
      if (lane_ok && ncell < a.n_cells) {
        const int64_t nbase = rs * (d.p * at.y) + ps * (d.p * at.z + t) + d.p * at.x;
        // (cell rows: measured faster without the operand's and the conductivity's prefetch)
        if (!ROWS) prefetch_plane<n>(a.src, nbase, d.nd[0]);
        if (TLIN) prefetch_plane<n>(a.Tl, nbase, d.nd[0]);
        if (LAW == 3 && !ROWS) {
          const char *kq = reinterpret_cast<const char *>(a.kq + ncell * npt);
          for (int off = t * 128; off < npt * 4; off += n * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(kq + off));
        }
        if (LAW == 4 || LAW == 6 || LAW == 7) {
          constexpr int nf = LAW == 4 ? 5 : (LAW == 6 ? 8 : kTanFields2);
          constexpr int bytes = nf * npt * (int)sizeof(T);
          const char *cf = reinterpret_cast<const char *>(a.cf + ncell * nf * npt);
          for (int off = t * 128; off < bytes; off += n * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(cf + off));
        }
        if (GEO == 1) {
          const char *gq = reinterpret_cast<const char *>(a.g.q + ncell * 7 * npt);
          constexpr int bytes = 7 * npt * (int)sizeof(T);
          for (int off = t * 128; off < bytes; off += n * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(gq + off));
        }
      }
    }

    if (LAW == 8) {
      // ---- linearisation point: values at the q-points -> k(T_lin) (thread-private columns)
      psweep_b<n, kS, false>(Qt, Qt);
      psweep_a<n, kS, false>(Qt, Qt);
      T Tq[n][n];
      x_to_z1<n>(Qt, Tq, bufA, t);
      psweep_b<n, kS, false>(Tq, Tq);
#pragma unroll
      for (int j = 0; j < n; ++j)
#pragma unroll
        for (int i = 0; i < n; ++i) {
          T rhocp, kk, drhocp, dk;
          mat_eval<1>(a.m, Tq[j][i], rhocp, kk, drhocp, dk);
          coef[(j * n + i) * 32 + lane] = kk;
        }
    }
    if (TDEP) {
      // ---- linearisation point: values and reference gradients at the q-points
      T Dz[n][n];
      psweep_b<n, kS, false>(Qt, Qt);
      psweep_a<n, kS, false>(Qt, Qt);
      psweep_a<n, kD, false>(Qt, Dz);
      T Tq[n][n], Tz[n][n];
      x_to_z2<n>(Qt, Dz, Tq, Tz, bufA, bufB, t);
      psweep_b<n, kS, false>(Tq, Tq);
      psweep_b<n, kS, false>(Tz, Tz);
      T Ty[n][n], Tx[n][n];
      psweep_a<n, kD, false>(Tq, Ty);
      psweep_b<n, kD, false>(Tq, Tx);
      T To[n][n];
      if (LAW == 2 && a.m.need_told) {
        gather_column<n>(a.To, base, rs, ps, Qt, active);
        psweep_b<n, kS, false>(Qt, Qt);
        psweep_a<n, kS, false>(Qt, Qt);
        x_to_z1<n>(Qt, To, bufA, t);
        psweep_b<n, kS, false>(To, To);
      }
#pragma unroll
      for (int j = 0; j < n; ++j)
#pragma unroll
        for (int i = 0; i < n; ++i) {
          T rhocp, kk, drhocp, dk;
          mat_eval<LAW>(a.m, Tq[j][i], rhocp, kk, drhocp, dk);
          const int pt = j * n + i;
          coef[(0 * n * n + pt) * 32 + lane] = kk;
          coef[(1 * n * n + pt) * 32 + lane] = dk * Tx[j][i];
          coef[(2 * n * n + pt) * 32 + lane] = dk * Ty[j][i];
          coef[(3 * n * n + pt) * 32 + lane] = dk * Tz[j][i];
          if (LAW == 2) {
            T c = a.m.idt * rhocp;
            if (a.m.need_told) c += a.m.idt * drhocp * (Tq[j][i] - To[j][i]);
            coef[(4 * n * n + pt) * 32 + lane] = c;
          }
        }
    }

    // ---- operand: values and reference gradients at the q-points
    T U[n][n], Uz[n][n];
    {
      T Dz[n][n];
      psweep_b<n, kS, false>(Q, Q);
      psweep_a<n, kS, false>(Q, Q);
      psweep_a<n, kD, false>(Q, Dz);
      x_to_z2<n>(Q, Dz, U, Uz, bufA, bufB, t);
    }
    psweep_b<n, kS, false>(U, U);
    psweep_b<n, kS, false>(Uz, Uz);
    T Uy[n][n];
    psweep_a<n, kD, false>(U, Uy);

    T t0[LAW == 7 ? n : 1][LAW == 7 ? n : 1];  // LAW 7: k1 T_lin on the plane
    if constexpr (LAW == 7) {
#pragma unroll
      for (int j = 0; j < n; ++j)
        load_row<n>(a.cf + cc * kTanFields2 * npt + t * (n * n) + n * j, t0[j]);
    }

    // ---- quadrature-point operation (tangent_local_cell_operation), row by row: row j of U
    // turns into val + D_x^T f_x, those of Uy and Uz into f_y and f_z
#pragma unroll
    for (int j = 0; j < n; ++j) {
      T Ux[n];
      contract_row<n, kD, false>(U[j], Ux);
      const int64_t q0 = t * (n * n) + n * j;  // first point of the row within the cell
      T jxw[n], G[6][n];
      if constexpr (GEO == 0) {
        const T wjt = wt * mpdg::cw<T>(w_off(n) + j);
#pragma unroll
        for (int i = 0; i < n; ++i) {
          const T w = wjt * mpdg::cw<T>(w_off(n) + i);
          jxw[i] = a.g.detJ * w;
          G[0][i] = a.g.Gd[0] * w;
          G[3][i] = a.g.Gd[1] * w;
          G[5][i] = a.g.Gd[2] * w;
          G[1][i] = G[2][i] = G[4][i] = T(0);
        }
      } else if constexpr (GEO == 1) {
        const T *gb = a.g.q + cc * 7 * npt + q0;
        load_row<n>(gb, jxw);
#pragma unroll
        for (int f = 0; f < 6; ++f) load_row<n>(gb + (1 + f) * npt, G[f]);
      }
      // coefficient rows of the field laws
      constexpr int NC = LAW == 4 ? 5 : (LAW == 6 ? 8 : (LAW == 7 ? 4 : 1));
      T c[NC][n];
      if constexpr (LAW == 7) {
        // k1 T_lin of the row (c[0]) and its gradient: d/dx within the row, d/dy down the plane
        contract_row<n, kD, false>(t0[j], c[1]);
#pragma unroll
        for (int i = 0; i < n; ++i) {
          constexpr int full = tab_off(n, kD) + tab_full(n);
          c[0][i] = a.m.k_l + t0[j][i];
          c[2][i] = ctab<T>(full + j * n) * t0[0][i];
#pragma unroll
          for (int l = 1; l < n; ++l) c[2][i] = fma(ctab<T>(full + j * n + l), t0[l][i], c[2][i]);
        }
        load_row<n>(a.cf + (cc * kTanFields2 + 1) * npt + q0, c[3]);
      } else if constexpr (LAW == 4 || LAW == 6) {
        const T *cf = a.cf + cc * NC * npt + q0;
#pragma unroll
        for (int f = 0; f < NC; ++f) load_row<n>(cf + f * npt, c[f]);
      } else if constexpr (LAW == 3) {
        float kr[n];
        load_row<n>(a.kq + cc * npt + q0, kr);
#pragma unroll
        for (int i = 0; i < n; ++i) c[0][i] = (T)kr[i];
      }
      // GEO 2: the map's dx/dxi of the row and the two parts of dx/dzeta
      T Jx[3], Jz0[3], Jz1[3];
      const T wj = wt * mpdg::cw<T>(w_off(n) + j);
      if constexpr (GEO == 2) {
        const T eta = mpdg::cw<T>(xg_off(n) + j);
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          Jx[e] = fma(map(kMapB, e), eta, map(kMapA, e));
          Jz0[e] = fma(map(kMapF, e), eta, map(kMapD, e));
          Jz1[e] = fma(map(kMapH, e), eta, map(kMapE, e));
        }
      }
      T fx[n];
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const T uu = U[j][i], ux = Ux[i], uy = Uy[j][i], uz = Uz[j][i];
        T c0[3], c1[3], c2[3], s;  // GEO 2: cofactor columns, JxW G = s c_a.c_b
        if constexpr (GEO == 2) {
          const T xi = mpdg::cw<T>(xg_off(n) + i);
          T Jy[3], Jz[3];
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            Jy[e] = fma(map(kMapB, e), xi, map(kMapC, e));
            Jz[e] = fma(Jz1[e], xi, Jz0[e]);
          }
          cross(Jy, Jz, c0);
          cross(Jz, Jx, c1);
          cross(Jx, Jy, c2);
          const T det = Jx[0] * c0[0] + Jx[1] * c0[1] + Jx[2] * c0[2];
          const T w = wj * mpdg::cw<T>(w_off(n) + i);
          jxw[i] = w * det;
          s = w / det;
        }
        T f0, f1, f2, val;
        if constexpr (LAW == 4) {
          // rho_cp u / dt + rho_cp v.grad(u), and the flux k grad(u), from the fields
          val = a.m.idt * c[0][i] * uu + c[2][i] * ux + c[3][i] * uy + c[4][i] * uz;
          f0 = c[1][i] * ux;
          f1 = c[1][i] * uy;
          f2 = c[1][i] * uz;
        } else if constexpr (LAW == 6) {
          // c u + rho_cp b.grad(u), flux k grad(u) + dk grad(T_lin) u
          val = c[0][i] * uu + c[2][i] * ux + c[3][i] * uy + c[4][i] * uz;
          f0 = c[1][i] * ux + c[5][i] * uu;
          f1 = c[1][i] * uy + c[6][i] * uu;
          f2 = c[1][i] * uz + c[7][i] * uu;
        } else if constexpr (LAW == 7) {
          // linear-k tangent from its fields: flux k(T_lin) grad(u) + k1 grad(T_lin) u
          f0 = c[0][i] * ux + c[1][i] * uu;
          f1 = c[0][i] * uy + c[2][i] * uu;
          f2 = c[0][i] * uz + c[3][i] * uu;
          val = a.m.idt * (a.m.rho_l * a.m.cp_l) * uu * jxw[i];
        } else if constexpr (TDEP) {
          const int pt = j * n + i;
          const T kk = coef[(0 * n * n + pt) * 32 + lane];
          f0 = kk * ux + coef[(1 * n * n + pt) * 32 + lane] * uu;
          f1 = kk * uy + coef[(2 * n * n + pt) * 32 + lane] * uu;
          f2 = kk * uz + coef[(3 * n * n + pt) * 32 + lane] * uu;
          const T cval =
            LAW == 2 ? coef[(4 * n * n + pt) * 32 + lane] : a.m.idt * (a.m.rho_l * a.m.cp_l);
          val = cval * uu * jxw[i];
        } else {
          const T kk = LAW == 3 ? c[0][i] : (LAW == 8 ? coef[(j * n + i) * 32 + lane] : a.m.k_l);
          f0 = kk * ux;
          f1 = kk * uy;
          f2 = kk * uz;
          val = a.m.idt * (a.m.rho_l * a.m.cp_l) * uu * jxw[i];
        }
        if constexpr (GEO == 2) {
          T v[3];
#pragma unroll
          for (int e = 0; e < 3; ++e) v[e] = s * (c0[e] * f0 + c1[e] * f1 + c2[e] * f2);
          fx[i] = c0[0] * v[0] + c0[1] * v[1] + c0[2] * v[2];
          Uy[j][i] = c1[0] * v[0] + c1[1] * v[1] + c1[2] * v[2];
          Uz[j][i] = c2[0] * v[0] + c2[1] * v[1] + c2[2] * v[2];
        } else {
          const T Gi[6] = {G[0][i], G[1][i], G[2][i], G[3][i], G[4][i], G[5][i]};
          apply_G<GEO>(Gi, f0, f1, f2, fx[i], Uy[j][i], Uz[j][i]);
        }
        U[j][i] = val;
      }
      contract_row<n, kDT, true>(fx, U[j]);
    }

    // ---- integration
    psweep_a<n, kDT, true>(Uy, U);
    psweep_b<n, kST, false>(U, U);
    psweep_b<n, kST, false>(Uz, Uz);
    T Wz[n][n];
    z_to_x2<n>(U, Uz, Q, Wz, bufA, bufB, t);
    psweep_a<n, kDT, true>(Wz, Q);
    psweep_b<n, kST, false>(Q, Q);
    psweep_a<n, kST, false>(Q, Q);

    // ---- optional src.dst partial and the scatter (constrained rows skipped)
    if (!ROWS && a.fin != FIN_NONE && active) {
      T u[n][n];
      if constexpr (v2_dependent<T>())
        gather_live<n>(a.src, base, rs, ps, u, true);
      else
        gather_column<n>(a.src, base, rs, ps, u, true);
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j) {
          dot += cm.template at<n>(j, k) ? 0.0 : (double)u[k][j] * (double)Q[k][j];
        }
    }
    bool mine = active;
    if constexpr (n == 3) {
      // the last column of a cell and the first of its x-neighbour, the next lane, are the same
      // nodes: one lane adds both. At n = 3 that saves a third of the atomics (deformed FP32 on
      // 96^3 cells 0.207 against 0.213 ms); at n = 2, 4 the shuffles cost as much as they save.
      const int next_x = __shfl_down_sync(0xffffffffu, active ? cx : -1, 1);
      const bool join = active && t == n - 1 && next_x == cx + 1;
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j) {
          const T other = __shfl_down_sync(0xffffffffu, Q[k][j], 1);
          if (join) Q[k][j] += other;
        }
      mine = active && !(t == 0 && cw > 0 && cx > 0);
    }
    if (mine) {
      T *out = a.dst + base;
      if (!cm.any()) {
#pragma unroll
        for (int k = 0; k < n; ++k)
#pragma unroll
          for (int j = 0; j < n; ++j) atomic_add(out + (rs * j + ps * k), Q[k][j]);
      } else {
#pragma unroll
        for (int k = 0; k < n; ++k)
#pragma unroll
          for (int j = 0; j < n; ++j) {
            if (!cm.template at<n>(j, k)) atomic_add(out + (rs * j + ps * k), Q[k][j]);
          }
      }
    }
  }
  if (a.fin != FIN_NONE) {
    double v[1] = {dot}, tot[1];
    if (grid_sum<1>(v, a.partials, a.counter, tot)) {
      if (a.extra_dot) tot[0] += *a.extra_dot;
      if (a.fin == FIN_STORE) {
        *a.out = tot[0];
      } else {
        SolverState *s = a.st;
        s->pAp = tot[0];
        if (!(tot[0] > 0.0) || !isfinite(tot[0])) {
          s->done = 2;
          s->status = 5;
        } else {
          s->alpha = s->rz / tot[0];
        }
      }
    }
  }
}

// Conductivity at the quadrature points, kq[cell][q] = k(T_lin(x_q)) in FP32,
// for the coefficient-field (Picard) operator of the FP32 preconditioner.
template <int n, int LAW>
__global__ void __launch_bounds__(32 * kV2Warps) k_conductivity_q(CellArgs<double> a, float *kq)
{
  using T = double;
  constexpr int CW = v2_cells_per_warp<n>();
  constexpr int CS = v2_cell_stride<n>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = lane / n, t = lane % n;
  const bool lane_ok = cw < CW;
  T *bufA = reinterpret_cast<T *>(smem_raw) + (size_t)warp * (CW + 1) * CS + cw * CS;
  const MeshDims &d = a.d;
  const int64_t rs = d.nd[0], ps = (int64_t)d.nd[0] * d.nd[1];
  const int64_t stride = (int64_t)gridDim.x * kV2Warps * CW;
  const int64_t first = ((int64_t)blockIdx.x * kV2Warps + warp) * CW;  // the warp's first cell
  CellWalk at(d, first + cw, stride, a.n_cells);
  for (int64_t head = first; head < a.n_cells; head += stride) {
    const int64_t cell = head + cw;
    const bool active = lane_ok && cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    const int I = d.p * at.x + t, J0 = d.p * at.y, K0 = d.p * at.z;
    const int64_t base = I + rs * J0 + ps * K0;
    at.advance(d);
    T Q[n][n], P[n][n];
    gather_column<n>(a.Tl, base, rs, ps, Q, active);
    psweep_b<n, kS, false>(Q, Q);
    psweep_a<n, kS, false>(Q, Q);
    x_to_z1<n>(Q, P, bufA, t);
    psweep_b<n, kS, false>(P, P);
    if (active) {
      float *out = kq + cc * (n * n * n) + t * (n * n);
#pragma unroll
      for (int j = 0; j < n; ++j) {
        float r[n];
#pragma unroll
        for (int i = 0; i < n; ++i) {
          T rhocp, kk, drhocp, dk;
          mat_eval<LAW>(a.m, P[j][i], rhocp, kk, drhocp, dk);
          r[i] = (float)kk;
        }
        if constexpr (n == 4) {
          *reinterpret_cast<float4 *>(out + n * j) = make_float4(r[0], r[1], r[2], r[3]);
        } else {
#pragma unroll
          for (int i = 0; i < n; ++i) out[n * j + i] = r[i];
        }
      }
    }
  }
}

// Diagonal of the FP32 Picard operator (conductivity field kq at the q-points, no
// dk/dT term): diag_i = sum_q c JxW phi_i^2 + grad phi_i^T (kq G) grad phi_i, sum-
// factorised with the element-wise products P = S o S, Q = D o D, R = S o D of the 1D
// value and collocation-derivative matrices (transposed tables kPT, kQT, kRT):
// contraction along x and y on the quadrature planes, along z on the node columns.
//   A_PP = P_x C0 + Q_x Gxx   A_PQ = P_x Gyy   A_QP = P_x Gzz
//   Y_P = P_y A_PP + Q_y A_PQ   Y_Q = P_y A_QP   W = P_z Y_P + Q_z Y_Q
// plus on deformed cells the cross terms (2 kq Gxy ... in R products):
//   A_PR = R_x Gxy  A_RR = P_x Gyz  A_RP = R_x Gxz
//   Y_P += R_y A_PR   Y_R = R_y A_RR + P_y A_RP   W += R_z Y_R
// a.dst (FP32) accumulates; Dirichlet rows are skipped.
template <int n, int GEO>
__global__ void __launch_bounds__(32 * kV2Warps) k_diag_picard(CellArgs<float> a)
{
  using T = float;
  constexpr int CW = v2_cells_per_warp<n>();
  constexpr int CS = v2_cell_stride<n>();
  constexpr int npt = n * n * n;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = lane / n, t = lane % n;
  const bool lane_ok = cw < CW;
  T *wbuf = reinterpret_cast<T *>(smem_raw) + (size_t)warp * 2 * (CW + 1) * CS;
  T *bufA = wbuf + cw * CS;
  T *bufB = wbuf + (CW + 1) * CS + cw * CS;
  const T cval = a.m.idt * (a.m.rho_l * a.m.cp_l);
  const MeshDims &d = a.d;
  const int64_t rs = d.nd[0], ps = (int64_t)d.nd[0] * d.nd[1];
  const int64_t stride = (int64_t)gridDim.x * kV2Warps * CW;
  const int64_t first = ((int64_t)blockIdx.x * kV2Warps + warp) * CW;  // the warp's first cell
  CellWalk at(d, first + cw, stride, a.n_cells);
  for (int64_t head = first; head < a.n_cells; head += stride) {
    const int64_t cell = head + cw;
    const bool active = lane_ok && cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    const int I = d.p * at.x + t, J0 = d.p * at.y, K0 = d.p * at.z;
    const int64_t base = I + rs * J0 + ps * K0;
    at.advance(d);
    const ColumnMask cm(d, I, J0, K0, d.p);
    const T *gq = GEO == 1 ? a.g.q + cc * 7 * npt + t * n * n : nullptr;
    // q-point coefficients on the planes: thread t = q_z, registers [q_y][q_x]
    T APP[n][n], APQ[n][n], AQP[n][n], K[n][n];
    {
      T C0[n][n], Gxx[n][n], Gyy[n][n], Gzz[n][n];
#pragma unroll
      for (int j = 0; j < n; ++j) {
        load_row<n>(a.kq + cc * npt + t * n * n + n * j, K[j]);
        if constexpr (GEO == 1) {
          load_row<n>(gq + n * j, C0[j]);
          load_row<n>(gq + npt + n * j, Gxx[j]);
          load_row<n>(gq + 4 * npt + n * j, Gyy[j]);
          load_row<n>(gq + 6 * npt + n * j, Gzz[j]);
        }
#pragma unroll
        for (int i = 0; i < n; ++i) {
          if constexpr (GEO == 0) {
            T G[6];
            geo_at<n, GEO>(a.g, cc, i, j, t, C0[j][i], G);
            Gxx[j][i] = G[0];
            Gyy[j][i] = G[3];
            Gzz[j][i] = G[5];
          }
          C0[j][i] *= cval;
          Gxx[j][i] *= K[j][i];
          Gyy[j][i] *= K[j][i];
          Gzz[j][i] *= K[j][i];
        }
      }
      psweep_b<n, kPT, false>(C0, APP);
      psweep_b<n, kQT, true>(Gxx, APP);
      psweep_b<n, kPT, false>(Gyy, APQ);
      psweep_b<n, kPT, false>(Gzz, AQP);
    }
    T YP[n][n], YQ[n][n];
    psweep_a<n, kPT, false>(APP, YP);
    psweep_a<n, kQT, true>(APQ, YP);
    psweep_a<n, kPT, false>(AQP, YQ);
    T YR[n][n];
    if constexpr (GEO == 1) {
      T Gxy[n][n], Gxz[n][n], Gyz[n][n];
#pragma unroll
      for (int j = 0; j < n; ++j) {
        load_row<n>(gq + 2 * npt + n * j, Gxy[j]);
        load_row<n>(gq + 3 * npt + n * j, Gxz[j]);
        load_row<n>(gq + 5 * npt + n * j, Gyz[j]);
#pragma unroll
        for (int i = 0; i < n; ++i) {
          Gxy[j][i] *= T(2) * K[j][i];
          Gxz[j][i] *= T(2) * K[j][i];
          Gyz[j][i] *= T(2) * K[j][i];
        }
      }
      T A1[n][n], A2[n][n];
      psweep_b<n, kRT, false>(Gxy, A1);  // A_PR
      psweep_a<n, kRT, true>(A1, YP);
      psweep_b<n, kPT, false>(Gyz, A1);  // A_RR
      psweep_b<n, kRT, false>(Gxz, A2);  // A_RP
      psweep_a<n, kRT, false>(A1, YR);
      psweep_a<n, kPT, true>(A2, YR);
    }
    T XP[n][n], XQ[n][n];
    z_to_x2<n>(YP, YQ, XP, XQ, bufA, bufB, t);
    T W[n][n];
    psweep_a<n, kPT, false>(XP, W);
    psweep_a<n, kQT, true>(XQ, W);
    if constexpr (GEO == 1) {
      z_to_x1<n>(YR, XP, bufA, t);
      psweep_a<n, kRT, true>(XP, W);
    }
    if (active) {
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j)
          if (!cm.template at<n>(j, k)) atomicAdd(a.dst + base + (rs * j + ps * k), W[k][j]);
    }
  }
}

// a row of n values to global memory (as load_row reads it)
template <int n>
__device__ __forceinline__ void store_row(double *p, const double (&r)[n])
{
  if constexpr (n == 4) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(r[0]), "d"(r[1]),
                 "d"(r[2]), "d"(r[3])
                 : "memory");
  } else if constexpr (n == 2) {
    *reinterpret_cast<double2 *>(p) = make_double2(r[0], r[1]);
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) p[i] = r[i];
  }
}

// Tangent fields of the linear-k law at the linearisation point, built once per linearisation for
// LAW 7: out[cell][2][n^3] = {k1 T_lin, k1 dT_lin/dzeta} (k_vmult2 forms the other two derivatives
// on its planes). On the planes of k_vmult2 with 32-byte stores (128^3 cells of FE_Q(3): four
// fields on lines through shared memory 1.59 ms, on planes 1.14 ms, these two 0.63 ms).
template <int n>
__global__ void __launch_bounds__(32 * kV2Warps, 4) k_coef_lineark2(CellArgs<double> a, double *out)
{
  using T = double;
  constexpr int CW = v2_cells_per_warp<n>(), CS = v2_cell_stride<n>(), npt = n * n * n;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = lane / n, t = lane % n;
  const bool lane_ok = cw < CW;
  T *wbuf = reinterpret_cast<T *>(smem_raw) + (size_t)warp * 2 * (CW + 1) * CS;
  T *bufA = wbuf + cw * CS, *bufB = wbuf + (CW + 1) * CS + cw * CS;
  const MeshDims &d = a.d;
  const int64_t rs = d.nd[0], ps = (int64_t)d.nd[0] * d.nd[1];
  const int64_t stride = (int64_t)gridDim.x * kV2Warps * CW;
  const int64_t first = ((int64_t)blockIdx.x * kV2Warps + warp) * CW;  // the warp's first cell
  CellWalk at(d, first + cw, stride, a.n_cells);
  for (int64_t head = first; head < a.n_cells; head += stride) {
    const int64_t cell = head + cw;
    const bool active = lane_ok && cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    const int I = d.p * at.x + t, J0 = d.p * at.y, K0 = d.p * at.z;
    const int64_t base = I + rs * J0 + ps * K0;
    at.advance(d);
    T Q[n][n], Dz[n][n], Tq[n][n], Tz[n][n];
    gather_column<n>(a.Tl, base, rs, ps, Q, active);
    psweep_b<n, kS, false>(Q, Q);
    psweep_a<n, kS, false>(Q, Q);
    psweep_a<n, kD, false>(Q, Dz);
    x_to_z2<n>(Q, Dz, Tq, Tz, bufA, bufB, t);
    psweep_b<n, kS, false>(Tq, Tq);
    psweep_b<n, kS, false>(Tz, Tz);
    if (active) {
#pragma unroll
      for (int j = 0; j < n; ++j) {
        T *o = out + cc * kTanFields2 * npt + t * (n * n) + n * j;
#pragma unroll
        for (int i = 0; i < n; ++i) {
          Tq[j][i] *= a.m.k1;
          Tz[j][i] *= a.m.k1;
        }
        store_row<n>(o, Tq[j]);
        store_row<n>(o + npt, Tz[j]);
      }
    }
  }
}

// Y[a][i] += A[a][q] x[i] for the transposed product matrix of `kind` and the row q
template <int n, int kind>
__device__ __forceinline__ void add_outer(int q, const double (&x)[n], double (&Y)[n][n])
{
  constexpr int full = tab_off(n, kind) + tab_full(n);
#pragma unroll
  for (int a = 0; a < n; ++a)
#pragma unroll
    for (int i = 0; i < n; ++i) Y[a][i] = fma(ctab<double>(full + a * n + q), x[i], Y[a][i]);
}

// FP64 diagonal of the operator (k_diag's closed form) for the constant and the linear-k law on
// register planes: with P = S o S, Q = D o D, R = S o D (transposed tables) the x-contractions run
// within a row of the quadrature plane, the y-contractions add each finished row to the three planes
// that z contracts,
//   Y_P = P_y (P_x C0 + Q_x Gxx + R_x Bx) + Q_y P_x Gyy + R_y (R_x Gxy + P_x By)
//   Y_Q = P_y P_x Gzz      Y_R = P_y (R_x Gxz + P_x Bz) + R_y P_x Gyz
//   W = P_z Y_P + Q_z Y_Q + R_z Y_R
// so that no coefficient plane is kept (k_diag keeps ten in shared memory and takes 28 barriers a
// batch; the inverse diagonal on 64^3 cells of FE_Q(3) k(T) 673 -> 208 us, deformed 768 -> 394).
template <int n, int GEO, int LAW>
__global__ void __launch_bounds__(32 * kV2Warps, 4) k_diag2(CellArgs<double> a)
{
  static_assert(LAW == 0 || LAW == 1, "constant rho*cp laws");
  using T = double;
  constexpr int CW = v2_cells_per_warp<n>(), CS = v2_cell_stride<n>(), npt = n * n * n;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = lane / n, t = lane % n;
  const bool lane_ok = cw < CW;
  constexpr size_t kWarp = 2 * (CW + 1) * CS + (LAW == 1 ? 3 * n * n * 32 : 0);
  T *wbuf = reinterpret_cast<T *>(smem_raw) + (size_t)warp * kWarp;
  T *bufA = wbuf + cw * CS, *bufB = wbuf + (CW + 1) * CS + cw * CS;
  T *keep = wbuf + 2 * (CW + 1) * CS + lane;  // LAW 1: T_lin, d/dy, d/dz, thread-private columns
  const T cval = a.m.idt * (a.m.rho_l * a.m.cp_l);
  const MeshDims &d = a.d;
  const int64_t rs = d.nd[0], ps = (int64_t)d.nd[0] * d.nd[1];
  const int64_t stride = (int64_t)gridDim.x * kV2Warps * CW;
  const int64_t first = ((int64_t)blockIdx.x * kV2Warps + warp) * CW;  // the warp's first cell
  CellWalk at(d, first + cw, stride, a.n_cells);
  for (int64_t head = first; head < a.n_cells; head += stride) {
    const int64_t cell = head + cw;
    const bool active = lane_ok && cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    const int I = d.p * at.x + t, J0 = d.p * at.y, K0 = d.p * at.z;
    const int64_t base = I + rs * J0 + ps * K0;
    at.advance(d);
    const ColumnMask cm(d, I, J0, K0, d.p);
    if constexpr (LAW == 1) {
      T Q[n][n], Dz[n][n], Tq[n][n], Tz[n][n], Ty[n][n];
      gather_column<n>(a.Tl, base, rs, ps, Q, active);
      psweep_b<n, kS, false>(Q, Q);
      psweep_a<n, kS, false>(Q, Q);
      psweep_a<n, kD, false>(Q, Dz);
      x_to_z2<n>(Q, Dz, Tq, Tz, bufA, bufB, t);
      psweep_b<n, kS, false>(Tq, Tq);
      psweep_b<n, kS, false>(Tz, Tz);
      psweep_a<n, kD, false>(Tq, Ty);
#pragma unroll
      for (int j = 0; j < n; ++j)
#pragma unroll
        for (int i = 0; i < n; ++i) {
          keep[(0 * n * n + j * n + i) * 32] = Tq[j][i];
          keep[(1 * n * n + j * n + i) * 32] = Ty[j][i];
          keep[(2 * n * n + j * n + i) * 32] = Tz[j][i];
        }
    }
    T YP[n][n], YQ[n][n], YR[n][n];
#pragma unroll
    for (int j = 0; j < n; ++j)
#pragma unroll
      for (int i = 0; i < n; ++i) YP[j][i] = YQ[j][i] = YR[j][i] = T(0);
#pragma unroll
    for (int j = 0; j < n; ++j) {
      T C0[n], G[6][n], Tq[n], Tx[n], r[n];
      if constexpr (GEO == 1) {
        const T *gb = a.g.q + cc * 7 * npt + t * (n * n) + n * j;
        load_row<n>(gb, C0);
#pragma unroll
        for (int f = 0; f < 6; ++f) load_row<n>(gb + (1 + f) * npt, G[f]);
      } else {
#pragma unroll
        for (int i = 0; i < n; ++i) {
          T g[6];
          geo_at<n, GEO>(a.g, cc, i, j, t, C0[i], g);
#pragma unroll
          for (int f = 0; f < 6; ++f) G[f][i] = g[f];
        }
      }
      if constexpr (LAW == 1) {
#pragma unroll
        for (int i = 0; i < n; ++i) Tq[i] = keep[(j * n + i) * 32];
        contract_row<n, kD, false>(Tq, Tx);
      }
      T B[3][n];
#pragma unroll
      for (int i = 0; i < n; ++i) {
        T rhocp, kk, drhocp, dk;
        mat_eval<LAW>(a.m, LAW == 1 ? Tq[i] : T(0), rhocp, kk, drhocp, dk);
        C0[i] *= cval;
        if constexpr (LAW == 1) {
          const T Ty = keep[(n * n + j * n + i) * 32], Tz = keep[(2 * n * n + j * n + i) * 32];
          const T Gi[6] = {G[0][i], G[1][i], G[2][i], G[3][i], G[4][i], G[5][i]};
          apply_G<GEO>(Gi, dk * Tx[i], dk * Ty, dk * Tz, B[0][i], B[1][i], B[2][i]);
        }
#pragma unroll
        for (int f = 0; f < 6; ++f) G[f][i] *= kk;
        G[1][i] *= T(2);
        G[2][i] *= T(2);
        G[4][i] *= T(2);
      }
      contract_row<n, kPT, false>(C0, r);
      contract_row<n, kQT, true>(G[0], r);
      if constexpr (LAW == 1) contract_row<n, kRT, true>(B[0], r);
      add_outer<n, kPT>(j, r, YP);
      contract_row<n, kPT, false>(G[3], r);
      add_outer<n, kQT>(j, r, YP);
      contract_row<n, kPT, false>(G[5], r);
      add_outer<n, kPT>(j, r, YQ);
      if constexpr (GEO == 1 || LAW == 1) {
        if constexpr (GEO == 1) {
          contract_row<n, kRT, false>(G[1], r);
          if constexpr (LAW == 1) contract_row<n, kPT, true>(B[1], r);
        } else {
          contract_row<n, kPT, false>(B[1], r);
        }
        add_outer<n, kRT>(j, r, YP);
        if constexpr (GEO == 1) {
          contract_row<n, kRT, false>(G[2], r);
          if constexpr (LAW == 1) contract_row<n, kPT, true>(B[2], r);
        } else {
          contract_row<n, kPT, false>(B[2], r);
        }
        add_outer<n, kPT>(j, r, YR);
        if constexpr (GEO == 1) {
          contract_row<n, kPT, false>(G[4], r);
          add_outer<n, kRT>(j, r, YR);
        }
      }
    }
    T XP[n][n], XQ[n][n], W[n][n];
    z_to_x2<n>(YP, YQ, XP, XQ, bufA, bufB, t);
    psweep_a<n, kPT, false>(XP, W);
    psweep_a<n, kQT, true>(XQ, W);
    if constexpr (GEO == 1 || LAW == 1) {
      z_to_x1<n>(YR, XP, bufA, t);
      psweep_a<n, kRT, true>(XP, W);
    }
    if (active) {
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j)
          if (!cm.template at<n>(j, k)) atomic_add(a.dst + base + (rs * j + ps * k), W[k][j]);
    }
  }
}
template <int n, int LAW> constexpr size_t diag2_smem()
{
  return sizeof(double) * kV2Warps *
         ((size_t)2 * (v2_cells_per_warp<n>() + 1) * v2_cell_stride<n>() +
          (LAW == 1 ? 3 * n * n * 32 : 0));
}

// create_rhs on register-resident planes for laws with constant rho*cp (0, 1):
// dst += -R(T) = -sum_q [ (c (T - T_old) - q_h) phi_i JxW + k(T) grad T . G grad phi_i ]
// with c = rho*cp / dt (rhs_cell_loop, heat_diffuse_operator.cpp:393-529). The value
// term is linear in the nodal values, so w = c (T - T_old) - q is formed at the gather
// and interpolated once.
template <int n, int GEO, int LAW>
__global__ void __launch_bounds__(32 * kV2Warps) k_rhs2(CellArgs<double> a)
{
  static_assert(LAW == 0 || LAW == 1, "constant rho*cp laws");
  using T = double;
  constexpr int CW = v2_cells_per_warp<n>();
  constexpr int CS = v2_cell_stride<n>();
  constexpr int npt = n * n * n;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = lane / n, t = lane % n;
  const bool lane_ok = cw < CW;
  T *wbuf = reinterpret_cast<T *>(smem_raw) + (size_t)warp * 2 * (CW + 1) * CS;
  T *bufA = wbuf + cw * CS;
  T *bufB = wbuf + (CW + 1) * CS + cw * CS;
  const T c = a.m.idt * (a.m.rho_l * a.m.cp_l);
  const MeshDims &d = a.d;
  const int64_t rs = d.nd[0], ps = (int64_t)d.nd[0] * d.nd[1];
  const int64_t stride = (int64_t)gridDim.x * kV2Warps * CW;
  const int64_t first = ((int64_t)blockIdx.x * kV2Warps + warp) * CW;  // the warp's first cell
  CellWalk at(d, first + cw, stride, a.n_cells);
  for (int64_t head = first; head < a.n_cells; head += stride) {
    const int64_t cell = head + cw;
    const bool active = lane_ok && cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    const int I = d.p * at.x + t, J0 = d.p * at.y, K0 = d.p * at.z;
    const int64_t base = I + rs * J0 + ps * K0;
    at.advance(d);
    const ColumnMask cm(d, I, J0, K0, d.p);
    T Qt[n][n], Qw[n][n], Qq[n][n];
    gather_column<n>(a.Tl, base, rs, ps, Qt, active);
    gather_column<n>(a.To, base, rs, ps, Qw, active);
    // (one branch for the column: with the choice made node by node the source's loads came one
    // after the other, FE_Q(3) 64^3 cells 287 us against 139, deformed 382 against 280)
    if (!a.source.on && a.qs) {
      gather_column<n>(a.qs, base, rs, ps, Qq, active);
    } else {
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j)
          Qq[k][j] =
            a.source.on && active ? (T)source_at(a.source, base + (rs * j + ps * k)) : T(0);
    }
#pragma unroll
    for (int k = 0; k < n; ++k)
#pragma unroll
      for (int j = 0; j < n; ++j) Qw[k][j] = c * (Qt[k][j] - Qw[k][j]) - Qq[k][j];
    // w at the q-points
    T U[n][n];
    psweep_b<n, kS, false>(Qw, Qw);
    psweep_a<n, kS, false>(Qw, Qw);
    x_to_z1<n>(Qw, U, bufA, t);
    psweep_b<n, kS, false>(U, U);
    // T at the q-points: values, d/dy, d/dz (d/dx row by row below)
    T Tq[n][n], Fy[n][n], Fz[n][n];
    {
      T Dz[n][n];
      psweep_b<n, kS, false>(Qt, Qt);
      psweep_a<n, kS, false>(Qt, Qt);
      psweep_a<n, kD, false>(Qt, Dz);
      x_to_z2<n>(Qt, Dz, Tq, Fz, bufA, bufB, t);
    }
    psweep_b<n, kS, false>(Tq, Tq);
    psweep_b<n, kS, false>(Fz, Fz);
    psweep_a<n, kD, false>(Tq, Fy);
    // val = -w JxW, f = -k(T) G grad T; row j of U turns into val + D_x^T f_x
#pragma unroll
    for (int j = 0; j < n; ++j) {
      T Fx[n], jxw[n], G[6][n];
      contract_row<n, kD, false>(Tq[j], Fx);
      if constexpr (GEO == 0) {
#pragma unroll
        for (int i = 0; i < n; ++i) {
          T g[6];
          geo_at<n, GEO>(a.g, cc, i, j, t, jxw[i], g);
#pragma unroll
          for (int f = 0; f < 6; ++f) G[f][i] = g[f];
        }
      } else {
        const T *gb = a.g.q + cc * 7 * npt + t * (n * n) + n * j;
        load_row<n>(gb, jxw);
#pragma unroll
        for (int f = 0; f < 6; ++f) load_row<n>(gb + (1 + f) * npt, G[f]);
      }
#pragma unroll
      for (int i = 0; i < n; ++i) {
        T rhocp, kk, drhocp, dk;
        mat_eval<LAW>(a.m, Tq[j][i], rhocp, kk, drhocp, dk);
        kk = -kk;
        const T Gi[6] = {G[0][i], G[1][i], G[2][i], G[3][i], G[4][i], G[5][i]};
        apply_G<GEO>(Gi, kk * Fx[i], kk * Fy[j][i], kk * Fz[j][i], Fx[i], Fy[j][i], Fz[j][i]);
        U[j][i] = -U[j][i] * jxw[i];
      }
      contract_row<n, kDT, true>(Fx, U[j]);
    }
    // integration (as in k_vmult2)
    psweep_a<n, kDT, true>(Fy, U);
    psweep_b<n, kST, false>(U, U);
    psweep_b<n, kST, false>(Fz, Fz);
    T W[n][n], Wz[n][n];
    z_to_x2<n>(U, Fz, W, Wz, bufA, bufB, t);
    psweep_a<n, kDT, true>(Wz, W);
    psweep_b<n, kST, false>(W, W);
    psweep_a<n, kST, false>(W, W);
    if (active) {
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j)
          if (!cm.template at<n>(j, k)) atomic_add(a.dst + base + (rs * j + ps * k), W[k][j]);
    }
  }
}

}  // namespace mpdg
