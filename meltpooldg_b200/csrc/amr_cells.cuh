// Register-resident operator kernels on hanging-node meshes (mpdg_amr.cu): the work split of
// k_vmult2 (cell_kernels_v2.cuh), n lanes per cell, 32 / n cells per warp, with the cell's DoFs
// gathered through an index and the hanging interpolation applied in registers.
//
// The first form (one CTA of n^3 threads per cell, every sweep through shared memory, the 1D
// matrices indexed per thread) took 0.11 ms per application on 25.9 k cells of FE_Q(3), this one
// 0.03 ms: a sweep's coefficients are constant-bank operands, a thread's 16 points share one
// index computation, and there is no block-wide barrier. Cells with a hanging face or edge are
// stored before the others, so only the first warps run the interpolation.
#pragma once

#include "cell_kernels_v2.cuh"

namespace mpdg {

// DoF index entry of a cell: the DoF, or its complement where it is a Dirichlet DoF
__device__ __forceinline__ int amr_dof(int e) { return e < 0 ? ~e : e; }

struct AmrCellArgs {
  // [cell][i][k][j]: a thread's column of n^2 entries is contiguous
  const int *__restrict__ idx;
  const uint16_t *__restrict__ code;
  const double *src;  // (coherent loads: a dependent launch's predecessor writes it)
  const double *__restrict__ Tl;
  // the linearisation point's values and reference gradients at the q-points, [cell][4][n^3]
  const double *__restrict__ tf;
  double *dst;
  int64_t n_cells;
  double detJ, Gd[3];  // of a coarse cell
  double cval, k0, k1;
  double I[kMaxN * kMaxN];  // child interpolation I_0[j][a] = l_a(xi_j / 2); I_1 is its mirror image
};

// x <- I_s x or I_s^T x of one line where `on`
template <int n, bool TR>
__device__ __forceinline__ void hang_line(const double *I, bool upper, bool on, double (&x)[n])
{
  double r[n];
#pragma unroll
  for (int o = 0; o < n; ++o) {
    r[o] = 0.0;
#pragma unroll
    for (int l = 0; l < n; ++l) {
      const int j = TR ? l : o, a = TR ? o : l;  // entry I_s[j][a]
      r[o] = fma(upper ? I[(n - 1 - j) * n + (n - 1 - a)] : I[j * n + a], x[l], r[o]);
    }
  }
#pragma unroll
  for (int o = 0; o < n; ++o) x[o] = on ? r[o] : x[o];
}

// The hanging interpolation of a cell's nodal values on x-columns Q[k][j] (thread t = node t along
// x), or its transpose: along direction d, the lines on a hanging face normal to another direction
// and on a hanging edge parallel to d. The whole warp enters (the x-lines go through shared memory).
template <int n, bool TR>
__device__ __forceinline__ void hang_columns(const double *I, int code, double (&Q)[n][n],
                                             double *buf, int t)
{
  const int s[3] = {code & 1, (code >> 1) & 1, (code >> 2) & 1};
  const int own[3] = {s[0] ? n - 1 : 0, s[1] ? n - 1 : 0, s[2] ? n - 1 : 0};
  const bool f[3] = {(code >> 3 & 1) != 0, (code >> 4 & 1) != 0, (code >> 5 & 1) != 0};
  const bool e[3] = {(code >> 6 & 1) != 0, (code >> 7 & 1) != 0, (code >> 8 & 1) != 0};
  // along x, on z-planes: thread t = plane t, rows j
  auto along_x = [&]() {
    double P[n][n];
    x_to_z1<n>(Q, P, buf, t);
#pragma unroll
    for (int j = 0; j < n; ++j)
      hang_line<n, TR>(I, s[0] != 0,
                       (f[1] && j == own[1]) || (f[2] && t == own[2]) ||
                         (e[0] && j == own[1] && t == own[2]),
                       P[j]);
    z_to_x1<n>(P, Q, buf, t);
  };
  auto along_y = [&]() {
#pragma unroll
    for (int k = 0; k < n; ++k)
      hang_line<n, TR>(I, s[1] != 0,
                       (f[2] && k == own[2]) || (f[0] && t == own[0]) ||
                         (e[1] && k == own[2] && t == own[0]),
                       Q[k]);
  };
  auto along_z = [&]() {
#pragma unroll
    for (int j = 0; j < n; ++j) {
      double x[n];
#pragma unroll
      for (int k = 0; k < n; ++k) x[k] = Q[k][j];
      hang_line<n, TR>(I, s[2] != 0,
                       (f[0] && t == own[0]) || (f[1] && j == own[1]) ||
                         (e[2] && t == own[0] && j == own[1]),
                       x);
#pragma unroll
      for (int k = 0; k < n; ++k) Q[k][j] = x[k];
    }
  };
  if (!TR) {
    along_x();
    along_y();
    along_z();
  } else {
    along_z();
    along_y();
    along_x();
  }
}

// a thread's column of index entries
template <int n>
__device__ __forceinline__ void load_column_index(const int *__restrict__ p, int (&e)[n][n])
{
  if constexpr (n == 4 || n == 2) {
    int r[n * n];
#pragma unroll
    for (int i = 0; i < n * n / 4; ++i) {
      const int4 v = __ldg(reinterpret_cast<const int4 *>(p) + i);
      r[4 * i] = v.x;
      r[4 * i + 1] = v.y;
      r[4 * i + 2] = v.z;
      r[4 * i + 3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < n * n; ++i) e[i / n][i % n] = r[i];
  } else {
#pragma unroll
    for (int i = 0; i < n * n; ++i) e[i / n][i % n] = __ldg(p + i);
  }
}

// shared memory: two plane buffers per cell as in k_vmult2, and with EVAL the four coefficients
template <int n, bool EVAL> constexpr size_t amr_smem() { return v2_smem<n, double, EVAL ? 1 : 0>(); }

// what the CG iteration on the refined mesh keeps on the device
struct AmrCg {
  double rz, alpha, beta, rr, tol;
  int it, max_it, done, status;  // done: 0 running, 1 converged, 2 stopped with status
};

// dst += J src (Dirichlet rows skipped): TANGENT the k(T) tangent at T_lin, from the fields a.tf
// or (EVAL) from a.Tl evaluated in the kernel. With cg the sum src.dst is formed too and the last
// block sets alpha.
template <int n, bool TANGENT, bool EVAL>
__global__ void __launch_bounds__(32 * kV2Warps, 4)
  k_amr_apply(const __grid_constant__ AmrCellArgs a, AmrCg *cg, double *partials, unsigned *counter)
{
  using T = double;
  constexpr int CW = v2_cells_per_warp<n>(), CS = v2_cell_stride<n>(), npt = n * n * n;
  dependents_may_start();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = lane / n, t = lane % n;
  T *wbuf = reinterpret_cast<T *>(smem_raw) +
            (size_t)warp * (v2_smem_per_warp<n, T, EVAL ? 1 : 0>() / sizeof(T));
  T *bufA = wbuf + cw * CS, *bufB = wbuf + (CW + 1) * CS + cw * CS;
  T *coef = wbuf + 2 * (CW + 1) * CS;
  const T wt = cw_at<n, T>(w_off(n), t);
  double dot = 0.0;
  wait_for_predecessor();
  if (cg && cg->done) return;
  const int64_t stride = (int64_t)gridDim.x * kV2Warps * CW;
  for (int64_t head = ((int64_t)blockIdx.x * kV2Warps + warp) * CW; head < a.n_cells;
       head += stride) {
    const int64_t cell = head + cw;
    const bool active = cw < CW && cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    const int code = active ? a.code[cc] : 0;
    const bool hang = (code & 0x1F8) != 0, any_hang = __any_sync(0xffffffffu, hang);
    int e[n][n];
    load_column_index<n>(a.idx + cc * npt + t * n * n, e);
    // (inactive lanes read cell 0's nodes; loads without a condition are issued back to back)
    T Q[n][n];
#pragma unroll
    for (int k = 0; k < n; ++k)
#pragma unroll
      for (int j = 0; j < n; ++j) Q[k][j] = a.src[amr_dof(e[k][j])];
#pragma unroll
    for (int k = 0; k < n; ++k)
#pragma unroll
      for (int j = 0; j < n; ++j) Q[k][j] = active && e[k][j] >= 0 ? Q[k][j] : T(0);
    if constexpr (TANGENT && EVAL) {
      T R[n][n], Dz[n][n], Tq[n][n], Tz[n][n], Ty[n][n];
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j) R[k][j] = __ldg(a.Tl + amr_dof(e[k][j]));
      if (any_hang) hang_columns<n, false>(a.I, code, R, bufA, t);
      psweep_b<n, kS, false>(R, R);
      psweep_a<n, kS, false>(R, R);
      psweep_a<n, kD, false>(R, Dz);
      x_to_z2<n>(R, Dz, Tq, Tz, bufA, bufB, t);
      psweep_b<n, kS, false>(Tq, Tq);
      psweep_b<n, kS, false>(Tz, Tz);
      psweep_a<n, kD, false>(Tq, Ty);
#pragma unroll
      for (int j = 0; j < n; ++j) {
        T Tx[n];
        contract_row<n, kD, false>(Tq[j], Tx);
#pragma unroll
        for (int i = 0; i < n; ++i) {
          const int pt = j * n + i;
          coef[(0 * n * n + pt) * 32 + lane] = Tq[j][i];
          coef[(1 * n * n + pt) * 32 + lane] = Tx[i];
          coef[(2 * n * n + pt) * 32 + lane] = Ty[j][i];
          coef[(3 * n * n + pt) * 32 + lane] = Tz[j][i];
        }
      }
    }
    if (any_hang) hang_columns<n, false>(a.I, code, Q, bufA, t);
    T U[n][n], Uz[n][n], Uy[n][n];
    {
      T Dz[n][n];
      psweep_b<n, kS, false>(Q, Q);
      psweep_a<n, kS, false>(Q, Q);
      psweep_a<n, kD, false>(Q, Dz);
      x_to_z2<n>(Q, Dz, U, Uz, bufA, bufB, t);
    }
    psweep_b<n, kS, false>(U, U);
    psweep_b<n, kS, false>(Uz, Uz);
    psweep_a<n, kD, false>(U, Uy);
    // quadrature points: a cell of level l has edges h / 2^l, so JxW scales with 8^-l and JxW/h^2
    // with 2^-l
    const T s = ldexp(1.0, -((code >> 10) & 7)), s3 = s * s * s;
    const T cm = a.cval * a.detJ * s3 * wt, gx = a.Gd[0] * s * wt, gy = a.Gd[1] * s * wt,
            gz = a.Gd[2] * s * wt;
#pragma unroll
    for (int j = 0; j < n; ++j) {
      T Ux[n], c[TANGENT ? 4 : 1][n];
      contract_row<n, kD, false>(U[j], Ux);
      if constexpr (TANGENT && !EVAL) {
        const T *f = a.tf + cc * 4 * npt + t * n * n + n * j;
#pragma unroll
        for (int q = 0; q < 4; ++q) load_row<n>(f + q * npt, c[q]);
      }
      if constexpr (TANGENT && EVAL) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int i = 0; i < n; ++i) c[q][i] = coef[(q * n * n + j * n + i) * 32 + lane];
      }
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const T w = mpdg::cw<T>(w_off(n) + j) * mpdg::cw<T>(w_off(n) + i), u = U[j][i];
        T f0, f1, f2;
        if constexpr (TANGENT) {
          const T k = a.k0 + a.k1 * c[0][i], u1 = a.k1 * u;
          f0 = k * Ux[i] + c[1][i] * u1;
          f1 = k * Uy[j][i] + c[2][i] * u1;
          f2 = k * Uz[j][i] + c[3][i] * u1;
        } else {
          f0 = a.k0 * Ux[i];
          f1 = a.k0 * Uy[j][i];
          f2 = a.k0 * Uz[j][i];
        }
        U[j][i] = cm * w * u;
        Ux[i] = gx * w * f0;
        Uy[j][i] = gy * w * f1;
        Uz[j][i] = gz * w * f2;
      }
      contract_row<n, kDT, true>(Ux, U[j]);
    }
    psweep_a<n, kDT, true>(Uy, U);
    psweep_b<n, kST, false>(U, U);
    psweep_b<n, kST, false>(Uz, Uz);
    {
      T Wz[n][n];
      z_to_x2<n>(U, Uz, Q, Wz, bufA, bufB, t);
      psweep_a<n, kDT, true>(Wz, Q);
    }
    psweep_b<n, kST, false>(Q, Q);
    psweep_a<n, kST, false>(Q, Q);
    if (any_hang) hang_columns<n, true>(a.I, code, Q, bufA, t);
    load_column_index<n>(a.idx + cc * npt + t * n * n, e);
    if (cg) {
      T u[n][n];
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j) u[k][j] = a.src[amr_dof(e[k][j])];
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j)
          dot += active && e[k][j] >= 0 ? u[k][j] * Q[k][j] : T(0);
    }
    if (active) {
#pragma unroll
      for (int k = 0; k < n; ++k)
#pragma unroll
        for (int j = 0; j < n; ++j)
          if (e[k][j] >= 0) atomic_add(a.dst + e[k][j], Q[k][j]);
    }
  }
  if (cg) {
    double v[1] = {dot}, tot[1];
    if (grid_sum<1>(v, partials, counter, tot)) {
      if (!(tot[0] > 0.0)) {
        cg->done = 2;
        cg->status = 5;  // breakdown
      } else {
        cg->alpha = cg->rz / tot[0];
      }
    }
  }
}

// the linearisation point's values and reference gradients at the q-points of every cell
// (hanging interpolation applied), [cell][4][n^3]: the operator's T_lin evaluation, once per solve
template <int n>
__global__ void __launch_bounds__(32 * kV2Warps, 4)
  k_amr_tfields(const __grid_constant__ AmrCellArgs a, double *tf)
{
  using T = double;
  constexpr int CW = v2_cells_per_warp<n>(), CS = v2_cell_stride<n>(), npt = n * n * n;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cw = lane / n, t = lane % n;
  T *wbuf = reinterpret_cast<T *>(smem_raw) +
            (size_t)warp * (v2_smem_per_warp<n, T, 0>() / sizeof(T));
  T *bufA = wbuf + cw * CS, *bufB = wbuf + (CW + 1) * CS + cw * CS;
  const int64_t stride = (int64_t)gridDim.x * kV2Warps * CW;
  for (int64_t head = ((int64_t)blockIdx.x * kV2Warps + warp) * CW; head < a.n_cells;
       head += stride) {
    const int64_t cell = head + cw;
    const bool active = cw < CW && cell < a.n_cells;
    const int64_t cc = active ? cell : 0;
    const int code = active ? a.code[cc] : 0;
    const bool any_hang = __any_sync(0xffffffffu, (code & 0x1F8) != 0);
    int e[n][n];
    load_column_index<n>(a.idx + cc * npt + t * n * n, e);
    T R[n][n], Dz[n][n], Tq[n][n], Tz[n][n], Ty[n][n];
#pragma unroll
    for (int k = 0; k < n; ++k)
#pragma unroll
      for (int j = 0; j < n; ++j) R[k][j] = __ldg(a.Tl + amr_dof(e[k][j]));
    if (any_hang) hang_columns<n, false>(a.I, code, R, bufA, t);
    psweep_b<n, kS, false>(R, R);
    psweep_a<n, kS, false>(R, R);
    psweep_a<n, kD, false>(R, Dz);
    x_to_z2<n>(R, Dz, Tq, Tz, bufA, bufB, t);
    psweep_b<n, kS, false>(Tq, Tq);
    psweep_b<n, kS, false>(Tz, Tz);
    psweep_a<n, kD, false>(Tq, Ty);
    if (active) {
#pragma unroll
      for (int j = 0; j < n; ++j) {
        T Tx[n];
        contract_row<n, kD, false>(Tq[j], Tx);
        T *f = tf + cc * 4 * npt + t * n * n + n * j;
#pragma unroll
        for (int i = 0; i < n; ++i) {
          f[i] = Tq[j][i];
          f[npt + i] = Tx[i];
          f[2 * npt + i] = Ty[j][i];
          f[3 * npt + i] = Tz[j][i];
        }
      }
    }
  }
}

// ---- the Jacobi-CG iteration: scalars on the device, two vector kernels ----------------------
// x = 0, r = b, p = D r, Ap = 0
__global__ void k_amr_cg_init(int64_t n, const double *__restrict__ b,
                              const double *__restrict__ D, double *x, double *r, double *p,
                              double *Ap, AmrCg *cg, double *partials, unsigned *counter,
                              double rel, double abs_tol, int max_it)
{
  double v[2] = {0.0, 0.0};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double ri = b[i], zi = D[i] * ri;
    x[i] = 0.0;
    r[i] = ri;
    p[i] = zi;
    Ap[i] = 0.0;
    v[0] += ri * zi;
    v[1] += ri * ri;
  }
  double tot[2];
  if (grid_sum<2>(v, partials, counter, tot)) {
    cg->rz = tot[0];
    cg->rr = tot[1];
    cg->tol = fmax(abs_tol, rel * sqrt(tot[1]));
    cg->alpha = cg->beta = 0.0;
    cg->it = 0;
    cg->max_it = max_it;
    cg->status = 0;
    cg->done = sqrt(tot[1]) <= cg->tol ? 1 : 0;
    if (!cg->done && max_it <= 0) {
      cg->done = 2;
      cg->status = MPDG_ERR_NOT_CONVERGED;
    }
  }
}

// r -= alpha Ap with the sums r.r and r.D r; the last block tests the convergence
__global__ void k_amr_cg_update(int64_t n, const double *__restrict__ D, const double *Ap,
                                double *r, AmrCg *cg, double *partials, unsigned *counter)
{
  dependents_may_start();
  wait_for_predecessor();
  if (cg->done) return;
  const double alpha = cg->alpha;
  double v[2] = {0.0, 0.0};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double ri = r[i] - alpha * Ap[i];
    r[i] = ri;
    v[0] += ri * D[i] * ri;
    v[1] += ri * ri;
  }
  double tot[2];
  if (grid_sum<2>(v, partials, counter, tot)) {
    const int it = ++cg->it;
    cg->beta = tot[0] / cg->rz;
    cg->rz = tot[0];
    cg->rr = tot[1];
    if (!isfinite(tot[1])) {
      cg->done = 2;
      cg->status = MPDG_ERR_NAN;
    } else if (sqrt(tot[1]) <= cg->tol) {
      cg->done = 1;
    } else if (it >= cg->max_it) {
      cg->done = 2;
      cg->status = MPDG_ERR_NOT_CONVERGED;
    }
  }
}

// x += alpha p, p = D r + beta p, Ap = 0: x is updated where p is read anyway (the iteration that
// ends the solve leaves it to k_amr_cg_last)
__global__ void k_amr_cg_direction(int64_t n, const double *__restrict__ D, const double *r,
                                   double *x, double *p, double *Ap, const AmrCg *cg)
{
  dependents_may_start();
  wait_for_predecessor();
  if (cg->done) return;
  const double alpha = cg->alpha, beta = cg->beta;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double pi = p[i], xi = x[i], ri = r[i];  // (loaded before the stores)
    x[i] = xi + alpha * pi;
    p[i] = D[i] * ri + beta * pi;
    Ap[i] = 0.0;
  }
}

// x += alpha p of the iteration that ended the solve
__global__ void k_amr_cg_last(int64_t n, const double *__restrict__ p, double *x, const AmrCg *cg)
{
  const double alpha = cg->alpha;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    x[i] += alpha * p[i];
}

}  // namespace mpdg
