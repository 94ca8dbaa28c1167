// Host launchers of the cell kernels for one polynomial degree. Each
// cells_pN.cu translation unit includes this header and instantiates
// MPDG_DEFINE_DEGREE(n) so the degrees compile in parallel; the handle code
// reaches them through DegreeTable.
#pragma once

#include "cell_kernels.cuh"
#include "cell_kernels_lines.cuh"
#include "cell_kernels_v2.cuh"
#include "cell_kernels_f2.cuh"
#include "cell_kernels_tc.cuh"
#include "degree_table.hpp"
#include "resident.hpp"

#include <stdlib.h>
#include <algorithm>
#include <type_traits>

namespace mpdg {

// a persistent grid: the CTAs that the device holds at once, at most n_batches
template <typename... P, typename... A>
static cudaError_t launch_persistent(ResidentBlocks &resident, void (*kernel)(P...), int threads,
                                     size_t smem, int64_t n_batches, bool dependent,
                                     cudaStream_t s, const A &...args)
{
  int blocks = 0;
  const cudaError_t e = resident.get(kernel, threads, smem, &blocks);
  if (e != cudaSuccess) return e;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>(blocks, n_batches));
  if (dependent) return launch_dependent(kernel, g, threads, smem, s, args...);
  kernel<<<g, threads, smem, s>>>(args...);
  return cudaGetLastError();
}

// FP32 operator on the scalar register-resident kernel (default) or the packed-pair
// kernel (MPDG_FP32_PACKED=1); both compute the same operator. The packed kernel
// issues 31 % fewer instructions at p = 3, but a packed FMA occupies the FMA pipe
// for two cycles and its 210-255 registers per lane halve the resident warps, so
// it measured 1.3-1.5x slower (p = 2, 3; constant k, k(T) tangent, Picard).
static inline bool fp32_packed()
{
  static const int on = [] {
    const char *e = getenv("MPDG_FP32_PACKED");
    return (e && e[0] == '1') ? 1 : 0;
  }();
  return on != 0;
}

template <int n>
struct DegreeOps {
  static constexpr int CPB = cells_per_block(n);
  static constexpr int THREADS = block_threads(n);
  static constexpr int PLANE_THREADS = 32 * kV2Warps;  // register-plane kernels

  // CTAs' worth of work of the line kernels, and of the register-plane kernels
  static int64_t line_batches(int64_t cells) { return (cells + CPB - 1) / CPB; }
  static int64_t plane_batches(int64_t cells)
  {
    const int64_t groups = (cells + v2_cells_per_warp<n>() - 1) / v2_cells_per_warp<n>();
    return (groups + kV2Warps - 1) / kV2Warps;
  }

  static void upload(const double *tab, const float *tabf, const double *w, const float *wf)
  {
    cudaMemcpyToSymbol(c_tab_d, tab, sizeof(double) * kTabSize);
    cudaMemcpyToSymbol(c_tab_f, tabf, sizeof(float) * kTabSize);
    float2 tabf2[kTabSize];
    for (int i = 0; i < kTabSize; ++i) tabf2[i] = make_float2(tabf[i], tabf[i]);
    cudaMemcpyToSymbol(c_tab_f2, tabf2, sizeof(float2) * kTabSize);
    cudaMemcpyToSymbol(c_w_d, w, sizeof(double) * kWTabSize);
    cudaMemcpyToSymbol(c_w_f, wf, sizeof(float) * kWTabSize);
  }

  // register-plane kernels where a cell's planes fit the register file; the three-phase /
  // transport law with temperature dependence (LAW 5) runs the line kernel
  template <typename T, int LAW = 0>
  static constexpr bool use_v2()
  {
    return LAW != 5 && (sizeof(T) == 8 ? n <= 4 : n <= 5);
  }
  // the operator alone also with the constant law on a uniform box up to p = 5, which spills but
  // needs no per-point data (FP64 p = 4 on 64^3 cells 0.30 against 0.42 ms on lines, p = 5 on 53^3
  // 0.43 against 0.50 ms; FP32 p = 5 0.23 against 0.26 ms)
  // ... and not in FP32 at p = 4 on a deformed mesh, except for the operators that exist on planes
  // only (conductivity, LAW 3 and 8): a plane's rows of 5 values have no vector load and lie 100
  // bytes apart from lane to lane, a line's do not (planes against lines: constant law on 48^3 cells
  // 182, 162 us, on 6^3 11.2, 9.2; k(T) on 48^3 254, 209; liquid-solid on 30^3 172, 65, gas-liquid
  // 91, 51)
  template <typename T, int GEO, int LAW>
  static constexpr bool vmult_v2()
  {
    if (sizeof(T) == 4 && n == 5 && GEO == 1 && LAW != 3 && LAW != 8) return false;
    return use_v2<T, LAW>() || (GEO == 0 && LAW == 0 && n <= 6);
  }

  template <typename T, int GEO, int LAW>
  static cudaError_t vmult_t(const CellArgs<T> &a, cudaStream_t s, int sm)
  {
    if constexpr (std::is_same<T, float>::value && n <= 4 && (LAW == 0 || LAW == 1 || LAW == 3)) {
      if (fp32_packed()) {
        static ResidentBlocks cachep;
        auto kp = k_vmult2p<n, GEO, LAW>;
        const size_t smemp = v2_smem<n, F2, LAW>();
        return launch_persistent(cachep, kp, PLANE_THREADS, smemp,
                                 plane_batches((a.n_cells + 1) / 2), false, s, a);
      }
    }
    // at p = 5 only where the cells fill a round of the grid (8 warps per SM): below that the time
    // is one cell group's latency, which is longer with the spills (729 cells FP64 16.4 us, the
    // line kernel 12.3)
    const bool fills = n < 6 || a.n_cells >= (int64_t)sm * 8 * v2_cells_per_warp<n>();
    if constexpr (vmult_v2<T, GEO, LAW>()) {
      if (fills) return vmult_planes<T, GEO, LAW>(a, s, sm);
    }
    if constexpr (!vmult_v2<T, GEO, LAW>() || n == 6) return vmult_lines<T, GEO, LAW>(a, s, sm);
    return cudaErrorNotSupported;  // (not reached: fills is true below n = 6)
  }
  template <typename T, int GEO, int LAW>
  static cudaError_t vmult_planes(const CellArgs<T> &a, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache2;
    // deformed FP64: the geometry from the cell's vertices (p >= 2) instead of the stored one
    constexpr int G = v2_geometry<n, T, GEO, LAW>();
    auto k2 = k_vmult2<n, T, G, LAW>;
    const size_t smem2 = v2_smem<n, T, LAW, G>();
    const bool dependent = v2_dependent<T>() && a.dependent;
    return launch_persistent(cache2, k2, PLANE_THREADS, smem2, plane_batches(a.n_cells), dependent,
                             s, a);
  }
  template <typename T, int GEO, int LAW>
  static cudaError_t vmult_lines(const CellArgs<T> &a, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    auto k = k_vmult_lines<n, T, ln_geometry<T, GEO, LAW>(), LAW>;
    constexpr size_t smem = ln_smem<n, T>();
    return launch_persistent(cache, k, THREADS, smem, line_batches(a.n_cells), false, s, a);
  }
  template <typename T>
  static cudaError_t vmult(const CellArgs<T> &a, int geo, int law, cudaStream_t s, int sm)
  {
    if (law == 3) {
      if constexpr (use_v2<T>()) {
        return geo == 0 ? vmult_t<T, 0, 3>(a, s, sm) : vmult_t<T, 1, 3>(a, s, sm);
      } else {
        return cudaErrorNotSupported;
      }
    }
    if (law == 8) {  // the Picard operator from the gathered T_lin (linear-k law)
      if constexpr (use_v2<T>()) {
        return geo == 0 ? vmult_t<T, 0, 8>(a, s, sm) : vmult_t<T, 1, 8>(a, s, sm);
      } else {
        return cudaErrorNotSupported;
      }
    }
    if (law == 4) return geo == 0 ? vmult_t<T, 0, 4>(a, s, sm) : vmult_t<T, 1, 4>(a, s, sm);
    if (law == 5) return geo == 0 ? vmult_t<T, 0, 5>(a, s, sm) : vmult_t<T, 1, 5>(a, s, sm);
    if (law == 7) return geo == 0 ? vmult_t<T, 0, 7>(a, s, sm) : vmult_t<T, 1, 7>(a, s, sm);
    if (law == 6) {  // register-resident kernel only
      if constexpr (use_v2<T>()) {
        return geo == 0 ? vmult_t<T, 0, 6>(a, s, sm) : vmult_t<T, 1, 6>(a, s, sm);
      } else {
        return cudaErrorNotSupported;
      }
    }
    if (geo == 0) {
      if (law == 0) return vmult_t<T, 0, 0>(a, s, sm);
      if (law == 1) return vmult_t<T, 0, 1>(a, s, sm);
      return vmult_t<T, 0, 2>(a, s, sm);
    }
    if (law == 0) return vmult_t<T, 1, 0>(a, s, sm);
    if (law == 1) return vmult_t<T, 1, 1>(a, s, sm);
    return vmult_t<T, 1, 2>(a, s, sm);
  }
  static cudaError_t vmult_d(const CellArgs<double> &a, int geo, int law, cudaStream_t s, int sm)
  {
    return vmult<double>(a, geo, law, s, sm);
  }
  static cudaError_t vmult_f(const CellArgs<float> &a, int geo, int law, cudaStream_t s, int sm)
  {
    return vmult<float>(a, geo, law, s, sm);
  }

  template <int GEO, int LAW>
  static cudaError_t rhs_t(const CellArgs<double> &a, cudaStream_t s, int sm)
  {
    if constexpr (use_v2<double>() && (LAW == 0 || LAW == 1)) {
      static ResidentBlocks cache2;
      auto k2 = k_rhs2<n, GEO, LAW>;
      const size_t smem2 =
        sizeof(double) * kV2Warps * 2 * (v2_cells_per_warp<n>() + 1) * v2_cell_stride<n>();
      return launch_persistent(cache2, k2, PLANE_THREADS, smem2, plane_batches(a.n_cells), false, s,
                               a);
    }
    static ResidentBlocks cache;
    auto k = k_rhs<n, GEO, LAW>;
    const size_t smem = smem_rhs<n>();
    return launch_persistent(cache, k, THREADS, smem, line_batches(a.n_cells), false, s, a);
  }
  static cudaError_t rhs(const CellArgs<double> &a, int geo, int law, cudaStream_t s, int sm)
  {
    if (law == 4) return geo == 0 ? rhs_t<0, 4>(a, s, sm) : rhs_t<1, 4>(a, s, sm);
    if (law == 5) return geo == 0 ? rhs_t<0, 5>(a, s, sm) : rhs_t<1, 5>(a, s, sm);
    if (geo == 0) {
      if (law == 0) return rhs_t<0, 0>(a, s, sm);
      if (law == 1) return rhs_t<0, 1>(a, s, sm);
      return rhs_t<0, 2>(a, s, sm);
    }
    if (law == 0) return rhs_t<1, 0>(a, s, sm);
    if (law == 1) return rhs_t<1, 1>(a, s, sm);
    return rhs_t<1, 2>(a, s, sm);
  }

  template <int GEO, int LAW>
  static cudaError_t diag_t(const CellArgs<double> &a, cudaStream_t s, int sm)
  {
    if constexpr (use_v2<double>() && (LAW == 0 || LAW == 1)) {
      static ResidentBlocks cache2;
      auto k2 = k_diag2<n, GEO, LAW>;
      constexpr size_t smem2 = diag2_smem<n, LAW>();
      return launch_persistent(cache2, k2, PLANE_THREADS, smem2, plane_batches(a.n_cells), false, s,
                               a);
    } else {
      return diag_lines<GEO, LAW>(a, s, sm);
    }
  }
  template <int GEO, int LAW>
  static cudaError_t diag_lines(const CellArgs<double> &a, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    auto k = k_diag<n, GEO, LAW>;
    const size_t smem = smem_diag<n>();
    return launch_persistent(cache, k, THREADS, smem, line_batches(a.n_cells), false, s, a);
  }
  static cudaError_t diag(const CellArgs<double> &a, int geo, int law, cudaStream_t s, int sm)
  {
    if (law == 4) return geo == 0 ? diag_t<0, 4>(a, s, sm) : diag_t<1, 4>(a, s, sm);
    if (law == 5) return geo == 0 ? diag_t<0, 5>(a, s, sm) : diag_t<1, 5>(a, s, sm);
    if (geo == 0) {
      if (law == 0) return diag_t<0, 0>(a, s, sm);
      if (law == 1) return diag_t<0, 1>(a, s, sm);
      return diag_t<0, 2>(a, s, sm);
    }
    if (law == 0) return diag_t<1, 0>(a, s, sm);
    if (law == 1) return diag_t<1, 1>(a, s, sm);
    return diag_t<1, 2>(a, s, sm);
  }

  template <int GEO>
  static cudaError_t norm_t(const CellArgs<double> &a, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    auto k = k_norm<n, GEO>;
    const size_t smem = smem_norm<n>();
    return launch_persistent(cache, k, THREADS, smem, line_batches(a.n_cells), false, s, a);
  }
  static cudaError_t norm(const CellArgs<double> &a, int geo, int, cudaStream_t s, int sm)
  {
    return geo == 0 ? norm_t<0>(a, s, sm) : norm_t<1>(a, s, sm);
  }

  template <int LAW>
  static cudaError_t kq_t(const CellArgs<double> &a, float *kq, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    auto k = k_conductivity_q<n, LAW>;
    const size_t smem =
      sizeof(double) * kV2Warps * (v2_cells_per_warp<n>() + 1) * v2_cell_stride<n>();
    return launch_persistent(cache, k, PLANE_THREADS, smem, plane_batches(a.n_cells), false, s,
                             a, kq);
  }
  template <int GEO>
  static cudaError_t diag_picard_t(const CellArgs<float> &a, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    auto k = k_diag_picard<n, GEO>;
    const size_t smem =
      sizeof(float) * kV2Warps * 2 * (v2_cells_per_warp<n>() + 1) * v2_cell_stride<n>();
    return launch_persistent(cache, k, PLANE_THREADS, smem, plane_batches(a.n_cells), false, s,
                             a);
  }
  static cudaError_t diag_picard(const CellArgs<float> &a, int geo, cudaStream_t s, int sm)
  {
    return geo == 0 ? diag_picard_t<0>(a, s, sm) : diag_picard_t<1>(a, s, sm);
  }
  template <int GEO>
  static cudaError_t vmult_picard_rows_t(const CellArgs<float> &a, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    auto k = k_vmult2<n, float, GEO, 3, true>;
    const size_t smem = v2_smem<n, float, 3>();
    return launch_persistent(cache, k, PLANE_THREADS, smem, plane_batches(a.n_cells), false, s,
                             a);
  }
  static cudaError_t vmult_picard_rows(const CellArgs<float> &a, int geo, cudaStream_t s, int sm)
  {
    if constexpr (n == 4) {
      return geo == 0 ? vmult_picard_rows_t<0>(a, s, sm) : vmult_picard_rows_t<1>(a, s, sm);
    } else {
      (void)a, (void)geo, (void)s, (void)sm;
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t vmult_picard_tc(const CellArgs<float> &a, const float *gmat, int *err,
                                     cudaStream_t s, int sm)
  {
    if constexpr (n == 4) {
      static SharedLimit limit;
      auto k = k_vmult_picard_tc<n>;
      const cudaError_t e = limit.raise(k, optc::kSmem);
      if (e != cudaSuccess) return e;
      const int64_t nb = (int64_t)((a.d.m[0] + optc::kBX - 1) / optc::kBX) *
                         ((a.d.m[1] + optc::kBY - 1) / optc::kBY) *
                         ((a.d.m[2] + optc::kBZ - 1) / optc::kBZ);
      // one CTA per SM (two brick pipelines, 512 tensor-memory columns, ~161 KB shared)
      const int64_t nc = (nb + optc::kGroups - 1) / optc::kGroups;
      const int g = (int)std::min<int64_t>(nc, (int64_t)sm);
      k<<<g, optc::kThreads, optc::kSmem, s>>>(a, reinterpret_cast<const float4 *>(gmat), err);
      return cudaGetLastError();
    } else {
      (void)a, (void)gmat, (void)err, (void)s, (void)sm;
      return cudaErrorNotSupported;
    }
  }
  template <int GEO>
  static cudaError_t coef_tangent_t(const CellArgs<double> &a, double *out, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    auto k = k_coef_tangent<n, GEO>;
    const size_t smem = smem_coef_tangent<n>();
    return launch_persistent(cache, k, THREADS, smem, line_batches(a.n_cells), false, s, a, out);
  }
  static cudaError_t coef_tangent(const CellArgs<double> &a, double *out, int geo, cudaStream_t s,
                                  int sm)
  {
    return geo == 0 ? coef_tangent_t<0>(a, out, s, sm) : coef_tangent_t<1>(a, out, s, sm);
  }
  static cudaError_t coef_lineark(const CellArgs<double> &a, double *out, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    if constexpr (use_v2<double>()) {
      auto k = k_coef_lineark2<n>;
      constexpr size_t smem =
        sizeof(double) * kV2Warps * 2 * (v2_cells_per_warp<n>() + 1) * v2_cell_stride<n>();
      return launch_persistent(cache, k, PLANE_THREADS, smem, plane_batches(a.n_cells), false, s, a,
                               out);
    } else {
      auto k = k_coef_lineark<n>;
      const size_t smem = smem_coef_lineark<n>();
      return launch_persistent(cache, k, THREADS, smem, line_batches(a.n_cells), false, s, a, out);
    }
  }
  static cudaError_t field_values(const CellArgs<double> &a, const double *H, const double *vel,
                                  int64_t n_dofs, double *cf, cudaStream_t s, int sm)
  {
    static ResidentBlocks cache;
    auto k = k_field_values<n>;
    const size_t smem = smem_norm<n>();
    return launch_persistent(cache, k, THREADS, smem, line_batches(a.n_cells), false, s, a, H, vel,
                             n_dofs, cf);
  }
  static cudaError_t conductivity_q(const CellArgs<double> &a, float *kq, int law, cudaStream_t s,
                                    int sm)
  {
    if (law == 0) return kq_t<0>(a, kq, s, sm);
    if (law == 1) return kq_t<1>(a, kq, s, sm);
    return kq_t<2>(a, kq, s, sm);
  }

  static DegreeTable table()
  {
    DegreeTable t;
    t.n = n;
    t.upload = &upload;
    t.vmult_d = &vmult_d;
    t.vmult_f = &vmult_f;
    t.rhs = &rhs;
    t.diag = &diag;
    t.norm = &norm;
    t.coef_tangent = &coef_tangent;
    t.coef_lineark = &coef_lineark;
    t.field_values = &field_values;
    t.v2_d = use_v2<double>();
    t.v2_f = use_v2<float>();
    if constexpr (use_v2<float>()) {
      t.conductivity_q = &conductivity_q;
      t.diag_picard = &diag_picard;
    }
    if constexpr (n == 4) {
      t.vmult_picard_tc = &vmult_picard_tc;
      t.vmult_picard_rows = &vmult_picard_rows;
    }
    return t;
  }
};

}  // namespace mpdg

#define MPDG_DEFINE_DEGREE(N)                                            \
  namespace mpdg {                                                       \
  DegreeTable degree_table_##N() { return DegreeOps<N>::table(); }        \
  }
