// Weight gradients of the guess network's 3x3x3 convolutions,
// dW[co][ci][tap] = sum_p g[co][p] in[ci][p + shift(tap)], FP32 output gradients g, BF16 inputs,
// FP32 accumulation.
//
// A thread accumulates 4 output channels x 1 input channel x 27 taps in registers while it walks
// x-rows of its tile: per point 9 new inputs (the window slides) and 4 gradients come from shared
// memory for 108 FMAs, so the FMA pipe bounds the kernel (the first form kept 1 x 1 x 27
// accumulators and read 27 inputs per 27 FMAs, bound by shared memory: 16 -> 16 channels on 97^3
// points 1.88 ms, this one 0.36 ms, 12.6 GFLOP at 35 TFLOP/s; 16 -> 1 channel 1.81 -> 0.13 ms).
// Lanes are neighbouring input channels, stored contiguously per point, so the reads have no bank
// conflicts and the gradients are broadcast. Tensor cores were tried (an exact three-term BF16
// split of g): their FP32 accumulation truncates, and a walk of 32 tiles had 10 times this kernel's
// error against 64 bits (6e-7; the first form 1.1e-6).
//
// A CTA of 128 threads = CI input channels x CG groups of 4 output channels x PG row groups keeps
// its accumulators over a persistent walk of tiles, sums its row groups in shared memory and adds
// the result to dW once, with atomics (one set per CTA: with one per row group the 16 -> 1 layer
// took 0.40 ms); three CTAs per SM overlap one another's loads.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace nn_wg {

constexpr int kX = 15, kY = 4, kZ = 4;  // output tile; rows of kX points, kX a multiple of 3
constexpr int kHX = kX + 2, kHY = kY + 2, kHZ = kZ + 2, kHP = kHX * kHY * kHZ;
constexpr int kRows = kY * kZ;
constexpr int kThreads = 128;

struct Args {
  int nx, ny, nz;
  int ci, co;
  int ci_groups;  // blocks along the input channels; blockIdx.y = co block * ci_groups + ci block
  int up;         // the input is the coarse grid (sx, sy, sz), read nearest-neighbour
  int sx, sy, sz;
  const __nv_bfloat16 *in;  // [ceil(ci / 8)][points][8]
  const float *g;           // [co][points]
  float *dw, *db;           // [co][ci][27], [co]
};

template <int CI> __host__ __device__ constexpr int in_stride() { return CI; }
template <int CG> __host__ __device__ constexpr int g_stride() { return 4 * CG + 4; }
template <int CI, int CG> __host__ __device__ constexpr size_t smem_bytes()
{
  return sizeof(float) * ((size_t)kHP * in_stride<CI>() + (size_t)kRows * kX * g_stride<CG>());
}

template <int CI, int CG>
__global__ void __launch_bounds__(kThreads, 3) k_wgrad(const Args a)
{
  constexpr int PG = kThreads / (CI * CG), IS = in_stride<CI>(), GS = g_stride<CG>();
  static_assert(kRows % PG == 0, "whole rows per row group");
  static_assert(smem_bytes<CI, CG>() >= sizeof(float) * 27 * kThreads, "the final reduction's space");
  extern __shared__ __align__(16) float smem[];
  float *s_in = smem, *s_g = smem + kHP * IS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ci_l = tid % CI, cg = (tid / CI) % CG, pg = tid / (CI * CG);
  const int ci0 = (blockIdx.y % a.ci_groups) * CI, co0 = (blockIdx.y / a.ci_groups) * 4 * CG;
  const int64_t np = (int64_t)a.nx * a.ny * a.nz;
  const int64_t snp = a.up ? (int64_t)a.sx * a.sy * a.sz : np;
  const int tiles_x = (a.nx + kX - 1) / kX, tiles_y = (a.ny + kY - 1) / kY,
            tiles_z = (a.nz + kZ - 1) / kZ;
  const int64_t n_tiles = (int64_t)tiles_x * tiles_y * tiles_z;
  float acc[4][27];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int o = 0; o < 27; ++o) acc[c][o] = 0.f;
  // the bias gradient: a warp's share of the block's output channels
  constexpr int CW = CG;  // 4 CG channels over 4 warps
  const bool want_bias = ci0 == 0;
  float bias[CW];
#pragma unroll
  for (int c = 0; c < CW; ++c) bias[c] = 0.f;

  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int bx = (int)(tile % tiles_x) * kX;
    const int by = (int)((tile / tiles_x) % tiles_y) * kY;
    const int bz = (int)(tile / ((int64_t)tiles_x * tiles_y)) * kZ;
    __syncthreads();  // the last tile's reads
    // inputs with halo, zero outside the grid: 8 channels of a point per 16-byte vector
    constexpr int CH = CI >= 8 ? CI / 8 : 1;
    const uint4 *src = reinterpret_cast<const uint4 *>(a.in);
    for (int i = tid; i < kHP * CH; i += kThreads) {
      const int hp = i % kHP, c = i / kHP;
      const int gx = bx + hp % kHX - 1, gy = by + (hp / kHX) % kHY - 1,
                gz = bz + hp / (kHX * kHY) - 1;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (ci0 + 8 * c < a.ci && gx >= 0 && gx < a.nx && gy >= 0 && gy < a.ny && gz >= 0 &&
          gz < a.nz) {
        const int64_t p = a.up ? (gx >> 1) + (int64_t)a.sx * ((gy >> 1) + (int64_t)a.sy * (gz >> 1))
                               : gx + (int64_t)a.nx * (gy + (int64_t)a.ny * gz);
        v = __ldg(src + (int64_t)(ci0 / 8 + c) * snp + p);
      }
      float4 lo, hi;  // a BF16 value is the upper half of its FP32 one
      lo.x = __uint_as_float(v.x << 16);
      lo.y = __uint_as_float(v.x & 0xffff0000u);
      lo.z = __uint_as_float(v.y << 16);
      lo.w = __uint_as_float(v.y & 0xffff0000u);
      hi.x = __uint_as_float(v.z << 16);
      hi.y = __uint_as_float(v.z & 0xffff0000u);
      hi.z = __uint_as_float(v.w << 16);
      hi.w = __uint_as_float(v.w & 0xffff0000u);
      float4 *o = reinterpret_cast<float4 *>(s_in + hp * IS + 8 * c);
      o[0] = lo;
      if (CI >= 8) o[1] = hi;
    }
    // gradients, zero outside the grid, [row][x][channel]
    for (int i = lane; i < kRows * kX; i += 32) {
      const int x = bx + i % kX, r = i / kX, y = by + r % kY, z = bz + r / kY;
      const bool inside = x < a.nx && y < a.ny && z < a.nz;
      const int64_t p = x + (int64_t)a.nx * (y + (int64_t)a.ny * z);
#pragma unroll
      for (int c = 0; c < CW; ++c) {
        const int cl = warp * CW + c;
        const float v = inside && co0 + cl < a.co ? __ldg(a.g + (int64_t)(co0 + cl) * np + p) : 0.f;
        s_g[i * GS + cl] = v;
        bias[c] += v;
      }
    }
    __syncthreads();
    const int nv = a.nx - bx < kX ? a.nx - bx : kX;  // points of a row inside the grid
    for (int rr = 0; rr < kRows / PG; ++rr) {
      const int r = rr * PG + pg, ry = r % kY, rz = r / kY;
      if (by + ry >= a.ny || bz + rz >= a.nz) continue;
      const float *ip = s_in + ((rz * kHY + ry) * kHX) * IS + ci_l;
      const float *gp = s_g + r * kX * GS + 4 * cg;
      float w[3][9];  // the window's x-columns, column x in w[x % 3]
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        w[0][q] = ip[((q / 3 * kHY + q % 3) * kHX + 0) * IS];
        w[1][q] = ip[((q / 3 * kHY + q % 3) * kHX + 1) * IS];
      }
      for (int x0 = 0; x0 < nv; x0 += 3) {  // (past the grid's end the gradients are zero)
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          float(&wn)[9] = w[(u + 2) % 3];
#pragma unroll
          for (int q = 0; q < 9; ++q) wn[q] = ip[((q / 3 * kHY + q % 3) * kHX + x0 + u + 2) * IS];
          const float4 g4 = *reinterpret_cast<const float4 *>(gp + (x0 + u) * GS);
          const float gv[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
          for (int q = 0; q < 9; ++q)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
#pragma unroll
              for (int c = 0; c < 4; ++c)
                acc[c][dx + 3 * q] = fmaf(gv[c], w[(u + dx) % 3][q], acc[c][dx + 3 * q]);
        }
      }
    }
  }
  // sum the row groups in shared memory, then one atomic per weight and CTA
  constexpr int NW = CI * CG;  // threads of a row group
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    __syncthreads();
#pragma unroll
    for (int o = 0; o < 27; ++o) smem[o * kThreads + tid] = acc[c][o];
    __syncthreads();
    for (int i = tid; i < 27 * NW; i += kThreads) {
      const int t = i % NW, o = i / NW, ci = ci0 + t % CI, co = co0 + 4 * (t / CI) + c;
      float v = 0.f;
#pragma unroll
      for (int g = 0; g < PG; ++g) v += smem[o * kThreads + g * NW + t];
      if (co < a.co && ci < a.ci) atomicAdd(a.dw + ((int64_t)co * a.ci + ci) * 27 + o, v);
    }
  }
  if (want_bias) {
#pragma unroll
    for (int c = 0; c < CW; ++c) {
      float v = bias[c];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      const int co = co0 + warp * CW + c;
      if (lane == 0 && co < a.co) atomicAdd(a.db + co, v);
    }
  }
}

}  // namespace nn_wg
