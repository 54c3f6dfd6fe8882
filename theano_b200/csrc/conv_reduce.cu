// Second half of a forward / gradInputs launch whose reduction is split over CTAs.
//
// A layer with few output tiles (a small batch, the deep end of a network) leaves most SMs idle and
// walks a long reduction on the rest: 512 -> 512 filters 3x3 on one 14 x 14 image is 4 tiles of 144
// steps.  The convolution kernels then cut the reduction into slices, one work item per (tile, slice),
// and store float32 accumulators in slabs
//   partial[tile][slice][column / 4][row][4]          (row = accumulator lane of the tile)
// which both sides read and write in runs of 512 bytes.  This kernel adds the slices in order (the
// result does not depend on scheduling), applies the epilogue and writes the output.  Few bytes per thread and a dozen quotients to
// find its place: it was bound by integer divisions (a third of the instructions of a launch over 64 tiles of 128 x 256), and,
// where few tiles were split, by loads one after the other (a loop unrolled by eight takes five slices singly).  Now the host
// brings reciprocals, and the loads of up to eight slices, or of four slices of 16 columns, are in flight together.
// Convolution and reduction together (float32, one image, before -> now): 256 -> 512 3x3 at 28x28 14.8 -> 12.3 us, 512 -> 512 17.8 -> 15.2, with
// pooling 22.3 -> 19.8, 512 -> 512 at 14x14 12.7 -> 11.6, with pooling 15.5 -> 13.3.
#include "internal.h"
#include "ptx.cuh"

#include <algorithm>

namespace b200 {
namespace {

template <typename T> __device__ __forceinline__ float to_f(T v) { return static_cast<float>(v); }

constexpr int kReduceThreads = 128;

// How a launch is walked: units of (pixel tile, 32 rows, columns of a block).
struct ReduceWalk {
  Divisor row_chunks, col_blocks, per_w, per_h, tiles_w, tiles_h, tiles_co, groups;
  int units;
};

// One warp: 32 rows (a lane a row; pooled: a lane a 2x2 window) x 4 * QW columns; a block: four such side by side.
template <typename T, bool POOL, int QW>
__global__ void __launch_bounds__(kReduceThreads) conv_reduce_kernel(const __grid_constant__ ConvReduceParams p, const __grid_constant__ ReduceWalk walk) {
  constexpr int PL = POOL ? 2 : 1, ROWS = PL * PL, BATCH = 8 / (QW * ROWS) > 4 ? 8 : 4;
  pdl_enter();
  const long long slab = 1LL * p.rows * (p.bn_cols / 4);    // float4s of one slice
  const bool wide = p.out_sc == 1 && ((p.n_out * sizeof(T) | reinterpret_cast<uintptr_t>(p.out)) & 15) == 0;   // four columns are all in
  for (uint32_t unit = blockIdx.x; unit < static_cast<uint32_t>(walk.units); unit += gridDim.x) {
    const uint32_t u = quotient(unit, walk.col_blocks), cb = unit - u * walk.col_blocks.d;
    const uint32_t z = quotient(u, walk.row_chunks), idx = (u - z * walk.row_chunks.d) * 32 + (threadIdx.x & 31);
    const uint32_t tile = p.pair ? z >> 1 : z;
    const uint32_t tg = quotient(tile, walk.tiles_co), co_t = tile - tg * walk.tiles_co.d, tp = quotient(tg, walk.groups), g = tg - tp * walk.groups.d;
    const uint32_t pt = p.pair ? tp * 2 + (z & 1) : tp;
    const uint32_t th = quotient(pt, walk.tiles_w), tn = quotient(th, walk.tiles_h);
    const uint32_t ih = quotient(idx, walk.per_w), ni = quotient(ih, walk.per_h);
    const int ww = idx - ih * walk.per_w.d, hh = ih - ni * walk.per_h.d;
    const int w = (pt - th * walk.tiles_w.d) * walk.per_w.d + ww, h = (th - tn * walk.tiles_h.d) * walk.per_h.d + hh, n = tn * p.nb + ni;
    const int q0 = (cb * 4 + (threadIdx.x >> 5)) * QW, c0 = co_t * p.bn_cols + q0 * 4;          // c0: within the group
    if (static_cast<int>(ni) >= p.nb || w >= p.Wt / PL || h >= p.Ht / PL || n >= p.Nimg || q0 * 4 >= p.bn_cols || c0 >= p.n_out) continue;
    const int row = (ni * p.Hs + hh * PL) * p.Ws + ww * PL;
    const float4* base = reinterpret_cast<const float4*>(p.partial) + 1LL * z * p.splits * slab + 1LL * q0 * p.rows + row;
    const int qs = min(QW, min(p.bn_cols / 4 - q0, (p.n_out - c0 + 3) / 4));                     // groups of four columns that are there
    float4 acc[QW][ROWS];
#pragma unroll
    for (int q = 0; q < QW; ++q)
#pragma unroll
      for (int k = 0; k < ROWS; ++k) acc[q][k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!B200_IN_RANGE((reinterpret_cast<const float*>(base + (p.splits - 1) * slab + (qs - 1) * p.rows + (PL - 1) * (p.Ws + 1)) - p.partial) + 4 <= p.partial_elems, p.status)) continue;
    for (int s0 = 0; s0 < p.splits; s0 += BATCH) {
      float4 v[BATCH][QW][ROWS];
#pragma unroll
      for (int b = 0; b < BATCH; ++b)
#pragma unroll
        for (int q = 0; q < QW; ++q)
#pragma unroll
          for (int k = 0; k < ROWS; ++k)
            if (s0 + b < p.splits && q < qs) v[b][q][k] = __ldcg(base + (s0 + b) * slab + q * p.rows + (k >> 1) * p.Ws + (k & 1));
#pragma unroll
      for (int b = 0; b < BATCH; ++b) {
        if (s0 + b >= p.splits) break;
#pragma unroll
        for (int q = 0; q < QW; ++q)
#pragma unroll
          for (int k = 0; k < ROWS; ++k) {
            acc[q][k].x += v[b][q][k].x; acc[q][k].y += v[b][q][k].y; acc[q][k].z += v[b][q][k].z; acc[q][k].w += v[b][q][k].w;
          }
      }
    }
    long long at = p.out_off + n * p.out_sn + h * p.out_sh + w * p.out_sw + (1LL * g * p.n_out + c0) * p.out_sc;
#pragma unroll
    for (int q = 0; q < QW; ++q, at += 4 * p.out_sc) {
      if (q >= qs) break;
      const int c = c0 + 4 * q;
      float best[4];
#pragma unroll
      for (int k = 0; k < ROWS; ++k) {
        const float v[4] = {acc[q][k].x, acc[q][k].y, acc[q][k].z, acc[q][k].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (c + e >= p.n_out) continue;
          float f = p.epi.alpha * (c + e < p.n_real ? v[e] : 0.f);       // pad channels: 0 x infinity is NaN
          if (p.bias) f += to_f(static_cast<const T*>(p.bias)[g * p.n_out + c + e]);
          if (p.epi.residual && c + e < p.n_real) f += p.epi.beta * to_f(static_cast<const T*>(p.epi.residual)[at + e * p.out_sc]);
          if (p.relu) f = p.epi.lin * f + p.epi.abs * fabsf(f);
          // pooling compares stored values, as the unsplit epilogue does
          f = to_f(static_cast<T>(f));
          best[e] = k == 0 ? f : fmaxf(best[e], f);
        }
      }
      T* out = static_cast<T*>(p.out) + at;
      const long long last = at + ((c + 4 < p.n_out ? 4 : p.n_out - c) - 1) * p.out_sc;
      if (!B200_IN_RANGE(at >= 0 && last < p.out_elems, p.status)) continue;
      if (wide) {
        if (sizeof(T) == 4) {
          *reinterpret_cast<float4*>(out) = make_float4(best[0], best[1], best[2], best[3]);
        } else {
          __half2 h2[2] = {__floats2half2_rn(best[0], best[1]), __floats2half2_rn(best[2], best[3])};
          *reinterpret_cast<uint2*>(out) = *reinterpret_cast<uint2*>(h2);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c + e < p.n_out) out[e * p.out_sc] = static_cast<T>(best[e]);
      }
    }
  }
}

}  // namespace

// 16 columns per thread where that leaves every SM eight warps, else four.
cudaError_t launch_conv_reduce(const ConvReduceParams& p, int dtype, cudaStream_t s) {
  const int pl = p.epi.pool ? 2 : 1, cols = p.n_out < p.bn_cols ? p.n_out : p.bn_cols;
  const long long tiles = p.pair ? 2LL * p.tiles : p.tiles, rows = cdiv((p.wt / pl) * (p.th / pl) * p.nb, 32);
  if (tiles == 0 || rows == 0) return cudaSuccess;
  const bool many = !p.epi.pool && tiles * rows * cdiv(cols, 16) >= 8 * kB200Sms;
  const long long col_blocks = cdiv(cols, many ? 64 : 16), units = tiles * rows * col_blocks;
  if (units >= (1LL << 30)) return cudaErrorInvalidValue;
  ReduceWalk walk;
  walk.row_chunks = divisor(static_cast<uint32_t>(rows)); walk.col_blocks = divisor(static_cast<uint32_t>(col_blocks));
  walk.per_w = divisor(p.wt / pl); walk.per_h = divisor(p.th / pl);
  walk.tiles_w = divisor(p.tiles_w); walk.tiles_h = divisor(p.tiles_h); walk.tiles_co = divisor(p.tiles_co); walk.groups = divisor(p.groups);
  walk.units = static_cast<int>(units);
  const unsigned grid = static_cast<unsigned>(std::min<long long>(units, kChainedBlocks));
  const bool f16 = dtype == B200CONV_F16;
  auto launch = [&](auto kernel) { return launch_streaming(kernel, grid, kReduceThreads, 0, s, p, walk); };
  if (p.epi.pool) return f16 ? launch(conv_reduce_kernel<__half, true, 1>) : launch(conv_reduce_kernel<float, true, 1>);
  if (many) return f16 ? launch(conv_reduce_kernel<__half, false, 4>) : launch(conv_reduce_kernel<float, false, 4>);
  return f16 ? launch(conv_reduce_kernel<__half, false, 1>) : launch(conv_reduce_kernel<float, false, 1>);
}

}  // namespace b200
