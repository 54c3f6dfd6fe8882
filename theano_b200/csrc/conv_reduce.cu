// Second half of a forward / gradInputs launch whose reduction is split over CTAs.
//
// A layer with few output tiles (a small batch, the deep end of a network) leaves most SMs idle and
// walks a long reduction on the rest: 512 -> 512 filters 3x3 on one 14 x 14 image is 4 tiles of 144
// steps.  The convolution kernels then cut the reduction into slices, one work item per (tile, slice),
// and store float32 accumulators in slabs
//   partial[tile][slice][column / 4][row][4]          (row = accumulator lane of the tile)
// which both sides read and write in runs of 512 bytes.  This kernel adds the slices in order (the
// result does not depend on scheduling), applies the epilogue and writes the output.  It is bound by the
// latency of its loads (all slices of a thread are in flight together) and runs on all SMs.
#include "internal.h"
#include "ptx.cuh"

namespace b200 {
namespace {

template <typename T> __device__ __forceinline__ float to_f(T v) { return static_cast<float>(v); }

// Adds the slices of four columns of one row.
__device__ __forceinline__ float4 sum_slices(const float4* src, int slices, long long stride) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int s = 0; s < slices; ++s) {
    const float4 v = __ldcg(src + s * stride);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  return acc;
}

// One thread per (row, four columns); with pooling one per (2x2 window, four columns).  Block: 64 rows x 4
// column groups, so that a block writes 64 bytes per pixel.
template <typename T>
__global__ void __launch_bounds__(256) conv_reduce_kernel(const __grid_constant__ ConvReduceParams p) {
  pdl_enter();
  const int row_t = threadIdx.x & 63, q = blockIdx.y * 4 + (threadIdx.x >> 6);
  const uint32_t tile = blockIdx.z;
  const int pl = p.epi.pool ? 2 : 1;
  const int per_w = p.wt / pl, per_h = p.th / pl;
  const int idx = blockIdx.x * 64 + row_t;                  // dense index over the tile's (pooled) pixels
  if (idx >= per_w * per_h * p.nb || q * 4 >= p.bn_cols) return;
  const int ww = idx % per_w, hh = (idx / per_w) % per_h, ni = idx / (per_w * per_h);
  const int co_t = tile % static_cast<uint32_t>(p.tiles_co), g = tile / p.tiles_co % p.groups;
  const uint32_t pt = tile / (p.tiles_co * p.groups);
  const int w = (pt % p.tiles_w) * per_w + ww, h = (pt / p.tiles_w % p.tiles_h) * per_h + hh;
  const int n = pt / (p.tiles_w * p.tiles_h) * p.nb + ni;
  const int c0 = co_t * p.bn_cols + q * 4;                  // within the group
  if (w >= p.Wt / pl || h >= p.Ht / pl || n >= p.Nimg || c0 >= p.n_out) return;
  const long long slab = 1LL * p.rows * (p.bn_cols / 4);    // float4s of one slice
  const float4* base = reinterpret_cast<const float4*>(p.partial) + tile * p.splits * slab + 1LL * q * p.rows;
  T* out = static_cast<T*>(p.out) + p.out_off + n * p.out_sn + h * p.out_sh + w * p.out_sw + (1LL * g * p.n_out + c0) * p.out_sc;
  float best[4];
  for (int k = 0; k < pl * pl; ++k) {
    const int row = (ni * p.Hs + hh * pl + (k >> 1)) * p.Ws + ww * pl + (k & 1);
    if (!B200_IN_RANGE((reinterpret_cast<const float*>(base + row + (p.splits - 1) * slab) - p.partial) + 4 <= p.partial_elems, p.status)) return;
    const float4 a = sum_slices(base + row, p.splits, slab);
    const float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (c0 + e >= p.n_out) continue;
      float f = p.epi.alpha * (c0 + e < p.n_real ? v[e] : 0.f);       // pad channels: 0 x infinity is NaN
      if (p.bias) f += to_f(static_cast<const T*>(p.bias)[g * p.n_out + c0 + e]);
      if (p.epi.residual && c0 + e < p.n_real) f += p.epi.beta * to_f(static_cast<const T*>(p.epi.residual)[(out - static_cast<T*>(p.out)) + e * p.out_sc]);
      if (p.relu) f = p.epi.lin * f + p.epi.abs * fabsf(f);
      // pooling compares stored values, as the unsplit epilogue does
      f = to_f(static_cast<T>(f));
      best[e] = k == 0 ? f : fmaxf(best[e], f);
    }
  }
  const long long at = out - static_cast<T*>(p.out), last = at + ((c0 + 4 < p.n_out ? 4 : p.n_out - c0) - 1) * p.out_sc;
  if (!B200_IN_RANGE(at >= 0 && last < p.out_elems, p.status)) return;
  if (p.out_sc == 1 && ((p.n_out * sizeof(T) | reinterpret_cast<uintptr_t>(p.out)) & 15) == 0) { // four columns are all in
    if (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(out) = make_float4(best[0], best[1], best[2], best[3]);
    } else {
      __half2 h2[2] = {__floats2half2_rn(best[0], best[1]), __floats2half2_rn(best[2], best[3])};
      *reinterpret_cast<uint2*>(out) = *reinterpret_cast<uint2*>(h2);
    }
    return;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (c0 + e < p.n_out) out[e * p.out_sc] = static_cast<T>(best[e]);
}

}  // namespace

cudaError_t launch_conv_reduce(const ConvReduceParams& p, int dtype, cudaStream_t s) {
  const int pl = p.epi.pool ? 2 : 1;
  const long long tiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n * p.groups * p.tiles_co;
  if (tiles == 0) return cudaSuccess;
  if (tiles > 65535) return cudaErrorInvalidValue;
  const int cols = p.n_out < p.bn_cols ? p.n_out : p.bn_cols;
  const dim3 grid(((p.wt / pl) * (p.th / pl) * p.nb + 63) / 64, (cols + 15) / 16, static_cast<unsigned>(tiles));
  if (dtype == B200CONV_F16) return launch_streaming(conv_reduce_kernel<__half>, grid, 256, 0, s, p);
  return launch_streaming(conv_reduce_kernel<float>, grid, 256, 0, s, p);
}

}  // namespace b200
