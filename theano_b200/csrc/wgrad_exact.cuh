// Filter gradients of inputs with infinities or NaN.
//
// The gradWeights kernels cut the images into tiles of fixed shape and let zeros stand for the pixels of dy that a tile has too many:
// behind the last column or row, and in wgrad_rows.cu above the first one.  Those zeros meet real pixels of x.  A zero times a
// finite number adds nothing, but times an infinity or NaN it is NaN: an infinity in the last column of an image would make NaN
// of filter taps that never touch it, depending on which kernel runs.  So the reduction kernels take a sum that comes out NaN again,
// over the products that belong to it.  x outside of the image counts as zeros that take part, as in the reference's im2col form
// (theano/tensor/nnet/c_code/corr_gemm.c:31): an infinity in dy makes NaN of the taps that lie outside there.
//
// All finite: one comparison per sum.  Else warps look at the border of the channels that have a NaN: where it is finite the NaN
// is the sum's own, and stays.  Only where it is not, the sum is taken again, in double precision, up to the first product that is NaN.
// 64 -> 64 filters 3x3, 256 images of 56 x 56, float16 (77 us, finite): an infinity in dy 87 us, a NaN in dy 1.3 ms, all of x NaN 0.13 ms; an
// infinity at two borders of one channel 0.36 s, at two borders of every channel 0.5 s (256 -> 256 at 14x14, 128 images: 11 and 29 ms).
#pragma once
#include "internal.h"

namespace b200 {

// The code is inlined at the end of the kernels and kept short, without calls, stack or loops unrolled: what it adds to a kernel costs every
// launch, run or not (64 -> 64 3x3 at 28x28, 8 images, float16 gradWeights 8.88 us without it, 9.38 with twice the instructions or in
// functions, 8.97 as it is).
__device__ __forceinline__ float exact_load(const void* base, long long at, int f16) {
  return f16 ? __half2float(static_cast<const __half*>(base)[at]) : static_cast<const float*>(base)[at];
}

// Does channel c (of all groups) hold an infinity or NaN among the pixels that some tap does not reach: rows above the last tap's first
// one, below the first tap's last one, columns alike?  No others meet zeros that stand for dy, unless those stand behind pieces of rows
// (then all pixels count).  A whole warp.
__device__ __forceinline__ bool border_not_finite(const WgradSum& s, int c) {
  const int top = s.segments ? s.H : max(0, min(s.H, (s.kH - 1) * s.dilH - s.padH)), bottom = max(top, min(s.H, (s.Ho - 1) * s.sH - s.padH + 1));
  const int left = max(0, min(s.W, (s.kW - 1) * s.dilW - s.padW)), right = max(left, min(s.W, (s.Wo - 1) * s.sW - s.padW + 1));
  const unsigned cols = left + s.W - right, whole = static_cast<unsigned>(top + s.H - bottom) * s.W;      // whole rows, then columns of the others
#pragma unroll 1
  for (int n = 0; n < s.N; ++n) {
    bool found = false;
#pragma unroll 1
    for (unsigned p = threadIdx.x & 31; p < whole + (bottom - top) * cols; p += 32) {
      const bool row = p < whole;
      const unsigned q = row ? p : p - whole, width = row ? s.W : cols;
      int h = q / width, w = q - h * width;
      h += row ? (h >= top ? bottom - top : 0) : top;
      w += !row && w >= left ? right - left : 0;
      found |= !isfinite(exact_load(s.x, c * s.x_c + n * s.x_n + h * s.x_h + w * s.x_w, s.f16));
    }
    if (__any_sync(0xffffffffu, found)) return true;
  }
  return false;
}

// Sum of filter k and channel c (of all groups), filter element (i, j) in correlation order; a whole warp, the result in every lane.
__device__ __forceinline__ float exact_sum(const WgradSum& s, int k, int c, int i, int j) {
  int ow = (threadIdx.x & 31) - 32, oh = 0, n = 0;          // pixels lane, lane + 32, ...
  double sum = 0.;
#pragma unroll 1
  do {
    float a[2], b[2];                                       // loaded together
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      for (ow += 32; ow >= s.Wo; ow -= s.Wo)
        if (++oh == s.Ho) { oh = 0; ++n; }
      const int h = oh * s.sH + i * s.dilH - s.padH, w = ow * s.sW + j * s.dilW - s.padW;
      const bool on = n < s.N, inside = on && h >= 0 && h < s.H && w >= 0 && w < s.W;
      a[u] = on ? exact_load(s.dy, k * s.dy_c + n * s.dy_n + oh * s.dy_h + ow * s.dy_w, s.f16) : 0.f;
      b[u] = inside ? exact_load(s.x, c * s.x_c + n * s.x_n + h * s.x_h + w * s.x_w, s.f16) : 0.f;
    }
    sum += static_cast<double>(a[0]) * static_cast<double>(b[0]) + static_cast<double>(a[1]) * static_cast<double>(b[1]);
    if (__any_sync(0xffffffffu, isnan(sum))) break;         // the rest does not matter
  } while (__any_sync(0xffffffffu, n < s.N));
#pragma unroll 1
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  return static_cast<float>(sum);
}

// The NaN among a tile of sums of a block: filters k0 on, `pitch` apart, channels c0 on (of their groups) x taps in OIHW order.
__device__ __forceinline__ void exact_tile(const WgradSum& s, float* tile, int rows, int pitch, int channels, int k0, int c0) {
  const int taps = s.kH * s.kW, warps = blockDim.x >> 5, parts = max(1, warps / channels);      // warps per channel
#pragma unroll 1
  for (int unit = threadIdx.x >> 5; unit < channels * parts; unit += warps) {
    const int ch = unit / parts;
    int looked = -1;                                        // the group whose channel has been looked at
    bool suspect = false;
#pragma unroll 1
    for (int q = unit - ch * parts; q < rows * taps; q += parts) {
      const int row = q / taps, t = q - row * taps, k = k0 + row, g = k / s.Kg, c = g * s.Cg + c0 + ch;
      float* v = tile + row * pitch + ch * taps + t;
      if (!isnan(*v)) continue;
      if (g != looked) suspect = border_not_finite(s, c);
      looked = g;
      if (!suspect) continue;
      const int i = t / s.kW, j = t - i * s.kW;
      const float sum = exact_sum(s, k, c, s.flip ? s.kH - 1 - i : i, s.flip ? s.kW - 1 - j : j);
      if ((threadIdx.x & 31) == 0) *v = sum;
    }
  }
  __syncthreads();
}

}  // namespace b200
