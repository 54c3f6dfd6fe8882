// Layout of the float32 slabs that the gradWeights kernels write and the reduction kernels add up.
//
// One slab per split-K slice, taps * K * Cg elements (K: filters of all groups, Cg: channels per group):
//
//   [tap][channel / 4][filter][channel % 4]        (the last channels of a count that is no multiple of four: [filter][Cg % 4])
//
// An accumulator row is a TMEM lane: a warp reads 32 filters of 32 channels.  With the filter next to the innermost four
// channels each of its 16-byte stores covers 512 bytes in a row.  With a filter's channels in a row (the order of the
// result) every lane wrote its own 128-byte line in eight pieces of half a sector, and the read-out took 18000 of a CTA's
// 85000 clocks on 128 -> 128 filters 3x3 at 28x28 (256 images, float16), now 7500: 62 -> 59 us with the reduction.
#pragma once
#include "internal.h"
#include "ptx.cuh"

namespace b200 {

// Offset in a slab of channel c (within its group) of filter k (of all filters), tap t.
__host__ __device__ __forceinline__ long long slab_index(int t, int k, int c, int K, int Cg) {
  const int c4 = c & ~3, w = Cg - c4 < 4 ? Cg - c4 : 4;
  return 1LL * t * K * Cg + 1LL * c4 * K + 1LL * k * w + (c & 3);
}

// Channels wanted of filter kq (within its group): all, or the filter's block of merged groups of diag_k filters x diag_c channels.
__device__ __forceinline__ void diagonal_range(int diag_c, int diag_k, int kq, int Cg, int* lo, int* hi) {
  *lo = diag_c ? kq / diag_k * diag_c : 0;
  *hi = diag_c ? *lo + diag_c : Cg;
}

// Stores 32 channels from c0 on of one filter row; `slab` is the slice's slab plus its tap's offset, row k of K.
// [c_lo, c_hi): the channels that are wanted (block-diagonal filters want a part only).
__device__ __forceinline__ void store_slab_chunk(const uint32_t (&r)[32], float* slab, int c0, int c_lo, int c_hi, int Cg, int K, int k,
                                                 bool atomic, const float* partial, long long partial_elems, int* status) {
  const bool vec = ((1LL * K * Cg) & 3) == 0 && !atomic;
  if (vec && c_lo <= c0 && c0 + 32 <= c_hi) {               // whole: one address, K pieces apart (c_hi <= Cg)
    float* dst = slab + 1LL * c0 * K + 4LL * k;
    if (!B200_IN_RANGE(dst - partial >= 0 && (dst - partial) + 28LL * K + 4 <= partial_elems, status)) return;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      reinterpret_cast<float4*>(dst)[static_cast<unsigned>(j) * static_cast<unsigned>(K)] =
          make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
    return;
  }
#pragma unroll
  for (int j = 0; j < 32; j += 4) {
    const int c = c0 + j, w = min(4, Cg - c);
    if (c + 4 <= c_lo || c >= c_hi) continue;
    float* dst = slab + 1LL * c * K + 1LL * k * w;
    if (!B200_IN_RANGE(dst - partial >= 0 && (dst - partial) + w <= partial_elems, status)) continue;
    if (vec && w == 4) {
      *reinterpret_cast<float4*>(dst) =
          make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= w) continue;
        if (atomic) atomicAdd(dst + q, __uint_as_float(r[j + q]));
        else dst[q] = __uint_as_float(r[j + q]);
      }
    }
  }
}

}  // namespace b200
