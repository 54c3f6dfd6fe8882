// Memory-bound helper kernels: NCHW <-> channels-last transposes, filter packing for the
// implicit-GEMM kernels, bias conversion, 2x2 max pooling and the L2 flush.
#include <algorithm>

#include "internal.h"
#include "wgrad_exact.cuh"
#include "wgrad_slab.cuh"

namespace b200 {
namespace {

// in[b][r][s] -> out[b][s][r]; 32x32 tiles through shared memory so that both the read
// (along s) and the write (along r) are coalesced.  Rows r in [R, ld_out) are zero filled.
template <typename T>
__global__ void transpose_kernel(const T* __restrict__ in, T* __restrict__ out, int R, int S,
                                 int ld_in, int ld_out) {
  pdl_enter();
  __shared__ T tile[32][33];
  const long long b = blockIdx.z;
  const T* src = in + b * R * ld_in;
  T* dst = out + b * S * ld_out;
  const int r0 = blockIdx.y * 32, s0 = blockIdx.x * 32;
  for (int dr = threadIdx.y; dr < 32; dr += blockDim.y) {
    const int r = r0 + dr, s = s0 + threadIdx.x;
    tile[dr][threadIdx.x] = (r < R && s < S) ? src[1LL * r * ld_in + s] : T(0);
  }
  __syncthreads();
  for (int ds = threadIdx.y; ds < 32; ds += blockDim.y) {
    const int s = s0 + ds, r = r0 + threadIdx.x;
    if (s < S && r < ld_out) dst[1LL * s * ld_out + r] = tile[threadIdx.x][ds];
  }
}

// Filters OIHW w[K][Cg][kH][kW] -> dst[(tap*groups + g)][rows][ldc] (zero padded columns):
//   mode 0 (forward):        rows = filters of the group, cols = channels,
//                            tap t = i*kW + j multiplies the pixel at offset (i, j);
//   mode 1 (input gradient): rows = channels, cols = filters of the group.
// With flip the correlation tap t reads position taps - 1 - t of the filter.  With `merge` neighbouring groups as one, the
// bank is that of the layer's own groups and the packed form block-diagonal: a filter has channels of its own group only.
// A block moves a patch of filters x channels with all its taps through shared memory: the taps of a filter's consecutive
// channels are one run of OIHW, read in 16-byte pieces (elements at the ends of a run that lies off the 16-byte
// boundaries, all on their way together: one after the other they took eight latencies), and leave as 16-byte pieces of the destination's rows.  Every call on its own filters waits for this kernel, and
// what bounds it is latency: one round of loads (up to four pieces per thread) and one of stores.  Element by element it took
// 10 rounds of each.  Forward / gradInputs calls with the packing (a B200, before -> now): 64 -> 64 3x3 at 28x28, 8 images, float16 9.6 -> 9.1 /
// 11.9 -> 9.6 us; 100 -> 75 5x5, 37 images, float16 37.5 -> 28.5 / 35.4 -> 27.4; 256 -> 256 3x3 at 14x14, 128 images, float32 60.5 -> 56 / 66 -> 59.
// All banks of ResNet-50 in one launch (float16, both forms, 47 MB) 138 -> 65 us, of the VGG-16 stack (float32, 49 MB) 102 -> 80.
constexpr int kPackThreads = 256, kPackPieces = 4, kPackMaxK = 64;
template <typename T>
__device__ __forceinline__ void pack_filters_block(const PackJob& q, int bx, int by, int g) {
  extern __shared__ uint4 pack_smem[];
  __shared__ int4 row_of[kPackMaxK];            // per filter of the patch: shared-memory offset of (channel c0, tap 0), its channels [y, z)
  uint8_t* tile = reinterpret_cast<uint8_t*>(pack_smem);
  constexpr int V = 16 / static_cast<int>(sizeof(T));
  const int taps = q.taps, Kg = q.K / q.groups, Cs = q.Cg / q.merge, Ks = Kg / q.merge;
  const int k0 = by << q.log_k, c0 = bx << q.log_c, c_end = min(c0 + (1 << q.log_c), q.Cg), pitch = q.pieces * 16;
  const int nk = min(1 << q.log_k, Kg - k0);                   // <= 0 in patches that only pad
  const T* w = static_cast<const T*>(q.src);
  // channels of filter k0 + kk in this patch, and where they start
  auto run_of = [&](int kk, int* a, int* b) {
    const int k = k0 + kk, lo = q.merge > 1 ? k / Ks * Cs : 0;
    *a = max(c0, lo);
    *b = max(*a, min(c_end, lo + Cs));
    return w + ((1LL * g * Kg + k) * Cs + *a - lo) * taps;
  };
  if (threadIdx.x < (1 << q.log_k)) {
    int a = 0, b = 0, at = 0;
    if (static_cast<int>(threadIdx.x) < nk) {
      const T* run = run_of(threadIdx.x, &a, &b);
      at = threadIdx.x * pitch + threadIdx.x / V * 16 + static_cast<int>(reinterpret_cast<uintptr_t>(run) & 15) - (a - c0) * taps * static_cast<int>(sizeof(T));
    }
    row_of[threadIdx.x] = make_int4(at, a, b, 0);
  }
  for (int base = 0; base < nk * q.pieces; base += kPackThreads * kPackPieces) {
    uint4 v[kPackPieces];
    int to[kPackPieces];
#pragma unroll
    for (int u = 0; u < kPackPieces; ++u) {
      const int i = base + u * kPackThreads + threadIdx.x, kk = i / q.pieces;
      to[u] = -1;
      if (kk >= nk) continue;
      int a, b;
      const T* run = run_of(kk, &a, &b);
      const uintptr_t lo = reinterpret_cast<uintptr_t>(run), hi = reinterpret_cast<uintptr_t>(run + (b - a) * taps);
      const uintptr_t from = (lo & ~static_cast<uintptr_t>(15)) + (i - kk * q.pieces) * 16;
      if (from >= hi) continue;
      to[u] = (i + kk / V) * 16;
      if (from >= lo && from + 16 <= hi) {
        v[u] = *reinterpret_cast<const uint4*>(from);
        continue;
      }
      // an end of the run: its elements, all on their way together
      __align__(16) T part[V];
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const uintptr_t at = from + e * sizeof(T);
        part[e] = at >= lo && at < hi ? *reinterpret_cast<const T*>(at) : T(0);
      }
      v[u] = *reinterpret_cast<const uint4*>(part);
    }
#pragma unroll
    for (int u = 0; u < kPackPieces; ++u)
      if (to[u] >= 0) *reinterpret_cast<uint4*>(tile + to[u]) = v[u];
  }
  __syncthreads();
  const int rows = q.mode == 0 ? Kg : q.Cg, log_rows = q.mode == 0 ? q.log_k : q.log_c;
  const int log_v = (q.mode == 0 ? q.log_c : q.log_k) - (V == 8 ? 3 : 2), row0 = q.mode == 0 ? k0 : c0, col0 = q.mode == 0 ? c0 : k0;
  T* dst = static_cast<T*>(q.dst) + 1LL * g * rows * q.ldc;
  // whole patches of rows that start alike: no look-ups, neighbouring elements of a piece a constant apart
  const bool whole = q.merge == 1 && nk == 1 << q.log_k && c0 + (1 << q.log_c) <= q.Cg && (Cs * taps * sizeof(T)) % 16 == 0;
  const int first = row_of[0].x, apart = q.mode == 0 ? taps * static_cast<int>(sizeof(T)) : pitch;
  for (int o = threadIdx.x; o < taps << (log_rows + log_v); o += kPackThreads) {
    const int col = col0 + (o & ((1 << log_v) - 1)) * V, r = (o >> log_v) & ((1 << log_rows) - 1), t = o >> (log_rows + log_v);
    if (col >= q.ldc || row0 + r >= rows) continue;
    __align__(16) T v[V];
    if (whole) {
      const int k = q.mode == 0 ? r : col - k0, c = q.mode == 0 ? col - c0 : r;
      const uint8_t* at = tile + first + k * pitch + k / V * 16 + (c * taps + t) * static_cast<int>(sizeof(T));
#pragma unroll
      for (int e = 0; e < V; ++e) v[e] = *reinterpret_cast<const T*>(at + e * apart);
    } else
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const int c = q.mode == 0 ? col + e : c0 + r;
      const int4 f = row_of[q.mode == 0 ? r : col + e - k0];
      v[e] = c >= f.y && c < f.z ? *reinterpret_cast<const T*>(tile + f.x + ((c - c0) * taps + t) * static_cast<int>(sizeof(T))) : T(0);
    }
    const int tap = q.flip ? taps - 1 - t : t;
    *reinterpret_cast<uint4*>(dst + (1LL * tap * q.groups * rows + row0 + r) * q.ldc + col) = *reinterpret_cast<const uint4*>(v);
  }
}

template <typename T>
__device__ __forceinline__ void pack_job_block(const PackJob& q, int local) {
  const int bx = local % q.gx, by = local / q.gx % q.gy, bz = local / q.gx / q.gy;
  pack_filters_block<T>(q, bx, by, bz);
}

template <typename T>
__global__ void __launch_bounds__(kPackThreads) pack_filters_kernel(const __grid_constant__ PackJob q) {
  pdl_enter();
  pack_job_block<T>(q, blockIdx.x);
}

// Many filter banks in one launch: block b belongs to the job j with first_block[j] <= b < first_block[j + 1].
template <typename T>
__global__ void __launch_bounds__(kPackThreads) pack_filters_batch_kernel(const __grid_constant__ PackBatch b) {
  pdl_enter();
  int j = 0, end = b.njobs;
  while (j + 1 < end) {
    const int mid = (j + end) >> 1;
    if (static_cast<int>(blockIdx.x) >= b.jobs[mid].first_block) j = mid;
    else end = mid;
  }
  pack_job_block<T>(b.jobs[j], blockIdx.x - b.jobs[j].first_block);
}

// idx / d: a multiplication for 32-bit indices; those of more than 2^31 elements are divided.
__device__ __forceinline__ uint32_t over(uint32_t idx, const Divisor& d) { return quotient(idx, d); }
__device__ __forceinline__ long long over(long long idx, const Divisor& d) { return idx / d.d; }
constexpr long long kIndex32 = 1LL << 31;

// Few-channel layers ("row folding"): the image is copied channels-last with explicit zero
// columns left and right, [N][H][Wp][Cp], so that the kW * Cp values under one filter row are
// contiguous and can serve as one reduction block of the implicit GEMM.  One thread per output
// pixel; src is NCHW (nhwc_in = 0), channels-last [N][H][W][Cp] (1) or that off the 16-byte boundaries (2).
template <typename T, typename Index>
__global__ void pad_fold_kernel(const T* __restrict__ src, T* __restrict__ dst, Index total, Divisor by_H, Divisor by_Wp, int C,
                                int W, int Cp, int pad_l, int nhwc_in) {
  pdl_enter();
  const int H = by_H.d;
  for (Index idx = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const Index row = over(idx, by_Wp);
    const int n = static_cast<int>(over(row, by_H)), h = static_cast<int>(row - static_cast<Index>(n) * H);
    const int w = static_cast<int>(idx - row * by_Wp.d) - pad_l;
    const bool inside = w >= 0 && w < W;
    // A pixel is one to a few 16-byte pieces, each assembled in registers and stored once.  (Channel by channel, pixels of two pieces: 9 -> 80 3x3 at 14x46, 22 images,
    // float16, forward 19.3 -> 11.0 us from NCHW, 16.0 -> 8.8 from channels-last; 12 -> 40 at 56x56, 64 images, 52 -> 34.)
    constexpr int V = 16 / static_cast<int>(sizeof(T));
    const T* s = src + (nhwc_in ? ((1LL * n * H + h) * W + w) * Cp : (1LL * n * C * H + h) * W + w);
    for (int c0 = 0; c0 < Cp; c0 += V) {
      uint4 px = make_uint4(0, 0, 0, 0);
      if (inside) {
        if (nhwc_in == 1) {
          px = *reinterpret_cast<const uint4*>(s + c0);
          if (c0 + V > C) {
            T* v = reinterpret_cast<T*>(&px);
#pragma unroll
            for (int e = 0; e < V; ++e)
              if (c0 + e >= C) v[e] = T(0);
          }
        } else {
          T* v = reinterpret_cast<T*>(&px);
#pragma unroll
          for (int e = 0; e < V; ++e)
            if (c0 + e < C) v[e] = nhwc_in ? s[c0 + e] : s[1LL * (c0 + e) * H * W];
        }
      }
      *reinterpret_cast<uint4*>(dst + 1LL * idx * Cp + c0) = px;
    }
  }
}

// Folded filters: dst[i][k][j*Cp + c] = w[k][c][i'][j'] (zero elsewhere up to ld columns), where
// (i', j') = (i, j) or the flipped position.
template <typename T, typename Index>
__global__ void pack_filters_fold_kernel(const T* __restrict__ w, T* __restrict__ dst, int K, int C,
                                         int kH, int kW, int Cp, int ld, int flip) {
  pdl_enter();
  const Index total = static_cast<Index>(kH) * K * ld;
  for (Index idx = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const Index row = idx / ld;
    const int col = static_cast<int>(idx - row * ld), i = static_cast<int>(row / K), k = static_cast<int>(row - static_cast<Index>(i) * K);
    const int j = col / Cp, c = col % Cp;
    T v = T(0);
    if (j < kW && c < C) {
      const int wi = flip ? kH - 1 - i : i, wj = flip ? kW - 1 - j : j;
      v = w[((1LL * k * C + c) * kH + wi) * kW + wj];
    }
    dst[idx] = v;
  }
}

// Space-to-depth for stride-2 layers with very few channels (the 7x7 stride-2 stems): a 2 x 2 block
// of input pixels becomes one pixel of kS2dChannels channels,
//   dst[n][h2][q][(dy*2 + dx)*C + c] = src[n][c][2*h2 + dy][2*(q + q0) + dx]
// with zeros outside the image and in the unused channels.  The layer then is a stride-1 layer over
// dst whose filter rows span a few consecutive pixels: one contiguous reduction block per row.
// One thread per dst pixel; src is NCHW (nhwc_in = 0), channels-last [N][H][W][Cp_in] (1) or that off the 16-byte
// boundaries (2).
template <typename T, int C, typename Index>
__global__ void pad_s2d_kernel(const T* __restrict__ src, T* __restrict__ dst, Index total, Divisor by_H2, Divisor by_Wq, int H,
                               int W, int Cp_in, int q0, int nhwc_in) {
  pdl_enter();
  for (Index idx = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const Index row = over(idx, by_Wq);
    const int n = static_cast<int>(over(row, by_H2)), h2 = static_cast<int>(row - static_cast<Index>(n) * by_H2.d), q = static_cast<int>(idx - row * by_Wq.d);
    __align__(16) T v[kS2dChannels];
#pragma unroll
    for (int i = 0; i < kS2dChannels; ++i) v[i] = T(0);
#pragma unroll
    for (int par = 0; par < 4; ++par) {
      const int h = 2 * h2 + (par >> 1), w = 2 * (q + q0) + (par & 1);
      if (h < H && w >= 0 && w < W) {
        if (nhwc_in == 1 && Cp_in * sizeof(T) == 16) {     // one source pixel is one 16-byte load
          const uint4 px = *reinterpret_cast<const uint4*>(src + ((1LL * n * H + h) * W + w) * Cp_in);
          const T* e = reinterpret_cast<const T*>(&px);
#pragma unroll
          for (int c = 0; c < C; ++c) v[par * C + c] = e[c];
        } else {
#pragma unroll
          for (int c = 0; c < C; ++c)
            v[par * C + c] = nhwc_in ? src[((1LL * n * H + h) * W + w) * Cp_in + c]
                                     : src[((1LL * n * C + c) * H + h) * W + w];
        }
      }
    }
    uint4* d = reinterpret_cast<uint4*>(dst + 1LL * idx * kS2dChannels);
    const uint4* sv = reinterpret_cast<const uint4*>(v);
#pragma unroll
    for (int i = 0; i < (int)(kS2dChannels * sizeof(T) / 16); ++i) d[i] = sv[i];
  }
}

// Filters for the space-to-depth form: dst[t][k][j*kS2dChannels + (dy*2 + dx)*C + c] is the filter
// element that multiplies input pixel (2*(t + t0) + dy, 2*(j + q0) + dx) relative to the output
// position times the stride, i.e. tap (i, jj) = (2*(t + t0) + dy + padH, 2*(j + q0) + dx + padW);
// zero where that tap does not exist.
template <typename T, typename Index>
__global__ void pack_filters_s2d_kernel(const T* __restrict__ w, T* __restrict__ dst, int K, int C,
                                        int kH, int kW, int ntaps, int t0, int q0, int padH, int padW,
                                        int ld, int flip) {
  pdl_enter();
  const Index total = static_cast<Index>(ntaps) * K * ld;
  for (Index idx = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const Index row = idx / ld;
    const int col = static_cast<int>(idx - row * ld), t = static_cast<int>(row / K), k = static_cast<int>(row - static_cast<Index>(t) * K);
    const int j = col / kS2dChannels, r = col % kS2dChannels;
    T v = T(0);
    if (r < 4 * C) {
      const int par = r / C, c = r % C;
      const int i = 2 * (t + t0) + (par >> 1) + padH, jj = 2 * (j + q0) + (par & 1) + padW;
      if (i >= 0 && i < kH && jj >= 0 && jj < kW) {
        const int wi = flip ? kH - 1 - i : i, wj = flip ? kW - 1 - jj : jj;
        v = w[((1LL * k * C + c) * kH + wi) * kW + wj];
      }
    }
    dst[idx] = v;
  }
}

// Adds the slabs (wgrad_slab.cuh, rows of ld columns) of a gradient whose columns are not the filters' own channels: place(c, i', j') gives
// the slab tap and column of a filter element.  A block takes 32 filters of one element: neighbouring threads read neighbouring
// filters (16 bytes apart), eight threads share a sum (slabs l, l + 8, ..., then in order of l), so that a chain of loads
// is an eighth of the slices long.  `sum`: for sums that are NaN (wgrad_exact.cuh).
template <typename T, class Place>
__device__ __forceinline__ void reduce_gathered(const float* __restrict__ partial, T* __restrict__ dw, int splits, int K, int C, int kH, int kW,
                                                int ntaps, int ld, const WgradSum& sum, Place place) {
  __shared__ float part[8][32];
  const int kk = threadIdx.x & 31, lane = threadIdx.x >> 5, per_k = C * kH * kW, ktiles = (K + 31) / 32;
  const long long slab = 1LL * ntaps * K * ld;
  bool nan = false;
  for (long long tl = blockIdx.x; tl < 1LL * per_k * ktiles; tl += gridDim.x) {
    const int e = static_cast<int>(tl % per_k), k = static_cast<int>(tl / per_k) * 32 + kk;
    const int wj = e % kW, wi = (e / kW) % kH, c = e / (kW * kH);
    float acc = 0.f;
    if (k < K) {
      int t, col;
      place(c, wi, wj, &t, &col);
      const float* src = partial + slab_index(t, k, col, K, ld);
#pragma unroll 8
      for (int s = lane; s < splits; s += 8) acc += src[s * slab];
    }
    part[lane][kk] = acc;
    __syncthreads();
    if (lane == 0 && k < K) {
      for (int l = 1; l < 8; ++l) acc += part[l][kk];
      dw[1LL * k * per_k + e] = static_cast<T>(acc);
      nan |= isnan(acc);
    }
    __syncthreads();
  }
  if (!__syncthreads_or(nan)) return;
#pragma unroll 1
  for (long long tl = blockIdx.x; tl < 1LL * per_k * ktiles; tl += gridDim.x) {
    const int e = static_cast<int>(tl % per_k), k0 = static_cast<int>(tl / per_k) * 32, wj = e % kW, wi = e / kW % kH, c = e / kW / kH;
    bool looked = false, suspect = false;                   // the border of the channel
#pragma unroll 1
    for (int k = k0 + lane; k < min(K, k0 + 32); k += 8) {
      if (!isnan(static_cast<float>(dw[1LL * k * per_k + e]))) continue;
      if (!looked) suspect = border_not_finite(sum, c);
      looked = true;
      if (!suspect) break;
      const float v = exact_sum(sum, k, c, sum.flip ? kH - 1 - wi : wi, sum.flip ? kW - 1 - wj : wj);
      if (kk == 0) dw[1LL * k * per_k + e] = static_cast<T>(v);
    }
  }
}

// Filter gradient of the space-to-depth form: dw[k][c][i'][j'] = sum_s slab s[t][k][col] with
// (t, col) the place pack_filters_s2d_kernel gives tap (i, jj).
template <typename T>
__global__ void __launch_bounds__(256) wgrad_reduce_s2d_kernel(const float* __restrict__ partial, T* __restrict__ dw, int splits,
                                        int K, int C, int kH, int kW, int ntaps, int t0, int q0, int padH,
                                        int padW, int ld, int flip, const __grid_constant__ WgradSum sum) {
  pdl_enter();
  reduce_gathered(partial, dw, splits, K, C, kH, kW, ntaps, ld, sum, [=](int c, int wi, int wj, int* t, int* col) {
    const int i = flip ? kH - 1 - wi : wi, jj = flip ? kW - 1 - wj : wj;
    const int ah = i - padH, aw = jj - padW;                 // offsets from 2 * the output position
    const int th = ah >= 0 ? ah / 2 : -((1 - ah) / 2), tw = aw >= 0 ? aw / 2 : -((1 - aw) / 2);   // floor
    const int par = (ah - 2 * th) * 2 + (aw - 2 * tw);
    *t = th - t0;
    *col = (tw - q0) * kS2dChannels + par * C + c;
  });
}

// Folded filter gradient: dw[k][c][i'][j'] = sum_s slab s[i][k][j*Cp + c].
template <typename T>
__global__ void __launch_bounds__(256) wgrad_reduce_fold_kernel(const float* __restrict__ partial, T* __restrict__ dw,
                                         int splits, int K, int C, int kH, int kW, int Cp, int ld,
                                         int flip, const __grid_constant__ WgradSum sum) {
  pdl_enter();
  reduce_gathered(partial, dw, splits, K, C, kH, kW, kH, ld, sum, [=](int c, int wi, int wj, int* t, int* col) {
    *t = flip ? kH - 1 - wi : wi;
    *col = (flip ? kW - 1 - wj : wj) * Cp + c;
  });
}

// Grouped convolutions with few channels per group: m neighbouring groups are merged into one
// group with block-diagonal filters, so that a reduction block of the MMA is filled with real
// channels.  expand: wm[k][c'][t] = w[k][c' % Cg][t] if column block c'/Cg belongs to filter k's
// group, else 0 (wm has m*Cg columns).  extract is the inverse for the filter gradient.
template <typename T>
__global__ void merge_groups_kernel(const T* __restrict__ src, T* __restrict__ dst, int K, int Cg,
                                    int Kg, int m, int taps, int extract) {
  pdl_enter();
  const int CgE = Cg * m;
  const long long total = 1LL * K * (extract ? Cg : CgE) * taps;
  for (long long idx = blockIdx.x * 1LL * blockDim.x + threadIdx.x; idx < total;
       idx += 1LL * gridDim.x * blockDim.x) {
    const int t = idx % taps;
    if (extract) {
      const int c = (idx / taps) % Cg;
      const int k = idx / (1LL * taps * Cg);
      const int blk = (k % (Kg * m)) / Kg;
      dst[idx] = src[(1LL * k * CgE + blk * Cg + c) * taps + t];
    } else {
      const int ce = (idx / taps) % CgE;
      const int k = idx / (1LL * taps * CgE);
      const int blk = (k % (Kg * m)) / Kg;
      dst[idx] = (ce / Cg == blk) ? src[(1LL * k * Cg + ce % Cg) * taps + t] : T(0);
    }
  }
}

template <typename T>
__global__ void convert_bias_kernel(const T* __restrict__ b, float* __restrict__ dst, int n) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = static_cast<float>(b[i]);
}

// NCHW: one thread per output element.  NHWC: one thread per (pixel, channel) with the
// channel fastest, so neighbouring threads read neighbouring addresses.
template <typename T>
__global__ void maxpool2x2_nchw_kernel(const T* __restrict__ x, T* __restrict__ y, long long NC, int H, int W) {
  pdl_enter();
  const int Ho = H / 2, Wo = W / 2;
  const long long total = NC * Ho * Wo;
  for (long long idx = blockIdx.x * 1LL * blockDim.x + threadIdx.x; idx < total;
       idx += 1LL * gridDim.x * blockDim.x) {
    const int ow = idx % Wo;
    const int oh = (idx / Wo) % Ho;
    const long long nc = idx / (1LL * Wo * Ho);
    const T* p = x + (nc * H + 2 * oh) * W + 2 * ow;
    float m = static_cast<float>(p[0]);
    m = fmaxf(m, static_cast<float>(p[1]));
    m = fmaxf(m, static_cast<float>(p[W]));
    m = fmaxf(m, static_cast<float>(p[W + 1]));
    y[idx] = static_cast<T>(m);
  }
}

// Gradient of the 2x2 / stride 2 max pooling: gx = gy of its window if x equals the window maximum y, else 0;
// every element of gx is written.  One thread per input element.
template <typename T>
__global__ void maxpool2x2_grad_nchw_kernel(const T* __restrict__ x, const T* __restrict__ y,
                                            const T* __restrict__ gy, T* __restrict__ gx, long long NC, int H, int W) {
  pdl_enter();
  const int Ho = H / 2, Wo = W / 2;
  const long long total = NC * H * W;
  for (long long idx = blockIdx.x * 1LL * blockDim.x + threadIdx.x; idx < total;
       idx += 1LL * gridDim.x * blockDim.x) {
    const int w = idx % W, h = (idx / W) % H;
    const long long nc = idx / (1LL * W * H), o = (nc * Ho + h / 2) * Wo + w / 2;
    T g = static_cast<T>(0.f);
    if (h < 2 * Ho && w < 2 * Wo && static_cast<float>(x[idx]) == static_cast<float>(y[o])) g = gy[o];
    gx[idx] = g;
  }
}

// Channels-last forms: one thread per window and 16-byte piece of the channel vector, so that every access
// is 16 bytes wide, the four pixels' loads are in flight together and the index arithmetic is paid once per
// 16 to 32 elements (HBM bound: 64 x 128 x 112 x 112 float32 gradient 846 -> 176 us at 1.03 GB).
// A tensor that does not start on a 16-byte boundary is taken element by element (One).
template <typename T> struct One {
  static constexpr int n = 1;
  using type = T;
  T v;
  __device__ __forceinline__ void max(const One& o) { v = static_cast<T>(fmaxf(static_cast<float>(v), static_cast<float>(o.v))); }
  __device__ __forceinline__ static One route(const One& x, const One& y, const One& g) {
    return {static_cast<float>(x.v) == static_cast<float>(y.v) ? g.v : static_cast<T>(0.f)};
  }
};
template <typename T> struct Piece;               // 16 bytes of T
template <> struct Piece<float> {
  static constexpr int n = 4;
  using type = float;
  float4 v;
  __device__ __forceinline__ void max(const Piece& o) {
    v.x = fmaxf(v.x, o.v.x); v.y = fmaxf(v.y, o.v.y); v.z = fmaxf(v.z, o.v.z); v.w = fmaxf(v.w, o.v.w);
  }
  __device__ __forceinline__ static Piece route(const Piece& x, const Piece& y, const Piece& g) {
    return {make_float4(x.v.x == y.v.x ? g.v.x : 0.f, x.v.y == y.v.y ? g.v.y : 0.f, x.v.z == y.v.z ? g.v.z : 0.f,
                        x.v.w == y.v.w ? g.v.w : 0.f)};
  }
};
template <> struct Piece<__half> {
  static constexpr int n = 8;
  using type = __half;
  __align__(16) __half2 v[4];
  __device__ __forceinline__ void max(const Piece& o) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __hmax2(v[i], o.v[i]);
  }
  __device__ __forceinline__ static Piece route(const Piece& x, const Piece& y, const Piece& g) {
    Piece r;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half z = __float2half(0.f);
      r.v[i] = __halves2half2(__heq(__low2half(x.v[i]), __low2half(y.v[i])) ? __low2half(g.v[i]) : z,
                              __heq(__high2half(x.v[i]), __high2half(y.v[i])) ? __high2half(g.v[i]) : z);
    }
    return r;
  }
};
template <typename P, typename T> __device__ __forceinline__ P load_piece(const T* p) { return *reinterpret_cast<const P*>(p); }

template <typename P, typename Index, typename T = typename P::type>
__global__ void __launch_bounds__(256) maxpool2x2_nhwc_kernel(const T* __restrict__ x, T* __restrict__ y, Index total,
                                                              int H, int W, int pieces) {
  pdl_enter();
  constexpr int V = P::n;
  const Index idx = blockIdx.x * static_cast<Index>(256) + threadIdx.x;
  if (idx >= total) return;
  const Index Ho = H / 2, Wo = W / 2, Cv = pieces;
  const Index pix = idx / Cv, row = pix / Wo;
  const long long Cp = static_cast<long long>(pieces) * V;
  const int c = static_cast<int>(idx - pix * Cv) * V, ow = static_cast<int>(pix - row * Wo), oh = static_cast<int>(row % Ho);
  const long long n = row / Ho;
  const T* p = x + ((n * H + 2 * oh) * W + 2 * ow) * Cp + c;
  P m = load_piece<P>(p);
  const P a = load_piece<P>(p + Cp), b = load_piece<P>(p + W * Cp), d = load_piece<P>(p + W * Cp + Cp);
  m.max(a); m.max(b); m.max(d);
  *reinterpret_cast<P*>(y + static_cast<long long>(idx) * V) = m;
}

// The grid covers (H + 1) / 2 x (W + 1) / 2 windows: in an odd-sized image the last row / column belongs to no
// window and gets zeros.
template <typename P, typename Index, typename T = typename P::type>
__global__ void __launch_bounds__(256) maxpool2x2_grad_nhwc_kernel(const T* __restrict__ x, const T* __restrict__ y,
                                                                   const T* __restrict__ gy, T* __restrict__ gx,
                                                                   Index total, int H, int W, int pieces) {
  pdl_enter();
  constexpr int V = P::n;
  const Index idx = blockIdx.x * static_cast<Index>(256) + threadIdx.x;
  if (idx >= total) return;
  const int Ho = H / 2, Wo = W / 2;
  const Index Hc = (H + 1) / 2, Wc = (W + 1) / 2, Cv = pieces;
  const Index pix = idx / Cv, row = pix / Wc;
  const long long Cp = static_cast<long long>(pieces) * V;
  const int c = static_cast<int>(idx - pix * Cv) * V, ow = static_cast<int>(pix - row * Wc), oh = static_cast<int>(row % Hc);
  const long long n = row / Hc;
  const long long base = ((n * H + 2 * oh) * W + 2 * ow) * Cp + c;
  P r[4];
  memset(r, 0, sizeof r);
  if (oh < Ho && ow < Wo) {
    const long long o = ((n * Ho + oh) * Wo + ow) * Cp + c;
    const P m = load_piece<P>(y + o), g = load_piece<P>(gy + o);
    P v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = load_piece<P>(x + base + (k & 1) * Cp + (k >> 1) * W * Cp);
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = P::route(v[k], m, g);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (2 * oh + (k >> 1) < H && 2 * ow + (k & 1) < W)
      *reinterpret_cast<P*>(gx + base + (k & 1) * Cp + (k >> 1) * W * Cp) = r[k];
}

template <typename T, typename Index>
__global__ void pack_filters_merged_kernel(const T* __restrict__ w, T* __restrict__ dst, int K, int C, int kH,
                                           int kW, int flip, MergedTapTable tb, int nu, int ncls, int rows, int ldw) {
  pdl_enter();
  const Index total = static_cast<Index>(nu) * rows * ldw;
  for (Index idx = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const Index ur = idx / ldw;
    const int kf = static_cast<int>(idx - ur * ldw), u = static_cast<int>(ur / rows), row = static_cast<int>(ur - static_cast<Index>(u) * rows);
    const int cls = row / C, c = row % C;
    const int tap = cls < ncls ? tb.src[u][cls] : -1;     // rows past ncls * C are zero padding
    T v = T(0);
    if (tap >= 0 && kf < K) {
      const int i = tap / kW, j = tap % kW;
      const int pos = flip ? (kH - 1 - i) * kW + (kW - 1 - j) : tap;
      v = w[(1LL * kf * C + c) * kH * kW + pos];
    }
    dst[idx] = v;
  }
}

// NCHW output: one thread per element.  Channels-last output: one thread per pixel, which reads
// its C values (contiguous in tmp) and writes the whole padded channel vector in 16-byte pieces (nhwc = 1) or, into a
// tensor off the 16-byte boundaries (2), value by value.
template <typename T>
__global__ void depth_to_space_kernel(const T* __restrict__ tmp, T* __restrict__ dx, int N, int C, int H, int W,
                                      int sH, int sW, int Ct, int Cp, int nhwc) {
  pdl_enter();
  const int Hq = (H + sH - 1) / sH, Wq = (W + sW - 1) / sW;
  if (nhwc) {
    constexpr int kVec = 16 / static_cast<int>(sizeof(T));      // Cp is a multiple of kVec
    const long long total = 1LL * N * H * W;
    for (long long idx = blockIdx.x * 1LL * blockDim.x + threadIdx.x; idx < total;
         idx += 1LL * gridDim.x * blockDim.x) {
      const int w = idx % W, h = (idx / W) % H;
      const long long n = idx / (1LL * W * H);
      const int cls = (h % sH) * sW + (w % sW);
      const T* src = tmp + ((n * Hq + h / sH) * Wq + w / sW) * Ct + cls * C;
      T* dst = dx + idx * Cp;
      for (int c0 = 0; c0 < Cp; c0 += kVec) {
        __align__(16) T v[kVec];
#pragma unroll
        for (int q = 0; q < kVec; ++q) v[q] = c0 + q < C ? src[c0 + q] : T(0);
        if (nhwc == 1) {
          *reinterpret_cast<uint4*>(dst + c0) = *reinterpret_cast<const uint4*>(v);
        } else {
#pragma unroll
          for (int q = 0; q < kVec; ++q) dst[c0 + q] = v[q];
        }
      }
    }
    return;
  }
  const long long total = 1LL * N * C * H * W;
  for (long long idx = blockIdx.x * 1LL * blockDim.x + threadIdx.x; idx < total;
       idx += 1LL * gridDim.x * blockDim.x) {
    const int w = idx % W, h = (idx / W) % H, c = (idx / (1LL * W * H)) % C;
    const long long n = idx / (1LL * W * H * C);
    const int cls = (h % sH) * sW + (w % sW);
    dx[idx] = tmp[((n * Hq + h / sH) * Wq + w / sW) * Ct + cls * C + c];
  }
}

__global__ void fill_kernel(uint4* buf, size_t n16) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n16;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    buf[i] = make_uint4(0, 0, 0, 0);
}

int grid_for(long long total, int block) {
  long long g = (total + block - 1) / block;
  const long long cap = 148LL * 32;
  return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace

cudaError_t launch_transpose(const void* in, void* out, int B, int R, int S, int ld_in,
                             int ld_out, int dtype, cudaStream_t s) {
  if (B == 0 || S == 0 || ld_out == 0) return cudaSuccess;
  const int rows = R > ld_out ? R : ld_out;
  for (int b0 = 0; b0 < B; b0 += 65535) {  // gridDim.z limit
    const int nb = (B - b0) < 65535 ? (B - b0) : 65535;
    dim3 grid((S + 31) / 32, (rows + 31) / 32, nb), block(32, 8);
    if (dtype == B200CONV_F16)
      launch_streaming(transpose_kernel<__half>, grid, block, 0, s,
          static_cast<const __half*>(in) + 1LL * b0 * R * ld_in,
          static_cast<__half*>(out) + 1LL * b0 * S * ld_out, R, S, ld_in, ld_out);
    else
      launch_streaming(transpose_kernel<float>, grid, block, 0, s,
          static_cast<const float*>(in) + 1LL * b0 * R * ld_in,
          static_cast<float*>(out) + 1LL * b0 * S * ld_out, R, S, ld_in, ld_out);
  }
  return cudaGetLastError();
}

// Patch of a block: 64 (float16, up to 16 taps) or 32 columns of the destination and as many of its rows as make four pieces per thread,
// fewer while that makes fewer than `least` blocks: then rows down to runs of 64 bytes and blocks of 1.5 KB, at last columns down to 32 bytes.
// (With a row of 128 bytes to a block, 37 -> 418 1x1 took 418 blocks: forward at 8x8, 8 images, float16 8.6 us, 7.6 from 1 KB and 6.2 from 1.5 KB on; 2 -> 440
// 7.5, 6.2; 64 -> 64 3x3 7.7, 7.1.  From 2 KB on 100 -> 75 5x5, 37 images, goes from 33.9 to 34.5.)
int plan_pack(PackJob* q, int dtype, int least) {
  const int es = static_cast<int>(elem_size(dtype)), V = 16 / es, Kg = q->K / q->groups;
  const int cols = q->ldc, rows = q->mode == 0 ? Kg : q->Cg;
  int log_cols = es == 2 && q->taps <= 16 ? 6 : 5, log_rows = 0;
  while ((1 << (log_cols - 1)) >= cols && (1 << (log_cols - 1)) >= V) --log_cols;
  while (log_rows < 6 && (1 << log_rows) < rows && (q->taps * es << (log_cols + log_rows + 1)) <= kPackThreads * kPackPieces * 16) ++log_rows;
  auto blocks = [&] { return cdiv(cols, 1 << log_cols) * cdiv(rows, 1 << log_rows) * q->groups; };
  while (log_rows > 0 && blocks() < least && (q->taps * es << (log_cols + log_rows - 1)) >= 1536 && (q->mode == 0 || (q->taps * es << log_rows) > 64)) --log_rows;
  while ((es << log_cols) > 32 && 2 * blocks() < least) --log_cols;
  q->log_k = static_cast<uint8_t>(q->mode == 0 ? log_rows : log_cols);
  q->log_c = static_cast<uint8_t>(q->mode == 0 ? log_cols : log_rows);
  q->gx = static_cast<int>(cdiv(q->mode == 0 ? cols : rows, 1 << q->log_c));
  q->gy = static_cast<int>(cdiv(q->mode == 0 ? rows : cols, 1 << q->log_k));
  // a run that starts off a 16-byte boundary touches one piece more; an odd count, and a piece more every 16 bytes of filters: what a
  // warp gathers for 16-byte pieces of several rows lies in different banks
  q->pieces = static_cast<uint16_t>((((q->taps * es << q->log_c) + 15) / 16 + 1) | 1);
  return q->gx * q->gy * q->groups;
}
static size_t pack_smem_bytes(const PackJob& q) { return (static_cast<size_t>(q.pieces * 16) << q.log_k) + (16 << q.log_k) / 4; }

cudaError_t launch_pack_filters_batch(const PackBatch& b, int total_blocks, int dtype, cudaStream_t s) {
  if (b.njobs == 0 || total_blocks == 0) return cudaSuccess;
  size_t smem = 0;
  for (int j = 0; j < b.njobs; ++j) smem = std::max(smem, pack_smem_bytes(b.jobs[j]));
  if (dtype == B200CONV_F16) launch_chained(pack_filters_batch_kernel<__half>, total_blocks, kPackThreads, smem, s, b);
  else launch_chained(pack_filters_batch_kernel<float>, total_blocks, kPackThreads, smem, s, b);
  return cudaGetLastError();
}

cudaError_t launch_pack_filters(PackJob q, int dtype, cudaStream_t s) {
  if (1LL * q.taps * q.K * q.Cg == 0) return cudaSuccess;
  const int blocks = plan_pack(&q, dtype, kPackBlocks);
  q.first_block = 0;
  if (dtype == B200CONV_F16) launch_chained(pack_filters_kernel<__half>, blocks, kPackThreads, pack_smem_bytes(q), s, q);
  else launch_chained(pack_filters_kernel<float>, blocks, kPackThreads, pack_smem_bytes(q), s, q);
  return cudaGetLastError();
}

// 0: NCHW, 1: channels-last, 2: channels-last off the 16-byte boundaries (no wide access)
static int channels_last_form(int nhwc, const void* p) { return nhwc && !aligned16({p}) ? 2 : nhwc; }

cudaError_t launch_pad_fold(const void* src, void* dst, int N, int C, int H, int W, int Cp, int Wp,
                            int pad_l, int nhwc_in, int dtype, cudaStream_t s) {
  const long long total = 1LL * N * H * Wp;
  if (total == 0) return cudaSuccess;
  nhwc_in = channels_last_form(nhwc_in, src);
#define B200_FOLD(T, Index) \
  launch_streaming(pad_fold_kernel<T, Index>, grid_for(total, 256), 256, 0, s, static_cast<const T*>(src), static_cast<T*>(dst), \
                   static_cast<Index>(total), divisor(H), divisor(Wp), C, W, Cp, pad_l, nhwc_in)
  if (total < kIndex32) {
    if (dtype == B200CONV_F16) B200_FOLD(__half, uint32_t);
    else B200_FOLD(float, uint32_t);
  } else {
    if (dtype == B200CONV_F16) B200_FOLD(__half, long long);
    else B200_FOLD(float, long long);
  }
#undef B200_FOLD
  return cudaGetLastError();
}

cudaError_t launch_pack_filters_fold(const void* w, void* dst, int K, int C, int kH, int kW, int Cp,
                                     int ld, int flip, int dtype, cudaStream_t s) {
  const long long total = 1LL * kH * K * ld;
  if (total == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    total < kIndex32 ? launch_chained(pack_filters_fold_kernel<__half, uint32_t>, grid_for(total, 256), 256, 0, s, static_cast<const __half*>(w), static_cast<__half*>(dst), K, C, kH, kW, Cp, ld, flip)
                     : launch_chained(pack_filters_fold_kernel<__half, long long>, grid_for(total, 256), 256, 0, s, static_cast<const __half*>(w), static_cast<__half*>(dst), K, C, kH, kW, Cp, ld, flip);
  else
    total < kIndex32 ? launch_chained(pack_filters_fold_kernel<float, uint32_t>, grid_for(total, 256), 256, 0, s, static_cast<const float*>(w), static_cast<float*>(dst), K, C, kH, kW, Cp, ld, flip)
                     : launch_chained(pack_filters_fold_kernel<float, long long>, grid_for(total, 256), 256, 0, s, static_cast<const float*>(w), static_cast<float*>(dst), K, C, kH, kW, Cp, ld, flip);
  return cudaGetLastError();
}

// Blocks of reduce_gathered: one per element and 32 filters, at most what fills the device a few times.
static int gather_grid(int K, long long total) { return static_cast<int>(std::min<long long>(total / K * ((K + 31) / 32), 148 * 16)); }

cudaError_t launch_wgrad_reduce_s2d(const float* partial, void* dw, int splits, int K, int C, int kH,
                                    int kW, int ntaps, int t0, int q0, int padH, int padW, int ld, int flip,
                                    int dtype, const WgradSum& sum, cudaStream_t s) {
  const long long total = 1LL * K * C * kH * kW;
  if (total == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    launch_streaming(wgrad_reduce_s2d_kernel<__half>, gather_grid(K, total), 256, 0, s,
        partial, static_cast<__half*>(dw), splits, K, C, kH, kW, ntaps, t0, q0, padH, padW, ld, flip, sum);
  else
    launch_streaming(wgrad_reduce_s2d_kernel<float>, gather_grid(K, total), 256, 0, s,
        partial, static_cast<float*>(dw), splits, K, C, kH, kW, ntaps, t0, q0, padH, padW, ld, flip, sum);
  return cudaGetLastError();
}

template <typename T>
cudaError_t pad_s2d_typed(const void* src, void* dst, int N, int C, int H, int W, int Cp_in, int H2, int Wq,
                          int q0, int nhwc_in, cudaStream_t s) {
  const long long total = 1LL * N * H2 * Wq;
  const T* in = static_cast<const T*>(src);
  T* out = static_cast<T*>(dst);
  nhwc_in = channels_last_form(nhwc_in, src);
  const int grid = grid_for(total, 256);
#define B200_S2D(C)                                                                                                              \
  case C:                                                                                                                        \
    if (total < kIndex32)                                                                                                        \
      launch_streaming(pad_s2d_kernel<T, C, uint32_t>, grid, 256, 0, s, in, out, static_cast<uint32_t>(total), divisor(H2), divisor(Wq), H, W, Cp_in, q0, nhwc_in); \
    else                                                                                                                         \
      launch_streaming(pad_s2d_kernel<T, C, long long>, grid, 256, 0, s, in, out, total, divisor(H2), divisor(Wq), H, W, Cp_in, q0, nhwc_in); \
    break;
  switch (C) {   // the channel count as a constant keeps the assembled pixel in registers
    B200_S2D(1)
    B200_S2D(2)
    B200_S2D(3)
    B200_S2D(4)
    default: return cudaErrorInvalidValue;
  }
#undef B200_S2D
  return cudaGetLastError();
}

cudaError_t launch_pad_s2d(const void* src, void* dst, int N, int C, int H, int W, int Cp_in, int H2,
                           int Wq, int q0, int nhwc_in, int dtype, cudaStream_t s) {
  if (1LL * N * H2 * Wq == 0) return cudaSuccess;
  return dtype == B200CONV_F16 ? pad_s2d_typed<__half>(src, dst, N, C, H, W, Cp_in, H2, Wq, q0, nhwc_in, s)
                               : pad_s2d_typed<float>(src, dst, N, C, H, W, Cp_in, H2, Wq, q0, nhwc_in, s);
}

cudaError_t launch_pack_filters_s2d(const void* w, void* dst, int K, int C, int kH, int kW, int ntaps,
                                    int t0, int q0, int padH, int padW, int ld, int flip, int dtype,
                                    cudaStream_t s) {
  const long long total = 1LL * ntaps * K * ld;
  if (total == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    total < kIndex32 ? launch_chained(pack_filters_s2d_kernel<__half, uint32_t>, grid_for(total, 256), 256, 0, s, static_cast<const __half*>(w), static_cast<__half*>(dst), K, C, kH, kW, ntaps, t0, q0, padH, padW, ld, flip)
                     : launch_chained(pack_filters_s2d_kernel<__half, long long>, grid_for(total, 256), 256, 0, s, static_cast<const __half*>(w), static_cast<__half*>(dst), K, C, kH, kW, ntaps, t0, q0, padH, padW, ld, flip);
  else
    total < kIndex32 ? launch_chained(pack_filters_s2d_kernel<float, uint32_t>, grid_for(total, 256), 256, 0, s, static_cast<const float*>(w), static_cast<float*>(dst), K, C, kH, kW, ntaps, t0, q0, padH, padW, ld, flip)
                     : launch_chained(pack_filters_s2d_kernel<float, long long>, grid_for(total, 256), 256, 0, s, static_cast<const float*>(w), static_cast<float*>(dst), K, C, kH, kW, ntaps, t0, q0, padH, padW, ld, flip);
  return cudaGetLastError();
}

cudaError_t launch_wgrad_reduce_fold(const float* partial, void* dw, int splits, int K, int C, int kH,
                                     int kW, int Cp, int ld, int flip, int dtype, const WgradSum& sum, cudaStream_t s) {
  const long long total = 1LL * K * C * kH * kW;
  if (total == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    launch_streaming(wgrad_reduce_fold_kernel<__half>, gather_grid(K, total), 256, 0, s,
        partial, static_cast<__half*>(dw), splits, K, C, kH, kW, Cp, ld, flip, sum);
  else
    launch_streaming(wgrad_reduce_fold_kernel<float>, gather_grid(K, total), 256, 0, s,
        partial, static_cast<float*>(dw), splits, K, C, kH, kW, Cp, ld, flip, sum);
  return cudaGetLastError();
}

cudaError_t launch_merge_groups(const void* src, void* dst, int K, int Cg, int Kg, int m, int taps,
                                int extract, int dtype, cudaStream_t s) {
  const long long total = 1LL * K * (extract ? Cg : Cg * m) * taps;
  if (total == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    launch_streaming(merge_groups_kernel<__half>, grid_for(total, 256), 256, 0, s,
        static_cast<const __half*>(src), static_cast<__half*>(dst), K, Cg, Kg, m, taps, extract);
  else
    launch_streaming(merge_groups_kernel<float>, grid_for(total, 256), 256, 0, s,
        static_cast<const float*>(src), static_cast<float*>(dst), K, Cg, Kg, m, taps, extract);
  return cudaGetLastError();
}

namespace {
template <typename T>
__global__ void pad_bias_kernel(const T* __restrict__ b, T* __restrict__ dst, int n, int np) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < np) dst[i] = i < n ? b[i] : T(0);
}
}  // namespace
cudaError_t launch_pad_bias(const void* bias, void* dst, int n, int np, int dtype, cudaStream_t s) {
  if (dtype == B200CONV_F16)
    launch_chained(pad_bias_kernel<__half>, (np + 255) / 256, 256, 0, s, static_cast<const __half*>(bias), static_cast<__half*>(dst), n, np);
  else
    launch_chained(pad_bias_kernel<float>, (np + 255) / 256, 256, 0, s, static_cast<const float*>(bias), static_cast<float*>(dst), n, np);
  return cudaGetLastError();
}

cudaError_t launch_convert_bias(const void* bias, float* dst, int n, int dtype, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    launch_chained(convert_bias_kernel<__half>, (n + 255) / 256, 256, 0, s, static_cast<const __half*>(bias), dst, n);
  else
    launch_chained(convert_bias_kernel<float>, (n + 255) / 256, 256, 0, s, static_cast<const float*>(bias), dst, n);
  return cudaGetLastError();
}

namespace {
// Launches a channels-last pooling kernel with 32-bit indices where they suffice (64-bit divisions cost more
// than the memory accesses).
template <class Launch>
cudaError_t for_index(long long total, Launch launch) {
  const long long grid = (total + 255) / 256;
  if (grid >= (1LL << 31)) return cudaErrorInvalidValue;
  launch(static_cast<int>(grid), total < (1LL << 31));
  return cudaGetLastError();
}
template <typename P, typename T = typename P::type>
cudaError_t maxpool_nhwc(const T* x, T* y, int N, int H, int W, int Cp, cudaStream_t s) {
  const int pieces = Cp / P::n;
  const long long total = 1LL * N * (H / 2) * (W / 2) * pieces;
  return for_index(total, [&](int grid, bool small) {
    if (small) launch_streaming(maxpool2x2_nhwc_kernel<P, unsigned>, grid, 256, 0, s, x, y, static_cast<unsigned>(total), H, W, pieces);
    else launch_streaming(maxpool2x2_nhwc_kernel<P, long long>, grid, 256, 0, s, x, y, total, H, W, pieces);
  });
}
template <typename P, typename T = typename P::type>
cudaError_t maxpool_grad_nhwc(const T* x, const T* y, const T* gy, T* gx, int N, int H, int W, int Cp, cudaStream_t s) {
  const int pieces = Cp / P::n;
  const long long total = 1LL * N * ((H + 1) / 2) * ((W + 1) / 2) * pieces;
  return for_index(total, [&](int grid, bool small) {
    if (small)
      launch_streaming(maxpool2x2_grad_nhwc_kernel<P, unsigned>, grid, 256, 0, s, x, y, gy, gx, static_cast<unsigned>(total), H, W, pieces);
    else
      launch_streaming(maxpool2x2_grad_nhwc_kernel<P, long long>, grid, 256, 0, s, x, y, gy, gx, total, H, W, pieces);
  });
}
template <typename T>
cudaError_t maxpool_typed(const T* x, T* y, int N, int C, int H, int W, int nhwc, int Cp, cudaStream_t s) {
  if (!nhwc) {
    launch_streaming(maxpool2x2_nchw_kernel<T>, grid_for(1LL * N * C * (H / 2) * (W / 2), 256), 256, 0, s, x, y, 1LL * N * C, H, W);
    return cudaGetLastError();
  }
  return aligned16({x, y}) ? maxpool_nhwc<Piece<T>>(x, y, N, H, W, Cp, s) : maxpool_nhwc<One<T>>(x, y, N, H, W, Cp, s);
}
template <typename T>
cudaError_t maxpool_grad_typed(const T* x, const T* y, const T* gy, T* gx, int N, int C, int H, int W, int nhwc, int Cp,
                               cudaStream_t s) {
  if (!nhwc) {
    launch_streaming(maxpool2x2_grad_nchw_kernel<T>, grid_for(1LL * N * C * H * W, 256), 256, 0, s, x, y, gy, gx, 1LL * N * C, H, W);
    return cudaGetLastError();
  }
  return aligned16({x, y, gy, gx}) ? maxpool_grad_nhwc<Piece<T>>(x, y, gy, gx, N, H, W, Cp, s)
                                   : maxpool_grad_nhwc<One<T>>(x, y, gy, gx, N, H, W, Cp, s);
}
}  // namespace

cudaError_t launch_maxpool2x2(const void* x, void* y, int N, int C, int H, int W, int nhwc,
                              int Cp, int dtype, cudaStream_t s) {
  if (1LL * N * C * (H / 2) * (W / 2) == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    return maxpool_typed(static_cast<const __half*>(x), static_cast<__half*>(y), N, C, H, W, nhwc, Cp, s);
  return maxpool_typed(static_cast<const float*>(x), static_cast<float*>(y), N, C, H, W, nhwc, Cp, s);
}

cudaError_t launch_maxpool2x2_grad(const void* x, const void* y, const void* gy, void* gx, int N, int C,
                                   int H, int W, int nhwc, int Cp, int dtype, cudaStream_t s) {
  if (1LL * N * C * H * W == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    return maxpool_grad_typed(static_cast<const __half*>(x), static_cast<const __half*>(y), static_cast<const __half*>(gy),
                              static_cast<__half*>(gx), N, C, H, W, nhwc, Cp, s);
  return maxpool_grad_typed(static_cast<const float*>(x), static_cast<const float*>(y), static_cast<const float*>(gy),
                            static_cast<float*>(gx), N, C, H, W, nhwc, Cp, s);
}

cudaError_t launch_pack_filters_merged(const void* w, void* dst, int K, int C, int kH, int kW, int flip,
                                       const MergedTapTable& tb, int nu, int ncls, int rows, int ldw,
                                       int dtype, cudaStream_t s) {
  const long long total = 1LL * nu * rows * ldw;
  if (total == 0) return cudaSuccess;
  if (dtype == B200CONV_F16)
    total < kIndex32 ? launch_chained(pack_filters_merged_kernel<__half, uint32_t>, grid_for(total, 256), 256, 0, s, static_cast<const __half*>(w), static_cast<__half*>(dst), K, C, kH, kW, flip, tb, nu, ncls, rows, ldw)
                     : launch_chained(pack_filters_merged_kernel<__half, long long>, grid_for(total, 256), 256, 0, s, static_cast<const __half*>(w), static_cast<__half*>(dst), K, C, kH, kW, flip, tb, nu, ncls, rows, ldw);
  else
    total < kIndex32 ? launch_chained(pack_filters_merged_kernel<float, uint32_t>, grid_for(total, 256), 256, 0, s, static_cast<const float*>(w), static_cast<float*>(dst), K, C, kH, kW, flip, tb, nu, ncls, rows, ldw)
                     : launch_chained(pack_filters_merged_kernel<float, long long>, grid_for(total, 256), 256, 0, s, static_cast<const float*>(w), static_cast<float*>(dst), K, C, kH, kW, flip, tb, nu, ncls, rows, ldw);
  return cudaGetLastError();
}

cudaError_t launch_depth_to_space(const void* tmp, void* dx, int N, int C, int H, int W, int sH, int sW,
                                  int Ct, int Cp, int nhwc, int dtype, cudaStream_t s) {
  const long long total = 1LL * N * (nhwc ? 1 : C) * H * W;
  if (total == 0) return cudaSuccess;
  nhwc = channels_last_form(nhwc, dx);
  if (dtype == B200CONV_F16)
    launch_streaming(depth_to_space_kernel<__half>, grid_for(total, 256), 256, 0, s,
        static_cast<const __half*>(tmp), static_cast<__half*>(dx), N, C, H, W, sH, sW, Ct, Cp, nhwc);
  else
    launch_streaming(depth_to_space_kernel<float>, grid_for(total, 256), 256, 0, s,
        static_cast<const float*>(tmp), static_cast<float*>(dx), N, C, H, W, sH, sW, Ct, Cp, nhwc);
  return cudaGetLastError();
}

cudaError_t launch_fill_l2(void* buf, size_t bytes, cudaStream_t s) {
  fill_kernel<<<148 * 8, 256, 0, s>>>(static_cast<uint4*>(buf), bytes / 16);
  return cudaGetLastError();
}

}  // namespace b200
