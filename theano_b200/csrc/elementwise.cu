// Element-wise kernels on channels-last device tensors, and the per-channel sum.
//
// In compiled Theano graphs the convolution ops are separated by small Elemwise nodes (the bias
// add of a training graph, relu = 0.5 * (v + |v|), its gradient 0.5 * g + 0.5 * g * sgn(v), a
// residual add, a scale) and by the bias gradient Sum{axis=[0, 2, 3]}.  The reference's GPU
// back end keeps them on the device (theano/gpuarray/elemwise.py:86); these kernels do the same
// for tensors that live in HBM between two convolution ops, so that no activation travels to
// the host and back for a few arithmetic operations.  All of them are HBM bound.
#include "internal.h"

namespace b200 {
namespace {

template <typename T> struct Vec;                 // 16 bytes of T
template <> struct Vec<float> { static constexpr int n = 4; };
template <> struct Vec<__half> { static constexpr int n = 8; };

template <typename T> __device__ __forceinline__ void load16(const T* p, float (&f)[Vec<T>::n]);
template <> __device__ __forceinline__ void load16<float>(const float* p, float (&f)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
template <> __device__ __forceinline__ void load16<__half>(const __half* p, float (&f)[8]) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __half22float2(h[i]);
    f[2 * i] = t.x; f[2 * i + 1] = t.y;
  }
}
template <typename T> __device__ __forceinline__ void store16(T* p, const float (&f)[Vec<T>::n]);
template <> __device__ __forceinline__ void store16<float>(float* p, const float (&f)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
}
template <> __device__ __forceinline__ void store16<__half>(__half* p, const float (&f)[8]) {
  uint4 v;
  __half2* h = reinterpret_cast<__half2*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = v;
}

// 16 bytes, or one element
template <typename T, int V> __device__ __forceinline__ void load(const T* p, float (&f)[V]) {
  if constexpr (V == 1) f[0] = static_cast<float>(*p);
  else load16<T>(p, f);
}
template <typename T, int V> __device__ __forceinline__ void store(T* p, const float (&f)[V]) {
  if constexpr (V == 1) *p = static_cast<T>(f[0]);
  else store16<T>(p, f);
}

__device__ __forceinline__ float apply(int op, float a, float b) {
  switch (op) {
    case kEwAdd: return a + b;
    case kEwMul: return a * b;
    case kEwSub: return a - b;
    case kEwRSub: return b - a;
    case kEwDiv: return a / b;
    case kEwRDiv: return b / a;
    case kEwMax: return fmaxf(a, b);
    case kEwAbs: return fabsf(a);
    case kEwSgn: return a > 0.f ? 1.f : (a < 0.f ? -1.f : 0.f);
    case kEwNeg: return -a;
    default: return a;
  }
}

// out = op(a, b); b is a tensor of a's shape (b_kind 0), the scalar `s` (1), a float32 vector with
// one value per stored channel (2: element i belongs to channel i % Cp) or absent (3).  Pad
// channels are written as 0 so that the tensor stays a valid channels-last operand.
// HBM bound; what keeps it off that bound is bytes in flight per thread, so a thread takes four vectors
// whose loads are issued together, and a tensor without pad channels whose operand needs no channel index
// (PLAIN) computes none.  Unary op, 411 MB float32 in and out: 158 -> 133 us.  V is a vector's element count: 1 where
// a tensor does not start on a 16-byte boundary.
constexpr int kEwVecs = 4;
template <typename T, int V, bool PLAIN>
__global__ void __launch_bounds__(256) elementwise_kernel(const T* __restrict__ a, const T* __restrict__ b,
                                                          const float* __restrict__ chan, T* __restrict__ out,
                                                          long long nvec, int C, int Cp, int op, int b_kind, float s) {
  pdl_enter();
  const long long base = blockIdx.x * (256LL * kEwVecs) + threadIdx.x;
  float fa[kEwVecs][V], fb[kEwVecs][V];
#pragma unroll
  for (int k = 0; k < kEwVecs; ++k)
    if (base + k * 256 < nvec) load<T>(a + (base + k * 256) * V, fa[k]);
  if (b_kind == 0)
#pragma unroll
    for (int k = 0; k < kEwVecs; ++k)
      if (base + k * 256 < nvec) load<T>(b + (base + k * 256) * V, fb[k]);
#pragma unroll
  for (int k = 0; k < kEwVecs; ++k) {
    const long long i = base + k * 256;
    if (i >= nvec) return;
    float fo[V];
    const int c0 = PLAIN ? 0 : nvec < (1LL << 31) / V ? static_cast<int>(static_cast<unsigned>(i) * V % static_cast<unsigned>(Cp))
                                                      : static_cast<int>(i * V % Cp);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const float bv = b_kind == 0 ? fb[k][q] : b_kind == 1 ? s : !PLAIN && b_kind == 2 ? chan[c0 + q] : 0.f;
      fo[q] = PLAIN || c0 + q < C ? apply(op, fa[k][q], bv) : 0.f;
    }
    store<T>(out + i * V, fo);
  }
}

// Per-channel sum, stage 1: a block's 256 threads are `lanes` rows of threads over the pixels x `vecs`
// 16-byte pieces of the channel vector (256 / lanes of them at a time); block b takes the pixels
// (b * lanes + lane) + k * gridDim.x * lanes in that order, eight loads in flight, then adds its rows in
// lane order into partial[b][Cp].  V is a piece's element count: 1 for a tensor off the 16-byte boundaries.
template <typename T, int V>
__global__ void __launch_bounds__(256) channel_sum_partial_kernel(const T* __restrict__ x, float* __restrict__ partial,
                                                                  long long pixels, int Cp, int log_lanes) {
  pdl_enter();
  __shared__ float part[256][V + 1];
  const int cols = 256 >> log_lanes, lane = threadIdx.x >> (8 - log_lanes), col = threadIdx.x & (cols - 1);
  const int vecs = Cp / V;
  const long long step = 1LL * gridDim.x << log_lanes, first = (static_cast<long long>(blockIdx.x) << log_lanes) + lane;
  for (int v0 = 0; v0 < vecs; v0 += cols) {
    const int v = v0 + col;
    float acc[V];
#pragma unroll
    for (int q = 0; q < V; ++q) acc[q] = 0.f;
    if (v < vecs) {
      const T* src = x + 1LL * v * V;
#pragma unroll 8
      for (long long p = first; p < pixels; p += step) {
        float f[V];
        load<T>(src + p * Cp, f);
#pragma unroll
        for (int q = 0; q < V; ++q) acc[q] += f[q];
      }
    }
#pragma unroll
    for (int q = 0; q < V; ++q) part[threadIdx.x][q] = acc[q];
    __syncthreads();
    for (int i = threadIdx.x; i < cols * V; i += 256) {
      const int c = i / V, q = i % V;
      if (v0 + c < vecs) {
        float sum = 0.f;
        for (int l = 0; l < 1 << log_lanes; ++l) sum += part[l * cols + c][q];
        partial[1LL * blockIdx.x * Cp + (v0 + c) * V + q] = sum;
      }
    }
    __syncthreads();
  }
}
// Stage 2: 32 channels per block, 16 warps: warp w adds the blocks w, w + 16, ... and the warps' sums are added
// in warp order (the same result on every run); the result leaves in the data type.
template <typename T>
__global__ void __launch_bounds__(512) channel_sum_final_kernel(const float* __restrict__ partial, T* __restrict__ out,
                                                                int blocks, int C, int Cp) {
  pdl_enter();
  __shared__ float part[16][32];
  const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (c < C)
#pragma unroll 8
    for (int b = wp; b < blocks; b += 16) acc += partial[1LL * b * Cp + c];
  part[wp][lane] = acc;
  __syncthreads();
  if (wp == 0 && c < C) {
    for (int k = 1; k < 16; ++k) acc += part[k][lane];
    out[c] = static_cast<T>(acc);
  }
}

}  // namespace

cudaError_t launch_elementwise(const void* a, const void* b, const float* chan, void* out, long long elems, int C,
                               int Cp, int op, int b_kind, float s, int dtype, cudaStream_t st) {
  if (elems == 0) return cudaSuccess;
  const bool wide = aligned16({a, b, out});
  const int V = !wide ? 1 : dtype == B200CONV_F16 ? 8 : 4;
  const long long nvec = elems / V;              // Cp is a multiple of V, so elems is
  const long long grid = (nvec + 256 * kEwVecs - 1) / (256 * kEwVecs);
  if (grid >= (1LL << 31)) return cudaErrorInvalidValue;
  const bool plain = C == Cp && b_kind != 2;
#define B200_EW(T, V, PLAIN)                                                                                   \
  launch_streaming(elementwise_kernel<T, V, PLAIN>, static_cast<int>(grid), 256, 0, st,                        \
      static_cast<const T*>(a), static_cast<const T*>(b), chan, static_cast<T*>(out), nvec, C, Cp, op, b_kind, s)
  if (dtype == B200CONV_F16) {
    if (!wide) B200_EW(__half, 1, false);
    else if (plain) B200_EW(__half, 8, true);
    else B200_EW(__half, 8, false);
  } else {
    if (!wide) B200_EW(float, 1, false);
    else if (plain) B200_EW(float, 4, true);
    else B200_EW(float, 4, false);
  }
#undef B200_EW
  return cudaGetLastError();
}

// Four blocks per SM once there are 64 pixels for each: the partial sums stay few (stage 2 reads them all).
int channel_sum_blocks(long long pixels) {
  const long long b = (pixels + 63) / 64;
  return static_cast<int>(b < 1 ? 1 : b > 148 * 4 ? 148 * 4 : b);
}

cudaError_t launch_channel_sum(const void* x, float* partial, void* out, long long pixels, int C, int Cp, int dtype,
                               cudaStream_t st) {
  const int blocks = channel_sum_blocks(pixels);
  const bool wide = aligned16({x});
  const int vecs = wide ? Cp / (dtype == B200CONV_F16 ? 8 : 4) : Cp;
  int log_lanes = 0;                             // as many rows of threads over the pixels as the channel vector leaves
  while (log_lanes < 8 && (vecs << (log_lanes + 1)) <= 256) ++log_lanes;
#define B200_SUM(T, V) \
  launch_streaming(channel_sum_partial_kernel<T, V>, blocks, 256, 0, st, static_cast<const T*>(x), partial, pixels, Cp, log_lanes)
  if (dtype == B200CONV_F16) {
    if (wide) B200_SUM(__half, 8);
    else B200_SUM(__half, 1);
  } else {
    if (wide) B200_SUM(float, 4);
    else B200_SUM(float, 1);
  }
#undef B200_SUM
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (dtype == B200CONV_F16)
    launch_chained(channel_sum_final_kernel<__half>, (C + 31) / 32, 512, 0, st, partial, static_cast<__half*>(out), blocks, C, Cp);
  else
    launch_chained(channel_sum_final_kernel<float>, (C + 31) / 32, 512, 0, st, partial, static_cast<float*>(out), blocks, C, Cp);
  return cudaGetLastError();
}

}  // namespace b200
