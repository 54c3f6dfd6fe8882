// Implicit-GEMM convolution on the 5th-generation tensor cores (tcgen05 + TMEM).
//
//   out[pixel, co] = sum over taps t, channels c of  view_t[pixel + offset_t, c] * filt_t[co, c]
//
// The accumulator tile is 128 output pixels (TMEM lanes) x BN output channels (TMEM
// columns, float32).  A pixel tile is a box bw x bh x bn of the output grid (columns, rows,
// images); for one tap and one block of 32 float32 / 64 float16 channels the activation
// operand is a single TMA box of a channels-last view, landing in shared memory as 128-byte
// rows in the 128-byte-swizzled K-major layout the MMA reads.  Zero padding is the TMA
// out-of-bounds fill; stride > 1 is expressed by views that start at a parity offset with
// doubled pitches; dilation and the input-gradient case only change the tap offsets.
// The same kernel therefore serves forward and gradInputs.
//
// Warp roles (672 threads, one CTA per SM, persistent over tiles):
//   warps 0, 18-20  TMA producers   warp 1   MMA issuer + TMEM owner
//   warps 2-17 epilogue: TMEM -> registers -> (+bias, ReLU) -> global (NCHW or channels-last)
// Shared-memory stages are recycled through full/empty mbarriers; two TMEM accumulators
// let the epilogue of tile i overlap the main loop of tile i+1.
#include "internal.h"
#include "ptx.cuh"

namespace b200 {
namespace {

constexpr int kRows = 128;            // accumulator lanes = pixels per tile
constexpr int kRowBytes = 128;        // one swizzle row: 32 tf32 or 64 f16 channels
constexpr int kABytes = kRows * kRowBytes;
constexpr int kEpilogueWarps = 16;
// One thread gets a TMA box accepted about every 300 clocks, whatever its size; a stage is two
// boxes and at most 512 clocks of MMAs.  Four producer warps share the issue: warp 0 and the
// three warps after the epilogue warps; producer pw issues the activation box (pw even) or the
// filter box (pw odd) of every second stage (parity pw / 2).
constexpr int kProducers = 4;
constexpr int kFirstExtraProducer = 2 + kEpilogueWarps;
constexpr int kThreads = 32 * (kFirstExtraProducer + kProducers - 1);
constexpr int kSmemBudget = 200 * 1024;

template <int BN> constexpr int stage_bytes() { return kABytes + BN * kRowBytes; }
template <int BN> constexpr int num_stages() {
  return (kSmemBudget / stage_bytes<BN>()) > 8 ? 8 : (kSmemBudget / stage_bytes<BN>());
}

// Transpose buffers of the epilogue warps, 32 rows x 64 bytes each (float32; a float16 chunk is 64 bytes of a row already)
template <MmaKind KIND> constexpr int transpose_bytes() { return KIND == MmaKind::TF32 ? 2048 : 0; }

struct Bars {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
};

template <typename T> struct OutPack;
template <> struct OutPack<float> {
  static __device__ __forceinline__ void store(float* p, float v) { *p = v; }
};
template <> struct OutPack<__half> {
  static __device__ __forceinline__ void store(__half* p, float v) { *p = __float2half_rn(v); }
};

template <MmaKind KIND, int BN>
__global__ void __launch_bounds__(kThreads, 1)
conv_umma_kernel(const __grid_constant__ UmmaConvParams p) {
  using OutT = typename std::conditional<KIND == MmaKind::TF32, float, __half>::type;
  constexpr int kStages = num_stages<BN>();
  constexpr int kBK = KIND == MmaKind::TF32 ? 32 : 64;   // channels per stage
  constexpr uint32_t kIdesc = instr_desc(KIND == MmaKind::TF32, false, false, kRows, BN);
  constexpr uint32_t kTmemCols = 2 * BN < 32 ? 32 : 2 * BN;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* transposes = smem + kStages * stage_bytes<BN>();
  Bars* bars = reinterpret_cast<Bars*>(transposes + kEpilogueWarps * transpose_bytes<KIND>());

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int rows_used = p.bw * p.bh * p.bn;
  const uint32_t tx_bytes = rows_used * kRowBytes + BN * kRowBytes;
  const uint32_t kiters = p.ntaps * p.kblocks;
  // tile counts fit 32 bits (the launcher checks): 64-bit divisions per tile would cost each
  // role about a thousand clocks, a fifth of a small tile
  const uint32_t total = static_cast<uint32_t>(p.tiles_w) * p.tiles_h * p.tiles_n * p.groups * p.tiles_co * p.splits;
  const uint32_t splits = p.splits;            // work item = (tile, slice of the reduction), slices of a tile side by side

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->acc_full[b], 1);
      mbar_init(&bars->acc_empty[b], kEpilogueWarps);
    }
    bars->abort = 0;
    mbar_fence_init();
  }
  // descriptors, beside the set-up and the wait for the kernel before (they are parameters, not global data)
  if (warp == 2 && lane == 0) {
    for (int v = 0; v < p.nviews; ++v) tma_prefetch_desc(&p.views[v]);
    tma_prefetch_desc(&p.wmap);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  // Rows of the A stage that no TMA box ever writes must not hold NaN patterns that would
  // spill into *valid* lanes: they cannot (each accumulator lane depends on its own A row
  // only), so they are left as they are.
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  pdl_enter();              // the next kernel may start once this CTA holds its TMEM; nothing global was touched before

  if (warp == 0 || warp >= kFirstExtraProducer) {
    // every lane follows the loop (warp-uniform control flow and addresses), one elected lane issues
    const bool leader = elect_one();
    const int pw = warp == 0 ? 0 : warp - kFirstExtraProducer + 1;
    const bool b_box = (pw & 1) != 0;
    const uint32_t my_parity = pw >> 1;
    int stage = 0;
    uint32_t phase = 0, idx = 0;
    bool ok = true;
    for (uint32_t item = blockIdx.x; item < total && ok; item += gridDim.x) {
      const uint32_t t = quotient(item, p.walk.splits), slice = item - t * splits;
      const uint32_t k0 = splits == 1 ? 0 : kiters * slice / splits, k1 = splits == 1 ? kiters : kiters * (slice + 1) / splits;
      const TileAt at = tile_at(p.walk, t);
      const int co_t = at.co_t, g = at.g, w0 = at.w * p.bw, h0 = at.h * p.bh, n0 = at.n * p.bn;
      uint32_t k = k0;
      const int tap0 = k0 ? k0 / p.kblocks : 0;
      for (int tap = tap0, kb = k0 - tap0 * p.kblocks; k < k1 && ok; ++tap, kb = 0) {
        const ConvTap tp = p.taps[tap];
        for (; kb < p.kblocks && k < k1; ++kb, ++idx, ++k) {
          if ((idx & 1) == my_parity) {
            if (!uniform_wait(&bars->empty[stage], phase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
            uint8_t* sa = smem + stage * stage_bytes<BN>();
            if (leader) {
              if (!b_box) {
                mbar_expect_tx(&bars->full[stage], tx_bytes);
                tma_load_5d(sa, &p.views[tp.view], &bars->full[stage], kb * kBK, g, w0 + tp.dw,
                            h0 + tp.dh, n0);
              } else {
                tma_load_3d(sa + kABytes, &p.wmap, &bars->full[stage], kb * kBK, co_t * BN,
                            tp.wmat * p.groups + g);
              }
            }
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else if (warp == 1) {
    const bool leader = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int it = 0;
    const uint64_t desc_bits = smem_desc(0, 16, 1024);
    const uint32_t desc_hi = static_cast<uint32_t>(desc_bits >> 32);
    const uint32_t lo_base = static_cast<uint32_t>(desc_bits) + (smem_u32(smem) >> 4);
    uint32_t seen = 0, acc_seen = 0;             // next stage / next accumulator already seen ready (mbar_look)
    for (uint32_t item = blockIdx.x; item < total && ok; item += gridDim.x, ++it) {
      const uint32_t tile = quotient(item, p.walk.splits), slice = item - tile * splits;
      const uint32_t k0 = splits == 1 ? 0 : kiters * slice / splits, k1 = splits == 1 ? kiters : kiters * (slice + 1) / splits;
      const int buf = it & 1;
      const uint32_t aphase = (it >> 1) & 1;
      if (!wait_seen(acc_seen, &bars->acc_empty[buf], aphase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem + buf * BN;
      uint32_t idesc = kIdesc;
      if (p.n_mma % BN) idesc = with_columns(kIdesc, mma_columns(p.n_mma, (tile - quotient(tile, p.walk.tiles_co) * p.tiles_co) * BN, BN, false));
      for (uint32_t k = k0; k < k1; ++k) {
        if (!wait_seen(seen, &bars->full[stage], phase, bars, p.wait_clocks)) { ok = false; break; }
        tc_fence_after();
        // 8 tf32 / 16 f16 channels = 32 bytes along the swizzled row per MMA: only the address
        // field of the descriptors changes (by 2 units of 16 bytes)
        const uint32_t a_lo = lo_base + stage * (stage_bytes<BN>() >> 4);
        const uint32_t b_lo = a_lo + (kABytes >> 4);
        if (leader) {
          umma_words<KIND>(d_tmem, a_lo, b_lo, desc_hi, idesc, k != k0);
          umma_words<KIND>(d_tmem, a_lo + 2, b_lo + 2, desc_hi, idesc, 1u);
        }
        __syncwarp();
        const int cur = stage;
        if (++stage == kStages) { stage = 0; phase ^= 1; }
        seen = mbar_look(&bars->full[stage], phase);
        if (k + 1 == k1) acc_seen = mbar_look(&bars->acc_empty[(it + 1) & 1], (((it + 1) >> 1) & 1) ^ 1);
        if (leader) {
          umma_words<KIND>(d_tmem, a_lo + 4, b_lo + 4, desc_hi, idesc, 1u);
          umma_words<KIND>(d_tmem, a_lo + 6, b_lo + 6, desc_hi, idesc, 1u);
          umma_commit(&bars->empty[cur]);
        }
      }
      if (ok && leader) umma_commit(&bars->acc_full[buf]);
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else {
    // Epilogue, 16 warps: warp w reads TMEM lanes [32*(w%4), +32) (the hardware's rule) and, of
    // those rows, every fourth 32-column chunk.  One warp keeps only a few stores in flight, so
    // the SM's store bandwidth is reached through the number of warps.
    const int quad = warp & 3;
    const int sub = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    uint8_t* mine = transposes + (warp - 2) * transpose_bytes<KIND>();
    const int rw = row % p.bw, rh = (row / p.bw) % p.bh, rn = row / (p.bw * p.bh);
    OutT* out = static_cast<OutT*>(p.out);
    const bool rowwise = p.out_sc == 1 && ((p.n_out * sizeof(OutT) | reinterpret_cast<uintptr_t>(p.out)) & 15) == 0;
    const bool transposed = KIND == MmaKind::TF32 && rowwise && total > gridDim.x;
    bool ok = true;
    int it = 0;
    for (uint32_t item = blockIdx.x; item < total && ok; item += gridDim.x, ++it) {
      const int buf = it & 1;
      const uint32_t aphase = (it >> 1) & 1;
      const TileAt at = tile_at(p.walk, quotient(item, p.walk.splits));
      const int co_t = at.co_t, g = at.g, w = at.w * p.bw + rw, h = at.h * p.bh + rh, n = at.n * p.bn + rn;
      const bool valid = row < rows_used && w < p.Wt && h < p.Ht && n < p.Nimg;
      if (!warp_wait_or_abort(&bars->acc_full[buf], aphase, bars, lane, p.wait_clocks)) { ok = false; break; }
      tc_fence_after();
      OutT* pix = out + (p.out_off + n * p.out_sn + h * p.out_sh + w * p.out_sw) + 1LL * g * p.n_out * p.out_sc;
      const OutT* res = p.epi.residual ? static_cast<const OutT*>(p.epi.residual) + (pix - out) : nullptr;
      const int co_base = co_t * BN;
      // element offsets of the four rows that this lane helps to write, -1: no pixel
      long long rows[4] = {-1, -1, -1, -1};
      if (transposed)
#pragma unroll
        for (int i = 0; i < 4; ++i) rows[i] = __shfl_sync(0xffffffffu, valid ? static_cast<long long>(pix - out) : -1LL, i * 8 + (lane >> 2));
      const int first_ch = (sub - it * min(BN / 32, (p.n_out - co_base + 31) / 32)) & 3;      // the warps take turns on narrow tiles
      if (splits > 1) {       // raw accumulators; conv_reduce.cu adds the slices and applies the epilogue
        float4* dst = reinterpret_cast<float4*>(p.partial) + static_cast<long long>(item) * (kRows * BN / 4) + row;
#pragma unroll 1
        for (int ch = first_ch; ch < BN / 32 && co_base + ch * 32 < p.n_out; ch += kEpilogueWarps / 4) {
          uint32_t r[32];
          tmem_ld32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + buf * BN + ch * 32, r);
          tmem_ld_wait();
          if (!valid) continue;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (B200_IN_RANGE((reinterpret_cast<float*>(dst + (ch * 8 + j) * kRows) - p.partial) + 4 <= p.partial_elems, p.status))
              dst[(ch * 8 + j) * kRows] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                      __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
        }
      } else
#pragma unroll 1
      for (int ch = first_ch; ch < BN / 32; ch += kEpilogueWarps / 4) {
        const int co0 = co_base + ch * 32;          // first channel (within the group) of the chunk
        if (co0 >= p.n_out) break;
        uint32_t r[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + buf * BN + ch * 32, r);
        tmem_ld_wait();
        if (!valid && !transposed) continue;
        zero_pad_columns(r, co0, p.n_real);
        const OutT* bias = p.bias ? static_cast<const OutT*>(p.bias) + g * p.n_out + co0 : nullptr;
        if (transposed) {
          // Four lanes write 64 bytes of a row side by side.  With each lane writing its own row an instruction touched 32 lines and half of
          // each sector, 2400 clocks per 128 x 32 block: more than the MMAs of a shallow reduction.  (64 -> 128 3x3 stride 2 at
          // 56x56, 256 images: 106 -> 91 us.  Float16 gained nothing: half as many pieces; nor did a CTA's only tile.)
#pragma unroll
          for (int j0 = 0; j0 < 32; j0 += 16) {
            if (co0 + j0 >= p.n_out) break;
#pragma unroll
            for (int piece = 0; piece < 4; ++piece) {
              float f[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int j = j0 + 4 * piece + q;
                f[q] = p.epi.alpha * __uint_as_float(r[j]);
                if (bias && co0 + j < p.n_out) f[q] += static_cast<float>(bias[j]);
                if (res && valid && co0 + j < p.n_real) f[q] += p.epi.beta * static_cast<float>(res[co0 + j]);
                if (p.relu) f[q] = p.epi.lin * f[q] + p.epi.abs * fabsf(f[q]);
              }
              *reinterpret_cast<float4*>(mine + lane * 64 + ((piece ^ ((lane >> 1) & 3)) << 4)) = make_float4(f[0], f[1], f[2], f[3]);
            }
            __syncwarp();
            const int cp = co0 + j0 + (lane & 3) * 4;                    // this lane's channels of the rows it writes
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int srow = i * 8 + (lane >> 2);
              const float4 v = *reinterpret_cast<const float4*>(mine + srow * 64 + (((lane & 3) ^ ((srow >> 1) & 3)) << 4));
              if (rows[i] >= 0 && cp < p.n_out && B200_IN_RANGE(rows[i] + cp + 4 <= p.out_elems, p.status))
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + rows[i] + cp) = v;
            }
            __syncwarp();
          }
        } else if (rowwise) {   // n_out is a whole number of 16-byte pieces: a piece is all in or all out
#pragma unroll
          for (int j = 0; j < 32; j += 16 / sizeof(OutT)) {
            if (co0 + j >= p.n_out) break;
            float f[16 / sizeof(OutT)];
#pragma unroll
            for (int q = 0; q < 16 / (int)sizeof(OutT); ++q) {
              f[q] = p.epi.alpha * __uint_as_float(r[j + q]);
              if (bias) f[q] += static_cast<float>(bias[j + q]);
              if (res && co0 + j + q < p.n_real) f[q] += p.epi.beta * static_cast<float>(res[co0 + j + q]);
              if (p.relu) f[q] = p.epi.lin * f[q] + p.epi.abs * fabsf(f[q]);
            }
            if (!B200_IN_RANGE((pix - out) + co0 + j >= 0 && (pix - out) + co0 + j + 16 / (long long)sizeof(OutT) <= p.out_elems, p.status))
              continue;
            if (sizeof(OutT) == 4) {
              *reinterpret_cast<float4*>(pix + co0 + j) = make_float4(f[0], f[1], f[2], f[3]);
            } else {
              uint4 pk;
              uint32_t* pw = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                __half2 h2 = __floats2half2_rn(f[2 * q], f[2 * q + 1]);
                pw[q] = *reinterpret_cast<uint32_t*>(&h2);
              }
              *reinterpret_cast<uint4*>(pix + co0 + j) = pk;
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (co0 + j < p.n_out) {
              float v = p.epi.alpha * __uint_as_float(r[j]);
              if (bias) v += static_cast<float>(bias[j]);
              if (res && co0 + j < p.n_real) v += p.epi.beta * static_cast<float>(res[(co0 + j) * p.out_sc]);
              if (p.relu) v = p.epi.lin * v + p.epi.abs * fabsf(v);
              if (B200_IN_RANGE((pix - out) + (co0 + j) * p.out_sc >= 0 && (pix - out) + (co0 + j) * p.out_sc < p.out_elems, p.status))
                OutPack<OutT>::store(pix + (co0 + j) * p.out_sc, v);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty[buf]);
    }
    if (!ok && lane == 0) report_status(p.status, kStatusTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (bars->abort) abort_grace(p.wait_clocks);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

template <MmaKind KIND, int BN> constexpr int smem_bytes() { return num_stages<BN>() * stage_bytes<BN>() + kEpilogueWarps * transpose_bytes<KIND>() + sizeof(Bars) + 1024; }
template <MmaKind KIND, int BN>
cudaError_t configure() {
  static PerDeviceOnce configured;
  return configured.ensure([] { return cudaFuncSetAttribute(conv_umma_kernel<KIND, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<KIND, BN>()); });
}

template <MmaKind KIND, int BN>
cudaError_t launch_one(const UmmaConvParams& p, long long total, int num_sms, cudaStream_t s) {
  constexpr int smem = smem_bytes<KIND, BN>();
  cudaError_t e = configure<KIND, BN>();
  if (e != cudaSuccess) return e;
  const int grid = static_cast<int>(total < num_sms ? total : num_sms);
  launch_chained(conv_umma_kernel<KIND, BN>, grid, kThreads, smem, s, p);
  return cudaGetLastError();
}

}  // namespace

// Accumulator width: the smallest of 32/64/128/256 columns that holds the group's outputs.
int conv_umma_bn(int n_out) { return n_out <= 32 ? 32 : n_out <= 64 ? 64 : n_out <= 128 ? 128 : 256; }

cudaError_t load_conv_umma(int dtype, int bn) {
  const bool f16 = dtype == B200CONV_F16;
  switch (bn) {
    case 32: return f16 ? configure<MmaKind::F16, 32>() : configure<MmaKind::TF32, 32>();
    case 64: return f16 ? configure<MmaKind::F16, 64>() : configure<MmaKind::TF32, 64>();
    case 128: return f16 ? configure<MmaKind::F16, 128>() : configure<MmaKind::TF32, 128>();
    default: return f16 ? configure<MmaKind::F16, 256>() : configure<MmaKind::TF32, 256>();
  }
}

cudaError_t launch_conv_umma(const UmmaConvParams& p, int dtype, int num_sms, cudaStream_t s) {
  const long long total = 1LL * p.tiles_w * p.tiles_h * p.tiles_n * p.groups * p.tiles_co * p.splits;
  if (total == 0 || p.ntaps == 0) return cudaSuccess;
  if (total >= (1LL << 31)) return cudaErrorInvalidValue;
  const bool f16 = dtype == B200CONV_F16;
#define B200_CASE(BNV)                                                                  \
  case BNV:                                                                             \
    return f16 ? launch_one<MmaKind::F16, BNV>(p, total, num_sms, s)                    \
               : launch_one<MmaKind::TF32, BNV>(p, total, num_sms, s);
  switch (p.bn_cols) {
    B200_CASE(32)
    B200_CASE(64)
    B200_CASE(128)
    B200_CASE(256)
  }
#undef B200_CASE
  return cudaErrorInvalidValue;
}

}  // namespace b200
