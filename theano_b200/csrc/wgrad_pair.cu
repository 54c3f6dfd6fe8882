// Filter gradient on pairs of CTAs (tcgen05.mma.cta_group::2), layers with at least 256
// filters and 256 channels per group.
//
//   dW[tap][k, c] = sum over output pixels q of  dy[q, k] * x_view_tap[q + offset_tap, c]
//
// One CTA with a 128 x 256 accumulator needs, per stage of 64 float16 pixels, 16 KB of dy and 32 KB of x from
// L2 for 512 clocks of MMAs (float32: twice both): 94 B/clk where an SM gets 73.  Here two CTAs of a cluster compute a tile of
// 256 filters x 256 channels together: each loads the dy rows of ITS 128 filters and HALF of the x tile
// (128 channels) into its own shared memory with plain TMA loads, one thread of the even CTA issues MMAs
// of M = 256 over both CTAs' operands, and each CTA's TMEM receives its 128 filter rows x 256 channels.
// Per CTA that is 32 KB per 512 clocks: 64 B/clk.  No load is shared between CTAs by the copy engine.
// A thread gets a box accepted every 200 to 300 clocks: a stage's four (float32: eight) boxes of 8 KB are spread over
// four producer warps.  256 -> 256 filters 3x3 at 14x14, 128 images, float32: 62.5 us with the tap groups of one CTA, whose
// 128 x 128 MMAs read 128 B/clk of operands from shared memory beside the copies' writes, 51 us here (64 B/clk).
//
// Work items, split-K slices, slab layout and the reduction kernel are those of wgrad_umma.cu; an item is
// (256-filter tile, 256-channel tile, group, tap, slice) and both CTAs of a pair walk the same items.
#include "internal.h"
#include "ptx.cuh"
#include "wgrad_slab.cuh"

namespace b200 {
namespace {

constexpr int kEpilogueWarps = 16;
constexpr int kProducers = 4;                          // warp 0 and the last three warps; box j of a stage belongs to producer j % 4
constexpr int kFirstExtraProducer = 2 + kEpilogueWarps;
constexpr int kThreads = 32 * (kFirstExtraProducer + kProducers - 1);
constexpr int kPix = 64;                               // reduction rows (pixels) per stage
static_assert(kPix == kWgradPixF32 && kPix == kWgradPixF16Wide, "the pixel box of a stage");
constexpr int kBoxBytes = kPix * 128;                  // one TMA box: 64 pixels x 128 bytes of channels
constexpr int kBN = 256;
constexpr int kMaxStages = 6;

template <MmaKind KIND> constexpr int atom() { return KIND == MmaKind::TF32 ? 32 : 64; }
template <MmaKind KIND> constexpr int half_boxes() { return 128 / atom<KIND>(); }               // of dy (128 filters), and of x (128 channels)
template <MmaKind KIND> constexpr int stage_bytes() { return 2 * half_boxes<KIND>() * kBoxBytes; }   // 32 / 64 KB
template <MmaKind KIND> constexpr int num_stages() { return 192 * 1024 / stage_bytes<KIND>(); }     // 6 / 3

struct alignas(16) Bars {
  uint64_t full[kMaxStages];        // even CTA: both CTAs' boxes of a stage have landed
  uint64_t empty[kMaxStages];       // each CTA: the MMAs reading the stage are done
  uint64_t acc_full[2];          // each CTA: the item's accumulator is complete
  uint64_t acc_empty[2];         // even CTA: both CTAs' epilogues have read the accumulator
  uint32_t tmem_base;
  volatile int abort;
};

struct Item {
  int kt, ct, g, tap, sp;
  uint32_t t_begin, t_end;
};

__device__ __forceinline__ Item decode(uint32_t it, const UmmaWgradParams& p, uint32_t per_split, uint32_t pix_tiles) {
  Item r;
  const uint32_t a = quotient(it, p.walk.splits), b = quotient(a, p.walk.taps), c = quotient(b, p.walk.groups);
  r.sp = it - a * p.walk.splits.d;
  r.tap = a - b * p.walk.taps.d;
  r.g = b - c * p.walk.groups.d;
  r.kt = quotient(c, p.walk.ctiles);
  r.ct = c - r.kt * p.walk.ctiles.d;
  r.t_begin = r.sp * per_split;
  r.t_end = r.t_begin + per_split < pix_tiles ? r.t_begin + per_split : pix_tiles;
  return r;
}

// The MMAs of an item's pixel tiles: KS steps of a stage as straight-line code, 0: any number.
template <MmaKind KIND, int KS>
__device__ __forceinline__ bool mma_tiles(Bars* bars, uint32_t d_tmem, uint32_t lo_base, uint32_t desc_hi, int ksteps, int ntiles, int& stage,
                                          uint32_t& phase, uint32_t& seen, bool leader, long long limit) {
  constexpr int kK = KIND == MmaKind::TF32 ? 8 : 16;               // reduction rows per MMA
  constexpr uint32_t kStep = (kK * 128) >> 4;
  constexpr uint32_t kIdesc = instr_desc(KIND == MmaKind::TF32, true, true, 256, kBN);
  const uint32_t lane = leader;
  uint32_t acc = 0u;
  for (int t = 0; t < ntiles; ++t) {
    if (!wait_seen(seen, &bars->full[stage], phase, bars, limit)) return false;
    tc_fence_after();
    const uint32_t a_lo = lo_base + stage * (stage_bytes<KIND>() >> 4);
    const uint32_t b_lo = a_lo + ((half_boxes<KIND>() * kBoxBytes) >> 4);
    const int half = (KS ? KS : ksteps) / 2;
    auto steps = [&](int k0, int k1) {
      if (KS) {
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
          if (ks >= k0 && ks < k1) umma_words_if<KIND, true>(lane, d_tmem, a_lo + ks * kStep, b_lo + ks * kStep, desc_hi, kIdesc, ks ? 1u : acc);
      } else {
        for (int ks = k0; ks < k1; ++ks) umma_words_if<KIND, true>(lane, d_tmem, a_lo + ks * kStep, b_lo + ks * kStep, desc_hi, kIdesc, ks ? 1u : acc);
      }
    };
    steps(0, half);
    const int cur = stage;
    if (++stage == num_stages<KIND>()) { stage = 0; phase ^= 1; }
    seen = mbar_look(&bars->full[stage], phase);
    steps(half, KS ? KS : ksteps);
    if (leader) umma_commit_pair(&bars->empty[cur]);
    acc = 1u;
  }
  return true;
}

template <MmaKind KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
wgrad_pair_kernel(const __grid_constant__ UmmaWgradParams p) {
  constexpr int kK = KIND == MmaKind::TF32 ? 8 : 16;               // reduction rows per MMA
  constexpr int kHalf = half_boxes<KIND>(), kBoxes = 2 * kHalf, kStages = num_stages<KIND>(), kStageBytes = stage_bytes<KIND>();
  // float16: 8-row groups 1024 bytes apart, 16-byte swizzle; float32: 4-row groups 512 bytes apart, 32-byte swizzle
  constexpr uint32_t kSbo = KIND == MmaKind::TF32 ? 512 : 1024;
  constexpr uint64_t kLayout = KIND == MmaKind::TF32 ? kSwizzle128Base32 : kSwizzle128;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Bars* bars = reinterpret_cast<Bars*>(smem + kStages * kStageBytes);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const uint32_t pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int rows_used = p.bw * p.bh * p.bn;
  const int ksteps = (rows_used + kK - 1) / kK;
  const uint32_t pix_tiles = static_cast<uint32_t>(p.tiles_w) * p.tiles_h * p.tiles_n;
  const uint32_t per_split = (pix_tiles + p.splits - 1) / p.splits;
  const uint32_t total = static_cast<uint32_t>(p.ktiles) * p.ctiles * p.groups * p.ntaps * p.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->acc_full[b], 1);
      mbar_init(&bars->acc_empty[b], 2);                           // one arrival per CTA of the pair
    }
    bars->abort = 0;
    mbar_fence_init();
  }
  // descriptors, beside the set-up and the wait for the kernel before (they are parameters, not global data)
  if (warp == 2 && lane == 0) {
    for (int v = 0; v < p.nviews; ++v) tma_prefetch_desc(&p.x_views[v]);
    tma_prefetch_desc(&p.dy_map);
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars->tmem_base, 512);
    tmem_relinquish_pair();
  }
  // Reduction rows past the pixel box are never written by TMA: clear them once so that the last MMA
  // of a stage (which reads whole groups of 16 rows) adds zeros.
  if (rows_used < ksteps * kK) {
    const int tail_rows = ksteps * kK - rows_used;
    const int boxes = kStages * kBoxes;
    for (int i = threadIdx.x; i < boxes * tail_rows * 8; i += kThreads) {
      const int box = i / (tail_rows * 8), rem = i % (tail_rows * 8);
      *(reinterpret_cast<uint4*>(smem + box * kBoxBytes + (rows_used + rem / 8) * 128) + rem % 8) = make_uint4(0, 0, 0, 0);
    }
    fence_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                              // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  pdl_enter();              // the next kernel may start once this CTA holds its TMEM; nothing global was touched before

  if (warp == 0 || warp >= kFirstExtraProducer) {
    const int pw = warp == 0 ? 0 : warp - kFirstExtraProducer + 1;
    const bool leader = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const uint32_t tx = 2u * kBoxes * rows_used * 128;            // both CTAs' boxes (out-of-range parts arrive as zeros)
    for (uint32_t it = pair; it < total && ok; it += npairs) {
      const Item w = decode(it, p, per_split, pix_tiles);
      const ConvTap tp = p.taps[w.tap];
      const int k0 = w.kt * 256 + rank * 128, c0 = w.ct * kBN + rank * 128;
      const uint32_t trow = quotient(w.t_begin, p.walk.tiles_w);
      int tn = quotient(trow, p.walk.tiles_h), th_ = trow - tn * p.tiles_h, tw = w.t_begin - trow * p.tiles_w;
      for (uint32_t t = w.t_begin; t < w.t_end; ++t) {
        const int w0 = tw * p.bw, h0 = th_ * p.bh, n0 = tn * p.bn;
        if (++tw == p.tiles_w) {
          tw = 0;
          if (++th_ == p.tiles_h) { th_ = 0; ++tn; }
        }
        if (!uniform_wait(&bars->empty[stage], phase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
        uint8_t* sa = smem + stage * kStageBytes;
        if (leader) {
          if (rank == 0 && pw == 0) mbar_expect_tx(&bars->full[stage], tx);
#pragma unroll
          for (int j = pw; j < kBoxes; j += kProducers) {
            if (j < kHalf) tma_load_5d_pair(sa + j * kBoxBytes, &p.dy_map, &bars->full[stage], k0 + j * atom<KIND>(), w.g, w0, h0, n0);
            else tma_load_5d_pair(sa + j * kBoxBytes, &p.x_views[tp.view], &bars->full[stage], c0 + (j - kHalf) * atom<KIND>(), w.g, w0 + tp.dw, h0 + tp.dh, n0);
          }
        }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else if (warp == 1) {
    if (rank == 0) {
      const bool leader = elect_one();
      int stage = 0, n = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t seen = 0;                                             // the next stage already seen full (mbar_look)
      const uint64_t desc_bits = smem_desc(0, kBoxBytes, kSbo, kLayout);
      const uint32_t desc_hi = static_cast<uint32_t>(desc_bits >> 32);
      const uint32_t lo_base = static_cast<uint32_t>(desc_bits) + (smem_u32(smem) >> 4);
      for (uint32_t it = pair; it < total && ok; it += npairs, ++n) {
        const Item w = decode(it, p, per_split, pix_tiles);
        const int buf = n & 1, ntiles = static_cast<int>(w.t_end - w.t_begin);
        const uint32_t aphase = (n >> 1) & 1;
        if (!uniform_wait(&bars->acc_empty[buf], aphase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem + buf * kBN;
        if (ksteps == 8) ok = mma_tiles<KIND, 8>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, leader, p.wait_clocks);
        else if (ksteps == 7) ok = mma_tiles<KIND, 7>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, leader, p.wait_clocks);
        else if (ksteps == 4) ok = mma_tiles<KIND, 4>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, leader, p.wait_clocks);
        else ok = mma_tiles<KIND, 0>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, leader, p.wait_clocks);
        if (ok && leader) umma_commit_pair(&bars->acc_full[buf]);
      }
      if (!ok && leader) report_status(p.status, kStatusTimeout);
    }
  } else {
    // Epilogue, 16 warps: warp w reads TMEM lanes [32 * (w % 4), +32) = 32 of this CTA's 128 filter rows and,
    // of those, every fourth 32-column chunk; rows go to the item's slab.
    const int quad = warp & 3;
    const int sub = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    bool ok = true;
    int n = 0;
    const int K = p.Kg * p.groups;
    for (uint32_t it = pair; it < total; it += npairs, ++n) {
      const Item w = decode(it, p, per_split, pix_tiles);
      const int buf = n & 1;
      const uint32_t aphase = (n >> 1) & 1;
      wait_or_walk_on(ok, &bars->acc_full[buf], aphase, bars, lane, p.wait_clocks);
      tc_fence_after();
      const int kq = w.kt * 256 + static_cast<int>(rank) * 128 + row;
      const bool valid = kq < p.Kg;
      float* slab = p.partial + (1LL * (p.atomic ? 0 : w.sp) * p.taps_total + p.taps[w.tap].wmat) * K * p.Cg;
      int c_lo, c_hi;
      diagonal_range(p.diag_c, p.diag_k, kq, p.Cg, &c_lo, &c_hi);
#pragma unroll 1
      for (int ch = sub; ch < kBN / 32; ch += kEpilogueWarps / 4) {
        const int c0 = w.ct * kBN + ch * 32;
        if (c0 >= p.Cg) break;
        uint32_t r[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + buf * kBN + ch * 32, r);
        tmem_ld_wait();
        if (valid) store_slab_chunk(r, slab, c0, c_lo, c_hi, p.Cg, K, w.g * p.Kg + kq, p.atomic, p.partial, p.partial_elems, p.status);
      }
      // every epilogue warp of this CTA has read its part: one arrival per CTA on the even CTA's barrier
      tc_fence_before();
      named_barrier(5, 32 * kEpilogueWarps);
      if (warp == 2 && lane == 0) mbar_arrive_leader(&bars->acc_empty[buf]);
    }
    if (!ok && lane == 0) report_status(p.status, kStatusTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (bars->abort) abort_grace(p.wait_clocks);
  cluster_sync_all();                        // no CTA of the pair leaves (or frees TMEM) while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 512);
  }
}

template <MmaKind KIND>
cudaError_t launch_one(const UmmaWgradParams& p, long long total, int num_sms, cudaStream_t s) {
  constexpr int smem = num_stages<KIND>() * stage_bytes<KIND>() + sizeof(Bars) + 1024;
  static PerDeviceOnce configured;
  cudaError_t e = configured.ensure([] {
    return cudaFuncSetAttribute(wgrad_pair_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (e != cudaSuccess) return e;
  const long long pairs = std::min<long long>(total, num_sms / 2);
  launch_chained(wgrad_pair_kernel<KIND>, static_cast<int>(2 * pairs), kThreads, smem, s, p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_wgrad_pair(const UmmaWgradParams& params, int dtype, int num_sms, cudaStream_t s) {
  UmmaWgradParams p = params;
  p.walk = item_walk(p.splits, p.ntaps, p.groups, p.ctiles, p.tiles_w, p.tiles_h);
  const long long total = 1LL * p.ktiles * p.ctiles * p.groups * p.ntaps * p.splits;
  if (total == 0) return cudaSuccess;
  if (total >= (1LL << 31) || 1LL * p.tiles_w * p.tiles_h * p.tiles_n >= (1LL << 31) || p.bw * p.bh * p.bn > kPix)
    return cudaErrorInvalidValue;
  return dtype == B200CONV_F16 ? launch_one<MmaKind::F16>(p, total, num_sms, s) : launch_one<MmaKind::TF32>(p, total, num_sms, s);
}

}  // namespace b200
