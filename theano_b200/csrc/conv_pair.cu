// The per-tap implicit GEMM (conv_umma.cu) on pairs of CTAs: tcgen05.mma.cta_group::2, M = 256, at least 128 filters.
//
// Two CTAs of a cluster compute two neighbouring pixel tiles (128 rows each) for the same filters.  Per tap and 128 bytes of channels
// each loads the box of its own pixels and half of the filter tile; one thread of the even CTA issues the MMAs over both CTAs'
// operands, and each CTA's TMEM receives its own accumulator rows.  What bounds the one-CTA form with 256 filters is L2: 48 KB per
// 512 clocks of MMAs are 96 B/clk, where an SM receives 73; in a pair it is 32 KB, 64 B/clk.
//
// Tiles beyond whole waves are cut: 98 pair tiles on 74 pairs of SMs take as long as 148.  The reduction of the first `cut` tiles goes to
// `splits` pairs each, which leave float32 accumulators in global memory; each pair then takes a whole tile.  Whoever leaves the last slice
// of a CTA's half of a cut tile (an atomic count, nobody waits) adds the slices in order and writes the result, beside the MMAs of its
// whole tile.  Where no whole tile follows, conv_reduce.cu does it, on all SMs.  (pair_cut() in api.cu decides.)
//
// Warp roles (608 threads): warps 0 and 18 TMA producers (pixels, filters: the issue of a box takes a thread about 300 clocks), warp 1
// MMA issuer of the even CTA and TMEM owner, 16 epilogue warps.  Two accumulators, so that a tile's read-out runs beside the next tile's MMAs; the
// results leave as staged TMA stores, 128 bytes of channels per group of four warps.  Nothing is multicast.
//
// Measured (a B200, filters packed, one-CTA kernel -> pairs): float16, 256 images, 3x3 256 -> 256 at 14x14 48 -> 43 us (37 without any
// loads), 512 -> 512 at 7x7 (106 pair tiles, 32 of them cut in two) 52 -> 42, strided 1024 -> 2048 1x1 52 -> 45; float32 256 -> 256 at 14x14, 128 images
// (98 tiles, 24 cut in three) 58 -> 42, 512 -> 512, 64 images 100 -> 76.  With the slices added by a kernel of its own the cut ones took 46, 51 and 82.
// With 2x2 max pooling in the epilogue (slab kernel on pairs -> here), float32, 64 images: 512 -> 512 at 28x28 365 -> 312, at 14x14 103 -> 85,
// 256 -> 256 at 56x56 346 -> 329.
// Flattened 1x1 layers stay with gemm_pair.cu (256 -> 1024 at 14x14 33 us here, 31 there).
#include "internal.h"
#include "ptx.cuh"

#include <algorithm>

namespace b200 {
namespace {

constexpr int kRows = 128;                                     // pixels of a CTA's tile
constexpr int kABytes = kRows * 128;
constexpr int kEpilogueWarps = 16;
constexpr int kFilterProducer = 2 + kEpilogueWarps;      // warp index: streams the filter tiles (warp 0 the pixels)
constexpr int kThreads = 32 * (kFilterProducer + 1);
constexpr int kStoreBytes = kRows * 128;                       // one staged chunk: 128 bytes of channels of the CTA's pixels
constexpr int kMaxStages = 6;
template <int BN> constexpr int stage_bytes() { return kABytes + BN / 2 * 128; }
template <int BN> constexpr int num_stages() { return 160 * 1024 / stage_bytes<BN>() < kMaxStages ? 160 * 1024 / stage_bytes<BN>() : kMaxStages; }

struct alignas(16) Bars {
  uint64_t full[kMaxStages];        // even CTA: both CTAs' boxes of a stage have landed
  uint64_t empty[kMaxStages];       // each CTA: the MMAs that read the stage are done
  uint64_t acc_full[2];             // each CTA: the tile's accumulator is complete
  uint64_t acc_empty[2];            // even CTA: both CTAs' epilogues have read the accumulator
  uint32_t tmem_base;
  volatile int abort, last;         // last: this CTA's slice of a cut tile was the last to arrive
};

// Work item: a tile (of a pair) and the stages [k0, k1) of its reduction; slice < 0: all of them.  The slices of the cut tiles come first.
struct Item { uint32_t tile, k0, k1; int slice; };
__device__ __forceinline__ Item item_of(const UmmaConvParams& p, uint32_t item, uint32_t kiters) {
  const uint32_t splits = p.splits, slices = p.cut * splits;
  if (item >= slices) return Item{item - slices + p.cut, 0, kiters, -1};
  const uint32_t t = quotient(item, p.walk.splits), s = item - t * splits;
  return Item{t, kiters * s / splits, kiters * (s + 1) / splits, static_cast<int>(s)};
}

// The larger of each of the float or half numbers in 16 bytes.
template <class T>
__device__ __forceinline__ uint4 larger(uint4 a, uint4 b) {
  if (sizeof(T) == 4) {
    auto most = [](uint32_t x, uint32_t y) { return __float_as_uint(fmaxf(__uint_as_float(x), __uint_as_float(y))); };
    return make_uint4(most(a.x, b.x), most(a.y, b.y), most(a.z, b.z), most(a.w, b.w));
  }
  __half2 *ah = reinterpret_cast<__half2*>(&a), *bh = reinterpret_cast<__half2*>(&b);
#pragma unroll
  for (int e = 0; e < 4; ++e) ah[e] = __hmax2(ah[e], bh[e]);
  return a;
}

template <MmaKind KIND, int BN>
__global__ void __launch_bounds__(kThreads, 1)
conv_pair_kernel(const __grid_constant__ UmmaConvParams p) {
  using OutT = typename std::conditional<KIND == MmaKind::TF32, float, __half>::type;
  constexpr int kStages = num_stages<BN>();
  constexpr int kBK = KIND == MmaKind::TF32 ? 32 : 64;          // channels per stage, and of a staged chunk
  constexpr uint32_t kIdesc = instr_desc(KIND == MmaKind::TF32, false, false, 2 * kRows, BN);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* staging = smem + kStages * stage_bytes<BN>();
  Bars* bars = reinterpret_cast<Bars*>(staging + 4 * kStoreBytes);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const uint32_t first = blockIdx.x >> 1, stride = gridDim.x >> 1;
  const int rows_used = p.bw * p.bh * p.bn;
  const uint32_t tx_bytes = 2 * (rows_used * 128 + BN / 2 * 128);                 // both CTAs' boxes
  const uint32_t kiters = p.ntaps * p.kblocks;
  const uint32_t co_groups = static_cast<uint32_t>(p.tiles_co) * p.groups, tiles_wh = static_cast<uint32_t>(p.tiles_w) * p.tiles_h;
  const uint32_t tiles = (tiles_wh * p.tiles_n + 1) / 2 * co_groups;              // counts fit 32 bits (the launcher checks)
  const uint32_t total = p.cut * p.splits + tiles - p.cut;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->acc_full[b], 1);
      mbar_init(&bars->acc_empty[b], 2);
    }
    bars->abort = 0;
    mbar_fence_init();
  }
  // descriptors, beside the set-up and the wait for the kernel before (they are parameters, not global data)
  if (warp == 2 && lane == 0) {
    for (int v = 0; v < p.nviews; ++v) tma_prefetch_desc(&p.views[v]);
    tma_prefetch_desc(&p.wmap);
    tma_prefetch_desc(&p.out_map);
  }
  if (warp == 1) {                                               // the same warp in both CTAs
    tmem_alloc_pair(&bars->tmem_base, 2 * BN);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                            // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  pdl_enter();              // the next kernel may start once this CTA holds its TMEM; nothing global was touched before

  if (warp == 0 || warp == kFilterProducer) {
    // all lanes follow the loop, one elected lane issues
    const bool leader = elect_one();
    const bool b_box = warp != 0;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (uint32_t item = first; item < total && ok; item += stride) {
      const Item w = item_of(p, item, kiters);
      const TileAt at = tile_at<true>(p.walk, w.tile, rank);     // behind the last tile of an odd count: an image that is not there, zeros
      const int co_t = at.co_t, g = at.g, w0 = at.w * p.bw, h0 = at.h * p.bh, n0 = at.n * p.bn;
      const int row0 = co_t * BN + static_cast<int>(rank) * (mma_columns(p.n_mma, co_t * BN, BN, true) / 2);
      uint32_t k = w.k0;
      const int tap0 = k ? k / p.kblocks : 0;
      for (int tap = tap0, kb = k - tap0 * p.kblocks; k < w.k1 && ok; ++tap, kb = 0) {
        const ConvTap tp = p.taps[tap];
        for (; kb < p.kblocks && k < w.k1; ++kb, ++k) {
          if (!uniform_wait(&bars->empty[stage], phase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
          uint8_t* sa = smem + stage * stage_bytes<BN>();
          if (leader) {
            if (!b_box) {
              if (rank == 0) mbar_expect_tx(&bars->full[stage], tx_bytes);
              tma_load_5d_pair(sa, &p.views[tp.view], &bars->full[stage], kb * kBK, g, w0 + tp.dw, h0 + tp.dh, n0);
            } else {
              tma_load_3d_pair(sa + kABytes, &p.wmap, &bars->full[stage], kb * kBK, row0, tp.wmat * p.groups + g);
            }
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else if (warp == 1) {
    if (rank == 0) {                                             // the even CTA issues for both
      const bool leader = elect_one();
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint64_t desc_bits = smem_desc(0, 16, 1024);
      const uint32_t desc_hi = static_cast<uint32_t>(desc_bits >> 32);
      const uint32_t lo_base = static_cast<uint32_t>(desc_bits) + (smem_u32(smem) >> 4);
      uint32_t seen = 0, acc_seen = 0;           // next stage / next accumulator already seen ready (mbar_look)
      for (uint32_t item = first; item < total && ok; item += stride, ++it) {
        const Item w = item_of(p, item, kiters);
        const int buf = it & 1;
        const uint32_t aphase = (it >> 1) & 1;
        uint32_t idesc = kIdesc;
        if (p.n_mma % BN) idesc = with_columns(kIdesc, mma_columns(p.n_mma, (w.tile - quotient(w.tile, p.walk.tiles_co) * p.tiles_co) * BN, BN, true));
        if (!wait_seen(acc_seen, &bars->acc_empty[buf], aphase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem + buf * BN;
        for (uint32_t k = w.k0; k < w.k1; ++k) {
          if (!wait_seen(seen, &bars->full[stage], phase, bars, p.wait_clocks)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_lo = lo_base + stage * (stage_bytes<BN>() >> 4), b_lo = a_lo + (kABytes >> 4);
          if (leader) {
            umma_words<KIND, true>(d_tmem, a_lo, b_lo, desc_hi, idesc, k != w.k0);
            umma_words<KIND, true>(d_tmem, a_lo + 2, b_lo + 2, desc_hi, idesc, 1u);
          }
          __syncwarp();
          const int cur = stage;
          if (++stage == kStages) { stage = 0; phase ^= 1; }
          seen = mbar_look(&bars->full[stage], phase);
          if (k + 1 == w.k1) acc_seen = mbar_look(&bars->acc_empty[(it + 1) & 1], (((it + 1) >> 1) & 1) ^ 1);
          if (leader) {
            umma_words<KIND, true>(d_tmem, a_lo + 4, b_lo + 4, desc_hi, idesc, 1u);
            umma_words<KIND, true>(d_tmem, a_lo + 6, b_lo + 6, desc_hi, idesc, 1u);
            umma_commit_pair(&bars->empty[cur]);
          }
        }
        if (ok && leader) umma_commit_pair(&bars->acc_full[buf]);
      }
      if (!ok && leader) report_status(p.status, kStatusTimeout);
    }
  } else {
    // Warp w reads TMEM lanes [32 * (w % 4), +32); the four groups of four warps take 128-byte channel chunks in turn, stage them (swizzled
    // like the store map expects) and one thread per group stores the box.  A group waits for its buffer only before refilling it.
    const int quad = warp & 3, grp = (warp - 2) >> 2;
    const int row = quad * 32 + lane;                            // this lane's pixel of the CTA's tile
    const bool issuer = quad == 0 && lane == 0;
    const bool plain = p.epi.alpha == 1.f && !p.bias && !p.relu;
    uint8_t* stg = staging + grp * kStoreBytes;
    uint8_t* srow = stg + row * 128;
    bool ok = true, stored = false;
    int it = 0, turn = 0;
    for (uint32_t item = first; item < total; item += stride, ++it) {
      const Item w = item_of(p, item, kiters);
      const TileAt at = tile_at<true>(p.walk, w.tile, rank);
      const int co_t = at.co_t, g = at.g, w0 = at.w * p.bw, h0 = at.h * p.bh, n0 = at.n * p.bn;
      const int buf = it & 1;
      wait_or_walk_on(ok, &bars->acc_full[buf], (it >> 1) & 1, bars, lane, p.wait_clocks);
      tc_fence_after();
      const int co_base = co_t * BN;
      const uint32_t lane_base = tmem + buf * BN + (static_cast<uint32_t>(quad * 32) << 16);
      // slices of this CTA's half of a cut tile, one after the other
      float4* slabs = reinterpret_cast<float4*>(p.partial) + (static_cast<long long>(w.tile) * 2 + rank) * p.splits * (kRows * BN / 4) + row;
      const bool present = row < rows_used && n0 < p.Nimg;
      bool finish = true;
      if (w.slice >= 0) {
        // raw accumulators
        float4* dst = slabs + w.slice * (kRows * BN / 4);
#pragma unroll 1
        for (int ch = grp; ch < BN / 32 && co_base + ch * 32 < p.n_out; ch += 4) {
          uint32_t r[32];
          tmem_ld32(lane_base + ch * 32, r);
          tmem_ld_wait();
          if (!present) continue;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (B200_IN_RANGE((reinterpret_cast<float*>(dst + (ch * 8 + j) * kRows) - p.partial) + 4 <= p.partial_elems, p.status))
              dst[(ch * 8 + j) * kRows] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                      __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
        }
        tc_fence_before();
        __threadfence();
        named_barrier(5, 32 * kEpilogueWarps);
        if (warp == 2 && lane == 0) {
          mbar_arrive_leader(&bars->acc_empty[buf]);
          // the count of the tile's slices that have arrived goes back to zero with the last one
          bars->last = p.arrivals && atomicInc(p.arrivals + w.tile * 2 + rank, p.splits - 1) == static_cast<uint32_t>(p.splits) - 1;
        }
        named_barrier(5, 32 * kEpilogueWarps);
        finish = bars->last;
        if (finish) __threadfence();
      }
      if (finish) {
        const int nstaged = min(BN / kBK, (p.n_out - co_base + kBK - 1) / kBK);
        for (int ch = (grp - turn) & 3; ch < nstaged; ch += 4) {
          const int co0 = co_base + ch * kBK;
          const OutT* bias = p.bias ? static_cast<const OutT*>(p.bias) + g * p.n_out + co0 : nullptr;
          if (stored) {                                          // the buffer's previous box must have been read
            if (issuer) bulk_wait_read<0>();
            named_barrier(1 + grp, 128);
          }
          stored = true;
#pragma unroll
          for (int part = 0; part < kBK / 32; ++part) {
            uint32_t r[32];
            if (w.slice < 0) {
              tmem_ld32(lane_base + ch * kBK + part * 32, r);
              tmem_ld_wait();
            } else {
              // the slices in order, whichever arrived last; eight loads in flight
              const float4* src = slabs + (ch * kBK + part * 32) / 4 * kRows;
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = 0;
#pragma unroll 1
              for (int s = 0; s < (present ? p.splits : 0); ++s, src += kRows * BN / 4) {
                float4 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __ldcg(src + j * kRows);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  r[4 * j] = __float_as_uint(__uint_as_float(r[4 * j]) + v[j].x); r[4 * j + 1] = __float_as_uint(__uint_as_float(r[4 * j + 1]) + v[j].y);
                  r[4 * j + 2] = __float_as_uint(__uint_as_float(r[4 * j + 2]) + v[j].z); r[4 * j + 3] = __float_as_uint(__uint_as_float(r[4 * j + 3]) + v[j].w);
                }
              }
              __syncwarp();
            }
            zero_pad_columns(r, co0 + part * 32, p.n_real);
            const OutT* bp = bias ? bias + part * 32 : nullptr;
            if (!plain) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                float f = p.epi.alpha * __uint_as_float(r[j]);
                if (bp) f += static_cast<float>(bp[j]);
                if (p.relu) f = p.epi.lin * f + p.epi.abs * fabsf(f);
                r[j] = __float_as_uint(f);
              }
            }
            if (row >= rows_used) continue;
            if (sizeof(OutT) == 4) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                *reinterpret_cast<uint4*>(srow + ((j ^ (row & 7)) << 4)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint32_t h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  __half2 h2 = __floats2half2_rn(__uint_as_float(r[8 * j + 2 * q]), __uint_as_float(r[8 * j + 2 * q + 1]));
                  h[q] = *reinterpret_cast<uint32_t*>(&h2);
                }
                *reinterpret_cast<uint4*>(srow + (((part * 4 + j) ^ (row & 7)) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
              }
            }
          }
          if (p.epi.pool) {
            // 2x2 max pooling of the staged chunk, as in conv_slab.cu: the tile's sides are even, the maxima stay in registers until all rows
            // are read, then go to the front of the buffer
            named_barrier(1 + grp, 128);
            const int pw = p.bw >> 1, ph = p.bh >> 1, prows = p.bn * ph * pw;
            uint4 keep[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int i = row + u * 128, pr = i >> 3, piece = i & 7;
              if (pr < prows) {
                const int pl = pr / pw, w2 = pr - pl * pw, img = pl / ph, d00 = (img * p.bh + 2 * (pl - img * ph)) * p.bw + 2 * w2;
                uint4 m = *reinterpret_cast<const uint4*>(stg + d00 * 128 + ((piece ^ (d00 & 7)) << 4));
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                  const int dk = d00 + (k & 1) + (k >> 1) * p.bw;
                  m = larger<OutT>(m, *reinterpret_cast<const uint4*>(stg + dk * 128 + ((piece ^ (dk & 7)) << 4)));
                }
                keep[u] = m;
              }
            }
            named_barrier(1 + grp, 128);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int i = row + u * 128, pr = i >> 3, piece = i & 7;
              if (pr < prows) *reinterpret_cast<uint4*>(stg + pr * 128 + ((piece ^ (pr & 7)) << 4)) = keep[u];
            }
          }
          fence_async_smem();
          named_barrier(1 + grp, 128);
          if (issuer && n0 < p.Nimg && B200_IN_RANGE(w0 >= 0 && w0 < p.Wt && h0 >= 0 && h0 < p.Ht && n0 >= 0 && co0 >= 0, p.status)) {
            if (p.epi.pool) tma_store_4d(&p.out_map, stg, g * p.n_out + co0, w0 >> 1, h0 >> 1, n0);
            else tma_store_4d(&p.out_map, stg, g * p.n_out + co0, w0, h0, n0);
            bulk_commit();
          }
        }
        turn += nstaged;
      }
      if (w.slice >= 0) continue;
      tc_fence_before();
      // one arrival per CTA: sixteen releases at cluster scope, one per warp, cost 2000 clocks a tile (256 -> 1024 1x1 46 -> 33 us)
      named_barrier(5, 32 * kEpilogueWarps);
      if (warp == 2 && lane == 0) mbar_arrive_leader(&bars->acc_empty[buf]);
    }
    if (!ok && lane == 0) report_status(p.status, kStatusTimeout);
    if (lane == 0) bulk_wait<0>();           // this thread's stores (if it issued any) have left shared memory
  }

  tc_fence_before();
  __syncthreads();
  if (bars->abort) abort_grace(p.wait_clocks);
  cluster_sync_all();                        // no CTA of the pair leaves (or frees TMEM) while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 2 * BN);
  }
}

template <MmaKind KIND, int BN> constexpr int smem_bytes() { return num_stages<BN>() * stage_bytes<BN>() + 4 * kStoreBytes + static_cast<int>(sizeof(Bars)) + 1024; }

template <MmaKind KIND, int BN>
cudaError_t launch_one(const UmmaConvParams& p, long long items, int num_sms, cudaStream_t s) {
  constexpr int smem = smem_bytes<KIND, BN>();
  static_assert(smem <= 227 * 1024, "shared memory");
  static PerDeviceOnce configured;
  cudaError_t e = configured.ensure([] { return cudaFuncSetAttribute(conv_pair_kernel<KIND, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  if (e != cudaSuccess) return e;
  const int pairs = static_cast<int>(std::min<long long>(items, num_sms / 2));
  launch_linked(true, conv_pair_kernel<KIND, BN>, 2 * pairs, kThreads, smem, s, 2, p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_conv_pair(const UmmaConvParams& p, int dtype, int num_sms, cudaStream_t s) {
  const long long tiles = (1LL * p.tiles_w * p.tiles_h * p.tiles_n + 1) / 2 * p.groups * p.tiles_co;
  if (tiles == 0 || p.ntaps == 0) return cudaSuccess;
  if (num_sms < 2 || p.cut < 0 || p.cut > tiles || p.splits < 1 || (p.cut > 0 && !p.partial)) return cudaErrorInvalidValue;
  const long long items = 1LL * p.cut * p.splits + tiles - p.cut;
  if (items >= (1LL << 30)) return cudaErrorInvalidValue;
  const bool f16 = dtype == B200CONV_F16;
  if (p.bn_cols == 256) return f16 ? launch_one<MmaKind::F16, 256>(p, items, num_sms, s) : launch_one<MmaKind::TF32, 256>(p, items, num_sms, s);
  if (p.bn_cols == 128) return f16 ? launch_one<MmaKind::F16, 128>(p, items, num_sms, s) : launch_one<MmaKind::TF32, 128>(p, items, num_sms, s);
  return cudaErrorInvalidValue;
}

}  // namespace b200
