// Implicit-GEMM convolution with activation reuse across filter taps (tcgen05 + TMEM).
//
// When every tap reads the same channels-last view (stride-1 forward, every parity class of
// gradInputs) the operand rows of different taps are the same pixels shifted by a constant: with
// the output tile laid out on the slab's own pixel grid (tile width + halo columns), tap (dh, dw)
// is the slab advanced by dh * Ws + dw rows.  So one TMA box brings the slab (tile + halo, 128
// bytes of channels per pixel) once per channel block, and each tap's MMA reads it through a
// shared-memory descriptor that starts at the tap's row offset.  Only the filter tile is fetched
// per tap.  Accumulator rows that fall on halo columns / rows are computed and thrown away.
//
// A CTA keeps up to 512 TMEM columns of accumulators (two 128 x 256 tiles, or four 128 x 128 ...)
// so that a filter tile serves up to 512 output pixels.  Warp roles: warp 0 streams the activation
// slabs, warp 19 the filter tiles (TMA producers), warp 1 issues the MMAs and owns the TMEM, 16 epilogue
// warps; warp 18 is a second MMA issuer: with two or more accumulators per tile each issuer takes half
// of them (different TMEM columns, the same operands, the same order of accumulation).  Producer and
// issuer loops are followed by all 32 lanes of their warp; one elected lane issues.
//
// PAIR: two CTAs of a cluster work on two neighbouring pixel tiles and the same filters as one MMA unit (cta_group::2, M = 256).
// What bounds the one-CTA form is shared memory, 128 B/clk: four 128 x 256 x 8 tf32 MMAs (512 clocks) read 48 KB and
// the next filter tile's 32 KB are written beside them, 640 clocks; with 128 filters the operands alone take as long as the
// MMA.  In a pair each CTA loads, and its MMAs read, half of the filter tile: 32 + 16 KB, 384 clocks.
#include "internal.h"
#include "ptx.cuh"

namespace b200 {
namespace {

constexpr int kEpilogueWarps = 16;
constexpr int kSecondIssuer = 2 + kEpilogueWarps;     // warp index
constexpr int kFilterProducer = kSecondIssuer + 1;    // warp index: streams the filter tiles (warp 0 the slabs)
constexpr int kThreads = 32 * (kFilterProducer + 1);
constexpr int kMaxBStages = 8;
constexpr int kMaxSlabStages = 6;

struct alignas(16) Bars {
  uint64_t slab_full[kMaxSlabStages];
  uint64_t slab_empty[kMaxSlabStages];
  uint64_t b_full[kMaxBStages];
  uint64_t b_empty[kMaxBStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
};

template <typename T> __device__ __forceinline__ void store_out(T* p, float v);
template <> __device__ __forceinline__ void store_out<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void store_out<__half>(__half* p, float v) { *p = __float2half_rn(v); }

// Slice of a tile's reduction: channel blocks kb0..kb1, tap groups from tg0 in the first, up to tg1 in the last (inclusive).
struct Range { int kb0, kb1, tg0, tg1; };
__device__ __forceinline__ Range slice_range(const SlabConvParams& p, uint32_t slice) {
  const uint32_t stages_kb = p.tap_groups, stages_all = stages_kb * p.kblocks;
  if (p.splits == 1) return Range{0, p.kblocks - 1, 0, static_cast<int>(stages_kb) - 1};
  const uint32_t a = stages_all * slice / p.splits, b = stages_all * (slice + 1) / p.splits - 1;
  return Range{static_cast<int>(a / stages_kb), static_cast<int>(b / stages_kb), static_cast<int>(a % stages_kb), static_cast<int>(b % stages_kb)};
}

struct IssueLoop {
  const SlabConvParams& p;
  Bars* bars;
  uint8_t *smem, *bring;
  uint32_t tmem;
  int a_begin, na;
  uint32_t first, stride, total;
  bool dbl, leader;
  long long* trace;
};

// The MMAs of one issuing warp, all its tiles.  All 32 lanes follow the loop and wait on the barriers; one elected lane
// issues the MMAs and their commits.  A lone lane (code under `if (lane == 0)`) computes every descriptor on the
// per-thread datapath and moves it to uniform registers per MMA, which costs more clocks than a 128 x 64 or 128 x 128
// MMA runs.
// NT taps per filter stage, NA accumulators: a stage is straight-line code; 0: any number, in loops.  In loops the
// branches and the look-ups of each tap's shift take the warp longer than narrow MMAs run, and the wait at the head of
// each stage drains the tensor pipe.  The loop alone, operands always there, clocks per MMA in loops / straight-line
// with mbar_look(): 128 x 64 float32, three taps per stage, one accumulator 83 / 66, one for each issuer 59.5 / 48.3 (what the
// operands' reads take); one tap per stage and one accumulator: 128 x 32 133 / 71, 128 x 128 140 / 88, 128 x 256 147 / 132.
// No branch may stand among the elected lane's instructions: with the release of the slab under an `if` there, one
// tap per stage took 130 clocks again.
template <MmaKind KIND, int BN, bool PAIR, int NT, int NA>
__device__ __forceinline__ bool issue_tiles(const IssueLoop& w) {
  constexpr uint32_t kIdesc = instr_desc(KIND == MmaKind::TF32, false, false, PAIR ? 256 : 128, BN);
  constexpr int kBBytes = (PAIR ? BN / 2 : BN) * 128;
  constexpr bool kTogether = NT >= 4;      // many MMAs: issued by the whole warp (umma_words_if), under a branch their descriptors spill
  const SlabConvParams& p = w.p;
  Bars* bars = w.bars;
  const bool leader = w.leader;
  const int ncls = p.ncls, na = NA ? NA : w.na;
  const uint64_t desc_bits = smem_desc(0, 16, 1024);
  const uint32_t desc_hi = static_cast<uint32_t>(desc_bits >> 32), desc_lo = static_cast<uint32_t>(desc_bits);
  const uint32_t slab0 = desc_lo + ((smem_u32(w.smem) + 16384u * w.a_begin) >> 4), ring0 = desc_lo + (smem_u32(w.bring) >> 4);
  const uint32_t slab_units = static_cast<uint32_t>(p.slab_bytes) >> 4, stage_units = static_cast<uint32_t>(p.tps * kBBytes) >> 4;
  const uint32_t acc_step = ncls * BN;             // columns from one accumulator to the next
  auto commit = [&](uint64_t* bar) {
    if (PAIR) umma_commit_pair(bar);
    else umma_commit(bar);
  };
  int sb = 0, bs = 0, it = 0;
  uint32_t sphase = 0, bphase = 0;
  uint32_t slab_seen = 0, b_seen = 0, acc_seen = 0;  // the next slab / filter stage / accumulator already seen ready (mbar_look)
  for (uint32_t item = w.first; item < w.total; item += w.stride, ++it) {
    const uint32_t tile = quotient(item, p.walk.splits);
    const Range r = slice_range(p, item - tile * p.splits);
    // a constant where the tiles are full, and for 32 columns, whose MMAs take 36 to 40 clocks whatever is left out of them: with a
    // descriptor from a register these took 4 % longer
    uint32_t idesc = kIdesc;
    if (BN > 32 && p.n_mma % BN) {
      const int co_t = tile - quotient(tile, p.walk.tiles_co) * p.tiles_co;
      idesc = with_columns(kIdesc, mma_columns(p.n_mma, co_t * BN, BN, PAIR));
    }
    // two accumulator sets when they fit the 512 TMEM columns: the epilogue of a tile then
    // runs beside the MMAs of the next one
    const int buf = w.dbl ? (it & 1) : 0;
    const uint32_t aphase = w.dbl ? ((it >> 1) & 1) : (it & 1);
    const uint32_t acc0 = w.tmem + buf * (p.n_acc * acc_step) + w.a_begin * acc_step;
    if (!wait_seen(acc_seen, &bars->acc_empty[buf], aphase ^ 1, bars, p.wait_clocks)) return false;
    acc_seen = 0;
    tc_fence_after();
    for (int kb = r.kb0; kb <= r.kb1; ++kb) {
      if (!wait_seen(slab_seen, &bars->slab_full[sb], sphase, bars, p.wait_clocks)) return false;
      if (w.trace && it == 0 && kb == r.kb0) w.trace[2] = clock64();
      const uint32_t slab_lo = slab0 + sb * slab_units;
      const int tap_begin = kb == r.kb0 ? r.tg0 * p.tps : 0;
      const int tap_end = kb == r.kb1 ? min(p.ntaps, (r.tg1 + 1) * p.tps) : p.ntaps;
      for (int tap0 = tap_begin; tap0 < tap_end; tap0 += NT ? NT : p.tps) {
        const int nt = NT ? NT : min(p.tps, p.ntaps - tap0);
        uint32_t info[NT ? NT : 1];
        if (NT) {
#pragma unroll
          for (int q = 0; q < NT; ++q) info[q] = p.tap_issue[tap0 + q];
        }
        if (!wait_seen(b_seen, &bars->b_full[bs], bphase, bars, p.wait_clocks)) return false;
        tc_fence_after();
        const uint32_t ring_lo = ring0 + bs * stage_units;
        // 0 for the first products of the slice, or of the tap's class
        const uint32_t more = kb != r.kb0 || (ncls == 1 && tap0 != tap_begin), rest = more | (ncls == 1);
        auto mma = [&](int q, uint32_t tap, int a, int kk) {
          const uint32_t a_lo = slab_lo + slab_tap_shift(tap) + a * (16384 >> 4);
          const uint32_t acc = acc0 + slab_tap_column(tap) + a * acc_step, b_lo = ring_lo + ((q * kBBytes) >> 4), adds = kk ? 1u : (q ? rest : more) | slab_tap_adds(tap);
          if (kTogether) umma_words_if<KIND, PAIR>(leader, acc, a_lo + 2 * kk, b_lo + 2 * kk, desc_hi, idesc, adds);
          else umma_words<KIND, PAIR>(acc, a_lo + 2 * kk, b_lo + 2 * kk, desc_hi, idesc, adds);
        };
        // a stage's MMAs from u0 to u1, numbered (tap, accumulator, 32 bytes of the channels)
        auto part = [&](int u0, int u1) {
#pragma unroll
          for (int q = 0; q < NT; ++q)
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) {
                const int u = (q * NA + a) * 4 + kk;
                if (u >= u0 && u < u1) mma(q, info[q], a, kk);
              }
        };
        constexpr int kAll = NT * NA * 4, kBefore = kAll >= 16 ? kAll - 8 : kAll > 4 ? kAll - 4 : 2;
        if (kTogether) part(0, kBefore);
        if (!kTogether && leader) {
          if (NT) {
            part(0, kBefore);
          } else {
            for (int q = 0; q < nt; ++q) {
              const uint32_t tap = p.tap_issue[tap0 + q];
              for (int a = 0; a < (q + 1 == nt ? na - 1 : na); ++a) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) mma(q, tap, a, kk);
              }
            }
          }
        }
        __syncwarp();
        const int cur = bs;
        if (++bs == p.b_stages) { bs = 0; bphase ^= 1; }
        b_seen = mbar_look(&bars->b_full[bs], bphase);
        if (tap0 + p.tps >= tap_end) {             // the channel block ends, perhaps the tile too
          const int ns = sb + 1 == p.s_stages ? 0 : sb + 1;
          slab_seen = mbar_look(&bars->slab_full[ns], ns ? sphase : sphase ^ 1);
          if (w.dbl && kb == r.kb1) acc_seen = mbar_look(&bars->acc_empty[(it + 1) & 1], (((it + 1) >> 1) & 1) ^ 1);
        }
        if (kTogether) part(kBefore, kAll);
        if (leader) {
          if (NT) {
            if (!kTogether) part(kBefore, kAll);
          } else {
            const uint32_t tap = p.tap_issue[tap0 + nt - 1];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) mma(nt - 1, tap, na - 1, kk);
          }
          commit(&bars->b_empty[cur]);
        }
      }
      if (leader) commit(&bars->slab_empty[sb]);
      if (++sb == p.s_stages) { sb = 0; sphase ^= 1; }
    }
    if (leader) commit(&bars->acc_full[buf]);
    if (w.trace && it == 0) w.trace[3] = clock64();
  }
  return true;
}

template <MmaKind KIND, int BN, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
conv_slab_kernel(const __grid_constant__ SlabConvParams p) {
  using OutT = typename std::conditional<KIND == MmaKind::TF32, float, __half>::type;
  constexpr int kBK = KIND == MmaKind::TF32 ? 32 : 64;
  constexpr int kBBytes = (PAIR ? BN / 2 : BN) * 128;   // filters this CTA loads per tap and channel block

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* bring = smem + p.s_stages * p.slab_bytes;    // the slab ring comes first
  const int stage_b = p.tps * kBBytes;                  // bytes of one filter stage: tps taps
  Bars* bars = reinterpret_cast<Bars*>(bring + p.b_stages * stage_b + p.stage_reserved);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  long long* trace = p.trace ? p.trace + blockIdx.x * 32 : nullptr;   // 32 slots per CTA
  if (trace && threadIdx.x == 0) {
    trace[0] = clock64();
    trace[7] = static_cast<long long>(global_ns());
  }
  const uint32_t slab_tx = static_cast<uint32_t>(p.nb * p.Hs * p.Ws) * 128u;
  // tile counts fit 32 bits (the launcher checks): 64-bit divisions per tile would cost each
  // role about a thousand clocks, a fifth of a small tile
  const uint32_t pix_tiles = static_cast<uint32_t>(p.tiles_w) * p.tiles_h * p.tiles_n;
  const uint32_t total = (PAIR ? (pix_tiles + 1) / 2 : pix_tiles) * p.groups * p.tiles_co * p.splits;
  // a pair's CTAs take the pixel tiles 2 i and 2 i + 1 (the second of an odd count's last pair lies behind the last
  // image: its loads read zeros and its stores are left out); splits is 1
  const uint32_t rank = PAIR ? cluster_ctarank() : 0;
  const uint32_t first = PAIR ? blockIdx.x >> 1 : blockIdx.x, stride = PAIR ? gridDim.x >> 1 : gridDim.x;
  // Work item = (tile, slice of the reduction), the slices of a tile side by side.  A slice is a range of
  // filter stages (channel block x group of tps taps), in the order the unsplit loop walks them.
  const uint32_t splits = p.splits;
  const int ncls = p.ncls;                              // accumulator (a, class q): columns (a * ncls + q) * BN
  const bool dbl = 2 * p.n_acc * ncls * BN <= 512;
  const int issuers = p.n_acc >= 2 ? 2 : 1;

  if (threadIdx.x == 0) {
    // operands are released, and accumulators handed over, when every issuer's MMAs are done
    for (int s = 0; s < kMaxSlabStages; ++s) {
      mbar_init(&bars->slab_full[s], 1);
      mbar_init(&bars->slab_empty[s], issuers);
    }
    for (int s = 0; s < kMaxBStages; ++s) {
      mbar_init(&bars->b_full[s], 1);
      mbar_init(&bars->b_empty[s], issuers);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->acc_full[b], issuers);
      mbar_init(&bars->acc_empty[b], PAIR ? 2 : 32 * kEpilogueWarps);     // a pair: one arrival per CTA, on the even one
    }
    bars->abort = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(&bars->tmem_base, 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(&bars->tmem_base, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();      // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  pdl_enter();              // the next kernel may start once this CTA holds its TMEM; nothing global was touched before
  if (trace && threadIdx.x == 0) trace[1] = clock64();

  if (warp == 0) {
    // Slab producer.  Every lane runs the loop (so that its control flow and address arithmetic are
    // warp-uniform); one elected lane issues the copies.  Slabs and filter tiles have a producer warp
    // each: one in-order producer stalled on a free slab buffer while the filter ring ran dry, and the
    // MMA warp then waited a full L2 latency for filters (a third of its loop on the 3x3 layers).
    const bool leader = elect_one();
    if (leader) tma_prefetch_desc(&p.view);
    int sb = 0;
    uint32_t sphase = 0;
    bool ok = true;
    for (uint32_t item = first; item < total && ok; item += stride) {
      const uint32_t t = quotient(item, p.walk.splits);
      const Range r = slice_range(p, item - t * splits);
      const TileAt at = tile_at<PAIR>(p.walk, t, rank);
      const int g = at.g, w0 = at.w * p.wt, h0 = at.h * p.th, n0 = at.n * p.nb;
      for (int kb = r.kb0; kb <= r.kb1; ++kb) {
        if (!uniform_wait(&bars->slab_empty[sb], sphase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
        if (leader) {
          if (rank == 0) mbar_expect_tx(&bars->slab_full[sb], PAIR ? 2 * slab_tx : slab_tx);      // both CTAs' bytes
          if (PAIR) tma_load_5d_pair(smem + sb * p.slab_bytes, &p.view, &bars->slab_full[sb], kb * kBK, g, w0 + p.dw_min, h0 + p.dh_min, n0);
          else tma_load_5d(smem + sb * p.slab_bytes, &p.view, &bars->slab_full[sb], kb * kBK, g, w0 + p.dw_min, h0 + p.dh_min, n0);
        }
        if (++sb == p.s_stages) { sb = 0; sphase ^= 1; }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else if (warp == kFilterProducer) {
    // Filter producer: the same walk over tiles, channel blocks and taps, filter tiles only.
    const bool leader = elect_one();
    if (leader) tma_prefetch_desc(&p.wmap);
    int bs = 0;
    uint32_t bphase = 0;
    bool ok = true;
    for (uint32_t item = first; item < total && ok; item += stride) {
      const uint32_t t = quotient(item, p.walk.splits);
      const Range r = slice_range(p, item - t * splits);
      const TileAt at = tile_at<PAIR>(p.walk, t, rank);
      const int co_t = at.co_t, g = at.g;
      // a pair's CTAs load one half each of what the tile's MMAs take (and rows that those leave out)
      const int row0 = co_t * BN + static_cast<int>(rank) * (mma_columns(p.n_mma, co_t * BN, BN, true) / 2);
      auto load = [&](uint8_t* dst, int kb, int mat) {
        if (PAIR) tma_load_4d_pair(dst, &p.wmap, &bars->b_full[bs], kb * kBK, row0, g, mat);
        else tma_load_4d(dst, &p.wmap, &bars->b_full[bs], kb * kBK, row0, g, mat);
      };
      for (int kb = r.kb0; kb <= r.kb1 && ok; ++kb) {
        const int tap_end = kb == r.kb1 ? min(p.ntaps, (r.tg1 + 1) * p.tps) : p.ntaps;
        for (int tap = kb == r.kb0 ? r.tg0 * p.tps : 0; tap < tap_end; tap += p.tps) {
          if (!uniform_wait(&bars->b_empty[bs], bphase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
          const int nt = min(p.tps, p.ntaps - tap);         // taps of this stage
          if (leader) {
            // A box takes the issuing thread about 400 clocks whatever its size, as long as the MMAs of two
            // 128 x 64 taps: neighbouring taps come as one box.  (The box of a last, shorter group reads on into
            // the next matrix or zeros; its bytes count too.)
            if (!p.tap_boxes) {
              if (rank == 0) mbar_expect_tx(&bars->b_full[bs], (PAIR ? 2 : 1) * p.tps * kBBytes);
              load(bring + bs * stage_b, kb, p.tap_wmat[tap]);
            } else {
              if (rank == 0) mbar_expect_tx(&bars->b_full[bs], (PAIR ? 2 : 1) * nt * kBBytes);
              for (int q = 0; q < nt; ++q) load(bring + bs * stage_b + q * kBBytes, kb, p.tap_wmat[tap + q]);
            }
          }
          if (++bs == p.b_stages) { bs = 0; bphase ^= 1; }
        }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else if (warp == 1 || warp == kSecondIssuer) {
    // this issuer's accumulators of every tile: [a_begin, a_begin + na)
    const int a_split = issuers == 2 ? (p.n_acc + 1) / 2 : p.n_acc;
    const int a_begin = warp == 1 ? 0 : a_split, na = warp == 1 ? a_split : p.n_acc - a_split;
    if (rank == 0 && na > 0) {                 // a pair: the even CTA issues for both
      const bool leader = elect_one();
      IssueLoop w{p, bars, smem, bring, tmem, a_begin, na, first, stride, total, dbl, leader, warp == 1 && leader ? trace : nullptr};
      const int nt = p.ntaps % p.tps == 0 ? p.tps : 0;       // 0: groups of taps of different sizes
      bool ok;
      if (nt == 1 && na == 1) ok = issue_tiles<KIND, BN, PAIR, 1, 1>(w);
      else if (nt == 1 && na == 2) ok = issue_tiles<KIND, BN, PAIR, 1, 2>(w);
      else if (nt == 2 && na == 1) ok = issue_tiles<KIND, BN, PAIR, 2, 1>(w);
      else if (nt == 2 && na == 2) ok = issue_tiles<KIND, BN, PAIR, 2, 2>(w);
      else if (nt == 3 && na == 1) ok = issue_tiles<KIND, BN, PAIR, 3, 1>(w);
      else if (nt == 3 && na == 2) ok = issue_tiles<KIND, BN, PAIR, 3, 2>(w);
      else if (BN <= 64 && nt == 4 && na == 1) ok = issue_tiles<KIND, BN, PAIR, BN <= 64 ? 4 : 0, 1>(w);
      else if (BN <= 64 && nt == 4 && na == 2) ok = issue_tiles<KIND, BN, PAIR, BN <= 64 ? 4 : 0, 2>(w);
      else if (BN <= 64 && nt == 5 && na == 1) ok = issue_tiles<KIND, BN, PAIR, BN <= 64 ? 5 : 0, 1>(w);
      else if (BN <= 64 && nt == 5 && na == 2) ok = issue_tiles<KIND, BN, PAIR, BN <= 64 ? 5 : 0, 2>(w);
      else if (BN <= 32 && nt == 9 && na == 1) ok = issue_tiles<KIND, BN, PAIR, BN <= 32 ? 9 : 0, 1>(w);
      else if (BN <= 32 && nt == 9 && na == 2) ok = issue_tiles<KIND, BN, PAIR, BN <= 32 ? 9 : 0, 2>(w);
      else ok = issue_tiles<KIND, BN, PAIR, 0, 0>(w);
      if (!ok && leader) report_status(p.status, kStatusTimeout);
    }
  } else if (warp < kSecondIssuer) {
    // 16 epilogue warps: warp w reads TMEM lanes [32*(w%4), +32) (the hardware's rule) and, of
    // those rows, every fourth 32-column chunk.  A single warp keeps only a few stores in flight,
    // so the store bandwidth of the SM is reached by the number of warps, not by wider stores.
    const int quad = warp & 3;
    const int sub = (warp - 2) >> 2;
    OutT* out = static_cast<OutT*>(p.out);
    const int per_img = p.Hs * p.Ws;
    // channels-last output whose 32-channel groups are 16-byte aligned: 16-byte stores
    const bool rowwise = p.out_sc == 1 && ((p.n_out * sizeof(OutT) | reinterpret_cast<uintptr_t>(p.out)) & 15) == 0;
    // Staged TMA stores (n_acc is 1, 2 or 4): this lane's dense row of the tile's staging buffer, -1 outside of the tile.  One number kept over
    // all tiles: with its six parts kept instead, the lanes' own stores below, which need none of them, were 10 to 35 % slower (32 filters at 112x112, 64
    // images, float32, NCHW output 187 -> 150 us, with a residual 369 -> 278; 8 groups of 32 at 28x28, 256 images, with a residual 754 -> 570).
    int staged_row = -1;
    if (p.tma_out) {
      const int pos = (sub & (p.n_acc - 1)) * 128 + quad * 32 + lane, ni = pos / per_img, rem = pos - ni * per_img, hh = rem / p.Ws, ww = rem - hh * p.Ws;
      if (ni < p.nb && hh < p.th && ww < p.wt) staged_row = (ni * p.th + hh) * p.wt + ww;
    }
    bool ok = true;
    int it = 0;
    int nstore = 0;                              // chunks this warp's group has staged so far
    for (uint32_t item = first; item < total; item += stride, ++it) {
      const TileAt at = tile_at<PAIR>(p.walk, quotient(item, p.walk.splits), rank);
      const int co_t = at.co_t, g = at.g, w0 = at.w * p.wt, h0 = at.h * p.th, n0 = at.n * p.nb;
      const int buf = dbl ? (it & 1) : 0;
      const uint32_t aphase = dbl ? ((it >> 1) & 1) : (it & 1);
      wait_or_walk_on(ok, &bars->acc_full[buf], aphase, bars, lane, p.wait_clocks);
      tc_fence_after();
      if (trace && it == 0 && threadIdx.x == 64) trace[4] = clock64();
      const int co_base = co_t * BN;
      const int nchunks = min(BN / 32, (p.n_out - co_base + 31) / 32);
      const uint32_t lane_base = tmem + buf * (p.n_acc * ncls * BN) + (static_cast<uint32_t>(quad * 32) << 16);

      if (splits > 1) {
        // raw accumulators; conv_reduce.cu adds the slices and applies the epilogue
        const int rows = p.n_acc * 128;
        for (int a = 0; a < p.n_acc; ++a) {
          const int pos = a * 128 + quad * 32 + lane, rem = pos % per_img;
          const bool inbox = pos / per_img < p.nb && rem / p.Ws < p.th && rem % p.Ws < p.wt;
          float4* dst = reinterpret_cast<float4*>(p.partial) + static_cast<long long>(item) * rows * (BN / 4) + pos;
#pragma unroll 1
          for (int ch = sub; ch < nchunks; ch += kEpilogueWarps / 4) {
            uint32_t r[32];
            tmem_ld32(lane_base + a * BN + ch * 32, r);
            tmem_ld_wait();
            if (!inbox) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (B200_IN_RANGE((reinterpret_cast<float*>(dst + (ch * 8 + j) * rows) - p.partial) + 4 <= p.partial_elems, p.status))
                dst[(ch * 8 + j) * rows] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                       __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
          }
        }
      } else if (p.tma_out) {
        // Groups of 4 * n_acc warps take whole 128-byte channel chunks of the tile: lane -> its pixel's
        // dense row of a staging buffer (16-byte pieces swizzled like the store map expects),
        // then one thread stores the box.  Bias and ReLU are applied on the way.  A group owns
        // `bufs` staging buffers and fills them in turn; before a buffer is refilled only the
        // store that last read it must have finished reading, so a store runs beside the next
        // chunk's (or the next tile's) TMEM reads instead of being waited for.
        const int a = sub & (p.n_acc - 1), log_acc = p.n_acc >> 1, grp = sub >> log_acc, ngrp = (kEpilogueWarps / 4) >> log_acc;
        const int gthreads = 128 * p.n_acc;
        const bool inbox = staged_row >= 0;
        const int drow = staged_row;
        const bool issuer = a == 0 && quad == 0 && lane == 0;   // issues all of the group's stores
        const bool plain = p.epi.alpha == 1.f && !p.bias && !p.relu;
        const int bufs = p.stage_nbuf >= 2 * ngrp ? 2 : 1;
        constexpr int kCh = 128 / static_cast<int>(sizeof(OutT));   // channels of one 128-byte staged row
        const int nstaged = min(BN / kCh, (p.n_out - co_base + kCh - 1) / kCh);
        for (int cc = grp; cc < nstaged * ncls; cc += ngrp, ++nstore) {
          const int cls = ncls > 1 ? cc / nstaged : 0, ch = cc - cls * nstaged;
          uint8_t* stg = smem + p.stage_off + (grp * bufs + (bufs == 2 ? (nstore & 1) : 0)) * p.stage_bytes;
          uint8_t* srow = stg + drow * 128;
          const int co0 = co_base + ch * kCh;
          const OutT* bias = p.bias ? static_cast<const OutT*>(p.bias) + g * p.n_out + co0 : nullptr;
          if (nstore >= bufs) {                // the buffer's previous box must have been read
            if (issuer) {
              if (bufs == 2) bulk_wait_read<1>();
              else bulk_wait_read<0>();
            }
            named_barrier(1 + grp, gthreads);
          }
#pragma unroll
          for (int part = 0; part < kCh / 32; ++part) {
            uint32_t r[32];
            tmem_ld32(lane_base + (a * ncls + cls) * BN + ch * kCh + part * 32, r);
            tmem_ld_wait();
            if (!inbox) continue;
            zero_pad_columns(r, co0 + part * 32, p.n_real);
            const OutT* bp = bias ? bias + part * 32 : nullptr;
            if (plain) {
              // no scale, bias or activation (gradInputs, bare forward): convert and stage only.
              // The epilogue warps are bound by their instruction issue, not by TMEM or shared memory.
              if (sizeof(OutT) == 4) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  *reinterpret_cast<uint4*>(srow + ((j ^ (drow & 7)) << 4)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
              } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  uint32_t h[4];
#pragma unroll
                  for (int q = 0; q < 4; ++q) {
                    __half2 h2 = __floats2half2_rn(__uint_as_float(r[8 * j + 2 * q]), __uint_as_float(r[8 * j + 2 * q + 1]));
                    h[q] = *reinterpret_cast<uint32_t*>(&h2);
                  }
                  *reinterpret_cast<uint4*>(srow + (((part * 4 + j) ^ (drow & 7)) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
                }
              }
            } else if (sizeof(OutT) == 4) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float f[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  f[q] = p.epi.alpha * __uint_as_float(r[4 * j + q]);
                  if (bp) f[q] += static_cast<float>(bp[4 * j + q]);
                  if (p.relu) f[q] = p.epi.lin * f[q] + p.epi.abs * fabsf(f[q]);
                }
                *reinterpret_cast<float4*>(srow + ((j ^ (drow & 7)) << 4)) = make_float4(f[0], f[1], f[2], f[3]);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint32_t h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  float f0 = p.epi.alpha * __uint_as_float(r[8 * j + 2 * q]);
                  float f1 = p.epi.alpha * __uint_as_float(r[8 * j + 2 * q + 1]);
                  if (bp) { f0 += static_cast<float>(bp[8 * j + 2 * q]); f1 += static_cast<float>(bp[8 * j + 2 * q + 1]); }
                  if (p.relu) {
                    f0 = p.epi.lin * f0 + p.epi.abs * fabsf(f0);
                    f1 = p.epi.lin * f1 + p.epi.abs * fabsf(f1);
                  }
                  __half2 h2 = __floats2half2_rn(f0, f1);
                  h[q] = *reinterpret_cast<uint32_t*>(&h2);
                }
                *reinterpret_cast<uint4*>(srow + (((part * 4 + j) ^ (drow & 7)) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
              }
            }
          }
          if (p.epi.pool) {
            // 2x2 max pooling of the staged chunk (Pool{ignore_border=True, mode='max'}, ws = stride = 2): the
            // tile's width and height are even, so every window lies inside it.  The group's threads read the
            // four staged rows of a window (16-byte pieces, un-swizzled by row), keep the maxima in registers
            // until every read is done, then write the pooled rows to the front of the same buffer, swizzled
            // for the pooled rows, and the store below moves a quarter of the bytes.
            named_barrier(1 + grp, gthreads);
            const int tig = a * 128 + quad * 32 + lane;
            const int pw = p.wt >> 1, ph = p.th >> 1;
            const int prows = p.nb * ph * pw;
            uint4 keep[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int i = tig + u * gthreads;
              if (i < prows * 8) {
                const int pr = i >> 3, piece = i & 7;
                const int w2 = pr % pw, h2 = (pr / pw) % ph, ni2 = pr / (pw * ph);
                const int d00 = (ni2 * p.th + 2 * h2) * p.wt + 2 * w2;
                uint4 m = *reinterpret_cast<const uint4*>(stg + d00 * 128 + ((piece ^ (d00 & 7)) << 4));
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                  const int dk = d00 + (k & 1) + (k >> 1) * p.wt;
                  const uint4 v = *reinterpret_cast<const uint4*>(stg + dk * 128 + ((piece ^ (dk & 7)) << 4));
                  if (sizeof(OutT) == 4) {
                    m.x = __float_as_uint(fmaxf(__uint_as_float(m.x), __uint_as_float(v.x)));
                    m.y = __float_as_uint(fmaxf(__uint_as_float(m.y), __uint_as_float(v.y)));
                    m.z = __float_as_uint(fmaxf(__uint_as_float(m.z), __uint_as_float(v.z)));
                    m.w = __float_as_uint(fmaxf(__uint_as_float(m.w), __uint_as_float(v.w)));
                  } else {
                    __half2* mh = reinterpret_cast<__half2*>(&m);
                    const __half2* vh = reinterpret_cast<const __half2*>(&v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) mh[e] = __hmax2(mh[e], vh[e]);
                  }
                }
                keep[u] = m;
              }
            }
            named_barrier(1 + grp, gthreads);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int i = tig + u * gthreads;
              if (i < prows * 8) {
                const int pr = i >> 3, piece = i & 7;
                *reinterpret_cast<uint4*>(stg + pr * 128 + ((piece ^ (pr & 7)) << 4)) = keep[u];
              }
            }
          }
          fence_async_smem();
          named_barrier(1 + grp, gthreads);
          // a tiled store must not start at a negative coordinate, and its staging rows must lie
          // inside the reserved shared memory
          if (issuer && (!PAIR || n0 < p.Nimg) && (ncls == 1 || (w0 < p.cls_W[cls] && h0 < p.cls_H[cls])) &&
              B200_IN_RANGE(g * p.n_out + co0 >= 0 && w0 >= 0 && h0 >= 0 && n0 >= 0 && w0 < p.Wt && h0 < p.Ht &&
                                      n0 < p.Nimg && ch * kCh + kCh <= BN, p.status)) {
            if (p.epi.pool) tma_store_4d(&p.out_map[0], stg, g * p.n_out + co0, w0 >> 1, h0 >> 1, n0);
            else tma_store_4d(&p.out_map[cls], stg, g * p.n_out + co0, w0, h0, n0);
            bulk_commit();
          }
        }
      } else
      for (int a = 0; a < p.n_acc; ++a) {
        // this lane's output pixel for accumulator a
        const int pos = a * 128 + quad * 32 + lane;        // position on the slab grid
        const int ni = pos / per_img, rem = pos % per_img;
        const int hh = rem / p.Ws, ww = rem % p.Ws;
        const int n = n0 + ni, h = h0 + hh, w = w0 + ww;
        const bool valid = ni < p.nb && hh < p.th && ww < p.wt && n < p.Nimg && h < p.Ht && w < p.Wt;
        OutT* pix = out + (p.out_off + n * p.out_sn + h * p.out_sh + w * p.out_sw) +
                    1LL * g * p.n_out * p.out_sc;
        const OutT* res = p.epi.residual ? static_cast<const OutT*>(p.epi.residual) + (pix - out) : nullptr;
        for (int ch = sub; ch < nchunks; ch += kEpilogueWarps / 4) {
          uint32_t r[32];
          tmem_ld32(lane_base + a * BN + ch * 32, r);
          tmem_ld_wait();
          if (!valid) continue;
          const int co0 = co_base + ch * 32;
          zero_pad_columns(r, co0, p.n_real);
          const OutT* bias = p.bias ? static_cast<const OutT*>(p.bias) + g * p.n_out + co0 : nullptr;
          if (rowwise) {   // n_out is a whole number of 16-byte pieces: a piece is all in or all out
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
                  store_out<OutT>(pix + (co0 + j) * p.out_sc, v);
              }
            }
          }
        }
      }
      tc_fence_before();
      if (PAIR) {
        named_barrier(5, 32 * kEpilogueWarps);
        if (warp == 2 && lane == 0) mbar_arrive_leader(&bars->acc_empty[buf]);
      } else {
        mbar_arrive(&bars->acc_empty[buf]);
      }
      if (trace && it == 0 && threadIdx.x == 64) trace[5] = clock64();
    }
    if (p.tma_out && lane == 0) bulk_wait<0>();  // this thread's stores (if it issued any) have left shared memory
    if (!ok && lane == 0) report_status(p.status, kStatusTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (bars->abort) abort_grace(p.wait_clocks);
  if (PAIR) cluster_sync_all();              // no CTA of the pair leaves (or frees TMEM) while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem, 512);
    else tmem_dealloc(tmem, 512);
  }
  if (trace && threadIdx.x == 0) {
    trace[6] = clock64();
    trace[8] = static_cast<long long>(global_ns());
  }
}

template <MmaKind KIND, int BN, bool PAIR>
cudaError_t configure() {
  static PerDeviceOnce configured;
  return configured.ensure([] {
    return cudaFuncSetAttribute(conv_slab_kernel<KIND, BN, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  });
}

template <MmaKind KIND, int BN, bool PAIR>
cudaError_t launch_one(const SlabConvParams& p, long long total, int num_sms, cudaStream_t s) {
  const int smem = p.s_stages * p.slab_bytes + p.b_stages * p.tps * (PAIR ? BN / 2 : BN) * 128 + p.stage_reserved + sizeof(Bars) + 1024;
  cudaError_t e = configure<KIND, BN, PAIR>();
  if (e != cudaSuccess) return e;
  const int units = PAIR ? num_sms / 2 : num_sms;
  const int grid = static_cast<int>(total < units ? total : units) * (PAIR ? 2 : 1);
  launch_linked(true, conv_slab_kernel<KIND, BN, PAIR>, grid, kThreads, smem, s, PAIR ? 2 : 1, p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t load_conv_slab(int dtype, int bn) {
  const bool f16 = dtype == B200CONV_F16;
  switch (bn) {
    case 32: return f16 ? configure<MmaKind::F16, 32, false>() : configure<MmaKind::TF32, 32, false>();
    case 64: return f16 ? configure<MmaKind::F16, 64, false>() : configure<MmaKind::TF32, 64, false>();
    case 128: return f16 ? configure<MmaKind::F16, 128, false>() : configure<MmaKind::TF32, 128, false>();
    default: return f16 ? configure<MmaKind::F16, 256, false>() : configure<MmaKind::TF32, 256, false>();
  }
}

cudaError_t launch_conv_slab(const SlabConvParams& p, int dtype, int bn, int num_sms, cudaStream_t s) {
  const long long pix = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
  const long long total = (p.pair ? (pix + 1) / 2 : pix) * p.groups * p.tiles_co * p.splits;
  if (total == 0 || p.ntaps == 0) return cudaSuccess;
  if (p.ncls < 1 || p.ncls > kMaxSlabClasses || (p.ncls > 1 && (p.splits != 1 || !p.tma_out || p.epi.pool))) return cudaErrorInvalidValue;
  if (total >= (1LL << 31) || (p.pair && (p.splits != 1 || num_sms < 2))) return cudaErrorInvalidValue;
  const bool f16 = dtype == B200CONV_F16;
#define B200_CASE(BNV)                                                                  \
  case BNV:                                                                             \
    return f16 ? launch_one<MmaKind::F16, BNV, false>(p, total, num_sms, s)             \
               : launch_one<MmaKind::TF32, BNV, false>(p, total, num_sms, s);
#define B200_PAIR(BNV)                                                                  \
  case BNV:                                                                             \
    return f16 ? launch_one<MmaKind::F16, BNV, true>(p, total, num_sms, s)              \
               : launch_one<MmaKind::TF32, BNV, true>(p, total, num_sms, s);
  if (p.pair) switch (bn) {
    B200_PAIR(64)
    B200_PAIR(128)
    B200_PAIR(256)
    default: return cudaErrorInvalidValue;
  }
  switch (bn) {
    B200_CASE(32)
    B200_CASE(64)
    B200_CASE(128)
    default:
    B200_CASE(256)
  }
#undef B200_CASE
#undef B200_PAIR
}

}  // namespace b200
