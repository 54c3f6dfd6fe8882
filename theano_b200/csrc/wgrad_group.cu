// Filter gradient on tcgen05 tensor cores with operand sharing across filter taps.
//
//   dW[tap][k, c] = sum over output pixels q of  dy[q, k] * x_view[q + (dh, dw)_tap, c]
//
// Work item = (128-filter tile, 128-channel tile, conv group, tap group, split-K slice).  A tap
// group holds up to four taps with the same view and row offset dh; their x operands are the same
// pixels shifted by dw.  The reduction pixels of a stage are a box of the output grid whose rows
// are widened by the column span of the taps (dy reads zeros there), so "shifted by dw" is a plain
// row offset into one shared-memory x tile: per stage one dy tile and one x tile are fetched and
// every tap of the group accumulates into its own 128 x 128 TMEM accumulator.  That divides the
// number of TMA boxes per MMA.  (MN-major operands run at the same rate as K-major ones: 64 clocks per 128 x 128 MMA,
// whatever the row offset.  Which of the three gradWeights kernels is fastest depends on the layer, so the first call
// of a geometry times those that apply.)
//
// Operands are MN-major (the pixel is the slow index of a channels-last row): float16 with the
// 16-byte swizzle, tf32 with the 32-byte-atom swizzle; row offsets that are not multiples of the
// swizzle period are fine because the hardware swizzles on absolute shared-memory address bits.
// Warp roles: warp 0 and the last three warps TMA producers, warp 1 MMA issuer and TMEM owner,
// 16 epilogue warps.
#include <algorithm>

#include "internal.h"
#include "ptx.cuh"
#include "wgrad_slab.cuh"

namespace b200 {
namespace {

constexpr int kEpilogueWarps = 16;
// A thread gets one TMA box accepted every ~300 clocks: the boxes of a stage are spread over
// several producer warps (warp 0 and the warps after the epilogue warps) and their lanes, box j
// to producer j % kProducers, lane j / kProducers.
constexpr int kProducers = 4;
constexpr int kFirstExtraProducer = 2 + kEpilogueWarps;
constexpr int kThreads = 32 * (kFirstExtraProducer + kProducers - 1);
constexpr int kBN = 128;                       // channels per accumulator
// A box holds the stage's pixel rows and room for the largest column offset (p.box_bytes, a multiple of the 1024-byte
// swizzle period); a stage holds the boxes that the layer's filters and channels fill (p.a_boxes + p.b_boxes of at most
// 128 / atom each).  What bounds a stage of a narrow layer is the latency of its boxes, so the ring is as deep as
// the shared memory allows: with room for 128 x 128 in every stage there were two stages for every layer.
// An MMA reads 128 rows and its columns whatever the layer has: behind a stage's boxes that is other operand data
// (allocated memory, rows and columns of the accumulator that nobody reads).
constexpr int kSmemBudget = 222 * 1024;
constexpr int kMaxStages = 6;

template <MmaKind KIND> constexpr int atom() { return KIND == MmaKind::TF32 ? 32 : 64; }
// Operand memory of a ring, the reach of the last stage's MMAs included.
int ring_bytes(int stages, int atom, int a_boxes, int b_boxes, int box_bytes) {
  const int full = 128 / atom;
  return ((stages - 1) * (a_boxes + b_boxes) + a_boxes + full) * box_bytes;
}

struct alignas(16) Bars {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full;
  uint64_t acc_empty;
  uint32_t tmem_base;
  volatile int abort;
};

struct Item {
  int kt, ct, g, grp, sp;
  uint32_t t_begin, t_end;
};

// 32-bit arithmetic throughout (the launcher checks the counts)
__device__ __forceinline__ Item decode(uint32_t it, const GroupWgradParams& p, uint32_t per_split,
                                       uint32_t pix_tiles) {
  Item r;
  const uint32_t a = quotient(it, p.walk.splits), b = quotient(a, p.walk.taps), c = quotient(b, p.walk.groups);
  r.sp = it - a * p.walk.splits.d;
  r.grp = a - b * p.walk.taps.d;
  r.g = b - c * p.walk.groups.d;
  r.kt = quotient(c, p.walk.ctiles);
  r.ct = c - r.kt * p.walk.ctiles.d;
  r.t_begin = r.sp * per_split;
  r.t_end = r.t_begin + per_split < pix_tiles ? r.t_begin + per_split : pix_tiles;
  return r;
}

// Layers with at most 64 channels (STACK): the NT taps become NT groups of columns of ONE MMA per swizzle atom of channels
// (64 in float16, 32 in tf32).  The x operand's leading-dimension offset (the distance between column groups)
// is set to the taps' row spacing, so that column group q reads the x tile q taps further: 128 x (64 NT)
// (tf32: at most two of 128 x (32 NT), kStackTwice) instead of NT half-empty 128 x 128 MMAs.
enum Stack { kWide = 0, kStack, kStackTwice };

struct IssueLoop {
  Bars* bars;
  uint32_t tmem, lo_base, desc_hi;
  uint32_t toff[4];                  // row offset of every tap's x operand, in descriptor address units
  int ksteps, ntiles, stages;
  uint32_t a_units, stage_units;     // of the dy boxes of a stage / of a stage
  uint32_t stack_delta, box2;        // added to the x descriptor of stacked taps / distance of their second atom of channels
  bool leader, timed;
  long long limit;
  // the pipeline position, carried across items
  int stage;
  uint32_t phase, seen;
  long long t_wait;
};

// The MMA issuer's loop over the pixel tiles (pipeline stages) of one work item with NT taps.  Returns false when a wait
// ran out.  Exactly KS reduction steps per stage as straight-line code, or any number (0) in blocks of four: the issuing
// thread must spend fewer clocks per MMA than the MMA takes (64 for 128 x 128 x 8 tf32), and a taken branch between
// two of them alone costs 65 to 85.
template <MmaKind KIND, int NT, int KS, Stack STACK>
__device__ __forceinline__ bool mma_item(IssueLoop& w) {
  constexpr int kK = KIND == MmaKind::TF32 ? 8 : 16, kAtom = atom<KIND>();
  constexpr uint32_t kStep = (kK * 128) >> 4;
  constexpr uint32_t kIdesc = instr_desc(KIND == MmaKind::TF32, true, true, 128, STACK == kWide ? kBN : NT == 1 ? 64 : kAtom * NT);
  Bars* bars = w.bars;
  const uint32_t lane = w.leader, tmem = w.tmem, desc_hi = w.desc_hi;
  const int ntiles = w.ntiles, stages = w.stages;
  uint32_t toff[NT];                 // of the x operand of each tap (the column groups' start, when stacked)
#pragma unroll
  for (int q = 0; q < NT; ++q) toff[q] = w.a_units + w.toff[q] + (STACK != kWide && NT > 1 ? w.stack_delta : 0u);
  int stage = w.stage;
  uint32_t phase = w.phase, seen = w.seen;
  const int ksteps = KS ? KS : w.ksteps, half = ksteps / 2;
  uint32_t acc = 0u;
  for (int t = 0; t < ntiles; ++t) {
    const long long tw = w.timed ? clock64() : 0;
    if (!wait_seen(seen, &bars->full[stage], phase, bars, w.limit)) return false;
    if (w.timed) w.t_wait += clock64() - tw;
    tc_fence_after();
    const uint32_t a_lo = w.lo_base + stage * w.stage_units;
    auto step = [&](int ks, uint32_t accumulate) {
      const uint32_t a = a_lo + ks * kStep;
      if (STACK == kWide) {
#pragma unroll
        for (int q = 0; q < NT; ++q) umma_words_if<KIND>(lane, tmem + q * kBN, a, a + toff[q], desc_hi, kIdesc, accumulate);
      } else {
        // (a single tap is stacked with nothing: its atoms are the column groups, as ever)
        umma_words_if<KIND>(lane, tmem, a, a + toff[0], desc_hi, kIdesc, accumulate);
        if (STACK == kStackTwice && NT > 1) umma_words_if<KIND>(lane, tmem + kAtom * NT, a, a + toff[0] + w.box2, desc_hi, kIdesc, accumulate);
      }
    };
    auto steps = [&](int k0, int k1) {
      if (KS) {
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
          if (ks >= k0 && ks < k1) step(ks, ks ? 1u : acc);
        return;
      }
      int ks = k0;
      for (; ks + 4 <= k1; ks += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) step(ks + u, ks + u ? 1u : acc);
      }
      for (; ks < k1; ++ks) step(ks, ks ? 1u : acc);
    };
    steps(0, half);
    const int cur = stage;
    const bool wrap = stage + 1 == stages;
    stage = wrap ? 0 : stage + 1;
    phase ^= wrap ? 1u : 0u;
    seen = mbar_look(&bars->full[stage], phase);
    steps(half, ksteps);
    umma_commit_if(lane, &bars->empty[cur]);
    acc = 1u;
  }
  w.stage = stage; w.phase = phase; w.seen = seen;
  return true;
}

template <MmaKind KIND, int NT, Stack STACK>
__device__ __forceinline__ bool mma_item_steps(IssueLoop& w) {
  // the usual numbers of steps: images of 7, 14, 28 and 56 columns / segments of 56
  if (w.ksteps == 8) return mma_item<KIND, NT, 8, STACK>(w);
  if (w.ksteps == 7) return mma_item<KIND, NT, 7, STACK>(w);
  return mma_item<KIND, NT, 0, STACK>(w);
}
template <MmaKind KIND, Stack STACK>
__device__ __forceinline__ bool mma_item_taps(IssueLoop& w, int ntap) {
  if (ntap == 1) return mma_item_steps<KIND, 1, STACK>(w);
  if (ntap == 2) return mma_item_steps<KIND, 2, STACK>(w);
  if (ntap == 3) return mma_item_steps<KIND, 3, STACK>(w);
  return mma_item_steps<KIND, 4, STACK>(w);
}

template <MmaKind KIND, Stack STACK>
__global__ void __launch_bounds__(kThreads, 1)
wgrad_group_kernel(const __grid_constant__ GroupWgradParams p) {
  constexpr int kAtom = atom<KIND>();
  constexpr int kABoxes = 128 / kAtom, kBBoxes = kBN / kAtom;
  const int box_bytes = p.box_bytes, stage_bytes = (p.a_boxes + p.b_boxes) * box_bytes;
  constexpr int kK = KIND == MmaKind::TF32 ? 8 : 16;
  constexpr uint32_t kSbo = KIND == MmaKind::TF32 ? 512 : 1024;
  constexpr uint64_t kLayout = KIND == MmaKind::TF32 ? kSwizzle128Base32 : kSwizzle128;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  Bars* bars = reinterpret_cast<Bars*>(smem + p.ring_bytes);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  // phase timing (optional): [0] MMA thread waiting for operands, [1] its whole loop,
  // [2] first producer waiting for a free stage, [3] its whole loop, [4] kernel start to end,
  // [9] / [10] GPU-wide timer at start / end
  long long* trace = p.trace ? p.trace + blockIdx.x * 16 : nullptr;
  const long long t_begin = trace ? clock64() : 0;
  if (trace && threadIdx.x == 0) trace[9] = static_cast<long long>(global_ns());
  const int ksteps = (p.rows_a + kK - 1) / kK;
  const uint32_t pix_tiles = static_cast<uint32_t>(p.tiles_w) * p.tiles_h * p.tiles_n;
  const uint32_t per_split = (pix_tiles + p.splits - 1) / p.splits;
  const uint32_t total = static_cast<uint32_t>(p.ktiles) * p.ctiles * p.groups * p.ngroups * p.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->acc_empty, 32 * kEpilogueWarps);
    bars->abort = 0;
    mbar_fence_init();
  }
  // descriptors, beside the set-up and the wait for the kernel before (they are parameters, not global data)
  if (warp == 2 && lane == 0) {
    for (int v = 0; v < p.nviews; ++v) tma_prefetch_desc(&p.x_views[v]);
    tma_prefetch_desc(&p.dy_map);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  // Rows past the boxes are never written by TMA.  The MMA reads whole groups of kK dy rows and,
  // for the x operand, up to the largest column offset further: clear those rows once.  (dy rows
  // there must be zero; the x rows only need to be finite.)
  {
    const int boxes = p.stages * (p.a_boxes + p.b_boxes);
    const int first = min(p.rows_a, p.rows_b);
    const int nrows = box_bytes / 128 - first;
    for (int i = threadIdx.x; i < boxes * nrows * 8; i += kThreads) {
      const int box = i / (nrows * 8), rem = i % (nrows * 8);
      const int stage_box = box % (p.a_boxes + p.b_boxes);
      const int row = first + rem / 8;
      const int written = stage_box < p.a_boxes ? p.rows_a : p.rows_b;
      if (row >= written)
        *(reinterpret_cast<uint4*>(smem + box * box_bytes + row * 128) + rem % 8) = make_uint4(0, 0, 0, 0);
    }
    fence_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  pdl_enter();              // the next kernel may start once this CTA holds its TMEM; nothing global was touched before

  if (warp == 0 || warp >= kFirstExtraProducer) {
    const int pw = warp == 0 ? 0 : warp - kFirstExtraProducer + 1;
    // every lane follows the loop (warp-uniform control flow and addresses); one elected lane issues
    // this warp's boxes of a stage: pw, pw + kProducers, ...
    const bool leader = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    long long t_wait = 0;
    for (uint32_t it = blockIdx.x; it < total && ok; it += gridDim.x) {
      const Item w = decode(it, p, per_split, pix_tiles);
      const int view = p.grp_view[w.grp], dh = p.grp_dh[w.grp], dwmin = p.view_dwmin[view];
      const int a_boxes = min(kABoxes, (p.Kg - w.kt * 128 + kAtom - 1) / kAtom);
      const int b_boxes = min(kBBoxes, (p.Cg - w.ct * kBN + kAtom - 1) / kAtom);
      const uint32_t tx = (a_boxes * p.rows_a + b_boxes * p.rows_b) * 128;
      // tile coordinates advance by counting: 64-bit divisions per stage would cost the producers
      // more clocks than the stage's MMAs take
      const uint32_t trow = quotient(w.t_begin, p.walk.tiles_w);
      int tn = quotient(trow, p.walk.tiles_h), th_ = trow - tn * p.tiles_h, tw = w.t_begin - trow * p.tiles_w;
      for (uint32_t t = w.t_begin; t < w.t_end; ++t) {
        const int w0 = tw * p.wt, h0 = th_ * p.th, n0 = tn * p.nb;
        if (++tw == p.tiles_w) {
          tw = 0;
          if (++th_ == p.tiles_h) { th_ = 0; ++tn; }
        }
        const long long tw0 = trace ? clock64() : 0;
        if (!uniform_wait(&bars->empty[stage], phase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
        if (trace) t_wait += clock64() - tw0;
        uint8_t* sa = smem + stage * stage_bytes;
        uint8_t* sb = sa + p.a_boxes * box_bytes;
        if (leader) {
          if (pw == 0) mbar_expect_tx(&bars->full[stage], tx);
          for (int j = pw; j < a_boxes + b_boxes; j += kProducers) {
            if (j < a_boxes)
              tma_load_5d(sa + j * box_bytes, &p.dy_map, &bars->full[stage], w.kt * 128 + j * kAtom, w.g,
                          w0, h0, n0);
            else
              tma_load_5d(sb + (j - a_boxes) * box_bytes, &p.x_views[view], &bars->full[stage],
                          w.ct * kBN + (j - a_boxes) * kAtom, w.g, w0 + dwmin, h0 + dh, n0);
          }
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
    if (trace && leader && pw == 0) { trace[2] = t_wait; trace[3] = clock64() - t_begin; }
  } else if (warp == 1) {
    // all lanes follow the loop and wait; one elected lane issues the MMAs and their commits
    const uint64_t desc_bits = smem_desc(0, box_bytes, kSbo, kLayout);
    IssueLoop w;
    w.bars = bars; w.tmem = tmem;
    w.lo_base = static_cast<uint32_t>(desc_bits) + (smem_u32(smem) >> 4);
    w.desc_hi = static_cast<uint32_t>(desc_bits >> 32);
    w.ksteps = ksteps; w.stages = p.stages;
    w.a_units = (p.a_boxes * box_bytes) >> 4; w.stage_units = stage_bytes >> 4;
    // stacked taps: the low descriptor word carries the leading-dimension offset in bits [16, 30)
    w.stack_delta = ((static_cast<uint32_t>(p.stack_step * 128) >> 4) - (static_cast<uint32_t>(box_bytes) >> 4)) << 16;
    w.box2 = static_cast<uint32_t>(box_bytes) >> 4;
    w.leader = elect_one(); w.timed = trace != nullptr;
    w.limit = p.wait_clocks;
    w.stage = 0; w.phase = 0; w.seen = 0; w.t_wait = 0;
    bool ok = true;
    int n = 0;
    for (uint32_t it = blockIdx.x; it < total && ok; it += gridDim.x, ++n) {
      const Item item = decode(it, p, per_split, pix_tiles);
      const int first_tap = p.grp_first[item.grp], ntap = p.grp_n[item.grp];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        w.toff[q] = q < ntap ? static_cast<uint32_t>(p.tap_off[first_tap + q]) * (128u >> 4) : 0u;
      if (!uniform_wait(&bars->acc_empty, (n & 1) ^ 1, bars, p.wait_clocks)) { ok = false; break; }
      tc_fence_after();
      w.ntiles = static_cast<int>(item.t_end - item.t_begin);
      ok = mma_item_taps<KIND, STACK>(w, ntap);
      if (ok && w.leader) umma_commit(&bars->acc_full);
    }
    if (!ok && w.leader) report_status(p.status, kStatusTimeout);
    if (trace && w.leader) { trace[0] = w.t_wait; trace[1] = clock64() - t_begin; }
  } else {
    const int quad = warp & 3;
    const int sub = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    const int K = p.Kg * p.groups;
    bool ok = true;
    int n = 0;
    for (uint32_t it = blockIdx.x; it < total && ok; it += gridDim.x, ++n) {
      const Item w = decode(it, p, per_split, pix_tiles);
      const int first_tap = p.grp_first[w.grp], ntap = p.grp_n[w.grp];
      if (!warp_wait_or_abort(&bars->acc_full, n & 1, bars, lane, p.wait_clocks)) { ok = false; break; }
      tc_fence_after();
      const int kq = w.kt * 128 + row;
      const bool valid = kq < p.Kg;
      int c_lo, c_hi;
      diagonal_range(p.diag_c, p.diag_k, kq, p.Cg, &c_lo, &c_hi);
      const int items = ntap * (kBN / 32);
#pragma unroll 1
      for (int item = sub; item < items; item += kEpilogueWarps / 4) {
        const int q = item / (kBN / 32), ch = item % (kBN / 32);
        const int c0 = w.ct * kBN + ch * 32;
        if (c0 >= p.Cg) continue;
        uint32_t r[32];
        // columns of tap q, channels 32 ch: side by side per tap, or per atom of channels and then per tap
        const int col = STACK != kWide ? (ch * 32 / kAtom) * (kAtom * ntap) + q * kAtom + ch * 32 % kAtom : q * kBN + ch * 32;
        tmem_ld32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + col, r);
        tmem_ld_wait();
        if (!valid) continue;
        float* slab = p.partial + (1LL * (p.atomic ? 0 : w.sp) * p.taps_total + p.tap_wmat[first_tap + q]) * K * p.Cg;
        store_slab_chunk(r, slab, c0, c_lo, c_hi, p.Cg, K, w.g * p.Kg + kq, p.atomic, p.partial, p.partial_elems, p.status);
      }
      tc_fence_before();
      mbar_arrive(&bars->acc_empty);
    }
    if (!ok && lane == 0) report_status(p.status, kStatusTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (bars->abort) abort_grace(p.wait_clocks);
  if (trace && threadIdx.x == 0) {
    trace[4] = clock64() - t_begin;
    trace[10] = static_cast<long long>(global_ns());
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <MmaKind KIND, Stack STACK>
cudaError_t launch_one(const GroupWgradParams& p, long long total, int num_sms, cudaStream_t s) {
  const int smem = p.ring_bytes + static_cast<int>(sizeof(Bars)) + 1024;
  static PerDeviceOnce configured;
  cudaError_t e = configured.ensure([] { return cudaFuncSetAttribute(wgrad_group_kernel<KIND, STACK>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024); });
  if (e != cudaSuccess) return e;
  const int grid = static_cast<int>(total < num_sms ? total : num_sms);
  launch_chained(wgrad_group_kernel<KIND, STACK>, grid, kThreads, smem, s, p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_wgrad_group(const GroupWgradParams& params, int dtype, int num_sms, cudaStream_t s) {
  GroupWgradParams p = params;
  p.walk = item_walk(p.splits, p.ngroups, p.groups, p.ctiles, p.tiles_w, p.tiles_h);
  const long long total = 1LL * p.ktiles * p.ctiles * p.groups * p.ngroups * p.splits;
  if (total == 0) return cudaSuccess;
  if (total >= (1LL << 31) || 1LL * p.tiles_w * p.tiles_h * p.tiles_n >= (1LL << 31)) return cudaErrorInvalidValue;
  const int at = dtype == B200CONV_F16 ? 64 : 32, kk = dtype == B200CONV_F16 ? 16 : 8;
  int reach = 0, ntaps = 0;                     // rows of an x tile that the MMAs read
  for (int g = 0; g < p.ngroups; ++g) ntaps += p.grp_n[g];
  for (int t = 0; t < ntaps; ++t) reach = std::max<int>(reach, p.tap_off[t]);
  reach += (p.rows_a + kk - 1) / kk * kk;
  p.box_bytes = round_up(std::max(reach, std::max(p.rows_a, p.rows_b)), 8) * 128;
  p.a_boxes = std::min(128 / at, (p.Kg + at - 1) / at);
  p.b_boxes = std::min(128 / at, (p.Cg + at - 1) / at);
  p.stages = kMaxStages;
  while (p.stages > 2 && ring_bytes(p.stages, at, p.a_boxes, p.b_boxes, p.box_bytes) > kSmemBudget) --p.stages;
  p.ring_bytes = ring_bytes(p.stages, at, p.a_boxes, p.b_boxes, p.box_bytes);
  if (p.ring_bytes > kSmemBudget) return cudaErrorInvalidValue;
  if (dtype == B200CONV_F16)
    return p.stack_step > 0 ? launch_one<MmaKind::F16, kStack>(p, total, num_sms, s) : launch_one<MmaKind::F16, kWide>(p, total, num_sms, s);
  if (p.stack_step <= 0) return launch_one<MmaKind::TF32, kWide>(p, total, num_sms, s);
  return p.Cg > at ? launch_one<MmaKind::TF32, kStackTwice>(p, total, num_sms, s) : launch_one<MmaKind::TF32, kStack>(p, total, num_sms, s);
}

}  // namespace b200
