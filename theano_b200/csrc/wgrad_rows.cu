// Filter gradient of narrow layers on tcgen05 tensor cores: the filter's rows and columns both inside one MMA.
//
//   dW[tap][k, c] = sum over output pixels q of  dy[q, k] * x_view[q + (dh, dw)_tap, c]
//
// A layer with at most 64 (float16) or 32 (float32) filters per group fills a half or a quarter of an MMA's 128 rows
// and few of its columns.  Here the taps fill the rest: the pixels of a tile lie on a grid of pitch P (the
// output width and the span of the filter's columns), so that a tap is a row offset into a shared-memory tile.
//   columns: the taps of a filter row are groups of columns of the x operand, stack_step grid positions apart;
//   rows:    128 / (channels of a swizzle atom) copies of the dy operand, a_step grid positions (one filter row) apart.
// Both are strides of the MN-major descriptors (the leading-dimension offset), nothing is copied.  With x taken at filter row i the copy r
// of dy, which lies r filter rows further on, gives filter row i - r:
//   sum over p of  dy[p + r * a_step] * x[p + offset_i]  =  sum over q of  dy[q] * x[q + offset_i - r * a_step].
// A filter of 3 x 3 is one 128 x 96 MMA per 8 float32 pixels of 32 channels, or two of 128 x 192 per 16 float16 pixels of
// 64, where a tap group per filter row takes three; and dy and x are read once per stage, not once per filter row.
// Measured (gradWeights with its reduction, before -> here): 32 groups of 8 x 8 channels 3x3, 256 images of 28 x 28, float32
// 180 -> 83 us (411 MB: 63 us at the rate of a copy); 64 -> 64 3x3 at 56x56, 256 images, float16 95 -> 73 us; the 7x7 stem on
// pixel blocks, 256 images of 224 x 224, 311 -> 183 us, 50 of them the pass that makes the blocks.
//
// The positions p of a tile are th grid rows from row h0 on, h0 >= -halo (the copies reach back halo rows); dy rows above and below the
// image and columns behind it arrive as zeros, so every product of a tap is counted in exactly one tile (pixels of x that are not finite meet
// those zeros: wgrad_exact.cuh); th * P is a multiple of an
// MMA's reduction steps.
//
// Work item = (channel tile, group, stride parity view, slice).  Warp roles: warp 0 loads dy, the last warp loads x, warp 1 issues the
// MMAs and owns the TMEM, 16 epilogue warps.
#include <algorithm>

#include "internal.h"
#include "ptx.cuh"
#include "wgrad_slab.cuh"

namespace b200 {
namespace {

constexpr int kEpilogueWarps = 16;
constexpr int kXProducer = 2 + kEpilogueWarps;         // warp index
constexpr int kThreads = 32 * (kXProducer + 1);
constexpr int kMaxStages = 6;
constexpr int kSmemBudget = 222 * 1024;

template <MmaKind KIND> constexpr int atom() { return KIND == MmaKind::TF32 ? 32 : 64; }

struct alignas(16) Bars {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full;
  uint64_t acc_empty;
  uint32_t tmem_base;
  volatile int abort;
};

struct Item {
  int ct, g, v, sp;
  uint32_t t_begin, t_end;
};
__device__ __forceinline__ Item decode(uint32_t it, const RowsWgradParams& p, uint32_t per_split, uint32_t tiles) {
  Item r;
  const uint32_t a = quotient(it, p.walk.splits), b = quotient(a, p.walk.taps), c = quotient(b, p.walk.groups);
  r.sp = it - a * p.walk.splits.d;
  r.v = a - b * p.walk.taps.d;
  r.g = b - c * p.walk.groups.d;
  r.ct = c;
  r.t_begin = r.sp * per_split;
  r.t_end = min(r.t_begin + per_split, tiles);
  return r;
}

struct IssueLoop {
  Bars* bars;
  uint32_t tmem, a0, b0, desc_hi;                // a0 / b0: low descriptor words of the first stage's operands
  uint32_t idesc, set_cols, stage_units;
  uint32_t set_off[kMaxRowSets];                 // x offset of each set of filter rows, descriptor units
  int ksteps, ntiles, stages;
  bool leader;
  long long limit;
  int stage;
  uint32_t phase, seen;
};

// The MMAs of an item with SETS sets of filter rows.  Returns false when a wait ran out.
template <MmaKind KIND, int SETS>
__device__ __forceinline__ bool mma_item(IssueLoop& w) {
  constexpr uint32_t kStep = ((KIND == MmaKind::TF32 ? 8 : 16) * 128) >> 4;
  Bars* bars = w.bars;
  const uint32_t lane = w.leader, idesc = w.idesc, desc_hi = w.desc_hi;
  const int ksteps = w.ksteps, ntiles = w.ntiles, stages = w.stages;
  uint32_t off[SETS], acc_col[SETS];
#pragma unroll
  for (int j = 0; j < SETS; ++j) { off[j] = w.set_off[j]; acc_col[j] = w.tmem + j * w.set_cols; }
  int stage = w.stage;
  uint32_t phase = w.phase, seen = w.seen;
  uint32_t acc = 0u;
  for (int t = 0; t < ntiles; ++t) {
    if (!wait_seen(seen, &bars->full[stage], phase, bars, w.limit)) return false;
    tc_fence_after();
    uint32_t a = w.a0 + stage * w.stage_units, b = w.b0 + stage * w.stage_units;
    auto step = [&](uint32_t accumulate) {
#pragma unroll
      for (int j = 0; j < SETS; ++j) umma_words_if<KIND>(lane, acc_col[j], a, b + off[j], desc_hi, idesc, accumulate);
      a += kStep;
      b += kStep;
    };
    // blocks of four steps, the look ahead before the last four to seven
    int ks = 0;
    for (; ks + 8 <= ksteps; ks += 4) {
      step(acc);
      acc = 1u;
      step(1u);
      step(1u);
      step(1u);
    }
    const int cur = stage;
    const bool wrap = stage + 1 == stages;
    stage = wrap ? 0 : stage + 1;
    phase ^= wrap ? 1u : 0u;
    seen = mbar_look(&bars->full[stage], phase);
    for (; ks < ksteps; ++ks) {
      step(acc);
      acc = 1u;
    }
    umma_commit_if(lane, &bars->empty[cur]);
  }
  w.stage = stage; w.phase = phase; w.seen = seen;
  return true;
}

template <MmaKind KIND>
__global__ void __launch_bounds__(kThreads, 1)
wgrad_rows_kernel(const __grid_constant__ RowsWgradParams p) {
  constexpr int kAtom = atom<KIND>(), kK = KIND == MmaKind::TF32 ? 8 : 16;
  constexpr uint32_t kSbo = KIND == MmaKind::TF32 ? 512 : 1024;
  constexpr uint64_t kLayout = KIND == MmaKind::TF32 ? kSwizzle128Base32 : kSwizzle128;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Bars* bars = reinterpret_cast<Bars*>(smem + p.ring_bytes);
  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const int stage_bytes = p.a_bytes + p.b_bytes;
  const uint32_t tiles = static_cast<uint32_t>(p.tiles_h) * p.Nimg;
  const uint32_t per_split = (tiles + p.splits - 1) / p.splits;
  const uint32_t total = static_cast<uint32_t>(p.ctiles) * p.groups * p.nviews * p.splits;

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
  // the columns' taps read up to (nt - 1) * stack_step rows behind the x box, against zeros of dy: never written by TMA, finite
  for (int s = 0; s < p.stages; ++s) {
    const int nrows = p.b_bytes / 128 - p.rows_b;
    uint4* dst = reinterpret_cast<uint4*>(smem + s * stage_bytes + p.a_bytes + p.rows_b * 128);
    for (int i = threadIdx.x; i < nrows * 8; i += kThreads) dst[i] = make_uint4(0, 0, 0, 0);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  pdl_enter();              // the next kernel may start once this CTA holds its TMEM; nothing global was touched before

  if (warp == 0 || warp == kXProducer) {
    const bool leader = elect_one(), is_x = warp != 0;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (uint32_t it = blockIdx.x; it < total && ok; it += gridDim.x) {
      const Item w = decode(it, p, per_split, tiles);
      int n = quotient(w.t_begin, p.walk.tiles_h), th_ = w.t_begin - n * p.tiles_h;
      for (uint32_t t = w.t_begin; t < w.t_end; ++t) {
        const int h0 = th_ * p.th - p.halo, n0 = n;
        if (++th_ == p.tiles_h) { th_ = 0; ++n; }
        if (!uniform_wait(&bars->empty[stage], phase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
        uint8_t* sa = smem + stage * stage_bytes;
        if (leader) {
          if (!is_x) {
            mbar_expect_tx(&bars->full[stage], static_cast<uint32_t>(p.rows_a + p.rows_b) * 128u);
            tma_load_5d(sa, &p.dy_map, &bars->full[stage], 0, w.g, 0, h0, n0);
          } else {
            tma_load_5d(sa + p.a_bytes, &p.x_views[w.v], &bars->full[stage], w.ct * kAtom, w.g, p.view_dw[w.v], h0 + p.view_dh[w.v], n0);
          }
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else if (warp == 1) {
    const uint64_t bits = smem_desc(0, 0, kSbo, kLayout);
    IssueLoop w;
    w.bars = bars; w.tmem = tmem;
    w.desc_hi = static_cast<uint32_t>(bits >> 32);
    // the low word carries the leading-dimension offset in bits [16, 30): the copies of dy / the columns' taps of x
    w.a0 = static_cast<uint32_t>(bits) + (smem_u32(smem) >> 4) + (static_cast<uint32_t>(p.a_step * 128) >> 4 << 16);
    w.b0 = static_cast<uint32_t>(bits) + (smem_u32(smem + p.a_bytes) >> 4) + (static_cast<uint32_t>(p.stack_step * 128) >> 4 << 16);
    w.stage_units = static_cast<uint32_t>(stage_bytes) >> 4;
    w.ksteps = p.th * p.pitch / kK; w.stages = p.stages;
    w.leader = elect_one();
    w.limit = p.wait_clocks;
    w.stage = 0; w.phase = 0; w.seen = 0;
    bool ok = true;
    int n = 0;
    for (uint32_t it = blockIdx.x; it < total && ok; it += gridDim.x, ++n) {
      const Item item = decode(it, p, per_split, tiles);
      if (!uniform_wait(&bars->acc_empty, (n & 1) ^ 1, bars, p.wait_clocks)) { ok = false; break; }
      tc_fence_after();
      w.ntiles = static_cast<int>(item.t_end) - static_cast<int>(item.t_begin);
      const int nt = p.view_nt[item.v], sets = p.view_sets[item.v];
      w.set_cols = nt * kAtom;
      w.idesc = instr_desc(KIND == MmaKind::TF32, true, true, 128, nt * kAtom);
#pragma unroll
      for (int j = 0; j < kMaxRowSets; ++j) w.set_off[j] = static_cast<uint32_t>(p.set_rows[item.v][j]) * (128u >> 4);
      if (sets == 1) ok = mma_item<KIND, 1>(w);
      else if (sets == 2) ok = mma_item<KIND, 2>(w);
      else if (sets == 3) ok = mma_item<KIND, 3>(w);
      else ok = mma_item<KIND, 4>(w);
      if (ok && w.leader) umma_commit(&bars->acc_full);
    }
    if (!ok && w.leader) report_status(p.status, kStatusTimeout);
  } else {
    const int quad = warp & 3, sub = (warp - 2) >> 2, row = quad * 32 + lane;
    const int copy = row / kAtom, kq = row % kAtom, K = p.Kg * p.groups;       // the warp's rows are all of one copy
    bool ok = true;
    int n = 0;
    int c_lo, c_hi;
    diagonal_range(p.diag_c, p.diag_k, kq, p.Cg, &c_lo, &c_hi);
    for (uint32_t it = blockIdx.x; it < total && ok; it += gridDim.x, ++n) {
      const Item w = decode(it, p, per_split, tiles);
      if (!warp_wait_or_abort(&bars->acc_full, n & 1, bars, lane, p.wait_clocks)) { ok = false; break; }
      tc_fence_after();
      const int nt = p.view_nt[w.v], chunks = kAtom / 32, items = p.view_sets[w.v] * nt * chunks;
#pragma unroll 1
      for (int i = sub; i < items; i += kEpilogueWarps / 4) {
        const int ch = i % chunks, q = i / chunks % nt, set = i / (chunks * nt);
        const int frow = p.set_base[w.v][set] - copy;                            // filter row of the view; before the set's first: not wanted
        const int c0 = w.ct * kAtom + ch * 32;
        if (frow < p.set_first[w.v][set] || c0 >= p.Cg) continue;
        uint32_t r[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + i * 32, r);
        tmem_ld_wait();
        if (kq >= p.Kg) continue;
        const int tap = p.tap_id[p.view_tap0[w.v] + frow * nt + q];
        float* slab = p.partial + (1LL * w.sp * p.taps_total + tap) * K * p.Cg;
        store_slab_chunk(r, slab, c0, c_lo, c_hi, p.Cg, K, w.g * p.Kg + kq, false, p.partial, p.partial_elems, p.status);
      }
      tc_fence_before();
      mbar_arrive(&bars->acc_empty);
    }
    if (!ok && lane == 0) report_status(p.status, kStatusTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (bars->abort) abort_grace(p.wait_clocks);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <MmaKind KIND>
cudaError_t launch_one(const RowsWgradParams& p, long long total, int num_sms, cudaStream_t s) {
  static PerDeviceOnce configured;
  cudaError_t e = configured.ensure([] { return cudaFuncSetAttribute(wgrad_rows_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024); });
  if (e != cudaSuccess) return e;
  launch_chained(wgrad_rows_kernel<KIND>, static_cast<int>(std::min<long long>(total, num_sms)), kThreads,
                 p.ring_bytes + static_cast<int>(sizeof(Bars)) + 1024, s, p);
  return cudaGetLastError();
}

}  // namespace

bool wgrad_rows_ring(RowsWgradParams* p, int dtype) {
  const int copies = dtype == B200CONV_F16 ? 2 : 4, steps = p->th * p->pitch;  // copies of dy; positions that the MMAs walk
  int reach = 0, nt = 0;
  for (int v = 0; v < p->nviews; ++v) {
    nt = std::max<int>(nt, p->view_nt[v]);
    for (int j = 0; j < p->view_sets[v]; ++j) reach = std::max<int>(reach, p->set_rows[v][j]);
  }
  p->a_bytes = round_up(p->rows_a, 8) * 128;
  p->b_bytes = round_up(std::max(p->rows_b, reach + steps + (nt - 1) * p->stack_step), 8) * 128;
  // a dy copy that is not wanted reads on behind its box: into x, the next stage or, of the last stage, this tail
  const int tail = std::max(0, ((copies - 1) * p->a_step + steps) * 128 - p->a_bytes - p->b_bytes);
  p->stages = kMaxStages;
  while (p->stages > 1 && p->stages * (p->a_bytes + p->b_bytes) + tail > kSmemBudget) --p->stages;
  p->ring_bytes = round_up(p->stages * (p->a_bytes + p->b_bytes) + tail, 16);
  return p->stages >= 2;
}

cudaError_t launch_wgrad_rows(const RowsWgradParams& params, int dtype, int num_sms, cudaStream_t s) {
  RowsWgradParams p = params;
  p.walk = item_walk(p.splits, p.nviews, p.groups, p.ctiles, 1, p.tiles_h);
  const long long total = 1LL * p.ctiles * p.groups * p.nviews * p.splits;
  if (total == 0) return cudaSuccess;
  if (total >= (1LL << 31) || 1LL * p.tiles_h * p.Nimg >= (1LL << 31)) return cudaErrorInvalidValue;
  return dtype == B200CONV_F16 ? launch_one<MmaKind::F16>(p, total, num_sms, s) : launch_one<MmaKind::TF32>(p, total, num_sms, s);
}

}  // namespace b200
