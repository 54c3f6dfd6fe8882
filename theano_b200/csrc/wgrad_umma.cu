// Filter gradient as an implicit GEMM on tcgen05 tensor cores.
//
//   dW[tap][k, c] = sum over output pixels q of  dy[q, k] * x_view_tap[q + offset_tap, c]
//
// Both operands are channels-last, so the reduction index (the pixel) is the slow index of
// each shared-memory row and the M/N index (filter k, channel c) is the contiguous one: the
// MMA reads both operands in MN-major form with a 128-byte swizzle (16-byte chunks for
// float16; 32-byte chunks for tf32, the only swizzled MN-major form tf32 has).  One TMA box brings
// kAtom (32 float32 / 64 float16) channels of up to 64 pixels; an operand of 128 filters or
// BN channels is a row of such boxes (leading-dimension offset = one box).
//
// Warp roles: warp 0 and the last three warps TMA producers, warp 1 MMA issuer and TMEM owner,
// 16 epilogue warps.
// Work item = (filter tile, channel tile, group, tap, split-K slice).  Each item reduces its
// slice of the pixel tiles into a TMEM accumulator (128 filters x BN channels, float32) and
// writes it to its own slab of the partial buffer (wgrad_slab.cuh).  A second kernel adds the slabs in
// slice order (so the result does not depend on scheduling) and writes OIHW.
#include "internal.h"
#include "ptx.cuh"
#include "wgrad_exact.cuh"
#include "wgrad_slab.cuh"

namespace b200 {
namespace {

constexpr int kEpilogueWarps = 16;            // a warp keeps only a few stores in flight: use many
// One thread gets a TMA box accepted every ~300 clocks whatever its size; the MMAs of a stage
// take less than the stage's 6-12 boxes would need from one thread.  Boxes are therefore spread
// over several producer warps (warp 0 and the warps after the epilogue warps) and over lanes
// within them: box j of a stage belongs to producer warp j % kProducers, lane j / kProducers.
constexpr int kProducers = 4;
constexpr int kFirstExtraProducer = 2 + kEpilogueWarps;
constexpr int kThreads = 32 * (kFirstExtraProducer + kProducers - 1);
// one TMA box in shared memory: the stage's reduction rows x 128 bytes
template <MmaKind KIND, int BN> constexpr int box_bytes() {
  return (KIND == MmaKind::TF32 ? kWgradPixF32 : BN >= 256 ? kWgradPixF16Wide : kWgradPixF16) * 128;
}
constexpr int kSmemBudget = 208 * 1024;

template <MmaKind KIND> constexpr int atom() { return KIND == MmaKind::TF32 ? 32 : 64; }
template <MmaKind KIND, int BN> constexpr int stage_bytes() {
  return (128 / atom<KIND>() + BN / atom<KIND>()) * box_bytes<KIND, BN>();
}
template <MmaKind KIND, int BN> constexpr int num_stages() {
  return (kSmemBudget / stage_bytes<KIND, BN>()) > 8 ? 8 : (kSmemBudget / stage_bytes<KIND, BN>());
}

struct Bars {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
};

struct Item {
  int kt, ct, g, tap, sp;
  uint32_t t_begin, t_end;  // pixel-tile range of the split
};

// 32-bit arithmetic throughout (the launcher checks the counts)
__device__ __forceinline__ Item decode(uint32_t it, const UmmaWgradParams& p, uint32_t per_split,
                                       uint32_t pix_tiles) {
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

// The MMA issuer's loop over the pixel tiles (pipeline stages) of one work item.  KS > 0: exactly KS
// reduction steps per stage, issued as straight-line code; KS == 0: `ksteps` steps in blocks of four.
// f16: 8-row groups 1024 bytes apart, 16-byte swizzle; tf32: 4-row groups 512 bytes apart, 32-byte
// swizzle; leading offset = next box (next kAtom channels).  Only the address field of the two
// descriptors changes from one MMA to the next: kK rows further.  Returns false when a wait ran out.
template <MmaKind KIND, int BN, int KS, bool TIMED>
__device__ __forceinline__ bool mma_tiles(Bars* bars, uint32_t d_tmem, uint32_t lo_base, uint32_t desc_hi,
                                          int ksteps, int ntiles, int& stage, uint32_t& phase, uint32_t& seen,
                                          long long& t_wait, bool leader, long long limit) {
  constexpr int kAtom = atom<KIND>();
  constexpr int kABoxes = 128 / kAtom;
  constexpr int kStages = num_stages<KIND, BN>();
  constexpr int kK = KIND == MmaKind::TF32 ? 8 : 16;
  constexpr uint32_t kStep = (kK * 128) >> 4;
  constexpr uint32_t kIdesc = instr_desc(KIND == MmaKind::TF32, true, true, 128, BN);
  uint32_t acc = 0u;
  for (int t = 0; t < ntiles; ++t) {
    const long long tw = TIMED ? clock64() : 0;
    if (!wait_seen(seen, &bars->full[stage], phase, bars, limit)) return false;
    if (TIMED) t_wait += clock64() - tw;
    tc_fence_after();
    const uint32_t a_lo = lo_base + stage * (stage_bytes<KIND, BN>() >> 4);
    const uint32_t b_lo = a_lo + ((kABoxes * box_bytes<KIND, BN>()) >> 4);
    const int half = (KS > 0 ? KS : ksteps) / 2;
    auto steps = [&](int k0, int k1) {
      if (KS > 0) {
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
          if (ks >= k0 && ks < k1)
            umma_words<KIND>(d_tmem, a_lo + ks * kStep, b_lo + ks * kStep, desc_hi, kIdesc, ks == 0 ? acc : 1u);
      } else {
        for (int ks = k0; ks < k1; ++ks)
          umma_words<KIND>(d_tmem, a_lo + ks * kStep, b_lo + ks * kStep, desc_hi, kIdesc, ks == 0 ? acc : 1u);
      }
    };
    if (leader) steps(0, half);
    __syncwarp();
    const int cur = stage;
    const bool wrap = stage + 1 == kStages;
    stage = wrap ? 0 : stage + 1;
    phase ^= wrap ? 1u : 0u;
    seen = mbar_look(&bars->full[stage], phase);
    if (leader) {
      steps(half, KS > 0 ? KS : ksteps);
      umma_commit(&bars->empty[cur]);
    }
    acc = 1u;
  }
  return true;
}

template <MmaKind KIND, int BN>
__global__ void __launch_bounds__(kThreads, 1)
wgrad_umma_kernel(const __grid_constant__ UmmaWgradParams p) {
  constexpr int kAtom = atom<KIND>();
  constexpr int kABoxes = 128 / kAtom, kBBoxes = BN / kAtom;
  constexpr int kStages = num_stages<KIND, BN>();
  constexpr int kBoxBytes = box_bytes<KIND, BN>();
  constexpr int kK = KIND == MmaKind::TF32 ? 8 : 16;       // reduction rows per MMA
  constexpr uint32_t kIdesc = instr_desc(KIND == MmaKind::TF32, true, true, 128, BN);
  constexpr uint32_t kSbo = KIND == MmaKind::TF32 ? 512 : 1024;
  constexpr uint64_t kLayout = KIND == MmaKind::TF32 ? kSwizzle128Base32 : kSwizzle128;
  constexpr bool kDouble = 2 * BN <= 512;
  constexpr uint32_t kTmemCols = 2 * BN > 512 ? 512 : 2 * BN;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  Bars* bars = reinterpret_cast<Bars*>(smem + kStages * stage_bytes<KIND, BN>());

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  // phase timing (optional): [0] MMA thread waiting for operands, [1] its whole loop,
  // [2] first producer waiting for a free stage, [3] its whole loop, [4] kernel start to end,
  // [9] / [10] GPU-wide timer at start / end
  long long* trace = p.trace ? p.trace + blockIdx.x * 16 : nullptr;
  const long long t_begin = trace ? clock64() : 0;
  if (trace && threadIdx.x == 0) trace[9] = static_cast<long long>(global_ns());
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
      mbar_init(&bars->acc_empty[b], 32 * kEpilogueWarps);
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
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  // Reduction rows past the pixel box are never written by TMA: clear them once so that the
  // last MMA of a stage (which reads whole groups of kK rows) adds zeros.
  if (rows_used < ksteps * kK) {
    const int tail_rows = ksteps * kK - rows_used;
    const int boxes = kStages * (kABoxes + kBBoxes);
    for (int i = threadIdx.x; i < boxes * tail_rows * 8; i += kThreads) {
      const int box = i / (tail_rows * 8), rem = i % (tail_rows * 8);
      uint4* dst = reinterpret_cast<uint4*>(smem + box * kBoxBytes + (rows_used + rem / 8) * 128) + rem % 8;
      *dst = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
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
      const ConvTap tp = p.taps[w.tap];
      // boxes that lie wholly past the channel counts are skipped (their accumulator rows /
      // columns are never stored)
      const int a_boxes = min(kABoxes, (p.Kg - w.kt * 128 + kAtom - 1) / kAtom);
      const int b_boxes = min(kBBoxes, (p.Cg - w.ct * BN + kAtom - 1) / kAtom);
      const uint32_t tx = (a_boxes + b_boxes) * rows_used * 128;
      // tile coordinates advance by counting: 64-bit divisions per stage would cost the producers
      // more clocks than the stage's MMAs take
      const uint32_t trow = quotient(w.t_begin, p.walk.tiles_w);
      int tn = quotient(trow, p.walk.tiles_h), th_ = trow - tn * p.tiles_h, tw = w.t_begin - trow * p.tiles_w;
      for (uint32_t t = w.t_begin; t < w.t_end; ++t) {
        const int w0 = tw * p.bw, h0 = th_ * p.bh, n0 = tn * p.bn;
        if (++tw == p.tiles_w) {
          tw = 0;
          if (++th_ == p.tiles_h) { th_ = 0; ++tn; }
        }
        const long long tw0 = trace ? clock64() : 0;
        if (!uniform_wait(&bars->empty[stage], phase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
        if (trace) t_wait += clock64() - tw0;
        uint8_t* sa = smem + stage * stage_bytes<KIND, BN>();
        uint8_t* sb = sa + kABoxes * kBoxBytes;
        if (leader) {
          if (pw == 0) mbar_expect_tx(&bars->full[stage], tx);
          for (int j = pw; j < a_boxes + b_boxes; j += kProducers) {
            if (j < a_boxes)
              tma_load_5d(sa + j * kBoxBytes, &p.dy_map, &bars->full[stage], w.kt * 128 + j * kAtom, w.g,
                          w0, h0, n0);
            else
              tma_load_5d(sb + (j - a_boxes) * kBoxBytes, &p.x_views[tp.view], &bars->full[stage],
                          w.ct * BN + (j - a_boxes) * kAtom, w.g, w0 + tp.dw, h0 + tp.dh, n0);
          }
        }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
    if (trace && leader && pw == 0) { trace[2] = t_wait; trace[3] = clock64() - t_begin; }
  } else if (warp == 1) {
    // all lanes follow the loop and wait; one elected lane issues the MMAs and their commits
    const bool leader = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int n = 0;
    long long t_wait = 0;
    const uint64_t desc_bits = smem_desc(0, kBoxBytes, kSbo, kLayout);
    const uint32_t desc_hi = static_cast<uint32_t>(desc_bits >> 32);
    const uint32_t lo_base = static_cast<uint32_t>(desc_bits) + (smem_u32(smem) >> 4);
    uint32_t seen = 0;                           // the next stage already seen full (mbar_look)
    for (uint32_t it = blockIdx.x; it < total && ok; it += gridDim.x, ++n) {
      const Item w = decode(it, p, per_split, pix_tiles);
      const int buf = kDouble ? (n & 1) : 0;
      const uint32_t aphase = kDouble ? ((n >> 1) & 1) : (n & 1);
      if (!uniform_wait(&bars->acc_empty[buf], aphase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem + buf * BN;
      const int ntiles = static_cast<int>(w.t_end - w.t_begin);
      // the usual step counts get straight-line MMA blocks
      if (trace) ok = mma_tiles<KIND, BN, 0, true>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, t_wait, leader, p.wait_clocks);
      else if (ksteps == 8) ok = mma_tiles<KIND, BN, 8, false>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, t_wait, leader, p.wait_clocks);
      else if (ksteps == 7) ok = mma_tiles<KIND, BN, 7, false>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, t_wait, leader, p.wait_clocks);
      else if (ksteps == 4) ok = mma_tiles<KIND, BN, 4, false>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, t_wait, leader, p.wait_clocks);
      else ok = mma_tiles<KIND, BN, 0, false>(bars, d_tmem, lo_base, desc_hi, ksteps, ntiles, stage, phase, seen, t_wait, leader, p.wait_clocks);
      if (ok && leader) umma_commit(&bars->acc_full[buf]);
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
    if (trace && leader) { trace[0] = t_wait; trace[1] = clock64() - t_begin; }
  } else {
    // warp w reads TMEM lanes [32*(w%4), +32) and every fourth 32-column chunk of them
    const int quad = warp & 3;
    const int sub = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    bool ok = true;
    int n = 0;
    const int K = p.Kg * p.groups;
    for (uint32_t it = blockIdx.x; it < total && ok; it += gridDim.x, ++n) {
      const Item w = decode(it, p, per_split, pix_tiles);
      const int buf = kDouble ? (n & 1) : 0;
      const uint32_t aphase = kDouble ? ((n >> 1) & 1) : (n & 1);
      if (!warp_wait_or_abort(&bars->acc_full[buf], aphase, bars, lane, p.wait_clocks)) { ok = false; break; }
      tc_fence_after();
      const int kq = w.kt * 128 + row;
      const bool valid = kq < p.Kg;
      float* slab = p.partial + (1LL * (p.atomic ? 0 : w.sp) * p.taps_total + p.taps[w.tap].wmat) * K * p.Cg;
      int c_lo, c_hi;
      diagonal_range(p.diag_c, p.diag_k, kq, p.Cg, &c_lo, &c_hi);
#pragma unroll 1
      for (int ch = sub; ch < BN / 32; ch += kEpilogueWarps / 4) {
        const int c0 = w.ct * BN + ch * 32;
        if (c0 >= p.Cg) break;
        uint32_t r[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(quad * 32) << 16) + buf * BN + ch * 32, r);
        tmem_ld_wait();
        if (valid) store_slab_chunk(r, slab, c0, c_lo, c_hi, p.Cg, K, w.g * p.Kg + kq, p.atomic, p.partial, p.partial_elems, p.status);
      }
      tc_fence_before();
      mbar_arrive(&bars->acc_empty[buf]);
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
    tmem_dealloc(tmem, kTmemCols);
  }
}

// out[k][c][tap] = sum over the slices of their slabs (wgrad_slab.cuh).  A block takes 2^log_k filters x 2^log_q groups
// of four channels x all taps, one thread per four channels and share of the slices; neighbouring threads take neighbouring filters, 16 bytes
// apart in a slab.  Each sum is split over 2^log_lanes threads: lane l takes the slabs l, l + lanes, ... in that order and the
// partial sums are then added in lane order, so the result does not depend on scheduling (it is the same on every run).
// The sums go to shared memory in output order [filter][channel][tap] (rows an odd number of words apart) and leave as
// one contiguous run per filter.
// The slabs are read once, from L2 or HBM; what bounds the kernel below a few megabytes is the length
// of the chain of loads in a thread, so a block is one round of loads (up to 640 threads) and long sums are split over lanes.
// diag_c / diag_k: only the diagonal blocks of merged groups are there and wanted (diag_c channels per filter, starting at the block of the
// filter), 0: all.  `sum`: for sums that are NaN (wgrad_exact.cuh).
template <typename T>
__global__ void __launch_bounds__(640, 2) wgrad_reduce_kernel(const float* __restrict__ partial, T* __restrict__ dw, int splits, int taps, int K,
                                                               int Cg, int Kg, int diag_c, int diag_k, int log_k, int log_q, int log_lanes,
                                                               const __grid_constant__ WgradSum sum) {
  pdl_enter();
  extern __shared__ float4 shared[];
  const int kt = 1 << log_k, nq = 1 << log_q, lanes = 1 << log_lanes;
  const int cols = diag_c ? diag_c : Cg;                      // channels per filter of the result
  const int pitch = (4 * nq * taps) | 1, units = (kt << log_q) * taps;
  float4* part = shared;                                      // [lane - 1][unit]
  float* tile = reinterpret_cast<float*>(shared + (lanes - 1) * units);
  const int lane = threadIdx.x / units, u = threadIdx.x - lane * units;
  const int kk = u & (kt - 1), q = (u >> log_k) & (nq - 1), t = u >> (log_k + log_q);
  const long long slab = 1LL * taps * K * Cg;
  const int qtiles = (cols + 4 * nq - 1) / (4 * nq);
  const bool whole = (((1LL * K * Cg) & 3) | (cols & 3) | (diag_c & 3)) == 0;
  const int k0 = static_cast<int>(blockIdx.x) / qtiles << log_k, c0 = static_cast<int>(blockIdx.x) % qtiles * 4 * nq;
  const int k = k0 + kk, co = c0 + 4 * q;                     // filter, first channel of the result
  const bool on = lane < lanes && k < K && co < cols;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (on) {
    const int c = co + (diag_c ? k % Kg / diag_k * diag_c : 0);
    if (whole) {
      const float4* src = reinterpret_cast<const float4*>(partial + slab_index(t, k, c, K, Cg)) + lane * (slab >> 2);
      const long long step = lanes * (slab >> 2);
      for (int s0 = lane; s0 < splits; s0 += 4 * lanes, src += 4 * step) {      // four loads in flight, also where there are three
        float4 v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (s0 + e * lanes < splits) v[e] = src[e * step];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (s0 + e * lanes < splits) { acc.x += v[e].x; acc.y += v[e].y; acc.z += v[e].z; acc.w += v[e].w; }
      }
    } else {
      float* a = &acc.x;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (co + e >= cols) continue;
        const float* src = partial + slab_index(t, k, c + e, K, Cg);
        for (int s = lane; s < splits; s += lanes) a[e] += src[s * slab];
      }
    }
    if (lane > 0) part[(lane - 1) * units + u] = acc;
  }
  if (lanes > 1) __syncthreads();
  bool nan = false;
  if (lane == 0 && on) {
    for (int l = 0; l < lanes - 1; ++l) {
      const float4 v = part[l * units + u];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    float* dst = tile + kk * pitch + 4 * q * taps + t;
    dst[0] = acc.x; dst[taps] = acc.y; dst[2 * taps] = acc.z; dst[3 * taps] = acc.w;
    nan = isnan(acc.x) || isnan(acc.y) || isnan(acc.z) || isnan(acc.w);
  }
  const int run = min(4 * nq, cols - c0) * taps;
  auto store = [&] {
#pragma unroll 1
    for (int row = threadIdx.x >> 5; row < kt && k0 + row < K; row += blockDim.x >> 5) {
      T* dst = dw + (1LL * (k0 + row) * cols + c0) * taps;
      for (int i = threadIdx.x & 31; i < run; i += 32) dst[i] = static_cast<T>(tile[row * pitch + i]);
    }
  };
  const bool any_nan = __syncthreads_or(nan);
  store();
  if (!any_nan) return;
  __syncthreads();
  exact_tile(sum, tile, min(kt, K - k0), pitch, min(4 * nq, cols - c0), k0, c0);
  store();
}

template <MmaKind KIND, int BN>
cudaError_t launch_one(const UmmaWgradParams& p, long long total, int num_sms, cudaStream_t s) {
  constexpr int smem = num_stages<KIND, BN>() * stage_bytes<KIND, BN>() + sizeof(Bars) + 1024;
  static PerDeviceOnce configured;
  cudaError_t e = configured.ensure([] { return cudaFuncSetAttribute(wgrad_umma_kernel<KIND, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  if (e != cudaSuccess) return e;
  const int grid = static_cast<int>(total < num_sms ? total : num_sms);
  launch_chained(wgrad_umma_kernel<KIND, BN>, grid, kThreads, smem, s, p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_wgrad_umma(const UmmaWgradParams& params, int dtype, int bn_cols, int num_sms,
                              cudaStream_t s) {
  UmmaWgradParams p = params;
  p.walk = item_walk(p.splits, p.ntaps, p.groups, p.ctiles, p.tiles_w, p.tiles_h);
  const long long total = 1LL * p.ktiles * p.ctiles * p.groups * p.ntaps * p.splits;
  if (total == 0) return cudaSuccess;
  if (total >= (1LL << 31) || 1LL * p.tiles_w * p.tiles_h * p.tiles_n >= (1LL << 31)) return cudaErrorInvalidValue;
  const bool f16 = dtype == B200CONV_F16;
#define B200_CASE(BNV)                                                                  \
  case BNV:                                                                             \
    return f16 ? launch_one<MmaKind::F16, BNV>(p, total, num_sms, s)                    \
               : launch_one<MmaKind::TF32, BNV>(p, total, num_sms, s);
  switch (bn_cols) {
    B200_CASE(64)
    B200_CASE(128)
    B200_CASE(256)
  }
#undef B200_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_wgrad_reduce(const float* partial, void* dw, int splits, int taps, int K, int Cg, int Kg, int diag_c, int diag_k,
                                int dtype, const WgradSum& sum, cudaStream_t s) {
  if (1LL * K * Cg == 0 || taps == 0) return cudaSuccess;
  const int cols = diag_c ? diag_c : Cg;
  // About four slabs per thread, at most 8 threads per sum; as many channels as make a filter's run 128 bytes; up to 32 filters
  // in a block of at most 640 threads, fewer while that leaves SMs without three blocks.  1x1 layers of few slices keep their filters, 512 bytes
  // of a slab in a row, and give up threads per sum instead: 256 -> 1024 at 14x14, 18 slices, float16, all of gradWeights 37.5 -> 33.3 us
  // (64 -> 64 at 56x56, 148 slices, that way 39.8 -> 45.5).  Where the line lies, by pinned slice counts, float16, 256 images: 128 -> 512 at 28x28 18 slices 58.0 -> 57.6, 24
  // 50.2 -> 50.0, 28 47.6 -> 49.4, 37 47.5 -> 50.1; 64 -> 64 24 96.4 -> 97.2, 28 83.8 -> 85.1; wide layers gain with any count (256 -> 1024 28 44.7 -> 40.4, but 14 to
  // 18 are faster).  The one seen to lose below it: 512 -> 2048 at 7x7, 64 images, float32, 6 slices 28.6 -> 29.7.
  const bool flat = taps == 1 && splits <= 24;
  int log_k = 5, log_q = 0, log_lanes = 0;
  while (log_lanes < 3 && splits > (4 << log_lanes)) ++log_lanes;
  while (log_q < 4 && (4 << log_q) < cols && (4 << log_q) * taps * static_cast<int>(elem_size(dtype)) < (flat ? 64 : 128)) ++log_q;
  auto blocks = [&] { return ((cols + (4 << log_q) - 1) / (4 << log_q)) * static_cast<long long>((K + (1 << log_k) - 1) >> log_k); };
  while (flat && log_lanes > 1 && (taps << (log_k + log_q + log_lanes)) > 640) --log_lanes;
  while (log_k > 2 && ((taps << (log_k + log_q + log_lanes)) > 640 || (1 << (log_k - 1)) >= K || blocks() < 3 * 148)) --log_k;
  while (log_lanes > 0 && (taps << (log_k + log_q + log_lanes)) > 640) --log_lanes;
  while (log_q > 0 && ((taps << (log_k + log_q + log_lanes)) > 640 || blocks() < 2 * 148)) --log_q;
  if (blocks() >= (1LL << 31)) return cudaErrorInvalidValue;
  const int units = taps << (log_k + log_q), threads = ((units << log_lanes) + 31) / 32 * 32, g = static_cast<int>(blocks());
  const size_t smem = sizeof(float4) * ((1 << log_lanes) - 1) * units + (sizeof(float) * (((4 << log_q) * taps) | 1) << log_k);
  if (dtype == B200CONV_F16)
    launch_streaming(wgrad_reduce_kernel<__half>, g, threads, smem, s, partial, static_cast<__half*>(dw), splits, taps, K, Cg, Kg, diag_c, diag_k, log_k, log_q, log_lanes, sum);
  else
    launch_streaming(wgrad_reduce_kernel<float>, g, threads, smem, s, partial, static_cast<float*>(dw), splits, taps, K, Cg, Kg, diag_c, diag_k, log_k, log_q, log_lanes, sum);
  return cudaGetLastError();
}

}  // namespace b200
