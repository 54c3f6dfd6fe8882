// Implicit GEMM for layers of at most 64 filters (per group): the columns of the filter inside one MMA.
//
// With N = 32 or 64 filters an MMA of 128 pixels is bound by its operands' reads of shared memory: the 128 rows of pixels, 4 KB per
// 32 bytes of channels, are read again for every filter tap.  Here a filter's columns j lie side by side along N, so that one MMA
// multiplies the pixels with a whole filter row,
//   D[position, j * bn + co] = sum over filter rows i, channels c of  x[position + i, c] * w[co, c, i, j],
// and the epilogue adds what belongs to one output: out[position, co] = sum over j of D[position + j, j * bn + co].  Neighbouring
// positions are neighbouring lanes, so these are shuffles inside a warp.  For that a row of positions must not straddle warps: the
// slab's pitch is 32, 16 or 8 positions, of which the filter's width less one are halo.  The A operand of every filter row then
// starts on a whole swizzle atom (8 rows), too; where each tap is a shift of its own, it starts anywhere.
//
// Measured (a B200, filters packed ahead, replayed as a graph, all in one build; slab kernel or its pairs, whichever is faster -> columns on single
// CTAs): 3x3 on 8 groups of 32 channels at 28x28, 256 images, float32 121 -> 88 us (the pixels alone take HBM 63); 32 -> 32 at 112x112, 64 images 58 -> 41;
// float16 64 -> 32 at 112x112 79 -> 40; 5x5 64 -> 16 at 56x56, 256 images 124 -> 45, float32 235 -> 91.  64 filters on single CTAs: float16 at 56x56, 256
// images 65 -> 68, float32 at 224x224, 16 images 132 -> 138: an MMA of 192 columns runs at its rate, but 72 KB of filters per 112 pixels
// come from L2.  On pairs (PAIR: two pixel tiles, M = 256, each CTA loading 32 of the 64 filters) the latter take 122, 64 images 507 -> 472, with pooling
// 456 -> 449, 128 -> 64 at 112x112, 64 images 235 -> 211; float16 at 56x56 80.
// What the steps gave, each in the build that brought it: filters that fit their ring whole and stay in it (`resident`) 64 -> 64 at 224x224, 64 images, on
// pairs 511 -> 459, the 8 groups 100 -> 91.  Tried there: 128 -> 64 with its filters whole beside two slabs and half of the staging 205 -> 216; a fourth slab
// for it, no change; its pixels for nothing, 197 -> 149; the 8 groups without their epilogue 97 -> 67.
//
// Warp roles (640 threads): warp 0 streams slabs (tile and halo, 128 bytes of channels per pixel), warp 19 filter rows, warps 1
// and 18 issue the MMAs of one accumulator each, 16 epilogue warps (TMEM -> shuffles -> staged TMA stores, with 2x2 max pooling,
// or, for the merged classes of a strided gradInputs, straight to the gradient's pixels).  Accumulator sets: `sets`, two to four of n_acc
// accumulators, sets * n_acc * kW * bn <= 512 columns.  The groups of epilogue warps that share no tile are `step`: with two or more each has a set of
// its own (sets = step), a single one takes two in turn.
#include "internal.h"
#include "ptx.cuh"

#include <type_traits>

namespace b200 {
namespace {

constexpr int kEpilogueWarps = 16;
constexpr int kSecondIssuer = 2 + kEpilogueWarps;     // warp index
constexpr int kFilterProducer = kSecondIssuer + 1;    // warp index
constexpr int kThreads = 32 * (kFilterProducer + 1);
constexpr int kMaxStages = kMaxColStages, kMaxSets = 4;

struct alignas(16) Bars {
  uint64_t slab_full[kMaxStages];
  uint64_t slab_empty[kMaxStages];
  uint64_t b_full[kMaxStages];
  uint64_t b_empty[kMaxStages];
  uint64_t acc_full[kMaxSets];
  uint64_t acc_empty[kMaxSets];
  uint32_t tmem_base;
  volatile int abort;
};

// Tile: one image's rows h0 .. h0 + th - 1, columns w0 .. w0 + wt - 1, of group g.  A pair's CTAs take two neighbouring ones (the second of an
// odd count's last pair lies behind the last image: its loads read zeros and its stores are left out).
struct Tile { int g, w0, h0, n; };
template <bool PAIR>
__device__ __forceinline__ Tile tile_of(const ColsConvParams& p, uint32_t t, uint32_t rank) {
  const uint32_t gt = quotient(t, p.by_groups), pt = PAIR ? 2 * gt + rank : gt, row = quotient(pt, p.by_tiles_w), n = quotient(row, p.by_tiles_h);
  return Tile{static_cast<int>(t - gt * p.groups), static_cast<int>(pt - row * p.tiles_w) * p.wt, static_cast<int>(row - n * p.tiles_h) * p.th, static_cast<int>(n)};
}

struct IssueLoop {
  const ColsConvParams& p;
  Bars* bars;
  uint32_t slab0, ring0, tmem;          // low descriptor words of the rings, accumulator a of set 0
  uint32_t first, stride, total;
  bool leader;
  uint32_t resident;                    // filters: the ring is one tile's, loaded once, its barriers stay in their first phase
};

// The MMAs of one issuing warp, all its tiles: RPS filter rows per filter stage as straight-line code, all 32 lanes in the loop, one
// elected lane issues (conv_slab.cu, issue_tiles()).  With a stage per filter row its four MMAs of 128 x 96 took 470 clocks, twice their own time.
template <MmaKind KIND, int RPS, bool PAIR>
__device__ __forceinline__ bool issue_tiles(const IssueLoop& w) {
  constexpr bool kTogether = RPS >= 4;
  const ColsConvParams& p = w.p;
  Bars* bars = w.bars;
  const bool leader = w.leader;
  const uint32_t n_cols = p.kW * p.bn, idesc = with_columns(instr_desc(KIND == MmaKind::TF32, false, false, PAIR ? 256 : 128, 256), n_cols);
  auto commit = [&](uint64_t* bar) {
    if (PAIR) umma_commit_pair(bar);
    else umma_commit(bar);
  };
  const uint32_t desc_hi = static_cast<uint32_t>(smem_desc(0, 16, 1024) >> 32);
  const uint32_t slab_units = static_cast<uint32_t>(p.slab_bytes) >> 4, row_units = (PAIR ? n_cols / 2 : n_cols) * 8, stage_units = RPS * row_units;
  int sb = 0, bs = 0, buf = 0;
  uint32_t sphase = 0, bphase = 0, aphase = 0, slab_seen = 0, b_seen = 0, acc_seen = 0;
  for (uint32_t t = w.first; t < w.total; t += w.stride) {
    if (!wait_seen(acc_seen, &bars->acc_empty[buf], aphase ^ 1, bars, p.wait_clocks)) return false;
    acc_seen = 0;
    tc_fence_after();
    const uint32_t acc = w.tmem + buf * p.n_acc * n_cols;
    for (int kb = 0; kb < p.kblocks; ++kb) {
      if (!wait_seen(slab_seen, &bars->slab_full[sb], sphase, bars, p.wait_clocks)) return false;
      const uint32_t slab_lo = w.slab0 + sb * slab_units;
      for (int i = 0; i < p.kH; i += RPS) {
        uint32_t a_lo[RPS];
#pragma unroll
        for (int q = 0; q < RPS; ++q) a_lo[q] = slab_lo + p.row_shift[i + q] * 8u;
        if (!wait_seen(b_seen, &bars->b_full[bs], bphase, bars, p.wait_clocks)) return false;
        tc_fence_after();
        const uint32_t b_lo = w.ring0 + bs * stage_units, more = (kb | i) != 0;
        // a stage's MMAs from u0 to u1, numbered (filter row, 32 bytes of the channels)
        auto part = [&](int u0, int u1) {
#pragma unroll
          for (int u = 0; u < RPS * 4; ++u) {
            if (u < u0 || u >= u1) continue;
            const uint32_t al = a_lo[u >> 2] + 2 * (u & 3), bl = b_lo + (u >> 2) * row_units + 2 * (u & 3), adds = u ? 1u : more;
            if (kTogether) umma_words_if<KIND, PAIR>(leader, acc, al, bl, desc_hi, idesc, adds);
            else umma_words<KIND, PAIR>(acc, al, bl, desc_hi, idesc, adds);
          }
        };
        constexpr int kBefore = RPS > 1 ? RPS * 4 - 4 : 2;
        if (kTogether) part(0, kBefore);
        else if (leader) part(0, kBefore);
        __syncwarp();
        const int cur = bs;
        if (++bs == p.b_stages) { bs = 0; bphase ^= w.resident ^ 1; }
        b_seen = mbar_look(&bars->b_full[bs], bphase);
        if (i + RPS >= p.kH) {
          const int ns = sb + 1 == p.s_stages ? 0 : sb + 1;
          slab_seen = mbar_look(&bars->slab_full[ns], ns ? sphase : sphase ^ 1);
          if (kb + 1 == p.kblocks) {
            const int nb = buf + 1 == p.sets ? 0 : buf + 1;
            acc_seen = mbar_look(&bars->acc_empty[nb], nb ? aphase ^ 1 : aphase);
          }
        }
        if (kTogether) part(kBefore, RPS * 4);
        if (leader) {
          if (!kTogether) part(kBefore, RPS * 4);
          if (!w.resident) commit(&bars->b_empty[cur]);
        }
      }
      if (leader) commit(&bars->slab_empty[sb]);
      if (++sb == p.s_stages) { sb = 0; sphase ^= 1; }
    }
    if (leader) commit(&bars->acc_full[buf]);
    if (++buf == p.sets) { buf = 0; aphase ^= 1; }
  }
  return true;
}

// What 16 filters of one output add up to: their columns of the accumulator, `step` apart per filter column, the j-th from the position
// j * dil to the right (in the same warp).  A whole warp.
template <int N>
__device__ __forceinline__ void add_columns(uint32_t col, int step, int dil, int j0, float (&f)[16]) {
  uint32_t r[N][16];
#pragma unroll
  for (int j = 0; j < N; ++j) tmem_ld16(col + (j0 + j) * step, r[j]);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if (j == 0 && j0 == 0) {
#pragma unroll
      for (int q = 0; q < 16; ++q) f[q] = __uint_as_float(r[0][q]);
    } else {
#pragma unroll
      for (int q = 0; q < 16; ++q) f[q] += __uint_as_float(__shfl_down_sync(0xffffffffu, r[j][q], (j0 + j) * dil));
    }
  }
}
__device__ __forceinline__ void column_sums(uint32_t col, int step, int dil, int kW, float (&f)[16]) {
  __syncwarp();
  if (kW == 3) {
    add_columns<3>(col, step, dil, 0, f);
    return;
  }
  add_columns<2>(col, step, dil, 0, f);
#pragma unroll 1
  for (int j = 2; j < kW; ++j) add_columns<1>(col, step, dil, j, f);
}

template <MmaKind KIND, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
conv_cols_kernel(const __grid_constant__ ColsConvParams p) {
  using OutT = typename std::conditional<KIND == MmaKind::TF32, float, __half>::type;
  constexpr int kBK = KIND == MmaKind::TF32 ? 32 : 64;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* bring = smem + p.s_stages * p.slab_bytes;
  const int n_cols = p.kW * p.bn, stage_b = p.rps * (PAIR ? n_cols / 2 : n_cols) * 128;      // a pair's CTAs load half of the filters each
  uint8_t* staging = bring + p.b_stages * stage_b;               // a multiple of 1024: bn is a multiple of 16
  Bars* bars = reinterpret_cast<Bars*>(staging + p.stage_nbuf * p.stage_bytes);

  const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
  const uint32_t pix_tiles = static_cast<uint32_t>(p.tiles_w) * p.tiles_h * p.Nimg, total = (PAIR ? (pix_tiles + 1) / 2 : pix_tiles) * p.groups;      // fits 32 bits (the launcher checks)
  const uint32_t rank = PAIR ? cluster_ctarank() : 0, first = PAIR ? blockIdx.x >> 1 : blockIdx.x, stride = PAIR ? gridDim.x >> 1 : gridDim.x;
  const int issuers = p.n_acc;                                   // 1 or 2
  const int nchunks = p.d2s ? 1 : (p.n_out + p.chunk_ch - 1) / p.chunk_ch;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(&bars->slab_full[s], 1);
      mbar_init(&bars->slab_empty[s], issuers);
      mbar_init(&bars->b_full[s], 1);
      mbar_init(&bars->b_empty[s], issuers);
    }
    for (int b = 0; b < kMaxSets; ++b) {
      mbar_init(&bars->acc_full[b], issuers);
      mbar_init(&bars->acc_empty[b], PAIR ? 2 * nchunks : nchunks * 4 * p.n_acc);       // the warps that read a tile; a pair: one arrival per CTA and chunk
    }
    bars->abort = 0;
    mbar_fence_init();
  }
  // descriptors, beside the set-up and the wait for the kernel before (they are parameters, not global data)
  if (warp == 2 && lane == 0) {
    tma_prefetch_desc(&p.view);
    tma_prefetch_desc(&p.wmap);
    if (!p.d2s) tma_prefetch_desc(&p.out_map);
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

  if (warp == 0) {
    const bool leader = elect_one();
    const uint32_t tx = static_cast<uint32_t>(p.pitch * p.Hs) * 128u;
    int sb = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (uint32_t t = first; t < total && ok; t += stride) {
      const Tile w = tile_of<PAIR>(p, t, rank);
      for (int kb = 0; kb < p.kblocks; ++kb) {
        if (!uniform_wait(&bars->slab_empty[sb], phase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
        if (leader) {
          if (rank == 0) mbar_expect_tx(&bars->slab_full[sb], PAIR ? 2 * tx : tx);      // both CTAs' bytes
          if (PAIR) tma_load_5d_pair(smem + sb * p.slab_bytes, &p.view, &bars->slab_full[sb], kb * kBK, w.g, w.w0 + p.dw_min, w.h0 + p.dh_min, w.n);
          else tma_load_5d(smem + sb * p.slab_bytes, &p.view, &bars->slab_full[sb], kb * kBK, w.g, w.w0 + p.dw_min, w.h0 + p.dh_min, w.n);
        }
        if (++sb == p.s_stages) { sb = 0; phase ^= 1; }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else if (warp == kFilterProducer) {
    // a stage is rps filter rows of one channel block: neighbours in the packed filters, they arrive as one box
    const bool leader = elect_one();
    int bs = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (uint32_t t = first; t < total && ok; t = p.resident ? total : t + stride) {
      const int g = t % static_cast<uint32_t>(p.groups);
      for (int kb = 0; kb < p.kblocks && ok; ++kb) {
        for (int i = 0; i < p.kH; i += p.rps) {
          if (!uniform_wait(&bars->b_empty[bs], phase ^ 1, bars, p.wait_clocks)) { ok = false; break; }
          if (leader) {
            if (rank == 0) mbar_expect_tx(&bars->b_full[bs], (PAIR ? 2 : 1) * stage_b);
            if (PAIR) tma_load_4d_pair(bring + bs * stage_b, &p.wmap, &bars->b_full[bs], kb * kBK, static_cast<int>(rank) * (p.bn / 2), g, p.row_mat[i]);
            else tma_load_4d(bring + bs * stage_b, &p.wmap, &bars->b_full[bs], kb * kBK, 0, g, p.row_mat[i]);
          }
          if (++bs == p.b_stages) { bs = 0; phase ^= 1; }
        }
      }
    }
    if (!ok && leader) report_status(p.status, kStatusTimeout);
  } else if (warp == 1 || warp == kSecondIssuer) {
    // Issuer a: accumulator a of every tile, all 32 lanes in the loop, one elected lane issues (conv_slab.cu).
    const int a = warp == 1 ? 0 : 1;
    if (rank == 0 && a < p.n_acc) {              // a pair: the even CTA issues for both
      const bool leader = elect_one();
      const uint32_t desc_lo = static_cast<uint32_t>(smem_desc(0, 16, 1024));
      const IssueLoop w{p, bars, desc_lo + ((smem_u32(smem) + 16384u * a) >> 4), desc_lo + (smem_u32(bring) >> 4), tmem + a * n_cols, first, stride, total, leader, p.resident ? 1u : 0u};
      bool ok;
      switch (p.rps) {
        case 2: ok = issue_tiles<KIND, 2, PAIR>(w); break;
        case 3: ok = issue_tiles<KIND, 3, PAIR>(w); break;
        case 4: ok = issue_tiles<KIND, 4, PAIR>(w); break;
        case 5: ok = issue_tiles<KIND, 5, PAIR>(w); break;
        default: ok = issue_tiles<KIND, 1, PAIR>(w); break;
      }
      if (!ok && leader) report_status(p.status, kStatusTimeout);
    }
  } else {
    // Warp w reads TMEM lanes [32 * (w % 4), +32) of accumulator a.  Groups of 4 * n_acc warps take one chunk of the channels of every
    // step-th tile each: beside one another they keep step tiles, in as many accumulator sets, in work.  A single warp's way through a
    // chunk is about 3000 clocks of latencies, so what counts is how many are on their way, and that nobody waits for tiles of others.
    const int quad = warp & 3, sub = (warp - 2) >> 2;
    const int a = sub % p.n_acc, grp = sub / p.n_acc, gthreads = 128 * p.n_acc;
    const int tig = a * 128 + quad * 32 + lane, hh = tig / p.pitch, ww = tig - hh * p.pitch;      // this lane's position on the slab's grid
    const bool inbox = hh < p.th && ww < p.wt;
    const int drow = hh * p.wt + ww;
    const bool issuer = tig == 0;
    const bool plain = p.epi.alpha == 1.f && !p.bias && !p.relu;
    const int row_bytes = p.chunk_ch * static_cast<int>(sizeof(OutT));
    // 16-byte pieces of a staged row are swizzled the way a store map of 128, 64 or 32 bytes expects
    const int sw_mask = row_bytes >= 128 ? 7 : row_bytes >= 64 ? 3 : 1, sw_shift = row_bytes >= 128 ? 0 : row_bytes >= 64 ? 1 : 2;
    auto piece_at = [&](int row, int piece) { return row * row_bytes + ((piece ^ ((row >> sw_shift) & sw_mask)) << 4); };
    const int my_row = drow * row_bytes, my_swizzle = (drow >> sw_shift) & sw_mask;
    constexpr int kPieces = 16 * static_cast<int>(sizeof(OutT)) / 16;                             // of 16 channels
    const int bufs = p.stage_nbuf / (nchunks * p.step), ch = nchunks == 2 ? grp & 1 : 0, mine = nchunks == 2 ? grp >> 1 : grp, co0 = ch * p.chunk_ch;
    bool ok = true;
    int buf = mine < p.sets ? mine : 0, nstore = 0;
    uint32_t phase = 0;
    for (uint32_t t = mine < p.step ? first + mine * stride : total; t < total; t += p.step * stride) {
      const Tile w = tile_of<PAIR>(p, t, rank);
      wait_or_walk_on(ok, &bars->acc_full[buf], phase, bars, lane, p.wait_clocks);
      tc_fence_after();
      const uint32_t acc0 = tmem + (buf * p.n_acc + a) * n_cols + p.col_first + (static_cast<uint32_t>(quad * 32) << 16);
      // the accumulator goes back as soon as its last columns are in registers
      auto release = [&] {
        tc_fence_before();
        if (PAIR) {
          named_barrier(5 + grp, gthreads);
          if (issuer) mbar_arrive_leader(&bars->acc_empty[buf]);
        } else {
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->acc_empty[buf]);
        }
      };
      if (p.d2s) {
        // classes of a stride-2 gradInputs: filter cls * C + c is channel c of the pixel (2 h + cls / 2, 2 w + cls % 2), whose stored channels
        // are 16 bytes; neighbouring lanes write neighbouring pixels
        {
          float f[16];
          column_sums(acc0, p.col_step, p.dil, p.kW, f);
          release();
          const int h = w.h0 + hh, x = w.w0 + ww;
          auto put = [&](auto channels) {
            constexpr int C = decltype(channels)::value, V = 16 / sizeof(OutT);
#pragma unroll
            for (int cls = 0; cls < 4; ++cls) {
              __align__(16) OutT px[V];
#pragma unroll
              for (int e = 0; e < V; ++e) px[e] = static_cast<OutT>(e < C ? f[(cls * C + e) & 15] : 0.f);
              const int H = 2 * h + (cls >> 1), W = 2 * x + (cls & 1);
              const long long at = ((1LL * w.n * p.d2s_H + H) * p.d2s_W + W) * V;
              if (!inbox || H >= p.d2s_H || W >= p.d2s_W || !B200_IN_RANGE(at >= 0 && at + V <= p.out_elems, p.status)) continue;
              if ((reinterpret_cast<uintptr_t>(p.out) & 15) == 0) {
                *reinterpret_cast<uint4*>(static_cast<OutT*>(p.out) + at) = *reinterpret_cast<const uint4*>(px);
              } else {
#pragma unroll
                for (int e = 0; e < V; ++e) static_cast<OutT*>(p.out)[at + e] = px[e];
              }
            }
          };
          switch (p.d2s_C) {
            case 1: put(std::integral_constant<int, 1>()); break;
            case 2: put(std::integral_constant<int, 2>()); break;
            case 3: put(std::integral_constant<int, 3>()); break;
            case 4: put(std::integral_constant<int, 4>()); break;
          }
        }
      } else {
        {
          uint8_t* stg = staging + (grp * bufs + (bufs == 2 ? nstore & 1 : 0)) * p.stage_bytes;
          if (nstore >= bufs) {                  // the buffer's previous box must have been read
            if (issuer) {
              if (bufs == 2) bulk_wait_read<1>();
              else bulk_wait_read<0>();
            }
            named_barrier(1 + grp, gthreads);
          }
#pragma unroll 1
          for (int c = 0; c < p.chunk_ch; c += 16) {
            float f[16];
            column_sums(acc0 + ch * p.chunk_step + c, p.col_step, p.dil, p.kW, f);
            if (c + 16 >= p.chunk_ch) release();
            if (p.n_real - co0 - c < 16) {
#pragma unroll
              for (int q = 0; q < 16; ++q)
                if (q >= p.n_real - co0 - c) f[q] = 0.f;       // pad channels: their filters are zero, but zero times an infinity is NaN
            }
            if (!plain) {
              const OutT* bias = p.bias ? static_cast<const OutT*>(p.bias) + w.g * p.n_out + co0 + c : nullptr;
#pragma unroll
              for (int q = 0; q < 16; ++q) {
                f[q] *= p.epi.alpha;
                if (bias && co0 + c + q < p.n_out) f[q] += static_cast<float>(bias[q]);
                if (p.relu) f[q] = p.epi.lin * f[q] + p.epi.abs * fabsf(f[q]);
              }
            }
            const int piece0 = c * static_cast<int>(sizeof(OutT)) / 16;
            if (inbox) {
#pragma unroll
              for (int j = 0; j < kPieces; ++j) {
                uint4 v;
                if (sizeof(OutT) == 4) {
                  v = make_uint4(__float_as_uint(f[4 * j]), __float_as_uint(f[4 * j + 1]), __float_as_uint(f[4 * j + 2]), __float_as_uint(f[4 * j + 3]));
                } else {
                  uint32_t h[4];
#pragma unroll
                  for (int q = 0; q < 4; ++q) {
                    __half2 h2 = __floats2half2_rn(f[(8 * j + 2 * q) & 15], f[(8 * j + 2 * q + 1) & 15]);
                    h[q] = *reinterpret_cast<uint32_t*>(&h2);
                  }
                  v = make_uint4(h[0], h[1], h[2], h[3]);
                }
                *reinterpret_cast<uint4*>(stg + my_row + (((piece0 + j) ^ my_swizzle) << 4)) = v;
              }
            }
          }
          if (p.epi.pool) {
            // 2x2 max pooling of the staged chunk: tiles have even sides, so every window lies inside one.  The maxima stay in registers until
            // all rows are read, then go to the front of the buffer.
            named_barrier(1 + grp, gthreads);
            const int pw = p.wt >> 1, prows = (p.th >> 1) * pw, pieces = row_bytes >> 4;
            uint4 keep[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int i = tig + u * gthreads;
              if (i < prows * pieces) {
                const int pr = i / pieces, piece = i - pr * pieces, h2 = pr / pw, d00 = 2 * h2 * p.wt + 2 * (pr - h2 * pw);
                uint4 m = *reinterpret_cast<const uint4*>(stg + piece_at(d00, piece));
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                  const uint4 v = *reinterpret_cast<const uint4*>(stg + piece_at(d00 + (k & 1) + (k >> 1) * p.wt, piece));
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
              if (i < prows * pieces) {
                const int pr = i / pieces;
                *reinterpret_cast<uint4*>(stg + piece_at(pr, i - pr * pieces)) = keep[u];
              }
            }
          }
          fence_async_smem();
          named_barrier(1 + grp, gthreads);
          if (issuer && (!PAIR || w.n < p.Nimg) && B200_IN_RANGE(w.w0 >= 0 && w.h0 >= 0 && w.w0 < p.Wt && w.h0 < p.Ht && w.n < p.Nimg && co0 < p.n_out, p.status)) {
            if (p.epi.pool) tma_store_4d(&p.out_map, stg, w.g * p.n_out + co0, w.w0 >> 1, w.h0 >> 1, w.n);
            else tma_store_4d(&p.out_map, stg, w.g * p.n_out + co0, w.w0, w.h0, w.n);
            bulk_commit();
          }
          ++nstore;
        }
      }
      if (p.sets == p.step || (buf ^= 1) == 0) phase ^= 1;       // the group's own set, or the two in turn
    }
    if (lane == 0) bulk_wait<0>();           // this thread's stores (if it issued any) have left shared memory
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
}

template <MmaKind KIND, bool PAIR>
cudaError_t launch_one(const ColsConvParams& p, long long total, int num_sms, cudaStream_t s) {
  static PerDeviceOnce configured;
  cudaError_t e = configured.ensure([] { return cudaFuncSetAttribute(conv_cols_kernel<KIND, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024); });
  if (e != cudaSuccess) return e;
  const int smem = p.s_stages * p.slab_bytes + p.b_stages * p.rps * p.kW * (PAIR ? p.bn / 2 : p.bn) * 128 + p.stage_nbuf * p.stage_bytes + static_cast<int>(sizeof(Bars)) + 1024;
  const int all = PAIR ? num_sms / 2 : num_sms, units = p.resident ? all / p.groups * p.groups : all, grid = static_cast<int>(total < units ? total : units) * (PAIR ? 2 : 1);
  launch_linked(true, conv_cols_kernel<KIND, PAIR>, grid, kThreads, smem, s, PAIR ? 2 : 1, p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_conv_cols(const ColsConvParams& p, int dtype, int num_sms, cudaStream_t s) {
  const long long pix_tiles = 1LL * p.tiles_w * p.tiles_h * p.Nimg, total = (p.pair ? (pix_tiles + 1) / 2 : pix_tiles) * p.groups;
  if (total == 0) return cudaSuccess;
  if (p.pair && (p.bn != 64 || p.d2s || p.n_acc != 1 || num_sms < 2)) return cudaErrorInvalidValue;
  if (total >= (1LL << 31) || p.n_acc < 1 || p.n_acc > 2 || p.sets < 2 || p.sets > kMaxSets || (p.step != p.sets && (p.step != 1 || p.sets != 2)) || p.sets * p.n_acc * p.kW * p.bn > 512 || p.kH > kMaxColTaps || p.rps < 1 || p.kH % p.rps || p.kW > kMaxColTaps ||
      p.s_stages < 2 || p.s_stages > kMaxStages || p.b_stages < (p.resident ? 1 : 2) || p.b_stages > kMaxStages ||
      (p.resident && (p.b_stages != p.kblocks * (p.kH / p.rps) || (p.pair ? num_sms / 2 : num_sms) < p.groups))) return cudaErrorInvalidValue;
  if (p.pair) return dtype == B200CONV_F16 ? launch_one<MmaKind::F16, true>(p, total, num_sms, s) : launch_one<MmaKind::TF32, true>(p, total, num_sms, s);
  return dtype == B200CONV_F16 ? launch_one<MmaKind::F16, false>(p, total, num_sms, s) : launch_one<MmaKind::TF32, false>(p, total, num_sms, s);
}

}  // namespace b200
