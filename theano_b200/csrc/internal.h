// Declarations shared by the translation units of libb200conv (not part of the C ABI).
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <initializer_list>

#include "../../include/b200conv.h"
#include "geometry.h"

namespace b200 {

// cudaFuncSetAttribute applies to the device that is current when it is called, so a process
// that opens contexts on several devices has to repeat it on each: one bit per device.
struct PerDeviceOnce {
  std::atomic<unsigned long long> done{0};
  // Runs `set()` (returning cudaError_t) unless it already ran on the current device.
  template <class F> cudaError_t ensure(F set) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ULL << dev : 0ULL;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    e = set();
    if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_release);
    return e;
  }
};

// Chained launches (programmatic dependent launch): the CTAs of a kernel start, set up their barriers and
// take their TMEM while the kernel before it in the stream drains, then wait in pdl_enter() until that
// one has finished and its writes are visible.  Rules that keep this safe:
//  * every kernel launched this way executes pdl_enter() before its first access to global memory, so
//    that "the kernel before has finished" implies the same for all earlier ones;
//  * a kernel that takes TMEM executes it after its allocation: the next kernel's CTAs, which may
//    allocate too and then wait, start only when all CTAs of this one have passed that point.
// Between two kernels of a stream this saves 1.5 to 3 us of launch latency and drain.
// launch_streaming() is for kernels that stream through L1: chained only while all their CTAs are
// resident at once (kChainedBlocks).  CTAs that start beside a tensor-core kernel leave the SM split as
// that kernel wants it, 228 KB of shared memory and 28 KB of L1, for as long as CTAs keep arriving, and
// with that little L1 too few loads are in flight: the pooling gradient of 64 x 128 x 112 x 112 after a
// convolution took 250 instead of 148 us.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif
template <class... Exp, class... Act>
cudaError_t launch_linked(bool chained, void (*kernel)(Exp...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, int cluster, Act&&... args) {
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = chained ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster; at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cfg.attrs = at; cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Exp>(args)...);
}

template <class... Exp, class... Act>
cudaError_t launch_chained(void (*kernel)(Exp...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Act&&... args) {
  return launch_linked(true, kernel, grid, block, smem, s, 1, args...);
}
// 148 (here and in the grids of the memory-bound kernels) are the SMs of a B200: these kernels fill the device whatever
// b200conv_set_sm_count leaves to the persistent ones.
constexpr unsigned kChainedBlocks = 148 * 8;      // of 256 threads
template <class... Exp, class... Act>
cudaError_t launch_streaming(void (*kernel)(Exp...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Act&&... args) {
  return launch_linked(grid.x * grid.y * grid.z <= kChainedBlocks, kernel, grid, block, smem, s, 1, args...);
}

// Kernels with 16-byte accesses take an element-wise form where a caller's tensor starts off the 16-byte boundaries.
inline bool aligned16(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}

// n / d for n < 2^31 by a multiplication (Granlund and Montgomery, "Division by invariant integers using multiplication")
struct Divisor { uint32_t d, mul, shift; };
inline Divisor divisor(uint32_t d) {
  if (d == 0) d = 1;                     // of launches that have nothing to do
  uint32_t shift = 0;
  while ((1ull << shift) < d) ++shift;
  return Divisor{d, static_cast<uint32_t>(((1ull << 32) * ((1ull << shift) - d)) / d + 1), shift};
}
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t quotient(uint32_t n, const Divisor& v) { return (__umulhi(n, v.mul) + n) >> v.shift; }
#endif

// How the convolution kernels walk their work items: (pixel tile, group, filter tile, slice of the reduction), the slice fastest.  Every
// role finds its place with these quotients once per tile; divided out, they cost a warp of the epilogue 2000 clocks, more than reading
// the accumulators of a 256 x 64 tile out and storing them (a B200: 64 -> 256 1x1 at 56x56, float16, 256 images 107 -> 95 us, 64 -> 64 48 -> 37;
// 3 -> 64 3x3 at 224x224, float32, 64 images 268 -> 202; 3 -> 64 7x7 stride 2 at 224x224, float16, 256 images 243 -> 194).
struct TileWalk { Divisor splits, tiles_co, groups, tiles_w, tiles_h; };
inline TileWalk tile_walk(int splits, int tiles_co, int groups, int tiles_w, int tiles_h) {
  return TileWalk{divisor(splits), divisor(tiles_co), divisor(groups), divisor(tiles_w), divisor(tiles_h)};
}
#ifdef __CUDACC__
struct TileAt { int co_t, g, w, h, n; };         // filter tile, group, pixel tile
template <bool PAIR = false> __device__ __forceinline__ TileAt tile_at(const TileWalk& k, uint32_t tile, uint32_t rank = 0) {
  const uint32_t tg = quotient(tile, k.tiles_co), tp = quotient(tg, k.groups), pt = PAIR ? 2 * tp + rank : tp;
  const uint32_t row = quotient(pt, k.tiles_w), n = quotient(row, k.tiles_h);
  return TileAt{static_cast<int>(tile - tg * k.tiles_co.d), static_cast<int>(tg - tp * k.groups.d), static_cast<int>(pt - row * k.tiles_w.d),
                static_cast<int>(row - n * k.tiles_h.d), static_cast<int>(n)};
}
#endif

// Codes a kernel writes to the device status word when it gives up.
enum : int { kStatusOk = 0, kStatusTimeout = 1, kStatusBadIndex = 2 };

// ---- implicit-GEMM convolution (conv_umma.cu) -----------------------------------------
// One "tap" of the reduction: a spatial offset into one activation view and the filter
// slice that multiplies it.
struct ConvTap {
  int16_t dh, dw;   // offset added to the output-tile origin (in the view's pixel grid)
  int16_t view;     // which activation tensor map
  int16_t wmat;     // which packed filter matrix
};

// Forward epilogue: y = act(alpha * conv + bias + beta * residual); with `relu` set
// act(v) = lin * v + abs * |v|  (ReLU: 0.5, 0.5; leaky ReLU of slope s: 0.5 * (1 + s), 0.5 * (1 - s),
// the reference's formula, theano/tensor/nnet/nnet.py:2242-2250), else the identity.  `residual` has
// the layout of the output.  Defaults (alpha 1, no residual, 0.5 / 0.5) reproduce bias + ReLU.
struct ConvEpilogue {
  const void* residual;
  float alpha, beta, lin, abs;
  int pool;          // 1: 2x2 max pooling (stride 2) of the activated result inside the epilogue; the output tensor has
                     // half the rows and columns (slab kernel with staged TMA stores only)
};
inline ConvEpilogue default_epilogue() { return ConvEpilogue{nullptr, 1.f, 0.f, 0.5f, 0.5f, 0}; }

struct alignas(64) UmmaConvParams {
  CUtensorMap views[kMaxViews];  // 5-D (c_in_group, group, w, h, n) channels-last views
  int nviews;
  CUtensorMap wmap;              // 3-D (k_red, n_out, wmat*groups + g) packed filters
  ConvTap taps[kMaxTaps];
  int ntaps;
  int kblocks;                   // ceil(reduction channels per group / channels per stage)
  int bn_cols;                   // accumulator columns of a tile (32, 64, 128 or 256)
  int splits;                    // slices of the reduction; > 1: float32 accumulators go to `partial` (conv_reduce.cu)
  int cut;                       // conv_pair.cu: that many tiles (of pairs), the first ones, are cut into `splits` slices
  unsigned int* arrivals;        // counts of their slices, zero between launches; null: conv_reduce.cu adds the slices
  float* partial;
  long long partial_elems;       // elements of `partial` (checked in the range-checked build)
  int groups;
  int Wt, Ht, Nimg;              // extent of the output pixel grid this launch covers
  int bw, bh, bn;                // pixel tile (bw*bh*bn <= 128 rows of the accumulator)
  int tiles_w, tiles_h, tiles_n, tiles_co;
  TileWalk walk;
  int n_out;                     // output channels per group as stored
  int n_mma;                     // those that the widths of the MMAs follow: n_out, or whole tiles
  int n_real;                    // of these, the ones with filters: the pad channels behind them are stored as 0
  void* out;
  const void* bias;              // per output channel (groups*n_out), in the data type, or null
  long long out_sn, out_sc, out_sh, out_sw, out_off;  // element strides / offset of `out`
  long long out_elems;           // elements of `out` this launch may touch (checked in the range-checked build)
  int relu;
  ConvEpilogue epi;
  int* status;
  long long wait_clocks;          // bound of every device-side wait, in SM clocks
  CUtensorMap out_map;            // conv_pair.cu: 4-D (channel, w, h, n) over the output, box (128 bytes, bw, bh, bn)
};

// Columns of the MMAs of a tile that starts at output channel `first` of n_out: an MMA takes clocks by its columns, and a layer of
// 75 filters need not pay for the 128 that its accumulator has room for.  Multiples of 16, on pairs of CTAs of 32.  (37 images of 27 x 33,
// 5x5, float16: 100 -> 75 filters on pairs 28.5 -> 26.0 us, 75 -> 100 on single CTAs 27.3 -> 26.6.)
#ifdef __CUDACC__
__host__ __device__
#endif
inline int mma_columns(int n_out, int first, int bn, bool pair) {
  const int step = pair ? 32 : 16, n = (n_out - first + step - 1) / step * step;
  return n < bn ? n : bn;
}
int conv_umma_bn(int n_out);      // accumulator columns that hold n_out outputs per group, at most 256
cudaError_t launch_conv_umma(const UmmaConvParams& p, int dtype, int num_sms, cudaStream_t s);
// The same on pairs of CTAs (conv_pair.cu): channels-last outputs of whole 128-byte channel rows, no residual, 128 or 256 accumulator columns.
cudaError_t launch_conv_pair(const UmmaConvParams& p, int dtype, int num_sms, cudaStream_t s);
// Puts the kernel's code on the device (it is otherwise loaded by its first launch, which needs memory): a launch that
// runs split loads the code of the whole reduction with it, to fall back to when there is no memory for the slices.
cudaError_t load_conv_umma(int dtype, int bn);
cudaError_t load_conv_slab(int dtype, int bn);

// ---- implicit GEMM with one activation slab per channel block (conv_slab.cu) ---------------
// For launches whose taps all read the same view: the slab (output tile plus halo) is loaded
// once per channel block and every tap is a row offset into it.
constexpr int kMaxSlabClasses = 4;
// A tap in one word: row offset of the tap inside the slab in 16-byte units, column of its class's accumulator, and
// whether its products add to earlier ones of the class (set for all but the first tap of each class where there are several).
inline uint32_t slab_tap(int row_shift, int column, bool adds) { return static_cast<uint32_t>(row_shift) * 8 | static_cast<uint32_t>(column) << 16 | (adds ? 1u << 31 : 0u); }
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t slab_tap_shift(uint32_t tap) { return tap & 0xFFFF; }
__device__ __forceinline__ uint32_t slab_tap_column(uint32_t tap) { return (tap >> 16) & 0x7FFF; }
__device__ __forceinline__ uint32_t slab_tap_adds(uint32_t tap) { return tap >> 31; }
#endif
struct alignas(64) SlabConvParams {
  CUtensorMap view;              // 5-D (c_in_group, group, w, h, n), box (kBK, 1, Ws, Hs, nb)
  CUtensorMap wmap;              // 4-D packed filters (k_red, n_out, group, tap), box (kBK, BN or half of it, 1, 1 or tps)
  uint32_t tap_issue[kMaxTaps];  // what the MMAs of the tap need (slab_tap)
  int16_t tap_wmat[kMaxTaps];
  // Output classes: the taps of class q add up in accumulators of their own, and the class has its own output tensor
  // (strided gradInputs: the stride's parity classes of dx, all from one slab of dy).  1: one output, no classes.
  int ncls;
  int cls_W[kMaxSlabClasses], cls_H[kMaxSlabClasses];    // output grid of the class (at most Wt x Ht)
  int ntaps;
  int kblocks;
  int groups;
  int Wt, Ht, Nimg;              // output grid
  int wt, th, nb;                // output columns / rows / images per tile
  int Ws, Hs;                    // slab columns / rows per image (tile + halo)
  int dw_min, dh_min;            // view coordinate of slab column / row 0 relative to the tile origin
  int tiles_w, tiles_h, tiles_n, tiles_co;
  TileWalk walk;
  int n_acc;                     // 128-row accumulators in use (<= 512 / BN)
  int slab_bytes;                // bytes of one slab buffer (1024-byte multiple)
  int b_stages;                  // filter-tile ring depth
  int s_stages;                  // slab ring depth (2 .. 6)
  int splits;                    // slices of the reduction; > 1: float32 accumulators go to `partial` (conv_reduce.cu)
  float* partial;
  long long partial_elems;       // elements of `partial` (checked in the range-checked build)
  int pair;                      // 1: CTA pairs (two pixel tiles side by side, M = 256); splits is 1
  int tap_boxes;                 // 1: one TMA box per tap; 0: the taps of a stage are neighbours in the packed filters
                                 // and arrive as one box (the map's box then is tps matrices deep)
  int tps;                       // filter taps per stage of the filter ring (narrow tiles: several taps share a barrier round)
  int tap_groups;                // stages of a channel block: ceil(ntaps / tps)
  int n_out, n_real;             // output channels per group as stored / with filters
  int n_mma;                     // those that the widths of the MMAs follow: n_out, or whole tiles
  void* out;
  const void* bias;
  long long out_sn, out_sc, out_sh, out_sw, out_off;
  long long out_elems;           // elements of `out` this launch may touch (checked in the range-checked build)
  int relu;
  ConvEpilogue epi;
  int* status;
  long long wait_clocks;          // bound of every device-side wait, in SM clocks
  long long* trace;              // optional: 9 clock64 stamps per CTA (phase timing), 32 slots apart, or null
  // Channels-last outputs are written by TMA: the epilogue warps put 128-byte channel chunks (32
  // float32 / 64 float16) of the tile into shared memory (rows = the tile's pixels, dense) and one
  // thread per chunk stores the box (chunk, wt, th, nb) through out_map.
  CUtensorMap out_map[kMaxSlabClasses];      // 4-D (channel, w, h, n) over the output view of each class
  int tma_out;                   // 1: epilogue through out_map, 0: direct stores
  int stage_off;                 // byte offset of the staging buffers in dynamic shared memory
  int stage_reserved;            // bytes set aside for them behind the filter ring (0: they reuse the
                                 // operand buffers, which are dead when a CTA's only tile is done)
  int stage_bytes;               // bytes of one staging buffer (1024-byte multiple)
  int stage_nbuf;                // staging buffers (a multiple of the number of warp groups)
};
constexpr int kSlabStageBytes = 64 * 1024;    // staging buffers of the TMA-store epilogue (all groups)
constexpr int kSlabSmemBudget = 220 * 1024;   // slab buffers + filter ring; the rest of the 227 KB
                                              // holds barriers and the epilogue's transpose tiles
cudaError_t launch_conv_slab(const SlabConvParams& p, int dtype, int bn, int num_sms, cudaStream_t s);

// ---- layers of at most 64 filters, the filter's columns inside one MMA (conv_cols.cu) ----------------
constexpr int kMaxColTaps = 8;   // filter rows, filter columns
constexpr int kMaxColStages = 8; // of a ring
struct alignas(64) ColsConvParams {
  CUtensorMap view;              // 5-D (c_in_group, group, w, h, n), box (kBK, 1, pitch, Hs, 1)
  CUtensorMap wmap;              // 4-D packed filters (k_red, n_out, group, tap), box (kBK, bn, 1, rps * kW)
  CUtensorMap out_map;           // 4-D (channel, w, h, n) over the output, box (chunk_ch, wt, th, 1), pooled: half of wt and th
  int kH, kW;
  int16_t row_mat[kMaxColTaps];  // filter row: its first packed matrix
  int16_t row_shift[kMaxColTaps];// and how many slab positions it lies behind the first
  int col_first, col_step, dil;  // accumulator column of the leftmost filter column, from there to the next (to the right), positions between them
  int bn;                        // accumulator columns per filter column (16, 32 or 64)
  int kblocks, groups;
  int Wt, Ht, Nimg;              // output grid
  int wt, th, pitch, Hs;         // tile, positions from one slab row to the next (8, 16 or 32), slab rows
  int dw_min, dh_min;            // view coordinate of slab column / row 0 relative to the tile origin
  int tiles_w, tiles_h;
  Divisor by_groups, by_tiles_w, by_tiles_h;
  int n_acc;                     // 128-row accumulators of a tile: 1 or 2
  int sets;                      // of accumulators: 2 to 4, and as many tiles apart are the ones of a group of epilogue warps (every tile, where it has no choice)
  int step;                      // that distance
  int slab_bytes, s_stages, b_stages;
  int rps;                       // filter rows per filter stage (a divisor of kH)
  int resident;                  // 1: the filter ring is the filters of one tile, loaded once (a CTA's tiles are of one group)
  int n_out, n_real;             // output channels per group as stored / with filters
  int pair;                      // 1: CTA pairs (two pixel tiles side by side, M = 256; 64 columns per filter column, 32 of them per CTA)
  int chunk_step;                // accumulator columns from one chunk to the next
  int chunk_ch;                  // channels of a staged row: 16 or 32
  int stage_bytes, stage_nbuf;   // staging buffers (one or two per group of epilogue warps)
  int d2s, d2s_C, d2s_H, d2s_W;  // 1: the filters are the four classes of a stride-2 gradInputs with d2s_C channels, `out` the H x W gradient itself
  void* out;
  long long out_elems;           // of `out` (checked in the range-checked build)
  const void* bias;
  int relu;
  ConvEpilogue epi;
  int* status;
  long long wait_clocks;         // bound of every device-side wait, in SM clocks
};
cudaError_t launch_conv_cols(const ColsConvParams& p, int dtype, int num_sms, cudaStream_t s);

// ---- reductions split over CTAs (conv_reduce.cu) --------------------------------------------
// The tile geometry is that of the slab kernel (rows of a tile on a grid of Ws x Hs positions per image, of
// which wt x th are the tile's); for the per-tap kernel Ws = wt and Hs = th.
struct ConvReduceParams {
  const float* partial;          // [tile][slice][bn_cols / 4][rows][4]
  int tiles;                     // the tiles that were split, from the first on; pair: both pixel tiles of each pair tile, side by side
  int pair;
  int splits, rows, bn_cols;
  int Ws, Hs, wt, th, nb;
  int tiles_w, tiles_h, tiles_n, tiles_co, groups;
  int Wt, Ht, Nimg, n_out, n_real;
  void* out;                     // strides of the pooled tensor when epi.pool
  const void* bias;
  long long out_sn, out_sc, out_sh, out_sw, out_off;
  int relu;
  ConvEpilogue epi;
  long long partial_elems, out_elems;      // of `partial` and of `out` that this launch may touch (range-checked build)
  int* status;
};
cudaError_t launch_conv_reduce(const ConvReduceParams& p, int dtype, cudaStream_t s);

// ---- 1x1 layers on CTA pairs (gemm_pair.cu): float16, tiles of 256 pixels x 256 filters ------------
struct alignas(64) PairGemmParams {
  CUtensorMap view;              // 5-D (c, group = 1, pixel, 1, 1) over the activations, box (64, 1, 128, 1, 1)
  CUtensorMap wmap;              // 3-D packed filters, box (64, 128, 1)
  CUtensorMap out_map;           // 4-D (channel, pixel, 1, 1) over the output, box (64, 128, 1, 1)
  int kblocks;                   // ceil(channels / 64)
  int tiles_pix, tiles_co;       // 256-pixel tiles, 256-filter tiles
  Divisor by_tiles_co;
  int pixels, n_out, n_real;
  int stages;                    // ring depth (2 .. 5)
  const void* bias;
  int relu;
  ConvEpilogue epi;
  int* status;
  long long wait_clocks;
};
int gemm_pair_smem_bytes(int stages);
cudaError_t launch_gemm_pair(const PairGemmParams& p, int num_sms, cudaStream_t s);

// How the gradWeights kernels walk theirs: (filter tile, channel tile, group, tap or what the kernel puts in its place, slice), the slice fastest,
// and pixel tiles within an image.  (Set by the launchers; a role looks once per item, but on small layers there is one item per CTA, and its first
// load waited 1000 clocks for the quotients.)
struct ItemWalk { Divisor splits, taps, groups, ctiles, tiles_w, tiles_h; };
inline ItemWalk item_walk(int splits, int taps, int groups, int ctiles, int tiles_w, int tiles_h) {
  return ItemWalk{divisor(splits), divisor(taps), divisor(groups), divisor(ctiles), divisor(tiles_w), divisor(tiles_h)};
}

// ---- implicit-GEMM filter gradient (wgrad_umma.cu) -------------------------------------
struct alignas(64) UmmaWgradParams {
  CUtensorMap dy_map;            // 5-D (k_in_group, group, wo, ho, n) over dy, box 32/64 channels
  CUtensorMap x_views[kMaxViews];// 5-D views over x (stride parity classes)
  ConvTap taps[kMaxTaps];        // wmat = flat filter tap index i*kW + j (after flip)
  int ntaps;
  int groups;
  int Kg, Cg;                    // filters / channels per group
  int Wo, Ho, Nimg;
  int bw, bh, bn;                // pixel box per stage (bw*bh*bn <= wgrad_pix(dtype))
  int tiles_w, tiles_h, tiles_n; // pixel tiles covering (Wo, Ho, N)
  int ktiles, ctiles;            // 128-filter tiles, BN-channel tiles
  int splits;                    // split-K slices
  float* partial;                // one float32 slab per slice (wgrad_slab.cuh)
  int diag_c, diag_k;            // merged groups of diag_k filters x diag_c channels: only their blocks are stored; 0: everything
  long long partial_elems;       // its extent (checked in the range-checked build)
  int taps_total;                // kH*kW
  int atomic;                    // 1: red.add into partial[0] instead of per-split slabs
  int nviews;                    // x_views in use
  ItemWalk walk;                 // set by the launcher
  int* status;
  long long wait_clocks;          // bound of every device-side wait, in SM clocks
  long long* trace;              // optional: 16 clock counters per CTA (phase timing), or null
};
// Pixels (reduction rows) per pipeline stage of the gradWeights kernels.  A float16 MMA consumes 16
// rows, a tf32 MMA 8: twice the rows for float16 give every stage the same number of MMAs, so that the
// issuing thread's per-stage hand-over (a few hundred clocks) weighs the same.
// With 256 channel columns a float16 stage of 128 pixels is 96 KB, and only two fit the shared memory: too
// few copies in flight for the latency of L2 and HBM.  Those launches use 64-pixel stages (four of them).
#ifndef B200_WGRAD_PIX_WIDE
#define B200_WGRAD_PIX_WIDE 64
#endif
constexpr int kWgradPixF32 = 64, kWgradPixF16 = 128, kWgradPixF16Wide = B200_WGRAD_PIX_WIDE;
inline int wgrad_pix(int dtype, int bn_cols = 0) {
  return dtype == B200CONV_F16 ? (bn_cols >= 256 ? kWgradPixF16Wide : kWgradPixF16) : kWgradPixF32;
}
cudaError_t launch_wgrad_umma(const UmmaWgradParams& p, int dtype, int bn_cols, int num_sms,
                              cudaStream_t s);
// The same work on pairs of CTAs (wgrad_pair.cu): 256-filter x 256-channel tiles, stages of 64 pixels;
// `ktiles` / `ctiles` count 256-wide tiles.
cudaError_t launch_wgrad_pair(const UmmaWgradParams& p, int dtype, int num_sms, cudaStream_t s);
// What the elements of a gradient are sums of (wgrad_exact.cuh): the operands with their strides in elements, and the geometry.
struct WgradSum {
  const void *x, *dy;
  long long x_n, x_c, x_h, x_w, dy_n, dy_c, dy_h, dy_w;
  int f16;                               // type of x and dy
  int Cg, Kg;                            // channels / filters per group (of a layer's own groups, not of merged ones)
  int N, H, W, Ho, Wo, kH, kW, sH, sW, dilH, dilW, padH, padW, flip;
  int segments;                          // 1: zeros for dy stand behind pieces of rows too, whose ends may lie anywhere in an image
};
// Sums split-K slabs and writes the OIHW gradient; diag_c / diag_k as above (Kg: filters per merged group).
cudaError_t launch_wgrad_reduce(const float* partial, void* dw, int splits, int taps, int K, int Cg, int Kg, int diag_c, int diag_k,
                                int dtype, const WgradSum& sum, cudaStream_t s);

// ---- filter gradient with tap groups sharing their operands (wgrad_group.cu) -------------
// Taps that read the same view with the same row offset differ only by a column offset.  With
// the reduction pixels laid out on a grid whose rows are padded by that column span, a tap's x
// operand is the shared x tile advanced by (dw - dw_min) rows, so one dy tile and one x tile per
// stage serve up to four taps (four 128 x 128 accumulators in TMEM).
constexpr int kMaxTapGroups = 32;
// (`nviews` stands behind the tables: before them, it moved them off the 8-byte boundaries that whole entries are read from, and gradWeights of 112 -> 16
// 3x3 stride 2 at 39x51, 126 images, float32, took 41.4 us in place of 37.6.)
struct alignas(64) GroupWgradParams {
  CUtensorMap dy_map;              // box (atom, 1, Wa, th, nb)
  CUtensorMap x_views[kMaxViews];  // box (atom, 1, Wb, th, nb), one per stride parity class
  int16_t grp_view[kMaxTapGroups], grp_dh[kMaxTapGroups], grp_first[kMaxTapGroups], grp_n[kMaxTapGroups];
  int16_t view_dwmin[kMaxViews];
  int16_t tap_off[kMaxTaps];       // dw - dw_min of the tap's view: row offset into the x tile
  int16_t tap_wmat[kMaxTaps];      // filter tap index in OIHW order (after flip)
  int stack_step;                  // > 0: at most 64 channels and the taps of every group this many rows apart:
                                   // a group's taps are column groups of one MMA, tf32: of one per 32 channels (0: one MMA per tap)
  int ngroups;
  int groups;                      // convolution groups
  int Kg, Cg;
  int Wo, Ho, Nimg;
  int Wa, Wb, th, nb;              // dy / x box widths, rows and images per stage
  int wt;                          // output columns owned by a tile (== Wo in full-width mode)
  int rows_a, rows_b;              // box rows Wa*th*nb, Wb*th*nb
  int box_bytes, a_boxes, b_boxes, stages, ring_bytes;      // shared-memory ring (set by launch_wgrad_group)
  int tiles_w, tiles_h, tiles_n;
  int ktiles, ctiles;
  int splits;
  float* partial;                  // one float32 slab per slice (wgrad_slab.cuh)
  int diag_c, diag_k;              // merged groups of diag_k filters x diag_c channels: only their blocks are stored; 0: everything
  long long partial_elems;         // its extent (checked in the range-checked build)
  int taps_total;
  int nviews;                      // x_views in use
  int atomic;
  ItemWalk walk;                 // set by the launcher
  int* status;
  long long wait_clocks;          // bound of every device-side wait, in SM clocks
  long long* trace;                // optional: 16 clock counters per CTA (phase timing), or null
};
cudaError_t launch_wgrad_group(const GroupWgradParams& p, int dtype, int num_sms, cudaStream_t s);

// ---- filter gradient of narrow layers, filter rows and columns inside one MMA (wgrad_rows.cu) -----
constexpr int kMaxRowSets = 4;       // sets of 128 / atom filter rows per view
struct alignas(64) RowsWgradParams {
  CUtensorMap dy_map;                // box (atom, 1, pitch, th + halo, 1)
  CUtensorMap x_views[kMaxViews];    // box (atom, 1, pitch, x rows, 1), one per stride parity class
  int nviews;
  int16_t view_dh[kMaxViews], view_dw[kMaxViews];      // offset of the x box from the tile's origin
  int16_t view_nt[kMaxViews], view_sets[kMaxViews];    // filter columns / sets of filter rows of the view
  int16_t view_tap0[kMaxViews];                        // of its taps in tap_id, [filter row][filter column]
  int16_t set_first[kMaxViews][kMaxRowSets], set_base[kMaxViews][kMaxRowSets];   // first / last filter row of the set
  int16_t set_rows[kMaxViews][kMaxRowSets];            // x row offset of its last filter row
  int16_t tap_id[kMaxTaps];          // filter tap index in OIHW order (after flip)
  int stack_step, a_step;            // grid positions between the filter's columns / rows
  int groups, Kg, Cg, Nimg, ctiles;
  int pitch, th, halo, tiles_h;      // grid pitch, rows per tile, rows that the copies of dy reach back, tiles per image
  int rows_a, rows_b;                // rows of the boxes in shared memory
  int a_bytes, b_bytes, stages, ring_bytes;            // set by wgrad_rows_ring
  int splits;
  float* partial;                    // one float32 slab per slice (wgrad_slab.cuh)
  long long partial_elems;           // its extent (checked in the range-checked build)
  int diag_c, diag_k;                // merged groups of diag_k filters x diag_c channels: only their blocks are stored; 0: everything
  int taps_total;
  ItemWalk walk;                 // set by the launcher
  int* status;
  long long wait_clocks;             // bound of every device-side wait, in SM clocks
};
bool wgrad_rows_ring(RowsWgradParams* p, int dtype);      // false: two stages do not fit
cudaError_t launch_wgrad_rows(const RowsWgradParams& p, int dtype, int num_sms, cudaStream_t s);

// ---- strided gradInputs with few channels: parity classes merged into channels ---------------
// src[u][cls] = filter tap (i * kW + j, correlation coordinates) that class `cls` applies at the
// merged offset u, or -1 when the class has no tap there.
constexpr int kMaxParityClasses = 16;
struct MergedTapTable {
  int16_t src[kMaxTaps][kMaxParityClasses];
};
// dst[u][cls * C + c][kf] (`rows` rows per offset, the ones past ncls * C zero; row length ldw, zero
// padded) = w[kf][c][tap src[u][cls]] (flipped storage position when flip), zero where src is -1.
cudaError_t launch_pack_filters_merged(const void* w, void* dst, int K, int C, int kH, int kW, int flip,
                                       const MergedTapTable& tb, int nu, int ncls, int rows, int ldw,
                                       int dtype, cudaStream_t s);
// dx[n][c][h][w] (or channels-last with Cp channels, pad channels zeroed) =
// tmp[n][h / sH][w / sW][((h % sH) * sW + w % sW) * C + c], tmp channels-last with Ct channels.
cudaError_t launch_depth_to_space(const void* tmp, void* dx, int N, int C, int H, int W, int sH, int sW,
                                  int Ct, int Cp, int nhwc, int dtype, cudaStream_t s);

// ---- layout kernels (layout.cu) ---------------------------------------------------------
// in[b][r][s] (row length ld_in) -> out[b][s][r] (row length ld_out, zero filled past R).
cudaError_t launch_transpose(const void* in, void* out, int B, int R, int S, int ld_in,
                             int ld_out, int dtype, cudaStream_t s);
// Filter packing; mode 0: forward (rows = filters, cols = channels), mode 1: input gradient (rows = channels, cols = filters).
// dst[(tap*groups+g)][rows][ldc].  Cg: channels per (merged) group; merge: how many of the bank's own groups make one.
struct PackJob {
  const void* src;
  void* dst;
  int K, Cg, groups, ldc;
  int gx, gy, first_block;             // blocks along channels and filters, first one in a batch
  uint16_t taps, merge, pieces;        // pieces: 16 bytes each, of a filter's run in a patch
  uint8_t flip, mode, log_k, log_c;    // filters and channels of a patch
};
inline PackJob pack_job(const void* w, void* dst, int K, int Cg, int taps, int groups, int flip, int mode, int ldc, int merge = 1) {
  PackJob q = {};
  q.src = w; q.dst = dst;
  q.K = K; q.Cg = Cg; q.groups = groups; q.ldc = ldc;
  q.taps = static_cast<uint16_t>(taps); q.merge = static_cast<uint16_t>(merge);
  q.flip = flip != 0; q.mode = static_cast<uint8_t>(mode);
  return q;
}
cudaError_t launch_pack_filters(PackJob q, int dtype, cudaStream_t s);
// Many filter banks packed by one launch (b200conv_prepack): plan_pack() gives the blocks that a job takes.
constexpr int kPackBatchJobs = 56;             // 56 x 64 bytes stay below the 4 KB kernel-parameter limit
struct PackBatch {
  PackJob jobs[kPackBatchJobs];
  int njobs;
};
static_assert(sizeof(PackBatch) <= 4096, "kernel parameters");
constexpr int kB200Sms = 148;                 // for how finely work is cut that the hardware deals out
constexpr int kPackBlocks = 2 * kB200Sms;      // blocks of a launch that are worth smaller patches
int plan_pack(PackJob* q, int dtype, int least);
cudaError_t launch_pack_filters_batch(const PackBatch& b, int total_blocks, int dtype, cudaStream_t s);
// Row folding for layers with very few input channels (see layout.cu).
cudaError_t launch_pad_fold(const void* src, void* dst, int N, int C, int H, int W, int Cp, int Wp,
                            int pad_l, int nhwc_in, int dtype, cudaStream_t s);
cudaError_t launch_pack_filters_fold(const void* w, void* dst, int K, int C, int kH, int kW, int Cp,
                                     int ld, int flip, int dtype, cudaStream_t s);
// Space-to-depth form of stride-2 layers with very few channels (see layout.cu).
constexpr int kS2dChannels = 16;   // channels of one 2 x 2 pixel block: 4 x C <= 16
constexpr int kS2dPixels = 4;      // consecutive blocks one filter row may span
cudaError_t launch_pad_s2d(const void* src, void* dst, int N, int C, int H, int W, int Cp_in, int H2,
                           int Wq, int q0, int nhwc_in, int dtype, cudaStream_t s);
cudaError_t launch_pack_filters_s2d(const void* w, void* dst, int K, int C, int kH, int kW, int ntaps,
                                    int t0, int q0, int padH, int padW, int ld, int flip, int dtype,
                                    cudaStream_t s);
cudaError_t launch_wgrad_reduce_s2d(const float* partial, void* dw, int splits, int K, int C, int kH,
                                    int kW, int ntaps, int t0, int q0, int padH, int padW, int ld, int flip,
                                    int dtype, const WgradSum& sum, cudaStream_t s);
cudaError_t launch_wgrad_reduce_fold(const float* partial, void* dw, int splits, int K, int C, int kH,
                                     int kW, int Cp, int ld, int flip, int dtype, const WgradSum& sum, cudaStream_t s);
// Block-diagonal filters for merged groups (extract = 0) and the inverse for the gradient (1).
cudaError_t launch_merge_groups(const void* src, void* dst, int K, int Cg, int Kg, int m, int taps,
                                int extract, int dtype, cudaStream_t s);
// n values followed by zeros up to np values.
cudaError_t launch_pad_bias(const void* bias, void* dst, int n, int np, int dtype, cudaStream_t s);
cudaError_t launch_convert_bias(const void* bias, float* dst, int n, int dtype, cudaStream_t s);
cudaError_t launch_maxpool2x2(const void* x, void* y, int N, int C, int H, int W, int nhwc,
                              int Cp, int dtype, cudaStream_t s);
cudaError_t launch_maxpool2x2_grad(const void* x, const void* y, const void* gy, void* gx, int N, int C,
                                   int H, int W, int nhwc, int Cp, int dtype, cudaStream_t s);
cudaError_t launch_fill_l2(void* buf, size_t bytes, cudaStream_t s);

// ---- element-wise kernels on channels-last tensors and the per-channel sum (elementwise.cu) ----
enum : int { kEwAdd = 0, kEwMul, kEwSub, kEwRSub, kEwDiv, kEwRDiv, kEwMax, kEwAbs, kEwSgn, kEwNeg, kEwCount };
// out = op(a, b) over `elems` stored elements (a multiple of Cp); b_kind 0: tensor, 1: scalar s, 2: float32 vector
// of Cp values indexed by the stored channel, 3: unary.
cudaError_t launch_elementwise(const void* a, const void* b, const float* chan, void* out, long long elems, int C,
                               int Cp, int op, int b_kind, float s, int dtype, cudaStream_t st);
int channel_sum_blocks(long long pixels);          // rows of Cp floats the partial buffer needs
cudaError_t launch_channel_sum(const void* x, float* partial, void* out, long long pixels, int C, int Cp, int dtype,
                               cudaStream_t st);

// ---- bounded-wait self-test (selftest.cu): one CTA waits, with `limit`, on a barrier nobody arrives on
cudaError_t launch_wait_selftest(int* status, unsigned int* arrivals, int narrivals, long long limit, cudaStream_t s);

// ---- CUDA-core direct kernels (conv_direct.cu) ---------------------------------------------
cudaError_t launch_direct_fwd(const b200conv_desc& d, const void* x, const void* w,
                              const float* bias, void* y, int relu, const ConvEpilogue& epi, cudaStream_t s);
cudaError_t launch_direct_dgrad(const b200conv_desc& d, const void* w, const void* dy, void* dx,
                                cudaStream_t s);
cudaError_t launch_direct_wgrad(const b200conv_desc& d, const void* x, const void* dy, void* dw,
                                cudaStream_t s);

}  // namespace b200
