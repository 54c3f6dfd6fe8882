// Which geometries the tensor-core kernels take, and how grouped layers are merged for them.  Plain integer
// rules without CUDA headers, so that a test can compile and enumerate them on any machine.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <initializer_list>

#include "../../include/b200conv.h"

namespace b200 {

constexpr int kMaxTaps = 64;
constexpr int kMaxViews = 9;

inline int round_up(int x, int m) { return (x + m - 1) / m * m; }
inline long long cdiv(long long a, long long b) { return (a + b - 1) / b; }
inline size_t elem_size(int dtype) { return dtype == B200CONV_F16 ? 2 : 4; }
// Channels-last tensors pad the channel count so that one pixel is a multiple of 16 bytes
// (tensor-map strides must be).
inline int pad_channels(int c, int dtype) { return round_up(c < 1 ? 1 : c, dtype == B200CONV_F16 ? 8 : 4); }

inline bool fits16(int v) { return v >= -32768 && v <= 32767; }

// Can the tensor-core kernels take this geometry?  (Otherwise the direct kernels do.)
inline bool umma_ok(const b200conv_desc& d) {
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  const size_t es = elem_size(d.dtype);
  if (d.N == 0 || d.C == 0 || d.K == 0) return false;
  if (d.kH * d.kW > kMaxTaps) return false;
  if (d.sH * d.sW > kMaxViews) return false;
  if (d.groups > 1 && ((Cg * es) % 16 || (Kg * es) % 16)) return false;
  if (Cg * es < 16 && d.groups > 1) return false;
  // tap offsets travel as 16-bit numbers; pixel coordinates as 32-bit ones
  const int reach_h = (d.kH - 1) * d.dilH + d.padH_l, reach_w = (d.kW - 1) * d.dilW + d.padW_l;
  if (!fits16(reach_h) || !fits16(reach_w)) return false;
  if (1LL * d.H + reach_h > (1 << 30) || 1LL * d.W + reach_w > (1 << 30)) return false;
  return true;
}

// `d` with m neighbouring groups as one (block-diagonal filters).
inline b200conv_desc merged_groups(const b200conv_desc& d, int m) {
  b200conv_desc r = d;
  r.groups = d.groups / m;
  return r;
}

// Grouped layers with fewer channels per group than one reduction block: how many neighbouring
// groups to merge into one; 1 = leave as is.
inline int merge_factor(const b200conv_desc& d) {
  if (d.groups <= 1 || d.C == 0 || d.K == 0) return 1;
  const int kBK = d.dtype == B200CONV_F16 ? 64 : 32;
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  int best = 1;
  for (int m = 2; m <= d.groups && Cg * m <= kBK && Kg * m <= 256; ++m)
    if (d.groups % m == 0) best = m;
  return best;
}

// The same for gradWeights, whose MMAs are 128 filters x channels: merging until both fill 128 leaves fewer,
// fuller MMAs and reads each operand row once instead of in 32-channel pieces (the off-diagonal blocks cost
// nothing extra: they fill rows and columns that would be empty).  32 groups of 8 -> 8 channels, 256 images of
// 28 x 28, float32: 590 us at one reduction block per group, 190 us at 128 channels.
// Of the divisors within these limits only those count whose merged layer the kernels take (whole 16-byte pieces
// per group, or one group left); where none does and the layer cannot run unmerged either, the limits of the other
// directions decide.
inline int merge_factor_wgrad(const b200conv_desc& d) {
  if (d.groups <= 1 || d.C == 0 || d.K == 0) return 1;
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  int best = 1;
  for (int m = 2; m <= d.groups && Cg * m <= 128 && Kg * m <= 128; ++m)
    if (d.groups % m == 0 && umma_ok(merged_groups(d, m))) best = m;
  return best > 1 || umma_ok(d) ? best : merge_factor(d);
}

// Tile of the columns kernel (conv_cols.cu) for taps that reach Eh rows and Ew columns beyond their first: the pitch that leaves the fewest
// accumulator rows to compute; at most `most_acc` accumulators of 128 rows, `n_cols` columns each; even 2: sides that pooling windows do not
// straddle.  `found` is false where no row fits a pitch, or no tile a box of 256 rows.
struct ColsTile {
  int wt, th, pitch, n_acc;
  bool found;
};
inline ColsTile cols_tile(int Wt, int Ht, int Eh, int Ew, int n_cols, int most_acc, int even) {
  ColsTile best = {0, 0, 0, 0, false};
  if (Eh > 256 - even) return best;
  long long least = 0;
  for (int pitch : {32, 16, 8})
    for (int n_acc = most_acc; n_acc >= 1; --n_acc) {
      const int widest = (pitch - Ew) / even * even, rows = 128 / pitch * n_acc, most = rows < 256 - Eh ? rows : 256 - Eh, tallest = most / even * even;
      if (widest < 1 || tallest < 1) continue;
      const int tw = static_cast<int>(cdiv(Wt, widest)), th_n = static_cast<int>(cdiv(Ht, tallest));
      // clocks of the MMAs: with two accumulators each has an issuer of its own; one alone waits for itself (71 against 117 clocks per 128 x 96)
      const long long work = 1LL * tw * th_n * n_acc * (n_cols > 128 ? 1 : n_acc == 2 ? 6 : 10);
      if (best.found && work >= least) continue;
      least = work;
      best = ColsTile{round_up(static_cast<int>(cdiv(Wt, tw)), even), round_up(static_cast<int>(cdiv(Ht, th_n)), even), pitch, n_acc, true};
    }
  return best;
}

}  // namespace b200
