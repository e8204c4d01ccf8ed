// How the two passes of a backward share the SMs.
#pragma once
#include "rows_gms.cuh"
#include "rows_wgrad.cuh"
#include "umma_gms3.cuh"
#include "umma_wgrad3.cuh"

namespace fgms {

constexpr double SHARED_ROWS = 126e6;  // bytes of rows that both passes of a backward find in L2

// SMs of the weight gradient where the two passes of a backward share the chip; 0: each has all of it.
//
// Side by side the passes overlap each other's fixed parts (launch, tile table, first rows; the sums' way out) and what they are
// bound by, reds of rows in the input gradient, instructions of the gathers in the weight gradient.  The weight gradient goes
// first, with one block per SM on its share; the input gradient's blocks find room on the others only.  Either pass takes about
// c + u * (128-pair units) / SMs microseconds; the share is the one at which the later one ends first.  Behind one another / started
// together but with all SMs each / with the share, in a row of launches: fp16 64 -> 64 0.93 M pairs 69.0 / 66.0 / 61.9 us, 137 k 19.8 / 18.9 / 15.2,
// 32 -> 32 9.1 M 254 / 252 / 237, 84 k 12.1 / 10.3 / 7.9; 128 -> 128 303 k 44.5 / 44.2 / 37.5.  A share a sixth off gives the gain away (64 -> 64
// 0.93 M pairs at 0.36 / 0.48 / 0.60 of the SMs 77.9 / 61.4 / 78.1).
//
// With the weight gradient on tcgen05 the model is fitted to the passes side by side: 770 backwards (34 maps of 300 to 4.6 M pairs, full, surface, LiDAR
// and scattered clouds, strided maps both ways; 16 to 256 channels) times 20 shares, a sixth of them kept back to check it.  It counts
//   * stages and tiles by the launch: below one each a pass gets no shorter;
//   * the sums' way out wherever a CTA goes on to another offset.  With offsets of few pairs (LiDAR, whose pairs lie in the centre and a few others) that is
//     every stage: 256 -> 128 on 25 k pairs of 20 k voxels 26.2 us without it, 17.8;
//   * rows that come from memory, where the operands fill a good part of L2 (`cold`): 128 -> 128 stride 2 on 200 k pairs 37.3 / 34.7.
// On average it ends 2.8 % above the best share (without the last two 5.0, with constants fitted to each pass by itself 7.7).  The
// input gradient, launched second, takes 1.5 to 5 us longer than by itself.  Of shares about as good the one nearest half of the SMs is taken; in fp16, where every
// block rounds its sums, a larger one has to gain.  Slower than without those two by more than 2 %: fp16 128 -> 128 on 26 k pairs of a scattered cloud 10.7 / 11.2 us, 160 -> 160
// on 1.13 M 195 / 200, 128 -> 64 transposed 25.7 / 26.3.
// No share where the fp32 rows of a map of many pairs a row exceed L2: side by side at different rows the passes drive each other's out of it.  128 -> 128 on
// 1.13 M pairs 284 / 242 us with / without, on 2.2 M 725 / 629, 64 -> 64 on 4.6 M 758 / 649; with rows of 108 MB 137 without, 133 with.  In fp16 it would be as good (128 ->
// 128 on 4.6 M 751 / 657), but with the blocks of all SMs rounding their sums the gradient would be a third less exact (3.75e-4 / 5.0e-4 against 64 bits).
// Rows of up to 64 channels on both sides keep the constants of each pass by itself, within
// 10 % of the best; 0.97 and 1.07 are the margins of "behind one another", and the terms for 48 channels, whose rows are copied
// with idle lanes, are fitted like the others.
inline int split_backward(long long pairs, int n_in, int n_out, int c_in, int c_out, int k_vol, bool f16, int sms, int max_smem) {
  G3Config g;
  W3Config w;
  const int es = f16 ? 2 : 4;
  if (!g3_plan(c_in, c_out, es, k_vol, max_smem, true, &g) || !w3_plan(c_in, c_out, es, k_vol, max_smem, &w) || sms < 16) return 0;
  const int first = sms / 4, last = sms - sms / 4, blocks = (c_in * es + 127) / 128;  // 128-byte blocks of an output row of the input gradient
  int best = 0;
  if (wh_supported(c_in, c_out, f16)) {
    const double both = c_in + c_out, area = (double)c_in * c_out, units = (double)pairs / 128 + k_vol;
    double c_d = 4, u_d = 0.1 + 0.1 * g.kch + 0.43 * blocks;
    if (rw_supported(c_out, c_in, f16)) c_d = 3.5, u_d = both * (f16 ? 0.0046 : 0.01);
    const double c_w = 5 + area / 2048, u_w = f16 ? 0.094 + 0.026 * area / 256 + 0.075 * ((c_in == 48) + (c_out == 48))
                                                  : 0.1 + 0.003 * both + 0.035 * area / 256 + 0.1 * ((c_in == 48) + (c_out == 48));
    // behind one another, where the input gradient on all SMs meets L2's rate of reds
    double least = 0.97 * (c_d + c_w - 2 + (1.07 * u_d + u_w) * units / sms);
    for (int s = first; s <= last; s += 2) {
      const double d = c_d + u_d * units / (sms - s), v = c_w + u_w * units / s, end = d > v ? d : v;
      if (end < least) { least = end; best = s; }
    }
    return best;
  }
  auto least_of = [](double a, double b) { return a < b ? a : b; };
  const double moved = ((double)n_in * c_in * 2 + (double)n_out * c_out) * es;  // bytes of rows, both sides' and the input gradient's
  const int rows = n_in > n_out ? n_in : n_out;
  if (!f16 && k_vol > 8 && pairs >= 4ll * rows && moved > SHARED_ROWS) return 0;
  // parts of the passes' rows that are met for the first time, as far as they come from memory then
  const double cold = least_of(1, moved / 32e6) / (pairs > 0 ? pairs : 1), new_in = least_of(n_in, pairs) * cold, new_out = least_of(n_out, pairs) * cold;
  // pairs of an offset that is not the centre of a submanifold map
  const bool centre = k_vol % 2 == 1 && k_vol > 1 && n_in == n_out && pairs > n_in;
  const double of_offset = centre ? (double)(pairs - n_in) / (k_vol - 1) : (double)pairs / k_vol;
  // 128-byte pieces of the two rows; a last one that is filled in part counts for half of the rest as well
  const double in = 0.5 * (g.kch + c_out * es / 128.0), out = 0.5 * (blocks + c_in * es / 128.0), tiles = (double)pairs / 128 + 0.5 * k_vol;
  const double c_d = 4.26 + 0.302 * in + 0.596 * out, u_d = 0.1465 + (0.186 + 0.013 * new_out) * in + (0.386 + 0.122 * new_in) * out;
  const double less = 0.03 / sms, more = (f16 ? 0.25 : 0.03) / sms;
  double least = 1e30, c_w = 0, u_w = 0, stages = 0;
  W3Parts parts = {0, 0};
  for (int s = first; s <= last; s += 2) {
    const W3Parts of_s = w3_parts(c_in, c_out, es, k_vol, pairs, s);  // the weight gradient's plan depends on its share
    if (!(of_s == parts)) {
      parts = of_s;
      w3_plan(c_in, c_out, es, k_vol, max_smem, &w);
      w3_split(c_in, c_out, es, k_vol, pairs, s, max_smem, &w);
      const double of_128 = w.pb / 128.0, per_offset = of_offset / w.pb + 0.5;
      const double sums = (w.n_buf == 1 ? 2.72 : 1.11) * w.c_a * w.c_b * es / 32768;  // their way out
      stages = ((double)pairs / w.pb + 0.5 * k_vol) * w.parts_a * w.parts_b;
      c_w = 5.97 + sums;
      u_w = 0.215 + of_128 * (0.212 + ((0.0764 + 0.2 * new_in) * w.pa + (0.0764 + 0.035 * new_out) * w.pbp) / w.pack) +
            11.4 * sums * least_of(1 / (per_offset * per_offset), 0.0932);
    }
    const double t_d = tiles / (sms - s), t_w = stages / s, d = c_d + u_d * (t_d > 1 ? t_d : 1), v = c_w + u_w * (t_w > 1 ? t_w : 1);
    const double end = (d > v ? d : v) * (2 * s > sms ? 1 + more * (2 * s - sms) : 1 + less * (sms - 2 * s));
    if (end < least) { least = end; best = s; }
  }
  return best;
}

}  // namespace fgms
