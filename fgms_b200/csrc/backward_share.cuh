// How the two passes of a backward share the SMs.
#pragma once
#include "rows_gms.cuh"
#include "rows_wgrad.cuh"
#include "umma_gms3.cuh"
#include "umma_wgrad3.cuh"

namespace fgms {

constexpr long long LONG_SUMS = 1 << 19;  // pairs beyond which fp32 gradients keep their shares

// The share of wide fp32 gradients over many pairs.  A tensor-memory accumulator rounds every sum down a little, by how many pairs it takes: with any
// other share than the one it has had a gradient differs by 2.8e-11 a pair at most (128 -> 128 on 1.13 M pairs 3.7e-5, whether it has become more exact or less),
// and single-precision results stay the same to 2e-5.  So these keep the shares of passes timed by themselves, fitted to 300 to 0.44 M pairs, and with them a
// few per cent: 128 -> 128 on 1.13 M pairs 284 us, 242 with all SMs for each pass; on 2.2 M 732 / 636; 64 -> 64 on 4.6 M 758 / 660.
inline int split_long_sums(long long pairs, int rows, int c_in, int c_out, int k_vol, const G3Config& g, int sms, int max_smem) {
  const int es = 4, blocks = (c_in * es + 127) / 128;
  const double units = (double)pairs / 128 + 0.5 * k_vol, in = 0.5 * (g.kch + c_out * es / 128.0), out = 0.5 * (blocks + c_in * es / 128.0);
  const double c_d = 5.6 + 0.19 * in + 0.2 * out, u_d = 0.05 + 0.182 * in + 0.397 * out;
  const double few = k_vol > 8 && pairs < 4ll * rows ? 1.2 : 1.0;  // rows that come from memory rather than from L2
  int best = 0;
  double least = 1e30;
  for (int s = sms / 4; s <= sms - sms / 4; s += 2) {
    W3Config w;
    w3_plan(c_in, c_out, es, k_vol, max_smem, &w);
    w3_split(c_in, c_out, es, k_vol, pairs, s, max_smem, &w);
    const double c_w = 5.9 + (w.n_buf == 1 ? 3.01 : 1.02) * w.c_a * w.c_b * es / 32768;
    const double u_w = few * w.parts_a * w.parts_b * (0.264 + 0.025 * (w.pa + w.pbp) / w.pack + 0.336 * (128.0 / w.pb));
    const double d = c_d + u_d * units / (sms - s), v = c_w + u_w * units / s, end = d > v ? d : v;
    if (end < least) { least = end; best = s; }
  }
  return best;
}

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
// With the weight gradient on tcgen05 the model is fitted to the passes side by side: 850 backwards (maps of 97 to 480 k voxels and 300 to 4.6 M pairs, full,
// surface, LiDAR and scattered clouds, strided maps both ways; 16 to 256 channels) times 20 shares, a sixth of them kept back to check it.  It counts
//   * stages and tiles by the launch: below one each a pass gets no shorter;
//   * the sums' way out where a CTA goes on to another offset.  With hardly more pairs than the centre's (LiDAR, whose other pairs lie in few offsets) that is
//     every stage: 256 -> 128 on 25 k pairs of 20 k voxels 26.2 us without it, 16.3;
//   * rows that come from memory, where the operands fill a good part of L2 (`cold`): 128 -> 128 stride 2 on 200 k pairs 37.3 / 34.6.
// On average it ends 3.0 % above the best share (without the last two 4.8, with constants fitted to each pass by itself 7.7).  The
// input gradient, launched second, takes 1.5 to 5 us longer than by itself.  Of shares about as good the one nearest half of the SMs is taken (fp32: a little
// more, where several stages hold an offset's few pairs); in fp16, where every block rounds its sums, a larger one has to gain.  Slower than without those two by
// more than 2 %: fp16 128 -> 128 on 26 k pairs of a scattered cloud 10.6 / 11.1 us, 160 -> 160 on 1.13 M 193 / 197, 256 -> 256 on 418 k 105.9 / 108.1.
// Where the rows of a map of many pairs a row exceed L2, two passes at different rows drive each other's out of it, and all SMs for each pass are better than any share:
// fp16 128 -> 128 on 4.6 M pairs 751 / 657 us, 256 -> 256 on 1.13 M 334 / 310.  But with the blocks of all SMs rounding their sums the gradient would be a third less exact
// (3.75e-4 / 5.0e-4 against 64 bits), and fp32 ones keep theirs (above).
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
  if (!f16 && pairs > LONG_SUMS) return split_long_sums(pairs, n_in > n_out ? n_in : n_out, c_in, c_out, k_vol, g, sms, max_smem);
  auto least_of = [](double a, double b) { return a < b ? a : b; };
  const double moved = ((double)n_in * c_in * 2 + (double)n_out * c_out) * es;  // bytes of rows, both sides' and the input gradient's
  const int rows = n_in > n_out ? n_in : n_out;
  const bool uneven = k_vol > 8 && pairs < 1.6 * rows;  // hardly more pairs than the centre's, those of LiDAR in few of the other offsets
  // parts of the passes' rows that are met for the first time, as far as they come from memory then
  const double cold = least_of(1, moved / 32e6) / (pairs > 0 ? pairs : 1), new_in = least_of(n_in, pairs) * cold, new_out = least_of(n_out, pairs) * cold;
  // pairs of an offset that is not the centre of a submanifold map
  const bool centre = k_vol % 2 == 1 && k_vol > 1 && n_in == n_out && pairs > n_in;
  const double of_offset = centre ? (double)(pairs - n_in) / (k_vol - 1) : (double)pairs / k_vol;
  // 128-byte pieces of the two rows; a last one that is filled in part counts for half of the rest as well
  const double in = 0.5 * (g.kch + c_out * es / 128.0), out = 0.5 * (blocks + c_in * es / 128.0), tiles = (double)pairs / 128 + 0.5 * k_vol;
  const double c_d = 3.09 + 0.289 * in + 0.594 * out, u_d = 0.144 + (0.192 + 0.009 * new_out) * in + (0.413 + 0.122 * new_in) * out;
  const double middle = (f16 ? 0.5 : 0.545) * sms, less = 0.06 / sms, more = (f16 ? 0.5 : 0.06) / sms;
  double least = 1e30, c_w = 0, u_w = 0, stages = 0;
  W3Parts parts = {0, 0};
  for (int s = first; s <= last; s += 2) {
    const W3Parts of_s = w3_parts(c_in, c_out, es, k_vol, pairs, s);  // the weight gradient's plan depends on its share
    if (!(of_s == parts)) {
      parts = of_s;
      w3_plan(c_in, c_out, es, k_vol, max_smem, &w);
      w3_split(c_in, c_out, es, k_vol, pairs, s, max_smem, &w);
      const double of_128 = w.pb / 128.0, per_offset = of_offset / w.pb + 0.5;
      const double sums = (w.n_buf == 1 ? 2.7 : 0.927) * w.c_a * w.c_b * es / 32768;  // their way out
      stages = ((double)pairs / w.pb + 0.5 * k_vol) * w.parts_a * w.parts_b;
      c_w = 5.19 + sums;
      const double runs = 1 / (per_offset * per_offset);  // of a CTA in a stage
      u_w = 0.183 + of_128 * (0.202 + ((0.1 + 0.19 * new_in) * w.pa + (0.1 + 0.032 * new_out) * w.pbp) / w.pack) +
            sums * (uneven ? 19 * least_of(runs, 0.064) : 3.65 * least_of(runs, 1));
    }
    const double t_d = tiles / (sms - s), t_w = stages / s, d = c_d + u_d * (t_d > 1 ? t_d : 1), v = c_w + u_w * (t_w > 1 ? t_w : 1);
    const double end = (d > v ? d : v) * (s > middle ? 1 + more * (s - middle) : 1 + less * (middle - s));
    if (end < least) { least = end; best = s; }
  }
  return best;
}

}  // namespace fgms
