// Host-side check of the shares of a backward (split_backward) over every channel pair, kernel volumes and maps from one pair to millions: a share leaves
// either pass a quarter of the SMs; wide layers have one; where the pairs of an offset do not fill a stage, a CTA of
// the weight gradient gets no more stages than where they do, as it takes each one's sums out; and fp32 sums over many pairs keep the share
// they have had.  Prints one line per violation; exit status 1 if there are any.
#include <cstdio>
#include <initializer_list>
#include "../../fgms_b200/csrc/backward_share.cuh"
using namespace fgms;

int main() {
  const int max_smem = 232448;  // B200: 227 KB per CTA
  int bad = 0, seen = 0;
  auto check = [&](bool ok, const char* what, long long pairs, int n_in, int n_out, int ci, int co, int kv, bool f16, int share) {
    ++seen;
    if (ok) return;
    if (bad++ < 20) std::printf("%s: %lld pairs, %d -> %d rows, %d -> %d, k_vol %d, %s: %d\n", what, pairs, n_in, n_out, ci, co, kv, f16 ? "fp16" : "tf32", share);
  };
  for (bool f16 : {true, false})
    for (int ci = 16; ci <= 256; ci += 16)
      for (int co = 16; co <= 256; co += 16) {
        const int es = f16 ? 2 : 4;
        G3Config g;
        W3Config w;
        const bool wide = g3_plan(ci, co, es, 27, max_smem, true, &g) && w3_plan(ci, co, es, 27, max_smem, &w) && !wh_supported(ci, co, f16);
        for (int sms : {148, 132, 16})
          for (int kv : {1, 8, 27, 125})
            for (long long pairs : {1ll, 127ll, 3000ll, 25506ll, 417600ll, 4570518ll, 2000000000ll})
              for (int rows : {1, 300, 20000, 480000}) {
                const int share = split_backward(pairs, rows, kv == 8 ? (rows + 3) / 4 : rows, ci, co, kv, f16, sms, max_smem);
                check(share == 0 || (share >= sms / 4 && share <= sms - sms / 4), "share", pairs, rows, rows, ci, co, kv, f16, share);
              }
        if (!wide) continue;
        // wide layers always have one: nine pairs a row, rows of twice and of half of L2, and a strided map of the same rows
        for (long long bytes : {252000000ll, 63000000ll}) {
          const int n = (int)(bytes / ((2 * ci + co) * es));
          const int subm = split_backward(9ll * n, n, n, ci, co, 27, f16, 148, max_smem), down = split_backward(n, n, n / 4, ci, co, 8, f16, 148, max_smem);
          check(subm > 0, "submanifold", 9ll * n, n, n, ci, co, 27, f16, subm);
          check(down > 0, "strided", n, n, n / 4, ci, co, 8, f16, down);
        }
        // 20 k voxels: 212 pairs an offset beside the centre, and the same pairs in a map without one
        const int few = split_backward(25506, 20000, 20000, ci, co, 27, f16, 148, max_smem), even = split_backward(25506, 20000, 20001, ci, co, 27, f16, 148, max_smem);
        if (ci * co >= 96 * 96) check(few >= even, "offsets of few pairs", 25506, 20000, 20000, ci, co, 27, f16, few);
      }
  // what some of them are: four and three stages a CTA; the one that fp32 sums over many pairs have had
  const int lidar = split_backward(25506, 20000, 20000, 256, 128, 27, true, 148, max_smem), large = split_backward(1126332, 120000, 120000, 128, 128, 27, false, 148, max_smem);
  check(lidar >= 77, "LiDAR", 25506, 20000, 20000, 256, 128, 27, true, lidar);
  check(large == 49, "large", 1126332, 120000, 120000, 128, 128, 27, false, large);
  std::printf("%d shares, %d violations\n", seen, bad);
  return bad ? 1 : 0;
}
