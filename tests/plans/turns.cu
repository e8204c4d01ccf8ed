// Host-side check of the order in which tiles are handed out by turns (Turns in common.cuh): for random lists of
// offsets, shares and numbers of workers every tile of every offset belongs to exactly one worker's turn, with and without
// `spread`.  Prints the first tile that does not; exit status 0: none.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>
#include "../../fgms_b200/csrc/common.cuh"

int main() {
  std::mt19937 rng(1);
  auto upto = [&](int n) { return (int)(rng() % (unsigned)(n + 1)); };
  long long tiles = 0;
  for (int round = 0; round < 20000; ++round) {
    const int segments = 1 + upto(8), top = upto(round % 3 ? 12 : 400), workers = 1 + upto(round % 2 ? 9 : 60);
    std::vector<int> start{0};
    for (int s = 0; s < segments; ++s) start.push_back(start.back() + (upto(3) ? upto(top) : 0));
    const int total = start.back(), share = (total + workers - 1) / workers;
    for (bool spread : {false, true}) {
      std::vector<int> seen(total, 0);
      for (int w = 0; w < workers; ++w) {
        int t = std::min(total, w * share);
        const int end = std::min(total, t + share);
        for (int seg = 0; t < end;) {
          while (t >= start[seg + 1]) ++seg;
          const int run = std::min(end, start[seg + 1]) - t;
          const fgms::Turns turns(start[seg], start[seg + 1], share, w, t, spread);
          for (int n = 0; n < run; ++n) {
            const int tile = turns.tile(n);
            if (tile < 0 || tile >= start[seg + 1] - start[seg] || seen[start[seg] + tile]++) {
              std::printf("round %d: tile %d of offset %d (%d tiles), worker %d of %d, share %d, spread %d\n", round, tile, seg,
                          start[seg + 1] - start[seg], w, workers, share, (int)spread);
              return 1;
            }
          }
          t += run;
        }
      }
      tiles += total;
      if (std::count(seen.begin(), seen.end(), 1) != total) { std::printf("round %d: a tile was left out\n", round); return 1; }
    }
  }
  std::printf("%lld tiles, each handed out once\n", tiles);
  return 0;
}
