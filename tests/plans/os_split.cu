// Host-side check of the deal of the output-stationary forward (os_split) over every channel pair, CTAs of one to forty tiles and
// kernel volumes from 1 to 4096: what is launched fits shared and tensor memory and starts on the boundaries its copies need; no more
// producer warps than ring slots, weight buffers a multiple of the pipelines where offsets are dealt out; a pipeline of an offset
// deal has a weight buffer and the rings hold three rows or nine stages; a deal of tiles is not slower than one pipeline by the cycles the
// rule goes by.  Prints one line per violation; exit status 1 if there are any.
#include <cstdio>
#include <initializer_list>
#include "../../fgms_b200/csrc/umma_osfwd.cuh"
using namespace fgms;

int main() {
  const int max_smem = 232448;  // B200: 227 KB per CTA
  int bad = 0, seen = 0;
  auto most = [](int a, int b, int c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); };
  for (int es : {2, 4})
    for (int ci = 16; ci <= 256; ci += 16)
      for (int co = 16; co <= 256; co += 16)
        for (int kv : {1, 2, 3, 8, 27, 125, 4096})
          for (int tiles = 1; tiles <= 40; ++tiles) {
            G3Config g;
            OsConfig c;
            if (!g3_plan(ci, co, es, kv, max_smem, false, &g) || !os_plan(ci, co, es, max_smem, &c)) continue;
            const int one_slots = c.n_stage;
            os_split(&c, tiles, kv, max_smem);
            ++seen;
            const int n = c.n_pipe, slots = c.n_stage / n, parts = c.by_offset ? n : 1;
            bool ok = n >= 1 && n <= OS_MAX_PIPES && slots >= 2 && c.n_stage <= OS_MAX_STAGES && c.n_prod >= 1 && c.n_prod <= slots &&
                      c.n_prod * n <= OS_PROD_WARPS && c.n_wbuf >= 1 && c.n_wbuf <= 2 * OS_MAX_PIPES && c.group >= 1 && c.group * parts <= OS_MAX_GROUP &&
                      c.group * parts * c.n_acc <= 512 && c.group * c.kch <= 64 && c.w_bytes % 1024 == 0 && c.smem <= max_smem &&
                      c.smem == 1024 + OS_EPI_WARPS * 4096 + OS_SHARED_BYTES + c.n_wbuf * c.w_bytes + c.n_stage * G3_STAGE_BYTES;
            if (c.by_offset) {
              ok = ok && n <= kv && tiles <= c.group && c.n_wbuf % n == 0 && (slots * n >= 9 || slots * n >= 3 * c.kch);
            } else {
              ok = ok && c.group % n == 0;
              int turns = 0;
              for (int t = tiles; t > 0; t -= c.group) turns += ((t < c.group ? t : c.group) + n - 1) / n;
              const int rows = c.kch > 3 ? 3300 : 3100;
              ok = ok && turns * most(550, rows / slots, 360 * n) <= tiles * most(550, rows / one_slots, 360);
            }
            if (!ok) {
              if (bad < 20)
                std::printf("es %d, %d -> %d, k_vol %d, %d tiles: %d pipelines %s, %d slots, %d weight buffers, group %d\n", es, ci, co, kv, tiles, n,
                            c.by_offset ? "by offset" : "by tile", slots, c.n_wbuf, c.group);
              ++bad;
            }
          }
  std::printf("%d plans, %d violations\n", seen, bad);
  return bad ? 1 : 0;
}
