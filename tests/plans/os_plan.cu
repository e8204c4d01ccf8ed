// Host-side check of the launch plan of the output-stationary forward over every channel pair: shared memory within the
// limit, no more producer warps than ring slots, accumulators within the 512 tensor-memory columns, and a plan for every shape
// that the scatter form has one for.  Prints one line per violation; exit status 1 if there are any.
#include <cstdio>
#include "../../fgms_b200/csrc/umma_osfwd.cuh"
using namespace fgms;

int main() {
  const int max_smem = 232448;  // B200: 227 KB per CTA
  int bad = 0, seen = 0;
  for (int es : {2, 4})
    for (int ci = 16; ci <= 256; ci += 16)
      for (int co = 16; co <= 256; co += 16) {
        G3Config g;
        OsConfig c;
        if (!g3_plan(ci, co, es, 27, max_smem, false, &g)) continue;
        ++seen;
        const bool ok = os_plan(ci, co, es, max_smem, &c) && c.smem <= max_smem && c.n_stage >= 2 && c.n_stage <= OS_MAX_STAGES &&
                        c.n_prod >= 1 && c.n_prod <= c.n_stage && c.n_prod <= OS_PROD_WARPS && c.group >= 1 && c.group <= OS_MAX_GROUP &&
                        c.group * c.n_acc <= 512 && c.n_acc >= co && c.group * c.kch <= 64 && c.w_bytes == ci * 128 * (c.n_acc * es / 128);
        if (!ok) { std::printf("es %d, %d -> %d\n", es, ci, co); ++bad; }
      }
  std::printf("%d shapes, %d violations\n", seen, bad);
  return bad ? 1 : 0;
}
