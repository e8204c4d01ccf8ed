// The tcgen05 kernels when a wait runs out (on a GPU): the tensor map that they load weights with brings half of each matrix, so
// that the load never completes, and the MMA lane waits a twentieth of a millisecond for it instead of a second.  Rows and map
// entries land as ever, no copy is under way when the kernel leaves.  Then the output is as it was, the run says that it
// gave up, and the launch behind it is right.  Exit status 0 if all of that holds.
#include <cstdio>
#include <cstring>
#include <vector>
#include "../../fgms_b200/csrc/umma_osfwd.cuh"
using namespace fgms;

#define CHECK(call)                                                                      \
  do {                                                                                   \
    const cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess) { std::printf("%s: %s\n", #call, cudaGetErrorString(e_)); return 2; } \
  } while (0)

static unsigned long long problems() {
  unsigned long long v = 0, z = 0;
  cudaMemcpyFromSymbol(&v, g_device_problems, sizeof(v));
  cudaMemcpyToSymbol(g_device_problems, &z, sizeof(z));
  return v;
}

// three launches on the same data, the second one with weights that do not arrive
template <typename Kernel, typename Params, typename Config>
static int check(const char* name, Kernel kernel, Params p, Config cfg, int grid, int threads, int max_smem, bool f16, bool mn_major, size_t out_bytes) {
  static std::atomic<int> granted[64];
  for (auto& g : granted) g = 0;
  if (ensure_smem(kernel, max_smem, granted)) return 1;
  const std::vector<unsigned char> before(out_bytes, 0x45);
  std::vector<unsigned char> out[3];
  unsigned long long said[3];
  for (int run = 0; run < 3; ++run) {
    const bool half = run == 1;
    CUtensorMap map;
    if (weight_tensor_map(&map, p.weights, half ? 2 * p.k_vol : p.k_vol, half ? p.c_in / 2 : p.c_in, p.c_out, f16, mn_major)) return 1;
    cfg.w_limit = half ? 100000 : umma::WAIT_LIMIT_CYCLES;
    CHECK(cudaMemcpy(p.dst, before.data(), out_bytes, cudaMemcpyHostToDevice));
    problems();
    CHECK(launch_pdl(kernel, grid, threads, (size_t)cfg.smem, nullptr, p, cfg, map));
    CHECK(cudaDeviceSynchronize());
    said[run] = problems();
    out[run].resize(out_bytes);
    CHECK(cudaMemcpy(out[run].data(), p.dst, out_bytes, cudaMemcpyDeviceToHost));
  }
  const bool ok = said[0] == 0 && said[1] > 0 && said[2] == 0 && out[0] != before && out[1] == before && out[2] == out[0];
  std::printf("%s: gave up %llu times, output %s: %s\n", name, said[1], out[1] == before ? "as it was" : "changed", ok ? "ok" : "FAILED");
  return ok ? 0 : 1;
}

// one offset, every row of both sides once: no element of the output is added to twice
template <bool F16>
static int forms(int c_in, int c_out, int sms, int max_smem) {
  const int es = F16 ? 2 : 4, n = sms * 128 * 14 + 37;  // more stages to a CTA than its ring holds
  const int tiles = (n + 127) / 128;
  std::vector<int> from(n), to(n), table((size_t)tiles * 128, -1);
  for (int i = 0; i < n; ++i) { from[i] = i; to[i] = n - 1 - i; table[n - 1 - i] = i; }
  // 1/4 in every element of rows and weights
  auto filled = [&](size_t elements) {
    std::vector<unsigned char> v(elements * es);
    for (size_t i = 0; i < elements; ++i) {
      if (F16) { const unsigned short h = 0x3400; std::memcpy(&v[2 * i], &h, 2); }
      else { const float f = 0.25f; std::memcpy(&v[4 * i], &f, 4); }
    }
    return v;
  };
  const int kpos_h[2] = {0, n};
  const std::vector<unsigned char> w = filled((size_t)c_in * c_out), x = filled((size_t)n * (c_in > c_out ? c_in : c_out));
  int *kpos, *imap, *omap, *nbr;
  void *weights, *src, *dst;
  CHECK(cudaMalloc(&kpos, 8)); CHECK(cudaMalloc(&imap, n * 4)); CHECK(cudaMalloc(&omap, n * 4)); CHECK(cudaMalloc(&nbr, table.size() * 4));
  CHECK(cudaMalloc(&weights, w.size())); CHECK(cudaMalloc(&src, x.size())); CHECK(cudaMalloc(&dst, x.size()));
  CHECK(cudaMemcpy(kpos, kpos_h, 8, cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(imap, from.data(), n * 4, cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(omap, to.data(), n * 4, cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(nbr, table.data(), table.size() * 4, cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(weights, w.data(), w.size(), cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(src, x.data(), x.size(), cudaMemcpyHostToDevice));
  const bool full = c_in * es % 128 == 0 && c_out * es % 128 == 0;
  int bad = 0;
  char name[96];
  for (int trans = 0; trans < 2; ++trans) {
    GmsParams p = {};
    p.weights = weights; p.src = src; p.dst = dst; p.kpos = kpos;
    p.gather_map = trans ? omap : imap; p.scatter_map = trans ? imap : omap;
    p.pairs = p.n_gather = p.n_scatter = n;
    p.k_dim = trans ? c_out : c_in; p.n_dim = trans ? c_in : c_out;
    p.c_in = c_in; p.c_out = c_out; p.k_vol = 1;
    G3Config cfg;
    if (!g3_plan(c_in, c_out, es, 1, max_smem, trans != 0, &cfg)) return 1;
    std::snprintf(name, sizeof(name), "%s %s %d -> %d", trans ? "input gradient" : "forward", F16 ? "fp16" : "tf32", c_in, c_out);
    auto kernel = trans ? (full ? umma_gms3_kernel<!F16, true, true> : umma_gms3_kernel<!F16, true, false>)
                        : (full ? umma_gms3_kernel<!F16, false, true> : umma_gms3_kernel<!F16, false, false>);
    bad |= check(name, kernel, p, cfg, sms, G3_THREADS, max_smem, F16, !trans, (size_t)n * p.n_dim * es);
  }
  OsParams p = {};
  p.weights = weights; p.src = src; p.dst = dst; p.nbr = nbr; p.nbr_stride = (long long)table.size();
  p.n_in = p.n_out = n; p.n_tiles = tiles;
  p.c_in = c_in; p.c_out = c_out; p.k_vol = 1;
  OsConfig cfg;
  if (!os_plan(c_in, c_out, es, max_smem, &cfg)) return 1;
  std::snprintf(name, sizeof(name), "output-stationary %s %d -> %d", F16 ? "fp16" : "tf32", c_in, c_out);
  bad |= check(name, umma_osfwd_kernel<!F16>, p, cfg, sms, OS_THREADS, max_smem, F16, true, (size_t)n * c_out * es);
  CHECK(cudaFree(kpos)); CHECK(cudaFree(imap)); CHECK(cudaFree(omap)); CHECK(cudaFree(nbr));
  CHECK(cudaFree(weights)); CHECK(cudaFree(src)); CHECK(cudaFree(dst));
  return bad;
}

// several pipelines: CTAs of up to `tiles` tiles and three offsets, the deal that the launcher makes
template <bool F16, int DEAL>
static int pipelines(int c_in, int c_out, int tiles, int sms, int max_smem) {
  const int es = F16 ? 2 : 4, k_vol = 3, n_tiles = sms * (tiles - 1) + sms / 2, n = n_tiles * 128 - 91;
  std::vector<int> table((size_t)k_vol * n_tiles * 128, -1);
  for (int k = 0; k < k_vol; ++k)
    for (int i = 0; i < n; ++i) table[(size_t)k * n_tiles * 128 + i] = (i + 1000 * k) % n;
  std::vector<unsigned char> v((size_t)n * (c_in > c_out ? c_in : c_out) * es);
  for (size_t i = 0; i < v.size(); i += es) {
    if (F16) { const unsigned short h = 0x3400; std::memcpy(&v[i], &h, 2); }
    else { const float f = 0.25f; std::memcpy(&v[i], &f, 4); }
  }
  const size_t w_bytes = (size_t)k_vol * c_in * c_out * es;
  if (w_bytes > v.size()) return 1;
  int* nbr;
  void *weights, *src, *dst;
  CHECK(cudaMalloc(&nbr, table.size() * 4)); CHECK(cudaMalloc(&weights, w_bytes)); CHECK(cudaMalloc(&src, v.size())); CHECK(cudaMalloc(&dst, v.size()));
  CHECK(cudaMemcpy(nbr, table.data(), table.size() * 4, cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(weights, v.data(), w_bytes, cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(src, v.data(), v.size(), cudaMemcpyHostToDevice));
  OsParams p = {};
  p.weights = weights; p.src = src; p.dst = dst; p.nbr = nbr; p.nbr_stride = (long long)n_tiles * 128;
  p.n_in = p.n_out = n; p.n_tiles = n_tiles; p.c_in = c_in; p.c_out = c_out; p.k_vol = k_vol;
  OsConfig cfg;
  if (!os_plan(c_in, c_out, es, max_smem, &cfg)) return 1;
  os_split(&cfg, tiles, k_vol, max_smem);
  char name[96];
  std::snprintf(name, sizeof(name), "output-stationary %s %d -> %d, %d pipelines by %s", F16 ? "fp16" : "tf32", c_in, c_out, cfg.n_pipe, cfg.by_offset ? "offset" : "tile");
  int bad = cfg.n_pipe < 2 || cfg.by_offset != (DEAL == OS_DEAL_OFFSETS);
  if (bad) std::printf("%s: not the deal that is to be checked\n", name);
  else bad = check(name, umma_osfwd_kernel<!F16, DEAL>, p, cfg, sms, OS_THREADS, max_smem, F16, true, (size_t)n * c_out * es);
  CHECK(cudaFree(nbr)); CHECK(cudaFree(weights)); CHECK(cudaFree(src)); CHECK(cudaFree(dst));
  return bad;
}

int main() {
  cudaDeviceProp prop;
  CHECK(cudaGetDeviceProperties(&prop, 0));
  const int sms = prop.multiProcessorCount, max_smem = (int)prop.sharedMemPerBlockOptin;
  return forms<true>(128, 128, sms, max_smem) | forms<false>(48, 80, sms, max_smem) | pipelines<true, OS_DEAL_TILES>(64, 64, 6, sms, max_smem) |
         pipelines<false, OS_DEAL_TILES>(48, 48, 3, sms, max_smem) | pipelines<true, OS_DEAL_OFFSETS>(128, 128, 1, sms, max_smem) |
         pipelines<false, OS_DEAL_OFFSETS>(48, 48, 1, sms, max_smem);
}
