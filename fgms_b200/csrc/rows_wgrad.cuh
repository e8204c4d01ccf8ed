// Weight gradient for short tf32 rows: every warp gathers both operands straight into registers.  (fp16 rows:
// rows_wgrad16.cuh.)
//
//   dw[k] (c_in x c_out) += sum over the pairs j of offset k of feats[in_map[j]]^T (x) out_grad[out_map[j]]
//
// The pair index is the contraction index of the product.  A warp-level MMA wants, in the lane (g, t) = (lane / 4,
// lane % 4), a few channels of a few pairs; which channel is row m of the product, and in which order the pairs are
// summed, is free.  So lane (g, t) loads the g-th eighth of the rows of pairs t, t + 4 of 8 with one or two vector loads
// each; eight lanes cover a row, a warp-wide load covers four consecutive pairs, and the loaded registers are the operands
// as they are.  Nothing passes through shared memory but the final sum of the block's warps; the tcgen05 form
// (umma_wgrad3.cuh) stages both in shared memory and is bound by the copy instructions.
//
// One block per SM takes a share of the pairs, its warps take the share's tiles of 16 in turn, and the block adds up its
// warps' fp32 sums when the offset changes.
#pragma once
#include "common.cuh"
#include "rows_gms.cuh"  // rw_mma, rw_max_regs
#include "umma.cuh"

namespace fgms {

// A row in the eight lanes that share it, in units of 16 channels.  A unit is two channels per lane, a register each.  A
// row of U units is loaded in pieces of 16 or 8 bytes per lane.
template <int U>
struct WgRow {
  static constexpr int REGS = 2 * U;  // registers per row and lane
  static constexpr int N16 = REGS / 4, N8 = (REGS % 4) / 2;
  static constexpr uint32_t BYTES = U * 64;
  // first channel of unit u in lane g, and the channels a lane holds side by side from there (2 per unit in a piece)
  __device__ static __forceinline__ int channel(int u, int g) {
    const int r = 2 * u;  // register of the unit
    if (r < 4 * N16) { const int q = r / 4; return q * 32 + g * 4 + r % 4; }
    return N16 * 32 + g * 2;
  }
  __device__ static __forceinline__ void load(const uint8_t* row, int g, uint32_t* v) {
#pragma unroll
    for (int q = 0; q < N16; ++q) rw_ld16(row + q * 128 + g * 16, v + 4 * q);
    if (N8) rw_ld8(row + N16 * 128 + g * 8, v + 4 * N16);
  }
};

template <int MU, int NU, int WARPS>
__global__ void __maxnreg__(rw_max_regs(WARPS * 32, true)) rows_wgrad_kernel(WgradParams p, bool spread) {
  using A = WgRow<MU>;
  using B = WgRow<NU>;
  constexpr int NT = 2 * NU, SUMS = MU * 4 * NT;  // n-tiles of 8 columns; accumulators per lane
  extern __shared__ float wg_smem[];               // [WARPS][SUMS][32], then the tile table
  int* tile_start = reinterpret_cast<int*>(wg_smem + WARPS * SUMS * 32);
  int* kpos_s = tile_start + p.k_vol + 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int n_seg = p.k_vol + 1;

  umma::griddep_wait();
  umma::griddep_launch_dependents();
  build_tile_table(16, p.kpos, p.pairs, p.k_vol, 0, kpos_s, tile_start);
  // Tiles by turns; spread (see Turns) when the rows exceed what L2 holds: with consecutive parts 61 MB of rows on either
  // side were read 5.6 times over (683 MB).
  const int total = tile_start[n_seg], share = (total + gridDim.x - 1) / gridDim.x;
  int t0 = min(total, (int)blockIdx.x * share);
  const int t1 = min(total, t0 + share);
  const uint8_t* feats = static_cast<const uint8_t*>(p.feats);
  const uint8_t* og = static_cast<const uint8_t*>(p.out_grad);

  while (t0 < t1) {
    // this block's turns inside one offset; warp w takes tiles w, w + WARPS, ... of them
    const int seg = find_segment(tile_start, n_seg, t0);
    const int run = min(t1, tile_start[seg + 1]) - t0;
    const Turns turns(tile_start[seg], tile_start[seg + 1], share, (int)blockIdx.x, t0, spread);
    const int j_begin = kpos_s[seg], j_end = kpos_s[seg + 1];
    t0 += run;
    float acc[MU][NT][4];
#pragma unroll
    for (int u = 0; u < MU; ++u)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[u][j][e] = 0.f;

    // Map entries of this lane's pairs t, t + 4, t + 8, t + 12 of a tile (-1 beyond the run).  The eight lanes of a row
    // read the same words: four broadcast loads, where handing the entries round by shuffles was 15 % slower.
    struct Entries { int i[4], o[4]; };
    auto load_entries = [&](int n, Entries& e) {
      const int j = (n < run ? j_begin + 16 * turns.tile(n) : j_end) + t4;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        e.i[q] = e.o[q] = -1;
        if (j + 4 * q < j_end) {
          e.i[q] = __ldg(p.in_map + j + 4 * q);
          e.o[q] = __ldg(p.out_map + j + 4 * q);
        }
      }
    };
    auto gather = [&](const Entries& e, uint32_t (&a)[4][A::REGS], uint32_t (&b)[4][B::REGS]) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool ok = (unsigned)e.i[q] < (unsigned)p.n_in && (unsigned)e.o[q] < (unsigned)p.n_out;
        if (!ok && g == 0 && (e.i[q] != -1 || e.o[q] != -1)) report_problem();  // pair skipped, counted once
#pragma unroll
        for (int r = 0; r < A::REGS; ++r) a[q][r] = 0u;
#pragma unroll
        for (int r = 0; r < B::REGS; ++r) b[q][r] = 0u;
        if (ok) {
          A::load(feats + (size_t)(unsigned)e.i[q] * A::BYTES, g, a[q]);
          B::load(og + (size_t)(unsigned)e.o[q] * B::BYTES, g, b[q]);
        }
      }
    };
    auto multiply = [&](const uint32_t (&a)[4][A::REGS], const uint32_t (&b)[4][B::REGS]) {
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int u = 0; u < MU; ++u) {
          const uint32_t fa[4] = {a[2 * s][2 * u], a[2 * s][2 * u + 1], a[2 * s + 1][2 * u], a[2 * s + 1][2 * u + 1]};
#pragma unroll
          for (int j = 0; j < NT; ++j) rw_mma(acc[u][j], fa, b[2 * s][j], b[2 * s + 1][j], true);
        }
    };
    if (warp < run) {
      uint32_t a0[4][A::REGS], b0[4][B::REGS], a1[4][A::REGS], b1[4][B::REGS];
      Entries e0, e1;
      load_entries(warp, e0);
      load_entries(warp + WARPS, e1);
      gather(e0, a0, b0);
      // two tiles per turn of the loop: the rows of one are on their way while the other is multiplied
      for (int n = warp;;) {
        load_entries(n + 2 * WARPS, e0);
        gather(e1, a1, b1);
        multiply(a0, b0);
        if ((n += WARPS) >= run) break;
        load_entries(n + 2 * WARPS, e1);
        gather(e0, a0, b0);
        multiply(a1, b1);
        if ((n += WARPS) >= run) break;
      }
      float* mine = wg_smem + warp * SUMS * 32 + lane;
#pragma unroll
      for (int u = 0; u < MU; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int j = 0; j < NT; ++j) mine[((u * 4 + e) * NT + j) * 32] = acc[u][j][e];
    }
    const int used = min(run, WARPS);
    __syncthreads();
    // element e = 2 h + c of n-tile j = 2 v + w: gradient row channel(u, g) + h, column channel(v, 2 t + c) + w.  The two
    // units of an even pair hold four consecutive columns, an odd last unit two: one vector red each.
    constexpr int GROUPS = (NU + 1) / 2;
    for (int item = threadIdx.x; item < MU * 4 * GROUPS * 32; item += WARPS * 32) {
      const int grp = (item >> 5) % GROUPS, ue = (item >> 5) / GROUPS, u = ue >> 2, e = ue & 3;
      const float* from = wg_smem + (ue * NT + grp * 4) * 32 + lane;
      const bool four = 2 * grp + 1 < NU;
      float s[4] = {0.f, 0.f, 0.f, 0.f};
      for (int w = 0; w < used; ++w)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < 2 || four) s[k] += from[(w * SUMS + k) * 32];
      const int row = A::channel(u, g) + (e >> 1), col = B::channel(2 * grp, 2 * t4 + (e & 1));
      const size_t at = ((size_t)seg * (MU * 16) + row) * (NU * 16) + col;
      if (four) {
        red_add_v4(p.dw + at, s[0], s[1], s[2], s[3]);
      } else {
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p.dw + at), "f"(s[0]), "f"(s[1]) : "memory");
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// Warps of the block: as many as the registers allow (sums, two tiles of rows, about fifty for the rest), 16 at most.
constexpr int rw_wgrad_regs(int mu, int nu) { return 8 * mu * nu + 16 * (mu + nu) + 50; }
constexpr int rw_wgrad_warps(int mu, int nu) {
  const int regs = (rw_wgrad_regs(mu, nu) + 7) / 8 * 8, fit = 65536 / (32 * regs) / 4 * 4;
  return fit > 16 ? 16 : fit;
}
// Shapes this kernel takes: multiples of 16 up to 64 channels on both sides whose sums and rows fit 255 registers.
inline bool rw_wgrad_supported(int c_in, int c_out) {
  if (c_in % 16 || c_out % 16 || c_in < 16 || c_out < 16 || c_in > 64 || c_out > 64) return false;
  return rw_wgrad_regs(c_in / 16, c_out / 16) <= 248;
}

template <int MU, int NU>
inline int rw_wgrad_launch_as(const WgradParams& p, cudaStream_t st, int sms, int max_smem) {
  if constexpr (rw_wgrad_regs(MU, NU) > 248) {
    return 1;
  } else {
    constexpr int WARPS = rw_wgrad_warps(MU, NU);
    auto kernel = rows_wgrad_kernel<MU, NU, WARPS>;
    const size_t smem = (size_t)WARPS * MU * 8 * NU * 128 + (size_t)(2 * p.k_vol + 3) * sizeof(int);
    if (smem > (size_t)max_smem) return 1;
    static std::atomic<int> granted[64];
    if (int rc = ensure_smem(kernel, max_smem, granted)) return rc;
    const long long tiles = (long long)p.pairs / 16 + p.k_vol + 1;
    const bool spread = spread_tiles((size_t)p.n_in * MU * 64 + (size_t)p.n_out * NU * 64);
    return launch_pdl(kernel, (int)(tiles < sms ? tiles : sms), WARPS * 32, smem, st, p, spread) == cudaSuccess ? 0 : -1;
  }
}
template <int MU>
inline int rw_wgrad_launch_n(const WgradParams& p, cudaStream_t st, int sms, int max_smem) {
  switch (p.c_out / 16) {
    case 1: return rw_wgrad_launch_as<MU, 1>(p, st, sms, max_smem);
    case 2: return rw_wgrad_launch_as<MU, 2>(p, st, sms, max_smem);
    case 3: return rw_wgrad_launch_as<MU, 3>(p, st, sms, max_smem);
    case 4: return rw_wgrad_launch_as<MU, 4>(p, st, sms, max_smem);
  }
  return 1;
}
// 0 launched, 1 not a shape of this kernel or a pointer is not 16-byte aligned, < 0 CUDA error
inline int launch_rows_wgrad(const WgradParams& p, cudaStream_t st, int sms, int max_smem) {
  if (!rw_wgrad_supported(p.c_in, p.c_out)) return 1;
  if ((long long)p.pairs > 0x7fffffffll - 65536) return 1;  // positions two turns past the end stay in an int
  if ((reinterpret_cast<uintptr_t>(p.feats) | reinterpret_cast<uintptr_t>(p.out_grad) | reinterpret_cast<uintptr_t>(p.dw)) & 15) return 1;
  switch (p.c_in / 16) {
    case 1: return rw_wgrad_launch_n<1>(p, st, sms, max_smem);
    case 2: return rw_wgrad_launch_n<2>(p, st, sms, max_smem);
    case 3: return rw_wgrad_launch_n<3>(p, st, sms, max_smem);
    case 4: return rw_wgrad_launch_n<4>(p, st, sms, max_smem);
  }
  return 1;
}

}  // namespace fgms
