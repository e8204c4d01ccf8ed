// Weight gradient for short rows: every warp gathers both operands straight into registers.
//
//   dw[k] (c_in x c_out, fp32 sums) += sum over the pairs j of offset k of feats[in_map[j]]^T (x) out_grad[out_map[j]]
//
// The pair index is the contraction index of the product.  A warp-level MMA wants, in the lane (g, t) = (lane / 4,
// lane % 4), a few channels of a few pairs; which channel is row m of the product, and in which order the pairs are
// summed, is free.  So lane (g, t) loads the g-th eighth of the rows of pairs t, t + 4, t + 8, t + 12 of a tile of 16
// (tf32: t, t + 4 of 8) with one or two vector loads each; eight lanes cover a row, a warp-wide load covers four
// consecutive pairs.  In fp16 two pairs' values of a channel are put side by side with one byte permutation per register;
// in tf32 the loaded registers are the operands.  Nothing passes through shared memory but the final sum of the block's
// warps, so the kernel runs at the rate of the two gathers; the tcgen05 form (umma_wgrad3.cuh) stages both in shared
// memory and was bound by the copy instructions (334 us on 9.1 M pairs of 32 -> 32 fp16, where two gathers of the same
// rows alone take about 110 us).
//
// One block per SM takes a share of the pairs, its warps take the share's tiles of 16 in turn, and the block adds up its
// warps' fp32 sums when the offset changes.  Where those sums go straight into an fp16 gradient every block's is rounded,
// and the pairs are shared out in units of 256 of one offset, the stages of the tcgen05 form, so that an offset of up to
// 256 pairs is rounded once.  Shares cut by single tiles split such an offset among up to six blocks: relative error of
// the gradient (32 -> 32, 27 offsets) 4.3e-4 against 2.1e-4 now for 80 pairs each, 4.7e-4 against 3.6e-4 for 1300,
// 4.7e-4 both for 35 000; the block's warps share a unit's tiles, so that costs little: 3.0 against 3.4 us, 5.4 / 4.7, 19.4 / 19.6.
#pragma once
#include "common.cuh"
#include "rows_gms.cuh"  // rw_mma, rw_max_regs
#include "umma.cuh"

namespace fgms {

// A row in the eight lanes that share it, in units of 16 channels.  A unit is two channels per lane: one register in
// fp16, two in tf32.  A row of U units is loaded in pieces of 16, 8 or 4 bytes per lane.
template <bool TF32, int U>
struct WgRow {
  static constexpr int RPU = TF32 ? 2 : 1;             // registers per unit
  static constexpr int REGS = U * RPU;                  // registers per row and lane
  static constexpr int N16 = REGS / 4, N8 = (REGS % 4) / 2, N4 = REGS % 2;
  static constexpr uint32_t BYTES = U * 16 * (TF32 ? 4 : 2);
  // first channel of unit u in lane g, and the channels a lane holds side by side from there (2 per unit in a piece)
  __device__ static __forceinline__ int channel(int u, int g) {
    const int r = u * RPU;  // register of the unit
    if (r < 4 * N16) { const int q = r / 4; return q * (64 / RPU) + g * (8 / RPU) + (r % 4) / RPU * 2; }
    const int base = N16 * (64 / RPU);
    if (N8 && r < 4 * N16 + 2) return base + g * (4 / RPU) + (r - 4 * N16) / RPU * 2;
    return base + N8 * (32 / RPU) + g * 2;
  }
  __device__ static __forceinline__ void load(const uint8_t* row, int g, uint32_t* v) {
#pragma unroll
    for (int q = 0; q < N16; ++q) rw_ld16(row + q * 128 + g * 16, v + 4 * q);
    if (N8) rw_ld8(row + N16 * 128 + g * 8, v + 4 * N16);
    if (N4) asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v[REGS - 1]) : "l"(row + N16 * 128 + N8 * 64 + g * 4));
  }
};

constexpr int WG_F16_UNIT = 4;  // log2 of a unit's tiles where block sums are rounded to fp16; single tiles elsewhere

template <bool TF32, int MU, int NU, int WARPS>
__global__ void __maxnreg__(rw_max_regs(WARPS * 32, true)) rows_wgrad_kernel(WgradParams p, bool spread) {
  static_assert(WARPS <= 1 << WG_F16_UNIT, "a full unit has a tile for every warp");
  using A = WgRow<TF32, MU>;
  using B = WgRow<TF32, NU>;
  constexpr int NT = 2 * NU, SUMS = MU * 4 * NT;  // n-tiles of 8 columns; accumulators per lane
  extern __shared__ float wg_smem[];               // [WARPS][SUMS][32], then the tile table
  int* tile_start = reinterpret_cast<int*>(wg_smem + WARPS * SUMS * 32);
  int* kpos_s = tile_start + p.k_vol + 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int n_seg = p.k_vol + 1;

  umma::griddep_wait();
  umma::griddep_launch_dependents();
  const int unit = !TF32 && p.dw_f16 != nullptr ? WG_F16_UNIT : 0;
  build_tile_table(16 << unit, p.kpos, p.pairs, p.k_vol, 0, kpos_s, tile_start);
  // Units by turns; spread (see Turns) when the rows exceed what L2 holds: with consecutive parts 61 MB of rows on either
  // side were read 5.6 times over (683 MB).
  const int total = tile_start[n_seg], share = (total + gridDim.x - 1) / gridDim.x;
  int t0 = min(total, (int)blockIdx.x * share);
  const int t1 = min(total, t0 + share);
  const uint8_t* feats = static_cast<const uint8_t*>(p.feats);
  const uint8_t* og = static_cast<const uint8_t*>(p.out_grad);

  while (t0 < t1) {
    // this block's turns inside one offset; warp w takes tiles w, w + WARPS, ... of their units
    const int seg = find_segment(tile_start, n_seg, t0);
    const int units = min(t1, tile_start[seg + 1]) - t0;
    const Turns turns(tile_start[seg], tile_start[seg + 1], share, (int)blockIdx.x, t0, spread);
    const int j_begin = kpos_s[seg], j_end = kpos_s[seg + 1];
    // a single unit may be the offset's last, partly filled one; of several at least one is full
    const int run = units > 1 ? units << unit : min(1 << unit, (j_end - j_begin + 15) / 16 - (turns.tile(0) << unit));
    t0 += units;
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
      const int j = (n < run ? j_begin + 16 * ((turns.tile(n >> unit) << unit) + (n & ((1 << unit) - 1))) : j_end) + t4;
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
      if constexpr (TF32) {
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int u = 0; u < MU; ++u) {
            const uint32_t fa[4] = {a[2 * s][2 * u], a[2 * s][2 * u + 1], a[2 * s + 1][2 * u], a[2 * s + 1][2 * u + 1]};
#pragma unroll
            for (int j = 0; j < NT; ++j) rw_mma(acc[u][j], fa, b[2 * s][j], b[2 * s + 1][j], true);
          }
      } else {
        uint32_t fb[NT][2];
#pragma unroll
        for (int v = 0; v < NU; ++v)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            fb[2 * v][h] = __byte_perm(b[2 * h][v], b[2 * h + 1][v], 0x5410);
            fb[2 * v + 1][h] = __byte_perm(b[2 * h][v], b[2 * h + 1][v], 0x7632);
          }
#pragma unroll
        for (int u = 0; u < MU; ++u) {
          const uint32_t fa[4] = {__byte_perm(a[0][u], a[1][u], 0x5410), __byte_perm(a[0][u], a[1][u], 0x7632),
                                  __byte_perm(a[2][u], a[3][u], 0x5410), __byte_perm(a[2][u], a[3][u], 0x7632)};
#pragma unroll
          for (int j = 0; j < NT; ++j) rw_mma(acc[u][j], fa, fb[j][0], fb[j][1], false);
        }
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
      if (!TF32 && p.dw_f16 != nullptr) {
        if (four) red_add_h4(p.dw_f16 + at, pack_half2(s[0], s[1]), pack_half2(s[2], s[3]));
        else atomicAdd(reinterpret_cast<__half2*>(p.dw_f16 + at), __floats2half2_rn(s[0], s[1]));
      } else if (four) {
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
constexpr int rw_wgrad_regs(bool tf32, int mu, int nu) { return 8 * mu * nu + 8 * (mu + nu) * (tf32 ? 2 : 1) + 50; }
constexpr int rw_wgrad_warps(bool tf32, int mu, int nu) {
  const int regs = (rw_wgrad_regs(tf32, mu, nu) + 7) / 8 * 8, fit = 65536 / (32 * regs) / 4 * 4;
  return fit > 16 ? 16 : fit;
}
// Shapes this kernel takes: multiples of 16 up to 64 channels on both sides whose sums and rows fit 255 registers.
inline bool rw_wgrad_supported(int c_in, int c_out, bool f16) {
  if (c_in % 16 || c_out % 16 || c_in < 16 || c_out < 16 || c_in > 64 || c_out > 64) return false;
  return rw_wgrad_regs(!f16, c_in / 16, c_out / 16) <= 248;
}

template <bool TF32, int MU, int NU>
inline int rw_wgrad_launch_as(const WgradParams& p, cudaStream_t st, int sms, int max_smem) {
  if constexpr (rw_wgrad_regs(TF32, MU, NU) > 248) {
    return 1;
  } else {
    constexpr int WARPS = rw_wgrad_warps(TF32, MU, NU);
    auto kernel = rows_wgrad_kernel<TF32, MU, NU, WARPS>;
    const size_t smem = (size_t)WARPS * MU * 8 * NU * 128 + (size_t)(2 * p.k_vol + 3) * sizeof(int);
    if (smem > (size_t)max_smem) return 1;
    static std::atomic<int> granted[64];
    if (int rc = ensure_smem(kernel, max_smem, granted)) return rc;
    const long long units = (long long)p.pairs / (p.dw_f16 != nullptr ? 16 << WG_F16_UNIT : 16) + p.k_vol + 1;
    const bool spread = spread_tiles((size_t)p.n_in * MU * 16 * (TF32 ? 4 : 2) + (size_t)p.n_out * NU * 16 * (TF32 ? 4 : 2));
    return launch_pdl(kernel, (int)(units < sms ? units : sms), WARPS * 32, smem, st, p, spread) == cudaSuccess ? 0 : -1;
  }
}
template <bool TF32, int MU>
inline int rw_wgrad_launch_n(const WgradParams& p, cudaStream_t st, int sms, int max_smem) {
  switch (p.c_out / 16) {
    case 1: return rw_wgrad_launch_as<TF32, MU, 1>(p, st, sms, max_smem);
    case 2: return rw_wgrad_launch_as<TF32, MU, 2>(p, st, sms, max_smem);
    case 3: return rw_wgrad_launch_as<TF32, MU, 3>(p, st, sms, max_smem);
    case 4: return rw_wgrad_launch_as<TF32, MU, 4>(p, st, sms, max_smem);
  }
  return 1;
}
template <bool TF32>
inline int rw_wgrad_launch(const WgradParams& p, cudaStream_t st, int sms, int max_smem) {
  switch (p.c_in / 16) {
    case 1: return rw_wgrad_launch_n<TF32, 1>(p, st, sms, max_smem);
    case 2: return rw_wgrad_launch_n<TF32, 2>(p, st, sms, max_smem);
    case 3: return rw_wgrad_launch_n<TF32, 3>(p, st, sms, max_smem);
    case 4: return rw_wgrad_launch_n<TF32, 4>(p, st, sms, max_smem);
  }
  return 1;
}

// 0 launched, 1 not a shape of this kernel or a pointer is not 16-byte aligned, < 0 CUDA error
inline int launch_rows_wgrad(const WgradParams& p, bool f16, cudaStream_t st, int sms, int max_smem) {
  if (!rw_wgrad_supported(p.c_in, p.c_out, f16)) return 1;
  if ((long long)p.pairs > 0x7fffffffll - 65536) return 1;  // positions two turns past the end stay in an int
  if ((reinterpret_cast<uintptr_t>(p.feats) | reinterpret_cast<uintptr_t>(p.out_grad) | reinterpret_cast<uintptr_t>(p.dw) |
       reinterpret_cast<uintptr_t>(p.dw_f16)) & 15) return 1;
  return f16 ? rw_wgrad_launch<false>(p, st, sms, max_smem) : rw_wgrad_launch<true>(p, st, sms, max_smem);
}

}  // namespace fgms
