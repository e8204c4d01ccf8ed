// Weight gradient for short rows: every warp gathers tiles of 16 pairs into a ring of its own in shared memory.
//
//   dw[k] (c_in x c_out, fp32 sums) += sum over the pairs j of offset k of feats[in_map[j]]^T (x) out_grad[out_map[j]]
//
// The pair index is the contraction index of the product.  A tile's rows lie in shared memory as they are in memory, pair by
// pair, and both operands of mma.sync are read out of them: in fp16 by ldmatrix.trans; in tf32 lane (g, t) = (lane / 4,
// lane % 4) reads the g-th eighth of the rows of pairs t and t + 4 of eight, 16 bytes at a time, which channel is row m of the
// product being free.  Copies (16-byte cp.async), map entries (4-byte cp.async, a ring's length ahead of the rows) and products
// of a warp overlap without registers to hold them: a form that gathered straight into registers had two tiles a warp in
// flight, waited for its entries' registers and spent 220 instructions a tile.  In a row of launches, that form / this one:
// fp16 9.1 M pairs 32 -> 32 198 / 99.5 us (two gathers of these rows from L2 at 17 TB/s: 69), 0.93 M pairs 64 -> 64 43.7 / 31.7,
// 48 -> 48 41.1 / 29.3, 16 -> 16 16.7 / 12.1, 0.14 M 64 -> 64 13.3 / 11.1, 84 k 32 -> 32 7.5 / 6.5; tf32 4.6 M pairs 32 -> 32 189 / 104,
// 0.59 M 28.1 / 18.3, 0.2 M 32 -> 64 17.7 / 14.0, 55 k 32 -> 32 7.6 / 6.7, 0.37 M 48 -> 48 23.9 / 22.6.
//
// What bounds it now: with 8 warps at fp16 64 -> 64 (two a scheduler; 128 of a lane's registers are sums) the matrix
// instructions' fixed issue latency (3.3 of 6.7 cycles an instruction, tensor pipe 45 % busy); with 16 warps at 32 -> 32
// the same (2.7) and the entries' and rows' latency (1.4); on few pairs the sum of the warps' results at the end of an
// offset, about 2 us each time.  Two warps that share a tile and split a side of dW between them (twice the warps at
// 64 -> 64) were slower, 34 and 39 us.  The ring's length does not matter from three tiles on (four here; 8.1 M pairs in
// spread order want the fourth: 113 us with three); tf32 has room for two or three, and fewer warps with longer rings are slower
// (0.59 M 32 -> 32 with 8 / 12 / 16 warps 19.9 / 19.5 / 18.3).
//
// One block per SM takes a share of the pairs, its warps take the share's tiles of 16 in turn, and the block adds up its
// warps' fp32 sums when the offset changes.  Where those sums go straight into an fp16 gradient every block's is rounded,
// and the pairs are shared out in units of 256 of one offset, a tile for every warp, so that an offset of up to
// 256 pairs is rounded once.  Shares cut by single tiles split such an offset among up to six blocks: relative error of
// the gradient (32 -> 32, 27 offsets) 4.3e-4 against 2.1e-4 in units for 80 pairs each, 4.7e-4 against 3.6e-4 for 1300.
#pragma once
#include "common.cuh"
#include "rows_gms.cuh"  // rw_mma, rw_max_regs
#include "umma.cuh"

namespace fgms {

constexpr int WH_UNIT = 4;       // log2 of a unit's tiles where block sums are rounded to fp16; single tiles elsewhere
constexpr int WH_MAX_DEPTH = 4;  // tiles of a ring

// One operand's rows of a tile in shared memory, in units of 16 channels.
template <bool TF32, int U>
struct WhRows {
  static constexpr int CHUNKS = (TF32 ? 4 : 2) * U;      // of 16 bytes, of a row
  static constexpr uint32_t BYTES = CHUNKS * 16;         // of a row in global memory
  // Of a row in shared memory.  fp16: the chunks of the eight rows that an ldmatrix reads together lie in different banks: rows
  // of 1, 2 or 4 units exchange their chunks by row number, rows of 3 units are an odd number of chunks apart.  tf32: four
  // rows that are read together lie 8 (24) banks apart.
  static constexpr uint32_t LD = TF32 ? BYTES + 32 : U == 3 ? BYTES + 16 : BYTES;
  static constexpr uint32_t TILE = 16 * LD;
  // Lanes that copy a row, a chunk each; three rounds of four for twelve chunks (in sixteen lanes of which four do nothing
  // 0.37 M pairs tf32 48 -> 48 24.3 us, 22.6 this way, 0.59 M 33.8 / 30.1; but six chunks in rounds of two 23.0 us, 18.5 in eight lanes).
  static constexpr int LANES = CHUNKS == 6 ? 8 : CHUNKS == 12 ? 4 : CHUNKS, PARTS = CHUNKS > LANES ? CHUNKS / LANES : 1;
  static constexpr int ROUNDS = 16 * LANES / 32;  // turns through a tile's rows
  __device__ static __forceinline__ uint32_t at(int row, int chunk) {
    const int x = TF32 ? 0 : U == 4 ? row & 7 : U == 2 ? (row >> 1) & 3 : U == 1 ? (row >> 2) & 1 : 0;
    return (uint32_t)row * LD + (uint32_t)((chunk ^ x) << 4);
  }
  // fp16: chunk 2 u further on than the one at `addr`; rows without padding are aligned to their length
  __device__ static __forceinline__ uint32_t unit(uint32_t addr, int u) { return U == 3 ? addr + 32 * u : addr ^ (32 * u); }
  // tf32: a row in the eight lanes that share it, two channels (registers) a lane and unit, read 16 or 8 bytes at a time.  First
  // channel of unit u in lane g, and the channels a lane holds side by side from there (2 per unit in a piece):
  static constexpr int REGS = 2 * U, N16 = REGS / 4, N8 = REGS % 4 / 2;
  __device__ static __forceinline__ int channel(int u, int g) {
    const int r = 2 * u;  // register of the unit
    if (r < 4 * N16) return r / 4 * 32 + g * 4 + r % 4;
    return N16 * 32 + g * 2;
  }
  __device__ static __forceinline__ void load(uint32_t row, int g, uint32_t (&v)[REGS]) {
#pragma unroll
    for (int q = 0; q < N16; ++q)
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[4 * q]), "=r"(v[4 * q + 1]), "=r"(v[4 * q + 2]), "=r"(v[4 * q + 3]) : "r"(row + q * 128 + g * 16) : "memory");
    if constexpr (N8 > 0) asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v[REGS - 2]), "=r"(v[REGS - 1]) : "r"(row + N16 * 128 + g * 8) : "memory");
  }
  // this lane's chunk of every row of a tile, from src + lane's chunk; `on` says what rows there are, the others become zeros
  template <bool WHOLE>
  __device__ static __forceinline__ void copy(uint32_t slot, const uint8_t* src, int e, int first, unsigned on, int lane) {
    const int r0 = lane / LANES, c = lane % LANES;
#pragma unroll
    for (int i = 0; i < ROUNDS; ++i) {
      const int row = r0 + i * (32 / LANES), idx = __shfl_sync(0xffffffffu, e, first + row);
      if (LANES > CHUNKS && c >= CHUNKS) continue;
      const uint8_t* from = src + (WHOLE || ((on >> row) & 1) ? (size_t)(unsigned)idx * BYTES : 0);
#pragma unroll
      for (int k = 0; k < PARTS; ++k) {
        const uint32_t to = slot + at(row, c + k * LANES);
        if (WHOLE) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from + k * LANES * 16) : "memory");
        else umma::cp_async16(to, from + k * LANES * 16, (on >> row) & 1);
      }
    }
  }
};

__device__ __forceinline__ void wh_ldmatrix(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}

// A tile's products with W_k^T, added to the input gradient: what rows_gms_kernel does, with the rows in shared memory.
template <int MU, int NU>
__device__ __forceinline__ void wh_dgrad(uint32_t rows, uint32_t to_rows, int lane, const uint32_t (&wt)[NU][2 * MU][2], __half* in_grad) {
  using S = RowShape<false, NU, MU>;
  using B = WhRows<false, NU>;
  const int g = lane >> 2, t4 = lane & 3;
  int to[2];
  uint32_t a[2][S::AR];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    to[h] = umma::ld_shared_i32(to_rows + (g + 8 * h) * 4);
#pragma unroll
    for (int q = 0; q < S::KFULL; ++q)
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(a[h][4 * q]), "=r"(a[h][4 * q + 1]), "=r"(a[h][4 * q + 2]), "=r"(a[h][4 * q + 3])
                   : "r"(rows + B::at(g + 8 * h, 4 * q + t4)) : "memory");
    if constexpr (S::KHALF > 0)
      asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(a[h][4 * S::KFULL]), "=r"(a[h][4 * S::KFULL + 1])
                   : "r"(rows + B::at(g + 8 * h, 4 * S::KFULL + (t4 >> 1)) + (t4 & 1) * 8) : "memory");
  }
  auto piece = [&](int j_first, auto n_tiles, __half* base) {
    constexpr int N = decltype(n_tiles)::value;
    float c[N][4];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) c[i][k] = 0.f;
#pragma unroll
    for (int s = 0; s < S::KSTEPS; ++s) {
      const uint32_t frag[4] = {a[0][2 * s], a[1][2 * s], a[0][2 * s + 1], a[1][2 * s + 1]};
#pragma unroll
      for (int i = 0; i < N; ++i) rw_mma(c[i], frag, wt[s][j_first + i][0], wt[s][j_first + i][1], false);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (to[h] < 0) continue;
      __half* o = base + (size_t)(unsigned)to[h] * (MU * 16);
      if (N == 4)
        red_add_h8(o, pack_half2(c[0][2 * h], c[1][2 * h]), pack_half2(c[N - 2][2 * h], c[N - 1][2 * h]), pack_half2(c[0][2 * h + 1], c[1][2 * h + 1]),
                   pack_half2(c[N - 2][2 * h + 1], c[N - 1][2 * h + 1]));
      else red_add_h4(o, pack_half2(c[0][2 * h], c[1][2 * h]), pack_half2(c[0][2 * h + 1], c[1][2 * h + 1]));
    }
  };
#pragma unroll
  for (int q = 0; q < S::NFULL; ++q) piece(q * S::TPF, std::integral_constant<int, S::TPF>(), in_grad + q * 32 + t4 * 8);
  if constexpr (S::NHALF > 0) piece(S::NFULL * S::TPF, std::integral_constant<int, 2>(), in_grad + S::NFULL * 32 + t4 * 4);
}

// The input gradient of the same pairs: in_grad[in_map[j]] += out_grad[out_map[j]] . W_k^T.
struct RowsDgrad {
  const void* weights;
  __half* in_grad;
};

// DGRAD (fp16): both gradients of a backward.  Side by side, the two passes each gather every pair's row of the output gradient, and
// the L2 that serves their gathers and reds bounds them; here a tile's rows are copied once, and its products with W_k^T come from the
// copy in shared memory.  Backwards of 32 -> 32, us, two kernels side by side / this one with the clearing and rounding of its sums:
// 9.6 M pairs 248 / 208, 1.13 M 32.3 / 31.1; 16 -> 32 on 1.13 M 29.3 / 25.1.  All SMs work on the weight gradient then, and rounded to
// fp16 by each block, as those of its share were, it would be less exact (error against 64 bits, 1.13 M pairs: 5.0e-4, 4.0e-4 before),
// so the sums stay fp32 in a workspace (2.1e-4).  Clusters of two blocks that round once were no more than even with the share
// (4.0e-4; on 9.6 M pairs 4.0e-4 against 3.8e-4).
template <bool TF32, int MU, int NU, int WARPS, int DEPTH, bool DGRAD>
__global__ void __maxnreg__(rw_max_regs(WARPS * 32, true)) rows_wgrad_kernel(WgradParams p, bool spread, RowsDgrad dg) {
  static_assert(!(TF32 && DGRAD), "fp16 only");
  static_assert(WARPS <= 1 << WH_UNIT, "a full unit has a tile for every warp");
  static_assert(DEPTH >= 2, "a tile is filled while another is used");
  using A = WhRows<TF32, MU>;
  using B = WhRows<TF32, NU>;
  constexpr uint32_t STAGE = A::TILE + B::TILE, ENTRIES = 128;
  constexpr int NT = 2 * NU, SUMS = MU * 4 * NT;  // n-tiles of 8 columns; accumulators per lane
  constexpr uint32_t RINGS = WARPS * (DEPTH * STAGE + (DEPTH - 1) * ENTRIES + (DGRAD ? DEPTH * 64 : 0)), ALL_SUMS = WARPS * SUMS * 128;
  extern __shared__ __align__(128) uint8_t wh_smem[];  // the warps' rings, later [WARPS][SUMS][32] sums; then the tile table
  int* tile_start = reinterpret_cast<int*>(wh_smem + (RINGS > ALL_SUMS ? RINGS : ALL_SUMS));
  int* kpos_s = tile_start + p.k_vol + 2;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_seg = p.k_vol + 1;

  umma::griddep_begin(0, p.alone);
  const int unit = !TF32 && p.dw_f16 != nullptr ? WH_UNIT : 0;
  build_tile_table(16 << unit, p.kpos, p.pairs, p.k_vol, 0, kpos_s, tile_start, DGRAD ? 2 : 1);
  // Units by turns; spread (see Turns) when the rows exceed what L2 holds.
  const int total = tile_start[n_seg], share = (total + gridDim.x - 1) / gridDim.x;
  int t0 = min(total, (int)blockIdx.x * share);
  const int t1 = min(total, t0 + share);

  const uint32_t ring = umma::smem_u32(wh_smem) + warp * DEPTH * STAGE;
  const uint32_t entries = umma::smem_u32(wh_smem) + WARPS * DEPTH * STAGE + warp * (DEPTH - 1) * ENTRIES + lane * 4;
  // rows of the input gradient of a slot's pairs, -1: none
  const uint32_t to_rows = umma::smem_u32(wh_smem) + WARPS * (DEPTH * STAGE + (DEPTH - 1) * ENTRIES) + warp * DEPTH * 64;
  const uint8_t* feats = static_cast<const uint8_t*>(p.feats) + lane % A::LANES * 16;
  const uint8_t* og = static_cast<const uint8_t*>(p.out_grad) + lane % B::LANES * 16;
  // ldmatrix: lanes 0-7, 8-15, 16-23, 24-31 name the rows of the four 8 x 8 matrices
  const uint32_t a_off = A::at((lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1);
  const uint32_t b_off = B::at((lane & 7) + (((lane >> 3) & 1) << 3), lane >> 4);
  const int32_t* __restrict__ map = lane < 16 ? p.in_map : p.out_map;
  const unsigned n_rows = lane < 16 ? p.n_in : p.n_out;

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

    // position of this lane's map entry of tile n: lanes 0-15 the input rows of its pairs, lanes 16-31 the output rows
    auto entry_at = [&](int n) {
      return (n < run ? j_begin + 16 * ((turns.tile(n >> unit) << unit) + (n & ((1 << unit) - 1))) : j_end) + (lane & 15);
    };
    auto fetch_entry = [&](int n, uint32_t slot) {
      const int j = entry_at(n);
      if (j < j_end) umma::cp_async4(slot, map + j);
      else umma::st_shared_i32(slot, -1);
    };
    auto start = [&](int e, uint32_t at) {  // the rows of a tile's entries on their way
      const unsigned in = __ballot_sync(0xffffffffu, (unsigned)e < n_rows), ok = in & (in >> 16) & 0xffffu;
      const uint32_t slot = ring + at;
      if (DGRAD && lane < 16) umma::st_shared_i32(to_rows + at / STAGE * 64 + lane * 4, (ok >> lane) & 1 ? e : -1);
      if (ok == 0xffffu) {
        A::template copy<true>(slot, feats, e, 0, ok, lane);
        B::template copy<true>(slot + A::TILE, og, e, 16, ok, lane);
      } else {  // the offset's last tile, or entries outside the tensors
        const unsigned there = __ballot_sync(0xffffffffu, e != -1), bad = ((there | there >> 16) & ~ok) & 0xffffu;
        if ((bad >> lane) & 1) {  // pair skipped, counted once in each pass
          report_problem();
          if (DGRAD) report_problem();
        }
        A::template copy<false>(slot, feats, e, 0, ok, lane);
        B::template copy<false>(slot + A::TILE, og, e, 16, ok, lane);
      }
    };
    uint32_t wt[DGRAD ? NU : 1][2 * MU][2];  // W_k^T as the B operand
    if constexpr (DGRAD)
      if (warp < run) rw_load_b<false, true, NU, MU>(static_cast<const uint8_t*>(dg.weights) + (size_t)seg * p.c_in * p.c_out * 2, p.c_out, lane, wt);
    if (warp < run) {
      // group d of a warp's copies: the rows of its tile d and the entries of its tile d + DEPTH - 1
      int e[DEPTH - 1];
#pragma unroll
      for (int d = 0; d < DEPTH - 1; ++d) {
        const int j = entry_at(warp + d * WARPS);
        e[d] = j < j_end ? __ldg(map + j) : -1;
      }
#pragma unroll
      for (int d = 0; d < DEPTH - 1; ++d) {
        if (warp + d * WARPS < run) start(e[d], d * STAGE);
        fetch_entry(warp + (d + DEPTH - 1) * WARPS, entries + d * ENTRIES);
        umma::cp_async_commit();
      }
      uint32_t put = (DEPTH - 1) * STAGE, get = 0, ent = 0;
#pragma unroll 1
      for (int n = warp; n < run; n += WARPS) {
        umma::cp_async_wait<DEPTH - 2>();
        __syncwarp();  // the tile has landed for every lane, and every lane is done with the slot that is filled next
        auto next_tile = [&]() {
          if (n + (DEPTH - 1) * WARPS < run) {
            start(umma::ld_shared_i32(entries + ent), put);
            fetch_entry(n + 2 * (DEPTH - 1) * WARPS, entries + ent);
            ent = ent == (DEPTH - 2) * ENTRIES ? 0 : ent + ENTRIES;
            put = put == (DEPTH - 1) * STAGE ? 0 : put + STAGE;
          }
          umma::cp_async_commit();
        };
        // operands first: the next tile's copies are prepared while they come
        if constexpr (TF32) {
          const int g = lane >> 2, t = lane & 3;
          const uint32_t sa = ring + get + t * A::LD, sb = ring + get + A::TILE + t * B::LD;
#pragma unroll
          for (int s = 0; s < 2; ++s) {  // eight pairs: t and t + 4
            uint32_t a[2][A::REGS], b[2][B::REGS];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              A::load(sa + (8 * s + 4 * h) * A::LD, g, a[h]);
              B::load(sb + (8 * s + 4 * h) * B::LD, g, b[h]);
            }
            if (s == 0) next_tile();
#pragma unroll
            for (int u = 0; u < MU; ++u) {
              const uint32_t fa[4] = {a[0][2 * u], a[0][2 * u + 1], a[1][2 * u], a[1][2 * u + 1]};
#pragma unroll
              for (int j = 0; j < NT; ++j) rw_mma(acc[u][j], fa, b[0][j], b[1][j], true);
            }
          }
        } else {
          uint32_t a[MU][4], b[NU][4];
          const uint32_t sa = ring + get + a_off, sb = ring + get + A::TILE + b_off;
#pragma unroll
          for (int v = 0; v < NU; ++v) wh_ldmatrix(B::unit(sb, v), b[v]);
#pragma unroll
          for (int u = 0; u < MU; ++u) wh_ldmatrix(A::unit(sa, u), a[u]);
          next_tile();
#pragma unroll
          for (int u = 0; u < MU; ++u)
#pragma unroll
            for (int j = 0; j < NT; ++j) rw_mma(acc[u][j], a[u], b[j / 2][2 * (j & 1)], b[j / 2][2 * (j & 1) + 1], false);
          if constexpr (DGRAD) wh_dgrad<MU, NU>(ring + get + A::TILE, to_rows + get / STAGE * 64, lane, wt, dg.in_grad);
        }
        get = get == (DEPTH - 1) * STAGE ? 0 : get + STAGE;
      }
    }
    umma::cp_async_wait_all();
    __syncthreads();  // every warp is done with its ring
    if (warp < run) {
      float* mine = reinterpret_cast<float*>(wh_smem) + warp * SUMS * 32 + lane;
#pragma unroll
      for (int u = 0; u < MU; ++u)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) mine[((u * 4 + e) * NT + j) * 32] = acc[u][j][e];
    }
    const int used = min(run, WARPS);
    __syncthreads();
    if constexpr (TF32) {
      // element e = 2 h + c of n-tile j = 2 v + w: gradient row channel(u, g) + h, column channel(v, 2 t + c) + w.  The two
      // units of an even pair hold four consecutive columns, an odd last unit two: one vector red each.
      constexpr int GROUPS = (NU + 1) / 2;
      const int g = lane >> 2, t = lane & 3;
      for (int item = threadIdx.x; item < MU * 4 * GROUPS * 32; item += WARPS * 32) {
        const int grp = (item >> 5) % GROUPS, ue = (item >> 5) / GROUPS, u = ue >> 2, e = ue & 3;
        const float* from = reinterpret_cast<const float*>(wh_smem) + (ue * NT + grp * 4) * 32 + lane;
        const bool four = 2 * grp + 1 < NU;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        for (int w = 0; w < used; ++w)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k < 2 || four) s[k] += from[(w * SUMS + k) * 32];
        float* at = p.dw + ((size_t)seg * (MU * 16) + A::channel(u, g) + (e >> 1)) * (NU * 16) + B::channel(2 * grp, 2 * t + (e & 1));
        if (four) red_add_v4(at, s[0], s[1], s[2], s[3]);
        else asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(at), "f"(s[0]), "f"(s[1]) : "memory");
      }
    } else {
      // element e = 2 h + c of n-tile j in lane (g, t): gradient row 16 u + 8 h + g, column 8 j + 2 t + c.  Four lanes' two
      // elements are eight consecutive columns.
      for (int item = threadIdx.x; item < MU * 2 * NT * 8; item += WARPS * 32) {
        const int g = item & 7, j = (item >> 3) % NT, uh = (item >> 3) / NT;
        const float* from = reinterpret_cast<const float*>(wh_smem) + (uh * 2 * NT + j) * 32 + 4 * g;
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int w = 0; w < used; ++w) {
          const float4 x = *reinterpret_cast<const float4*>(from + w * SUMS * 32);
          const float4 y = *reinterpret_cast<const float4*>(from + w * SUMS * 32 + NT * 32);
          s[0] += x.x; s[1] += y.x; s[2] += x.y; s[3] += y.y; s[4] += x.z; s[5] += y.z; s[6] += x.w; s[7] += y.w;
        }
        const size_t at = ((size_t)seg * (MU * 16) + 8 * uh + g) * (NU * 16) + 8 * j;
        if (p.dw_f16 != nullptr) {
          red_add_h8(p.dw_f16 + at, pack_half2(s[0], s[1]), pack_half2(s[2], s[3]), pack_half2(s[4], s[5]), pack_half2(s[6], s[7]));
        } else {
          red_add_v4(p.dw + at, s[0], s[1], s[2], s[3]);
          red_add_v4(p.dw + at + 4, s[4], s[5], s[6], s[7]);
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// Warps of the block: as many as the registers allow (sums, operands, about fifty for the rest), 16 at most; the ring as
// long as shared memory allows, with room for a block of the exchange beside it.
constexpr int wh_warps(bool tf32, int mu, int nu, bool dgrad = false) {
  const int regs = 8 * mu * nu + 4 * (mu + nu) + (tf32 ? 56 : 48) + (dgrad ? 4 * mu * nu + 4 * nu + 24 : 0), fit = 61440 / (32 * ((regs + 7) / 8 * 8)) / 4 * 4;
  return fit > 16 ? 16 : fit;
}
constexpr int wh_depth(bool tf32, int mu, int nu, bool dgrad = false) {
  const int stage = tf32 ? 1024 * (mu + nu + 1) : 512 * (mu + nu) + (mu == 3 ? 256 : 0) + (nu == 3 ? 256 : 0);
  const int fit = 200 * 1024 / (wh_warps(tf32, mu, nu, dgrad) * (stage + (dgrad ? 192 : 128)));
  return fit > WH_MAX_DEPTH ? WH_MAX_DEPTH : fit;
}
// Shapes this kernel takes: multiples of 16 up to 64 channels on both sides, in tf32 not 48 -> 64, 64 -> 48 and 64 -> 64.
inline bool wh_supported(int c_in, int c_out, bool f16) {
  if (c_in % 16 || c_out % 16 || c_in < 16 || c_out < 16 || c_in > 64 || c_out > 64) return false;
  return f16 || c_in + c_out < 112;
}

// Shapes of the kernel for both gradients: at most eight pairs of 16-channel units, so that W_k^T fits beside the sums in the
// registers of eight warps or more (64 -> 48 on 591 k pairs with the four that are left 52.6 us, 42.2 by two kernels; with the weights
// in shared memory 64 -> 64 67.7 / 61.6).  And the pairs from which clearing and rounding the sums, 2.5 us, are paid for, us by two
// kernels / this one: 32 -> 64 on 591 k pairs 27.1 / 28.0, on 1.13 M 45.8 / 45.1; 32 -> 32 on 364 k 14.6 / 15.9, on 591 k 19.7 / 20.5.
// Above the line 12 shapes on surfaces, scattered and full clouds and strided maps of 1.1 to 4.6 M pairs take 0.71 to 1.03 of two kernels' time, but for
// two kinds, which stay here because the sums are rounded once (2.1e-4 against 4.0e-4): 32 -> 48 submanifold up to 2.2 M pairs, 1.08 M 47.4 / 50.1; and
// stride-2 maps with no fewer input than output channels, whose input gradient is one red a row into memory: 32 -> 32 on 1.2 M 48.9 / 50.8, on
// 3 M 119 / 139, 64 -> 32 on 1.2 M 86.7 / 95.6.  (Transposed 64 -> 32 67.5 / 60.8, stride 2 32 -> 64 58.1 / 53.8.)
constexpr bool wh_both_shape(int mu, int nu) { return mu * nu <= 8; }
constexpr long long WH_BOTH_PAIRS = 1 << 20;

template <bool TF32, int MU, int NU, bool DGRAD>
inline int wh_launch_as(const WgradParams& p, const RowsDgrad& dg, cudaStream_t st, int sms, int max_smem) {
  if constexpr ((TF32 && MU + NU >= 7) || (DGRAD && !wh_both_shape(MU, NU))) {
    return 1;
  } else {
    constexpr int WARPS = wh_warps(TF32, MU, NU, DGRAD), DEPTH = wh_depth(TF32, MU, NU, DGRAD);
    auto kernel = rows_wgrad_kernel<TF32, MU, NU, WARPS, DEPTH, DGRAD>;
    constexpr size_t rings = (size_t)WARPS * (DEPTH * (WhRows<TF32, MU>::TILE + WhRows<TF32, NU>::TILE) + (DEPTH - 1) * 128 + (DGRAD ? DEPTH * 64 : 0));
    constexpr size_t sums = (size_t)WARPS * MU * 8 * NU * 128;
    const size_t smem = (rings > sums ? rings : sums) + (size_t)(2 * p.k_vol + 3) * sizeof(int);
    if (smem > (size_t)max_smem) return 1;
    static std::atomic<int> granted[64];
    if (int rc = ensure_smem(kernel, max_smem, granted)) return rc;
    // Shared memory for the block and 4 KB: the driver's own choice, the smallest share that holds the block, may have no room for
    // a block of the exchange (tf32 32 -> 32 takes 163.3 of 164 KB: the exchange waited for the weight gradient to end).
    const int percent = (int)((rings > sums ? rings : sums) + 4096) * 100 / (228 * 1024) + 1;
    static std::atomic<bool> carved[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
    if (!carved[dev].load(std::memory_order_acquire)) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, percent < 100 ? percent : 100) != cudaSuccess) return -1;
      carved[dev].store(true, std::memory_order_release);
    }
    const long long units = (long long)p.pairs / (!TF32 && p.dw_f16 != nullptr ? 16 << WH_UNIT : 16) + p.k_vol + 1;
    const bool spread = spread_tiles((size_t)p.n_in * WhRows<TF32, MU>::BYTES + (size_t)p.n_out * WhRows<TF32, NU>::BYTES);
    return launch_pdl(kernel, (int)(units < sms ? units : sms), WARPS * 32, smem, st, p, spread, dg) == cudaSuccess ? 0 : -1;
  }
}
template <bool TF32, int MU, bool DGRAD>
inline int wh_launch_n(const WgradParams& p, const RowsDgrad& dg, cudaStream_t st, int sms, int max_smem) {
  switch (p.c_out / 16) {
    case 1: return wh_launch_as<TF32, MU, 1, DGRAD>(p, dg, st, sms, max_smem);
    case 2: return wh_launch_as<TF32, MU, 2, DGRAD>(p, dg, st, sms, max_smem);
    case 3: return wh_launch_as<TF32, MU, 3, DGRAD>(p, dg, st, sms, max_smem);
    case 4: return wh_launch_as<TF32, MU, 4, DGRAD>(p, dg, st, sms, max_smem);
  }
  return 1;
}
template <bool TF32, bool DGRAD = false>
inline int wh_launch(const WgradParams& p, const RowsDgrad& dg, cudaStream_t st, int sms, int max_smem) {
  switch (p.c_in / 16) {
    case 1: return wh_launch_n<TF32, 1, DGRAD>(p, dg, st, sms, max_smem);
    case 2: return wh_launch_n<TF32, 2, DGRAD>(p, dg, st, sms, max_smem);
    case 3: return wh_launch_n<TF32, 3, DGRAD>(p, dg, st, sms, max_smem);
    case 4: return wh_launch_n<TF32, 4, DGRAD>(p, dg, st, sms, max_smem);
  }
  return 1;
}

// 0 launched, 1 not a shape of this kernel or a pointer is not 16-byte aligned, < 0 CUDA error
inline int launch_rows_wgrad(const WgradParams& p, bool f16, cudaStream_t st, int sms, int max_smem) {
  if (!wh_supported(p.c_in, p.c_out, f16)) return 1;
  if ((long long)p.pairs > 0x7fffffffll - 65536) return 1;  // positions a few turns past the end stay in an int
  if ((reinterpret_cast<uintptr_t>(p.feats) | reinterpret_cast<uintptr_t>(p.out_grad) | reinterpret_cast<uintptr_t>(p.dw) |
       reinterpret_cast<uintptr_t>(p.dw_f16)) & 15) return 1;
  return f16 ? wh_launch<false>(p, RowsDgrad(), st, sms, max_smem) : wh_launch<true>(p, RowsDgrad(), st, sms, max_smem);
}
// Whether one kernel takes both gradients of fp16 rows, the weight gradient's sums in fp32; the buffers are distinct.
inline bool rows_bwd_supported(int c_in, int c_out) { return wh_supported(c_in, c_out, true) && wh_both_shape(c_in / 16, c_out / 16); }
inline bool rows_bwd_takes(const WgradParams& p, const RowsDgrad& dg, int max_smem) {
  return rows_bwd_supported(p.c_in, p.c_out) && (long long)p.pairs <= 0x7fffffffll - 65536 &&
         ((reinterpret_cast<uintptr_t>(p.feats) | reinterpret_cast<uintptr_t>(p.out_grad) | reinterpret_cast<uintptr_t>(p.dw) |
           reinterpret_cast<uintptr_t>(dg.weights) | reinterpret_cast<uintptr_t>(dg.in_grad)) & 15) == 0 &&
         216 * 1024 + (size_t)(2 * p.k_vol + 3) * sizeof(int) <= (size_t)max_smem;
}
inline int launch_rows_bwd(const WgradParams& p, const RowsDgrad& dg, cudaStream_t st, int sms, int max_smem) {
  return wh_launch<false, true>(p, dg, st, sms, max_smem);
}

}  // namespace fgms
