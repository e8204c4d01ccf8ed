// Exact fp32 on the CUDA cores, fp32 storage: forward / dgrad up to 128 contraction channels (about 108 where there are at most
// four output channels: one lane a pair, and the rows of 32 of them exceed shared memory), and the weight gradient.
//
// The products of a ragged layer (20 -> 36 channels, 390 k pairs) are 7.5 us of FMA a pass, moving its rows 11-15 us;
// the tiles of simt_kernels.cuh, 64 x 64 whatever the width, read shared memory a word at a time and keep no row in
// flight, and take 61 / 100 / 124 us (forward, dgrad, weight gradient); here 33 / 32 / 38 us, 64 -> 64 on 591 k pairs
// 205 / 204 / 186 -> 157 / 156 / 152 us, 3 -> 64 69 / 86 / 199 -> 35 / 41 / 43 us.  Bound by the FMA pipe and what waits for it: a packed
// FMA takes 2.4 cycles a scheduler (3.1 where no operand is the last one's), and multiplications of addresses and copies of registers go through
// the same pipe (forward 64 -> 64: 38 of 54 M instructions there are the products, it is busy for 62 % of the time, 2.4 warps a scheduler
// wait for it or for shared memory); with short rows the instructions of a tile's gather and reds.
//
//   * the work of a pass is cut to the layer's width: four (forward) or eight by four (weight gradient) channels per
//     thread, as many threads side by side as the width needs, the others take further pairs;
//   * operands come from shared memory 16 bytes at a time, rows laid an odd number of 16-byte units apart so that the
//     lanes of a quarter warp meet different banks;
//   * rows are copied with cp.async a tile ahead, their map entries another tile ahead;
//   * products are packed FMAs, half the instructions: the forward sums even and odd contraction channels side by side (fma.rn.f32x2
//     on two halves of a 16-byte word: nothing to duplicate), the weight gradient two input channels, with the output channel in both halves.
//     Fewer instructions leave the two passes of a backward, which share the SMs, more of each other's: 64 -> 64 on 591 k pairs 365 -> 293 us,
//     20 -> 36 on 390 k 72.3 -> 67.7, 40 -> 33 on 208 k 91 -> 84.
//
// Weights kept in registers, a lane's share of the contraction each (16 to 24 channels by four), were slower: forward 20 -> 36 48.8 us, dgrad
// 64 -> 64 212.
#pragma once
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "umma.cuh"  // launch_pdl, griddep_*

namespace fgms {

constexpr int FF_WARPS = 4;
constexpr int FF_THREADS = FF_WARPS * 32;
constexpr int FF_MAX_K = 128;
constexpr int ff_gms_blocks(int pt) { return pt == 8 ? 3 : 4; }  // 64 accumulators, 16 weights and the walk do not fit 128 registers

__device__ __forceinline__ void ff_fma2(uint64_t& c, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t ff_mul2(uint64_t a, uint64_t b) {
  uint64_t c;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  return c;
}
__device__ __forceinline__ void ff_add2(uint64_t& c, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(c) : "l"(a)); }
__device__ __forceinline__ uint64_t ff_two(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float ff_half(uint64_t v, int h) { return __uint_as_float((uint32_t)(v >> (32 * h))); }
__device__ __forceinline__ void ff_lds2(uint32_t addr, uint64_t& a, uint64_t& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr) : "memory");
}
__device__ __forceinline__ float ff_sum(uint64_t v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
// off: writes zeros and reads nothing
__device__ __forceinline__ void ff_cp16(uint32_t dst, const float* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ff_cp4(uint32_t dst, const float* src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(on ? 4 : 0) : "memory");
}
__device__ __forceinline__ void ff_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ff_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint32_t ff_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Steps through a [rows][units] grid `step` cells at a time from cell `first`, without a division per cell.
struct Walk {
  int row, unit, d_row, d_unit, units;
  __device__ __forceinline__ Walk(int first, int step, int units_) : units(units_) {
    row = first / units; unit = first - row * units;
    d_row = step / units; d_unit = step - d_row * units;
  }
  __device__ __forceinline__ void next() {
    row += d_row; unit += d_unit;
    if (unit >= units) { unit -= units; ++row; }
  }
};

// `rows` rows of `cols` channels from column c0 on, to dst[row * ld + column]; rows idx[row] < 0 become zeros.  Channels
// [cols, cols_padded) of a staged row become zeros too.  `w` walks rows x (16-byte or 4-byte units of cols_padded).
__device__ __forceinline__ void ff_gather(uint32_t dst, int ld, const float* base, int row_len, int c0, int cols, const int* idx, int rows,
                                          Walk w, bool vec) {
  if (vec) {
    for (; w.row < rows; w.next()) {
      const int r = idx[w.row];
      ff_cp16(dst + 4 * (w.row * ld + 4 * w.unit), r < 0 ? base : base + (size_t)r * row_len + c0 + 4 * w.unit, r >= 0);
    }
  } else {
    for (; w.row < rows; w.next()) {
      const int r = idx[w.row];
      const bool on = r >= 0 && w.unit < cols;
      ff_cp4(dst + 4 * (w.row * ld + w.unit), on ? base + (size_t)r * row_len + c0 + w.unit : base, on);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// forward / dgrad
// ---------------------------------------------------------------------------------------------------------------------
struct FfPlan {
  int n_blocks, cg, pg, pt;  // blocks of 4 cg output columns; pg lanes groups x pt pairs per lane = pairs of a warp's tile
  int ld;                    // words of a staged row of either operand
  size_t smem;
};

// Lane (g, c) of a warp: pairs g + pg i of the tile (i < PT), columns 4 c .. 4 c + 3 of the block.  Column 4 c + i of the
// weights is staged as row i cg + c, its contraction channels consecutive, so that both operands are read along them.
// VEC: rows of both sides are whole 16-byte units that start on a 16-byte boundary, known at compile time; otherwise each
// side is asked for at run time.
template <bool TRANS, int PT, bool VEC>
__global__ void __launch_bounds__(FF_THREADS, ff_gms_blocks(PT)) ffma_gms_kernel(GmsParams p, FfPlan plan) {
  extern __shared__ __align__(16) int ff_smem_dyn[];
  int* tile_start = ff_smem_dyn;           // [k_vol + 2]
  int* kpos_s = tile_start + p.k_vol + 2;  // [k_vol + 1]
  const int cg = plan.cg, pg = plan.pg, ld = plan.ld, tile_pairs = pg * PT;
  float* bs = reinterpret_cast<float*>(ff_smem_dyn + (2 * p.k_vol + 3 + 3) / 4 * 4);  // [4 cg][ld]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* as = bs + 4 * cg * ld + warp * (2 * tile_pairs * ld + 3 * 64);  // [2][tile_pairs][ld]
  int* rows_g = reinterpret_cast<int*>(as + 2 * tile_pairs * ld);        // [64]
  int* rows_s = rows_g + 64;                                             // [2][64]

  const float* __restrict__ src = static_cast<const float*>(p.src);
  const float* __restrict__ weights = static_cast<const float*>(p.weights);
  float* dst = static_cast<float*>(p.dst);
  const int n_seg = p.k_vol + 1;

  umma::griddep_begin(TRANS && p.beside, p.alone);
  build_tile_table(tile_pairs, p.kpos, p.pairs, p.k_vol, p.dense_rows, kpos_s, tile_start);
  int t, t1;
  cta_tile_range(tile_start[n_seg], &t, &t1);
  if (t >= t1) {
    umma::griddep_end(TRANS && p.beside);
    return;
  }

  const int kp = (p.k_dim + 3) / 4 * 4;
  const bool vec_in = VEC || (p.k_dim % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0);
  const bool vec_out = VEC || (p.n_dim % 4 == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0);
  const Walk walk(lane, 32, vec_in ? kp / 4 : kp);
  const Walk walk_b(threadIdx.x, FF_THREADS, TRANS ? kp : 4 * cg);
  const int c = lane % cg, g = lane / cg;
  const bool active = g < pg;
  const uint32_t b_addr = ff_smem(bs) + 4 * (c * ld), b_step = 4 * (cg * ld);
  const uint32_t a_addr = ff_smem(as) + 4 * ((active ? g : 0) * ld), a_step = 4 * (pg * ld), a_buf = 4 * (tile_pairs * ld);

  int seg = find_segment(tile_start, n_seg, t);
  while (t < t1) {
    while (t >= tile_start[seg + 1]) ++seg;
    const int t_end = min(t1, tile_start[seg + 1]);
    const bool dense = seg == p.k_vol;
    const int j_base = dense ? 0 : kpos_s[seg], j_count = dense ? p.dense_rows : kpos_s[seg + 1] - j_base;
    const int lt0 = t - tile_start[seg] + warp, lt1 = t_end - tile_start[seg];
    const float* __restrict__ wk = weights + (size_t)(dense ? p.dense_weight : seg) * p.c_in * p.c_out;

    for (int block = 0; block < plan.n_blocks; ++block) {
      const int n0 = block * 4 * cg;
      // map entries of tile lt, two per lane; looked at only when its rows are fetched, a tile later
      int eg[2], es[2];
      auto has_pair = [&](int lt, int i) {
        return lt < lt1 && i < tile_pairs && (uint32_t)lt * (uint32_t)tile_pairs + (uint32_t)i < (uint32_t)j_count;
      };
      auto load_rows = [&](int lt) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = lane + 32 * h;
          eg[h] = es[h] = -1;
          if (has_pair(lt, i)) {
            const int j = j_base + lt * tile_pairs + i;
            eg[h] = dense ? j : __ldg(p.gather_map + j);
            es[h] = dense ? j : __ldg(p.scatter_map + j);
          }
        }
      };
      auto start = [&](int lt, int buf) {  // rows of the loaded entries on their way to `buf`
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if ((unsigned)eg[h] >= (unsigned)p.n_gather || (unsigned)es[h] >= (unsigned)p.n_scatter) {
            if (block == 0 && has_pair(lt, lane + 32 * h)) report_problem();  // pair skipped, counted once
            eg[h] = es[h] = -1;
          }
          rows_g[lane + 32 * h] = eg[h];
          rows_s[buf * 64 + lane + 32 * h] = es[h];
        }
        __syncwarp();
        if (lt < lt1) ff_gather(ff_smem(as) + buf * a_buf, ld, src, p.k_dim, 0, p.k_dim, rows_g, tile_pairs, walk, vec_in);
        ff_commit();
        __syncwarp();
      };
      load_rows(lt0);
      __syncthreads();  // the weights before these have been used
      {
        // the faster index runs along memory; eight loads of a thread under way together
        Walk w = walk_b;
        while (w.row < (TRANS ? 4 * cg : kp)) {
          float v[8];
          int at[8];
#pragma unroll
          for (int i = 0; i < 8; ++i, w.next()) {
            const int n = TRANS ? w.row : w.unit, k = TRANS ? w.unit : w.row;
            const bool in = n < 4 * cg && k < kp;
            v[i] = 0.f;
            at[i] = in ? ((n & 3) * cg + (n >> 2)) * ld + k : -1;
            if (in && k < p.k_dim && n0 + n < p.n_dim) v[i] = __ldg(wk + (TRANS ? (size_t)(n0 + n) * p.c_out + k : (size_t)k * p.c_out + n0 + n));
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (at[i] >= 0) bs[at[i]] = v[i];
        }
      }
      start(lt0, 0);
      load_rows(lt0 + FF_WARPS);
      __syncthreads();

      int buf = 0;
      for (int lt = lt0; lt < lt1; lt += FF_WARPS, buf ^= 1) {
        start(lt + FF_WARPS, buf ^ 1);
        load_rows(lt + 2 * FF_WARPS);
        ff_wait<1>();
        __syncwarp();
        uint64_t acc[PT][4];
        const uint32_t a0 = a_addr + buf * a_buf;
        // four channels of the contraction, `first`: the sums begin
        auto step = [&](uint32_t k, uint32_t off, auto first) {
          uint64_t b0[4], b1[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) ff_lds2(b_addr + j * b_step + k + off, b0[j], b1[j]);
#pragma unroll
          for (int i = 0; i < PT; ++i) {
            uint64_t x0, x1;
            ff_lds2(a0 + i * a_step + k + off, x0, x1);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if constexpr (decltype(first)::value) acc[i][j] = ff_mul2(x0, b0[j]);
              else ff_fma2(acc[i][j], x0, b0[j]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) ff_fma2(acc[i][j], x1, b1[j]);
          }
        };
        step(0u, 0u, std::true_type());
        uint32_t k = 16;
#pragma unroll 1
        for (; k + 16 < 4 * (uint32_t)kp; k += 32) {
          step(k, 0u, std::false_type());
          step(k, 16u, std::false_type());
        }
        if (k < 4 * (uint32_t)kp) step(k, 0u, std::false_type());
        const int n = n0 + 4 * c, valid = min(4, p.n_dim - n);
        if (active && valid > 0) {
#pragma unroll
          for (int i = 0; i < PT; ++i) {
            const int s = rows_s[buf * 64 + g + pg * i];
            if (s < 0) continue;
            const float v[4] = {ff_sum(acc[i][0]), ff_sum(acc[i][1]), ff_sum(acc[i][2]), ff_sum(acc[i][3])};
            float* o = dst + (size_t)s * p.n_dim + n;
            if (VEC) red_add_v4(o, v[0], v[1], v[2], v[3]);
            else scatter_add<4>(o, v, valid, vec_out);
          }
        }
        __syncwarp();  // the buffer and its rows are free
      }
      ff_wait<0>();
    }
    t = t_end;
  }
  umma::griddep_end(TRANS && p.beside);
}

// ---------------------------------------------------------------------------------------------------------------------
// weight gradient
// ---------------------------------------------------------------------------------------------------------------------
constexpr int FW_PAIRS = 64;    // pairs of a chunk in shared memory, and of a scheduling tile
constexpr int FW_BLOCK = 64;    // channels of a block of dW_k on either side

// Block threads: `slices` groups of rg x cg threads, each thread eight input by four output channels; slice s takes pairs
// s, s + slices, .. of a chunk.  Sums stay in registers over the block's whole run inside one offset, those of 21 to 64 pairs at a time and
// the total of these (relative error 64 -> 64 on 591 k pairs 6.5e-7 -> 1.9e-7, 20 -> 36 2.3e-7 -> 1.5e-7; the same time, but for three and five
// slices, of 21 and 26 pairs, 40 -> 32 on 418 k 52.1 -> 53.1 us; of 43 pairs 52.0, and a tenth less exact); then the slices meet
// in shared memory and leave with one red per value.
template <int BLOCKS>
__global__ void __launch_bounds__(FF_THREADS, BLOCKS) ffma_wgrad_kernel(WgradParams p) {
  extern __shared__ __align__(16) int ff_smem_dyn[];
  int* tile_start = ff_smem_dyn;
  int* kpos_s = tile_start + p.k_vol + 2;
  const int bm = min(FW_BLOCK, p.c_in), bn = min(FW_BLOCK, p.c_out);
  const int rg = (bm + 7) / 8, cg = (bn + 3) / 4, ld_a = 8 * rg, ld_g = 4 * cg;
  const int slices = FF_THREADS / (rg * cg), period = max(1, 32 * slices / FW_PAIRS);
  int* rows = ff_smem_dyn + (2 * p.k_vol + 3 + 3) / 4 * 4;                 // [2][in, out][FW_PAIRS]
  float* stage = reinterpret_cast<float*>(rows + 4 * FW_PAIRS);            // [2][FW_PAIRS][ld_a + ld_g]
  const int stage_words = FW_PAIRS * (ld_a + ld_g);

  const float* __restrict__ feats = static_cast<const float*>(p.feats);
  const float* __restrict__ og = static_cast<const float*>(p.out_grad);
  const int tid = threadIdx.x, n_seg = p.k_vol + 1;

  umma::griddep_begin(0, p.alone);
  build_tile_table(FW_PAIRS, p.kpos, p.pairs, p.k_vol, 0, kpos_s, tile_start);
  int t, t1;
  cta_tile_range(tile_start[n_seg], &t, &t1);
  if (t >= t1) return;
  const bool vec_a = p.c_in % 4 == 0 && (reinterpret_cast<uintptr_t>(feats) & 15) == 0;
  const bool vec_g = p.c_out % 4 == 0 && (reinterpret_cast<uintptr_t>(og) & 15) == 0;
  const bool vec_out = p.c_out % 4 == 0 && (reinterpret_cast<uintptr_t>(p.dw) & 15) == 0;
  const int c = tid % cg, r = tid / cg % rg, slice = tid / (rg * cg);

  int seg = find_segment(tile_start, n_seg, t);
  while (t < t1) {
    while (t >= tile_start[seg + 1]) ++seg;
    const int t_end = min(t1, tile_start[seg + 1]);
    const int lt0 = t - tile_start[seg], chunks = t_end - t;
    const int j0 = kpos_s[seg] + lt0 * FW_PAIRS, j_count = kpos_s[seg + 1] - j0;
    float* dwk = p.dw + (size_t)seg * p.c_in * p.c_out;

    for (int m0 = 0; m0 < p.c_in; m0 += FW_BLOCK) {
      for (int n0 = 0; n0 < p.c_out; n0 += FW_BLOCK) {
        const int cols_a = min(bm, p.c_in - m0), cols_g = min(bn, p.c_out - n0);
        const Walk walk_a(tid, FF_THREADS, vec_a ? cols_a / 4 : cols_a), walk_g(tid, FF_THREADS, vec_g ? cols_g / 4 : cols_g);
        int ei = -1, eo = -1;
        auto has_pair = [&](int chunk) {
          return tid < FW_PAIRS && chunk < chunks && (uint32_t)chunk * FW_PAIRS + (uint32_t)tid < (uint32_t)j_count;
        };
        auto load_rows = [&](int chunk) {
          ei = eo = -1;
          if (has_pair(chunk)) {
            const int j = j0 + chunk * FW_PAIRS + tid;
            ei = __ldg(p.in_map + j);
            eo = __ldg(p.out_map + j);
          }
        };
        auto store_rows = [&](int chunk) {
          if (tid < FW_PAIRS) {
            if ((unsigned)ei >= (unsigned)p.n_in || (unsigned)eo >= (unsigned)p.n_out) {
              if (m0 == 0 && n0 == 0 && has_pair(chunk)) report_problem();  // counted once per skipped pair
              ei = eo = -1;
            }
            rows[(chunk & 1) * 2 * FW_PAIRS + tid] = ei;
            rows[(chunk & 1) * 2 * FW_PAIRS + FW_PAIRS + tid] = eo;
          }
        };
        auto start = [&](int chunk) {
          if (chunk < chunks) {
            const int* idx = rows + (chunk & 1) * 2 * FW_PAIRS;
            const uint32_t a = ff_smem(stage + (chunk & 1) * stage_words);
            ff_gather(a, ld_a, feats, p.c_in, m0, cols_a, idx, FW_PAIRS, walk_a, vec_a);
            ff_gather(a + 4 * FW_PAIRS * ld_a, ld_g, og, p.c_out, n0, cols_g, idx + FW_PAIRS, FW_PAIRS, walk_g, vec_g);
          }
          ff_commit();
        };
        __syncthreads();  // the stages and rows of the block before are free
        load_rows(0);
        store_rows(0);
        load_rows(1);
        store_rows(1);
        load_rows(2);
        __syncthreads();
        start(0);

        // input channels 2 i and 2 i + 1, output channel j: the sums of the last few chunks, and of those before
        uint64_t acc[4][4], total[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = total[i][j] = 0ull;
        int until = period;
        for (int chunk = 0; chunk < chunks; ++chunk) {
          start(chunk + 1);
          ff_wait<1>();
          __syncthreads();  // the chunk has landed for every thread
          store_rows(chunk + 2);  // where this chunk's entries were: every thread has started it
          load_rows(chunk + 3);
          if (slice < slices) {
            const uint32_t a = ff_smem(stage + (chunk & 1) * stage_words + 8 * r);
            const float* b = stage + (chunk & 1) * stage_words + FW_PAIRS * ld_a + 4 * c;
#pragma unroll (BLOCKS <= 3 ? 8 : 4)
            for (int j = slice; j < FW_PAIRS; j += slices) {
              uint64_t x[4];
              ff_lds2(a + 4 * j * ld_a, x[0], x[1]);
              ff_lds2(a + 4 * j * ld_a + 16, x[2], x[3]);
              const float4 y = *reinterpret_cast<const float4*>(b + j * ld_g);
              const uint64_t y2[4] = {ff_two(y.x, y.x), ff_two(y.y, y.y), ff_two(y.z, y.z), ff_two(y.w, y.w)};
#pragma unroll
              for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) ff_fma2(acc[i][k], x[i], y2[k]);
            }
          }
          if (BLOCKS < 6 && (--until == 0 || chunk + 1 == chunks)) {
            until = period;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                ff_add2(total[i][j], acc[i][j]);
                acc[i][j] = 0ull;
              }
          }
          __syncthreads();  // the chunk's stage is free, the entries of chunk + 2 are visible
        }
        ff_wait<0>();
        const uint64_t(&sums)[4][4] = BLOCKS < 6 ? total : acc;  // six blocks an SM have a chunk each
        // slices meet: [slices][8 rg][4 cg] words, at most 32 per thread of the block
        if (slice < slices) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float4 v;
            v.x = ff_half(sums[i / 2][0], i & 1); v.y = ff_half(sums[i / 2][1], i & 1); v.z = ff_half(sums[i / 2][2], i & 1); v.w = ff_half(sums[i / 2][3], i & 1);
            *reinterpret_cast<float4*>(stage + (slice * ld_a + 8 * r + i) * ld_g + 4 * c) = v;
          }
        }
        __syncthreads();
        for (int e = tid; e < ld_a * cg; e += FF_THREADS) {
          const int m = e / cg, n = 4 * (e - m * cg);
          if (m >= cols_a || n >= cols_g) continue;
          float v[4] = {0.f, 0.f, 0.f, 0.f};
          for (int s = 0; s < slices; s += 4) {  // fours of slices first
            float4 x[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
              x[k] = s + k < slices ? *reinterpret_cast<const float4*>(stage + ((s + k) * ld_a + m) * ld_g + n) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[0] += (x[0].x + x[1].x) + (x[2].x + x[3].x); v[1] += (x[0].y + x[1].y) + (x[2].y + x[3].y);
            v[2] += (x[0].z + x[1].z) + (x[2].z + x[3].z); v[3] += (x[0].w + x[1].w) + (x[2].w + x[3].w);
          }
          scatter_add<4>(dwk + (size_t)(m0 + m) * p.c_out + n0 + n, v, min(4, cols_g - n), vec_out);
        }
      }
    }
    t = t_end;
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------------
inline size_t ff_table_bytes(int k_vol) { return (size_t)(2 * k_vol + 3 + 3) / 4 * 16; }

// The largest tile of which two blocks fit an SM and whose pairs leave no lane over.  A call so small that every tile has
// a block of its own takes smaller ones as long as that stays so: its time is one tile's chain of loads (14 k pairs
// 16 -> 16: 5.0 us, two smaller tiles in turn 6.4).  False: the contraction is too wide (simt_gms_kernel takes it).
inline bool ff_plan(int k_dim, int n_dim, int k_vol, long long pairs, int sms, FfPlan* out) {
  if (k_dim > FF_MAX_K) return false;
  FfPlan f;
  f.n_blocks = (n_dim + 63) / 64;
  f.cg = ((n_dim + f.n_blocks - 1) / f.n_blocks + 3) / 4;
  const int units = (k_dim + 3) / 4;
  f.ld = 4 * (units | 1);
  bool found = false;
  for (int pt = 8; pt >= 1; pt /= 2) {
    f.pt = pt;
    f.pg = 32 / f.cg < 64 / pt ? 32 / f.cg : 64 / pt;
    f.smem = ff_table_bytes(k_vol) + 16 * (size_t)f.cg * f.ld + FF_WARPS * (8 * (size_t)f.pg * pt * f.ld + 3 * 64 * 4);
    const bool whole = f.pg == 32 / f.cg && f.smem <= 113 * 1024;
    if (!found ? whole : pairs / (f.pg * pt) + k_vol + 1 <= (long long)sms * ff_gms_blocks(pt) && whole) {
      *out = f;
      found = true;
    } else if (found) {
      break;
    }
  }
  return found;
}

inline int ff_by_smem(size_t smem) { return (int)(227 * 1024 / (smem + 1024)); }  // blocks
// As many blocks as an SM holds by registers (`by_regs`, the launch bound) and by shared memory, not more than tiles.
inline int ff_grid(long long tiles, size_t smem, int by_regs, int sms) {
  const long long by_smem = ff_by_smem(smem), most = sms * (by_smem < by_regs ? by_smem : by_regs);
  return (int)(tiles < most ? tiles : most);
}

template <bool TRANS, int PT, bool VEC>
inline int ff_launch_gms(const GmsParams& p, const FfPlan& f, cudaStream_t st, int sms) {
  static std::atomic<int> granted[64];
  if (ensure_smem(ffma_gms_kernel<TRANS, PT, VEC>, (int)f.smem, granted)) return -1;
  // a call of few tiles: one to a block, not one to a warp, so that no block has to change its weights
  const long long tiles = ((long long)p.pairs + p.dense_rows) / (f.pg * PT) + p.k_vol + 1;
  const int grid = ff_grid(tiles, f.smem, ff_gms_blocks(PT), sms);
  return launch_pdl(ffma_gms_kernel<TRANS, PT, VEC>, grid, FF_THREADS, f.smem, st, p, f) == cudaSuccess ? 0 : -1;
}
template <bool TRANS, bool VEC>
inline int ff_launch_pt(const GmsParams& p, const FfPlan& f, cudaStream_t st, int sms) {
  switch (f.pt) {
    case 8: return ff_launch_gms<TRANS, 8, VEC>(p, f, st, sms);
    case 4: return ff_launch_gms<TRANS, 4, VEC>(p, f, st, sms);
    case 2: return ff_launch_gms<TRANS, 2, VEC>(p, f, st, sms);
    default: return ff_launch_gms<TRANS, 1, VEC>(p, f, st, sms);
  }
}

// 0 launched, 1 not a shape of this kernel, < 0 CUDA error
inline int launch_ffma_gms(const GmsParams& p, bool trans, cudaStream_t st, int sms) {
  FfPlan f;
  if (!ff_plan(p.k_dim, p.n_dim, p.k_vol, (long long)p.pairs + p.dense_rows, sms, &f)) return 1;
  const bool vec = p.k_dim % 4 == 0 && p.n_dim % 4 == 0 && ((reinterpret_cast<uintptr_t>(p.src) | reinterpret_cast<uintptr_t>(p.dst)) & 15) == 0;
  if (vec) return trans ? ff_launch_pt<true, true>(p, f, st, sms) : ff_launch_pt<false, true>(p, f, st, sms);
  return trans ? ff_launch_pt<true, false>(p, f, st, sms) : ff_launch_pt<false, false>(p, f, st, sms);
}

template <int BLOCKS>
inline int ff_launch_wgrad(const WgradParams& p, size_t smem, cudaStream_t st, int sms) {
  static std::atomic<int> granted[64];
  if (ensure_smem(ffma_wgrad_kernel<BLOCKS>, (int)smem, granted)) return -1;
  const int grid = ff_grid((long long)p.pairs / FW_PAIRS + p.k_vol, smem, BLOCKS, sms);
  return launch_pdl(ffma_wgrad_kernel<BLOCKS>, grid, FF_THREADS, smem, st, p) == cudaSuccess ? 0 : -1;
}
inline int launch_ffma_wgrad(const WgradParams& p, cudaStream_t st, int sms) {
  const int rg = ((p.c_in < FW_BLOCK ? p.c_in : FW_BLOCK) + 7) / 8, cg = ((p.c_out < FW_BLOCK ? p.c_out : FW_BLOCK) + 3) / 4;
  const size_t stages = 2 * FW_PAIRS * (size_t)(8 * rg + 4 * cg) * 4, sums = FF_THREADS * 32 * 4;
  const size_t smem = ff_table_bytes(p.k_vol) + 4 * FW_PAIRS * 4 + (stages > sums ? stages : sums);
  // Registers, in which reads of shared memory run ahead of the products, are worth more than warps: four blocks of 128 rather than six
  // of 80 (24 -> 24 on 296 k pairs 24.2 -> 22.1 us), three of 168 where shared memory holds no more (64 -> 64 on 591 k 161 -> 152).
  // A call that gives each of six blocks an SM a single chunk has them all the same: 4 -> 16 on 39 k pairs 7.4 us with four, 6.2.
  const long long tiles = (long long)p.pairs / FW_PAIRS + p.k_vol;
  if (ff_by_smem(smem) >= 6 && tiles > 4ll * sms && tiles <= 6ll * sms) return ff_launch_wgrad<6>(p, smem, st, sms);
  return ff_by_smem(smem) > 3 ? ff_launch_wgrad<4>(p, smem, st, sms) : ff_launch_wgrad<3>(p, smem, st, sms);
}

}  // namespace fgms
