// Forward / dgrad for short rows: every warp gathers, multiplies and scatters on its own, in registers.
//
//   out[scatter[j]] += src[gather[j]] . W_k        for the pairs j of every offset k
//
// What bounds a layer of short rows is how many row pieces the SMs can ask L2 for, not arithmetic: a kernel that only
// copies (gather a row, red it to its destination; no product) takes 143 us on 9.1 M pairs of 64-byte rows, 28 us on
// 0.93 M pairs of 128-byte rows, while the tcgen05 form (umma_gms3.cuh) takes 318 us and 35 us there (this kernel 141 and
// 37): its tiles pass through shared memory, tensor memory and a patch, and each of those hand-offs costs a fixed few hundred
// cycles per 128 rows whatever their length.  A product of 32 x 32 is 2 % of the warp-level matrix rate, so this kernel gives up
// the faster tensor path and keeps nothing between the gather and the red but registers:
//
//   * mma.sync takes A with four lanes per row.  The contraction index may be enumerated in any order as long as A and B
//     agree, so lane t of a row's four loads 16 consecutive bytes (half rows: 8) and those registers ARE the A operand.
//   * The output columns may be permuted likewise: column j of n-tile i belongs to the lane that then holds 16 (or 8)
//     consecutive bytes of the output row, which go out as one vector red.
//   * B (the weight matrix) stays in registers while consecutive tiles belong to one offset: up to 64 registers.
//
// No shared memory beyond the tile table, no barrier, no shuffle in the loop; 8 (tf32 64 -> 32) to 24 (fp16 16 -> 16) warps per
// SM, each with the rows of one tile in flight while it multiplies the one before.
#pragma once
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "umma.cuh"  // launch_pdl, griddep_*

namespace fgms {

constexpr int RW_WARPS = 4;
constexpr int RW_THREADS = RW_WARPS * 32;

// The kernels of a backward leave every SM room for one block of the exchange kernel (peer_exchange.cuh: 128 threads of 32
// registers, a little shared memory), which is meant to run beside them: registers per thread of `threads` resident ones,
// and the percentage of the SM's shared memory that is not cache.  With all registers taken (128 per thread at 32 -> 32) or
// with the 8 KB of shared memory the driver chooses by itself, the exchange waits for the input gradient to end (8.1 M
// pairs: 285 us); with both it is done after 90 us, and the input gradient takes the same 136 us (64 -> 64: 282).  From 20 %
// on the smaller cache shows: 64 -> 64 303 us.
constexpr int rw_max_regs(int threads, bool backward) {
  const int regs = (backward ? 65536 - 4096 : 65536) / threads / 8 * 8;
  return regs < 248 ? regs : 248;
}
constexpr int RW_SMEM_PERCENT = 8;

__device__ __forceinline__ void rw_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, bool tf32) {
  if (tf32)
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// rows are used once per pair and come back from L2: no L1 allocation (164 -> 143 us for the copy of 64-byte rows)
__device__ __forceinline__ void rw_ld16(const void* p, uint32_t* v) {
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p));
}
__device__ __forceinline__ void rw_ld8(const void* p, uint32_t* v) {
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(p));
}

// Shape of a row in the four lanes that share it.  KU / NU: contraction and output width in units of 16 channels.
// A piece is what one vector access of the four lanes covers: 64 bytes (fp16: 32 channels, tf32: 16), or for the last 16
// channels of an odd number of units in fp16 32 bytes.
template <bool TF32, int KU, int NU>
struct RowShape {
  static constexpr int ES = TF32 ? 4 : 2;
  static constexpr int KFULL = TF32 ? KU : KU / 2, KHALF = TF32 ? 0 : KU % 2;
  static constexpr int NFULL = TF32 ? NU : NU / 2, NHALF = TF32 ? 0 : NU % 2;
  static constexpr int KSTEPS = TF32 ? 2 * KU : KU;  // MMAs along the contraction: 8 channels (tf32) or 16
  static constexpr int NT = 2 * NU;                  // n-tiles of 8 columns
  static constexpr int TPF = TF32 ? 2 : 4;           // n-tiles per full piece
  static constexpr int AR = 2 * KSTEPS;              // A registers per row and lane
  static constexpr int CPF = TF32 ? 16 : 32;         // channels per full piece
};

// The weight matrix of an offset as the B operand: b[step][n-tile][2].  Lane (g, t) = (lane / 4, lane % 4).  Contraction
// order: MMA step s of full piece q takes channels CPF q + E t + (E / 2)(s % 2) .. of lane t, E = the channels of a 16-byte
// load.  Output order: column g of n-tile j of full piece q is channel CPF q + TPF g + j.
template <bool TF32, bool TRANS, int KU, int NU>
__device__ __forceinline__ void rw_load_b(const uint8_t* w, int c_out, int lane, uint32_t (&b)[RowShape<TF32, KU, NU>::KSTEPS][2 * NU][2]) {
  using S = RowShape<TF32, KU, NU>;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t ld = (uint32_t)c_out * S::ES;  // bytes of a row of W_k
  if (TRANS) {
    // B[k][n] = W[n][k]: 16 (8) consecutive bytes of row n hold every k of this lane in a piece
#pragma unroll
    for (int j = 0; j < S::NT; ++j) {
      const bool nf = j < S::NFULL * S::TPF;
      const int q = j / S::TPF, jj = j % S::TPF;
      const int n = nf ? q * S::CPF + S::TPF * g + jj : S::NFULL * S::CPF + 2 * g + (j - S::NFULL * S::TPF);
      const uint8_t* row = w + (size_t)n * ld;
#pragma unroll
      for (int kq = 0; kq < S::KFULL; ++kq) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(row + kq * 64 + t * 16));
        b[2 * kq][j][0] = v.x; b[2 * kq][j][1] = v.y; b[2 * kq + 1][j][0] = v.z; b[2 * kq + 1][j][1] = v.w;
      }
      if (S::KHALF) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(row + S::KFULL * 64 + t * 8));
        b[S::KSTEPS - 1][j][0] = v.x; b[S::KSTEPS - 1][j][1] = v.y;
      }
    }
  } else {
#pragma unroll
    for (int s = 0; s < S::KSTEPS; ++s) {
      const bool kf = s < 2 * S::KFULL;
      if (TF32) {
        const int k0 = (s / 2) * 16 + 4 * t + 2 * (s & 1);
        const uint8_t* r0 = w + (size_t)k0 * ld;
#pragma unroll
        for (int q = 0; q < S::NFULL; ++q) {
          const uint2 x = __ldg(reinterpret_cast<const uint2*>(r0 + q * 64 + g * 8));
          const uint2 y = __ldg(reinterpret_cast<const uint2*>(r0 + ld + q * 64 + g * 8));
          b[s][2 * q][0] = x.x; b[s][2 * q][1] = y.x; b[s][2 * q + 1][0] = x.y; b[s][2 * q + 1][1] = y.y;
        }
      } else {
        const int k0 = kf ? (s / 2) * 32 + 8 * t + 4 * (s & 1) : S::KFULL * 32 + 4 * t;
        const uint8_t* r0 = w + (size_t)k0 * ld;
        auto pair_up = [&](int j, uint32_t lo0, uint32_t lo1, uint32_t hi0, uint32_t hi1) {  // two columns of four k rows
          b[s][j][0] = __byte_perm(lo0, lo1, 0x5410); b[s][j][1] = __byte_perm(hi0, hi1, 0x5410);
          b[s][j + 1][0] = __byte_perm(lo0, lo1, 0x7632); b[s][j + 1][1] = __byte_perm(hi0, hi1, 0x7632);
        };
#pragma unroll
        for (int q = 0; q < S::NFULL; ++q) {
          uint2 v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = __ldg(reinterpret_cast<const uint2*>(r0 + (size_t)i * ld + q * 64 + g * 8));
          pair_up(4 * q, v[0].x, v[1].x, v[2].x, v[3].x);
          pair_up(4 * q + 2, v[0].y, v[1].y, v[2].y, v[3].y);
        }
        if (S::NHALF) {
          uint32_t v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = __ldg(reinterpret_cast<const uint32_t*>(r0 + (size_t)i * ld + S::NFULL * 64 + g * 4));
          pair_up(S::NT - 2, v[0], v[1], v[2], v[3]);
        }
      }
    }
  }
}

// MT: m-tiles of 16 pairs a warp works on at a time.
template <bool TF32, bool TRANS, int KU, int NU, int MT, int MIN_BLOCKS>
__global__ void __maxnreg__(rw_max_regs(RW_THREADS * MIN_BLOCKS, TRANS)) rows_gms_kernel(GmsParams p, bool spread) {
  using S = RowShape<TF32, KU, NU>;
  constexpr int TILE = 16 * MT;
  constexpr uint32_t K_BYTES = KU * 16 * S::ES, N_BYTES = NU * 16 * S::ES;
  extern __shared__ int rw_smem[];
  int* tile_start = rw_smem;                // [k_vol + 2]
  int* kpos_s = tile_start + p.k_vol + 2;   // [k_vol + 1]
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int n_seg = p.k_vol + 1;

  umma::griddep_begin(TRANS && p.beside, p.alone);
  build_tile_table(TILE, p.kpos, p.pairs, p.k_vol, p.dense_rows, kpos_s, tile_start);

  // warp `me` has the turns [me F, me F + F) of all tiles' turns
  const int total = tile_start[n_seg], warps = (int)gridDim.x * RW_WARPS, share = (total + warps - 1) / warps;
  const int me = (int)blockIdx.x * RW_WARPS + (int)(threadIdx.x >> 5);
  int tile = min((long long)total, (long long)me * share);
  const int tile_end = min(total, tile + share);
  if (tile >= tile_end) {
    umma::griddep_end(TRANS && p.beside);
    return;
  }
  int seg = find_segment(tile_start, n_seg, tile);

  const uint8_t* src = static_cast<const uint8_t*>(p.src) + t4 * 16;
  const uint8_t* src_half = static_cast<const uint8_t*>(p.src) + S::KFULL * 64 + t4 * 8;
  uint8_t* dst = static_cast<uint8_t*>(p.dst) + t4 * 16;
  uint8_t* dst_half = static_cast<uint8_t*>(p.dst) + S::NFULL * 64 + t4 * 8;

  while (tile < tile_end) {
    // this warp's turns inside one offset
    while (tile >= tile_start[seg + 1]) ++seg;
    const int run = min(tile_end, tile_start[seg + 1]) - tile;
    const bool dense = seg == p.k_vol;
    const int j_begin = dense ? 0 : kpos_s[seg], j_end = dense ? p.dense_rows : kpos_s[seg + 1];
    const Turns turns(tile_start[seg], tile_start[seg + 1], share, me, tile, spread);
    tile += run;

    // gather and scatter rows of pairs j0 + 16 m + g and + 8; -1: no pair there, or an entry outside the tensors
    struct Rows { int g[MT][2], s[MT][2]; };
    auto load_rows = [&](int j0, Rows& r) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int jj = j0 + 16 * m + 8 * h + g;
          r.g[m][h] = r.s[m][h] = -1;
          if (jj < j_end) {
            r.g[m][h] = dense ? jj : __ldg(p.gather_map + jj);
            r.s[m][h] = dense ? jj : __ldg(p.scatter_map + jj);
          }
        }
    };
    auto gather = [&](Rows& r, uint32_t (&a)[MT][2][S::AR]) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int gi = r.g[m][h], si = r.s[m][h];
          const bool ok = (unsigned)gi < (unsigned)p.n_gather && (unsigned)si < (unsigned)p.n_scatter;
          if (!ok) {
            if (t4 == 0 && (gi != -1 || si != -1)) report_problem();  // pair skipped, counted once
            r.s[m][h] = -1;
          }
#pragma unroll
          for (int q = 0; q < S::AR; ++q) a[m][h][q] = 0u;
          if (ok) {
            const size_t off = (size_t)(unsigned)gi * K_BYTES;
#pragma unroll
            for (int q = 0; q < S::KFULL; ++q) rw_ld16(src + off + q * 64, &a[m][h][4 * q]);
            if (S::KHALF) rw_ld8(src_half + off, &a[m][h][4 * S::KFULL]);
          }
        }
    };
    Rows r0, r1;
    auto pair_of = [&](int n) { return n < run ? j_begin + TILE * turns.tile(n) : j_end; };
    load_rows(pair_of(0), r0);
    load_rows(pair_of(1), r1);
    uint32_t b[S::KSTEPS][S::NT][2];
    rw_load_b<TF32, TRANS, KU, NU>(static_cast<const uint8_t*>(p.weights) + (size_t)(dense ? p.dense_weight : seg) * p.c_in * p.c_out * S::ES,
                                   p.c_out, lane, b);
    uint32_t a0[MT][2][S::AR], a1[MT][2][S::AR];
    gather(r0, a0);

    auto multiply = [&](const Rows& r, const uint32_t (&a)[MT][2][S::AR]) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        auto piece = [&](int j_first, auto n_tiles, uint8_t* base) {  // n-tiles of one piece of the output row
          constexpr int N = decltype(n_tiles)::value;
          float c[N][4];
#pragma unroll
          for (int i = 0; i < N; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) c[i][k] = 0.f;
#pragma unroll
          for (int s = 0; s < S::KSTEPS; ++s) {
            const uint32_t frag[4] = {a[m][0][2 * s], a[m][1][2 * s], a[m][0][2 * s + 1], a[m][1][2 * s + 1]};
#pragma unroll
            for (int i = 0; i < N; ++i) rw_mma(c[i], frag, b[s][j_first + i][0], b[s][j_first + i][1], TF32);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (r.s[m][h] < 0) continue;
            uint8_t* o = base + (size_t)(unsigned)r.s[m][h] * N_BYTES;
            if (TF32) red_add_v4(reinterpret_cast<float*>(o), c[0][2 * h], c[1][2 * h], c[0][2 * h + 1], c[1][2 * h + 1]);
            else if (N == 4)
              red_add_h8(reinterpret_cast<__half*>(o), pack_half2(c[0][2 * h], c[1][2 * h]), pack_half2(c[N - 2][2 * h], c[N - 1][2 * h]),
                         pack_half2(c[0][2 * h + 1], c[1][2 * h + 1]), pack_half2(c[N - 2][2 * h + 1], c[N - 1][2 * h + 1]));
            else red_add_h4(reinterpret_cast<__half*>(o), pack_half2(c[0][2 * h], c[1][2 * h]), pack_half2(c[0][2 * h + 1], c[1][2 * h + 1]));
          }
        };
#pragma unroll
        for (int q = 0; q < S::NFULL; ++q) piece(q * S::TPF, std::integral_constant<int, S::TPF>(), dst + q * 64);
        if (S::NHALF) piece(S::NFULL * S::TPF, std::integral_constant<int, 2>(), dst_half);
      }
    };
    // two tiles per turn: the rows of one are on their way while the other is multiplied, and the map entries of the
    // tile after next
    for (int n = 0;;) {
      Rows r2;
      gather(r1, a1);
      load_rows(pair_of(n + 2), r2);
      multiply(r0, a0);
      if (++n >= run) break;
      r0 = r2;
      gather(r0, a0);
      load_rows(pair_of(n + 2), r2);
      multiply(r1, a1);
      if (++n >= run) break;
      r1 = r2;
    }
  }
  umma::griddep_end(TRANS && p.beside);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// Registers a variant needs decide how many of its blocks an SM should hold (the limit the compiler works to): the
// weights, two tiles of gathered rows, one piece of accumulators, and about forty for indices and addresses.
constexpr int rw_m_tiles(bool tf32, int ku) { return (tf32 ? 4 * ku : 2 * ku) <= 4 ? 2 : 1; }
constexpr int rw_min_blocks(bool tf32, int ku, int nu) {
  const int regs = (tf32 ? 8 : 4) * ku * nu + 4 * (tf32 ? 4 * ku : 2 * ku) * rw_m_tiles(tf32, ku) + 16 + 44;
  return 65536 / (RW_THREADS * ((regs + 7) / 8 * 8));
}

// Shapes this kernel takes: multiples of 16 up to 64 channels on both sides whose weights fit 64 registers.
inline bool rw_supported(int k_dim, int n_dim, bool f16) {
  if (k_dim % 16 || n_dim % 16 || k_dim < 16 || n_dim < 16 || k_dim > 64 || n_dim > 64) return false;
  return (k_dim / 16) * (n_dim / 16) * (f16 ? 4 : 8) <= 64;
}

template <bool TF32, bool TRANS, int KU, int NU>
inline int rw_launch_as(const GmsParams& p, cudaStream_t st, int sms) {
  constexpr int MT = rw_m_tiles(TF32, KU);
  auto kernel = rows_gms_kernel<TF32, TRANS, KU, NU, MT, rw_min_blocks(TF32, KU, NU)>;
  const size_t smem = (size_t)(2 * p.k_vol + 3) * sizeof(int);
  static std::atomic<int> resident[64];  // blocks per SM, by device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  int occ = resident[dev].load(std::memory_order_acquire);
  if (occ == 0) {
    if (TRANS && cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, RW_SMEM_PERCENT) != cudaSuccess) return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, RW_THREADS, 0) != cudaSuccess || occ < 1) return -1;
    resident[dev].store(occ, std::memory_order_release);
  }
  // no more blocks than there are tiles (a segment's last tile may be partly filled)
  const long long tiles = ((long long)p.pairs + p.dense_rows) / (16 * MT) + p.k_vol + 1;
  const long long most = (long long)sms * occ, want = (tiles + RW_WARPS - 1) / RW_WARPS;
  const bool spread = spread_tiles((size_t)p.n_gather * KU * 16 * (TF32 ? 4 : 2) + (size_t)p.n_scatter * NU * 16 * (TF32 ? 4 : 2));
  return launch_pdl(kernel, (int)(want < most ? want : most), RW_THREADS, smem, st, p, spread) == cudaSuccess ? 0 : -1;
}

template <bool TF32, bool TRANS, int KU>
inline int rw_launch_n(const GmsParams& p, cudaStream_t st, int sms) {
  constexpr int PER = (TF32 ? 8 : 4) * KU;  // weight registers per 16 output channels
  switch (p.n_dim / 16) {
    case 1: return rw_launch_as<TF32, TRANS, KU, 1>(p, st, sms);
    case 2: return rw_launch_as<TF32, TRANS, KU, 2>(p, st, sms);
    case 3: if constexpr (3 * PER <= 64) return rw_launch_as<TF32, TRANS, KU, 3>(p, st, sms); else return 1;
    case 4: if constexpr (4 * PER <= 64) return rw_launch_as<TF32, TRANS, KU, 4>(p, st, sms); else return 1;
  }
  return 1;
}
template <bool TF32, bool TRANS>
inline int rw_launch(const GmsParams& p, cudaStream_t st, int sms) {
  switch (p.k_dim / 16) {
    case 1: return rw_launch_n<TF32, TRANS, 1>(p, st, sms);
    case 2: return rw_launch_n<TF32, TRANS, 2>(p, st, sms);
    case 3: return rw_launch_n<TF32, TRANS, 3>(p, st, sms);
    case 4: return rw_launch_n<TF32, TRANS, 4>(p, st, sms);
  }
  return 1;
}

// 0 launched, 1 not a shape of this kernel or a pointer is not 16-byte aligned, < 0 CUDA error
inline int launch_rows_gms(const GmsParams& p, bool trans, bool f16, cudaStream_t st, int sms) {
  if (!rw_supported(p.k_dim, p.n_dim, f16)) return 1;
  // tf32 32 -> 64, a pair of widths whose weights fill the 64 registers and whose scattered rows are the longer ones: from
  // about 32 k pairs on the tcgen05 form is the faster (this kernel / that one, 27 offsets: 4 k pairs 3.7 / 5.0 us, 11 k
  // 4.6 / 5.1, 21 k 5.6 / 5.9; with the weights of this kernel 32 k 7.5, 131 k 12.5, 200 k 17.7, 1 M 65 against 39 k 7.0, 137 k
  // 11.7, 208 k 15.4, 0.93 M 51.7).  The other widths stay here whatever their size.  Most are faster here throughout (32 -> 48
  // 208 k 14.6 / 14.9; fp16 32 -> 32 0.93 M 18.8 / 35.8); where weights fill the registers the two forms cross as well, and
  // the line is not drawn for them: tf32 64 -> 32 39 k 7.2 / 6.4, 208 k 13.9 / 13.6, 0.93 M 42.1 / 43.2; tf32 16 -> 64 21 k 5.1 / 5.9, 39 k
  // 7.5 / 7.0, 0.93 M 59.0 / 52.4; fp16 64 -> 64 11 k 4.3 / 4.6, 39 k 6.9 / 5.8, 208 k 12.6 / 11.4, 0.93 M 37.4 / 34.8
  if (!f16 && p.k_dim == 32 && p.n_dim == 64 && p.pairs >= (1 << 15)) return 1;
  if ((long long)p.pairs + p.dense_rows > 0x7fffffffll - 4096) return 1;  // positions two tiles past the end stay in an int
  if ((reinterpret_cast<uintptr_t>(p.src) | reinterpret_cast<uintptr_t>(p.weights) | reinterpret_cast<uintptr_t>(p.dst)) & 15) return 1;
  if (f16) return trans ? rw_launch<false, true>(p, st, sms) : rw_launch<false, false>(p, st, sms);
  return trans ? rw_launch<true, true>(p, st, sms) : rw_launch<true, false>(p, st, sms);
}

}  // namespace fgms
