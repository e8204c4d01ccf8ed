// Shared device-side pieces of the fgms_b200 kernels: the parameter block, the per-CTA tile
// table derived from `kpos`, bounds-checked map reads and the scatter-add primitives.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fgms {

// Number of problems kernels ran into (map entries out of range that were skipped, bounded
// waits that gave up).  Read and reset from the host through fgms_b200_device_status().
__device__ unsigned long long g_device_problems = 0ull;

__device__ __forceinline__ void report_problem() { atomicAdd(&g_device_problems, 1ull); }

// One gather -> GEMM -> scatter pass.  Forward and dgrad are the same pass with the two maps
// and the two channel counts exchanged and the weight matrix read transposed; the reference
// makes the same observation by passing its maps swapped (backend/spconv.cu:460).
struct GmsParams {
  const void* src;             // [n_gather , k_dim]  rows that are gathered
  const void* weights;         // [k_vol, c_in, c_out]
  void* dst;                   // [n_scatter, n_dim]  rows that are accumulated into
  const int32_t* kpos;         // [k_vol + 1]
  const int32_t* gather_map;   // [pairs]
  const int32_t* scatter_map;  // [pairs]
  int pairs;                   // entries the two maps hold: no position >= pairs is ever read
  int n_gather, n_scatter;
  int k_dim, n_dim;            // contraction width, output width
  int c_in, c_out;             // layout of `weights`
  int k_vol;
  int dense_rows;              // > 0: one more segment of `dense_rows` identity pairs ...
  int dense_weight;            // ... that uses this weight index (the "separate mid" term)
  int beside = 0;              // the kernel ahead in the stream is the weight gradient of the same backward: run beside it (griddep_begin)
  int alone = 0;               // SMs are to stay free: the kernel behind this one in the stream is not let go before this one ends
};

struct WgradParams {
  const void* feats;     // [n_in , c_in ]
  const void* out_grad;  // [n_out, c_out]
  float* dw;             // [k_vol, c_in, c_out] fp32 accumulator
  const int32_t* kpos;
  const int32_t* in_map;
  const int32_t* out_map;
  int pairs;  // entries the two maps hold
  int n_in, n_out, c_in, c_out, k_vol;
  // fp16 storage, tensor-core kernel only: add every CTA's fp32 partial sums, rounded to fp16, straight
  // into the fp16 gradient (dw is then unused)
  __half* dw_f16 = nullptr;
  int alone = 0;  // see GmsParams
};

// ---------------------------------------------------------------------------------------------
// Tile table.  Segment s < k_vol holds the pairs kpos[s] .. kpos[s+1] of kernel offset s; the
// optional last segment holds the identity pairs of the dense centre term.  Every segment is cut
// into tiles of TILE pairs that never straddle two segments — the property the reference gets by
// padding each offset to a multiple of 256 rows on the host (kpos_quantized, cpu-check.py:6-14)
// and searching the padded prefix sums per block (backend/utils.cuh:6-27).  Here each CTA derives
// the table from the unpadded `kpos` itself, so no padded rows are ever scheduled.
// ---------------------------------------------------------------------------------------------
// `kpos` comes from the caller's device memory and is not trusted: every entry is clamped to
// [0, pairs] (pairs = length of the maps) on its way into shared memory, so a stale or mismatched
// kpos can shorten segments but never moves a map read past the end of the maps.  A clamped entry
// is counted as a problem once per launch (`passes` times by a launch that does several passes' work).
__device__ __forceinline__ void build_tile_table(int TILE, const int32_t* __restrict__ kpos, int pairs, int k_vol,
                                                 int dense_rows, int* kpos_s /* [k_vol+1] */,
                                                 int* tile_start /* [k_vol+2] */, int passes = 1) {
  // The first warp does it alone, 32 segments at a time: both ends of a segment are loaded side by side, so the table
  // costs one trip to memory, one scan by shuffles and one barrier (three barriers and a second pass before).
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int carry = 0;
    for (int s0 = 0; s0 <= k_vol; s0 += 32) {
      const int s = s0 + lane;
      int v = 0;
      if (s <= k_vol) {
        const int first = __ldg(kpos + s), next = s < k_vol ? __ldg(kpos + s + 1) : 0;
        const int c = min(max(first, 0), pairs);
        if (first != c && blockIdx.x == 0 && blockIdx.y == 0)
          for (int r = 0; r < passes; ++r) report_problem();
        kpos_s[s] = c;
        const int cnt = s < k_vol ? min(max(next, 0), pairs) - c : dense_rows;
        v = cnt > 0 ? (cnt + TILE - 1) / TILE : 0;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
      }
      if (s <= k_vol) tile_start[s + 1] = v + carry;
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) tile_start[0] = 0;
  }
  __syncthreads();
}

// Segment that owns tile t (tile_start is non-decreasing; empty segments are skipped).
__device__ __forceinline__ int find_segment(const int* tile_start, int n_seg, int t) {
  int lo = 0, hi = n_seg;  // invariant: tile_start[lo] <= t < tile_start[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (tile_start[mid] <= t) lo = mid; else hi = mid;
  }
  return lo;
}

// Contiguous share of `total` tiles for this CTA (of the first row of a grid of two dimensions).
__device__ __forceinline__ void cta_tile_range(int total, int* t0, int* t1) {
  const unsigned g = gridDim.x, b = blockIdx.x;
  if (total <= 0x7fffffff / 1024 && g <= 1024) {  // a 64-bit division is a few hundred cycles
    *t0 = (int)((unsigned)total * b / g);
    *t1 = (int)((unsigned)total * (b + 1) / g);
  } else {
    *t0 = (int)((long long)total * b / g);
    *t1 = (int)((long long)total * (b + 1) / g);
  }
}

// Tiles handed out by turns.  All tiles' turns, offset after offset, are cut into shares of F consecutive ones; worker w
// (a warp or a block) has turns [w F, w F + F).  Without `spread` turns and tiles are the same thing: a worker takes a
// consecutive part of an offset's list.  With it the workers that share an offset step through its list side by side: at
// turn i (counted from the start of a worker's share) the offset's next tiles go to the `full` workers between its first
// and its last, from turn first_i on also to the first one, and until turn last_r also to the last one.  In a canonical
// map (ascending output rows inside an offset) all offsets are then at about the same rows at the same time, and a row is
// read from memory once and found in L2 by the other offsets.
struct Turns {
  int i0, full, first_i, last_r, me;
  // [s0, s1): the offset's turns; t: this worker's first turn inside it
  __host__ __device__ __forceinline__ Turns(int s0, int s1, int share, int worker, int t, bool spread) {
    const int first = s0 / share, last = (s1 - 1) / share;
    full = spread ? last - first - 1 : -1;
    first_i = s0 - first * share;
    last_r = s1 - last * share;
    me = worker - first;
    i0 = full < 0 ? t - s0 : t - worker * share;
  }
  // the offset's tile for this worker's n-th turn inside it
  __host__ __device__ __forceinline__ int tile(int n) const {
    const int i = i0 + n;
    if (full < 0) return i;  // consecutive parts, or the offset lies inside one share
    const int rank = me == 0 ? full : (me <= full ? me - 1 : full + (i >= first_i ? 1 : 0));
    return i * full + max(0, i - first_i) + min(i, last_r) + rank;
  }
};
// Spread when gathered and scattered rows together exceed half of L2 (a row read from both dies is held twice):
// 122 MB of 64-byte rows forward 163 -> 154 us, weight gradient 289 -> 200 us; rows that stay in L2 prefer consecutive
// parts (41 MB of tf32 rows 16.6 against 18.2 us).
inline bool spread_tiles(size_t row_bytes) { return row_bytes > ((size_t)64 << 20); }

// ---------------------------------------------------------------------------------------------
// element helpers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(__half v) { return __half2float(v); }

__device__ __forceinline__ void red_add(float* p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void red_add(__half* p, float v) { atomicAdd(p, __float2half_rn(v)); }

__device__ __forceinline__ void red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void red_add_h8(__half* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("red.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(a), "r"(b), "r"(c),
               "r"(d)
               : "memory");
}

__device__ __forceinline__ void red_add_h4(__half* p, uint32_t a, uint32_t b) {
  asm volatile("red.global.add.noftz.v2.f16x2 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}

// Add v[0..n) to consecutive elements starting at p.  `vec` says that p is suitably aligned for one
// vector red of N elements (16 bytes for four floats, 8 bytes for four halves) — decided once per
// launch from the channel count and the base address.
template <int N>
__device__ __forceinline__ void scatter_add(float* p, const float (&v)[N], int valid, bool vec) {
  if constexpr (N == 4) {
    if (vec && valid == 4) {
      red_add_v4(p, v[0], v[1], v[2], v[3]);
      return;
    }
  }
  {
#pragma unroll
    for (int c = 0; c < N; ++c)
      if (c < valid) red_add(p + c, v[c]);
  }
}
template <int N>
__device__ __forceinline__ void scatter_add(__half* p, const float (&v)[N], int valid, bool vec) {
  if constexpr (N == 4) {
    if (vec && valid == 4) {
      red_add_h4(p, pack_half2(v[0], v[1]), pack_half2(v[2], v[3]));
      return;
    }
  }
  {
#pragma unroll
    for (int c = 0; c < N; ++c)
      if (c < valid) red_add(p + c, v[c]);
  }
}

// Clears [a, a + a_bytes) and [b, b + b_bytes), 16 bytes per store; the buffers start on 16-byte boundaries.  One launch
// for both gradients of a backward (a fill each through PyTorch is 1.4 us on the device and 3 us on the host).
__global__ void __launch_bounds__(256) zero2_kernel(uint8_t* a, size_t a_bytes, uint8_t* b, size_t b_bytes) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // kernels before this one may still use the buffers
  const size_t na = a_bytes >> 4, n = na + (b_bytes >> 4), step = (size_t)gridDim.x * blockDim.x;
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (size_t i = i0; i < n; i += step)
    *reinterpret_cast<uint4*>(i < na ? a + 16 * i : b + 16 * (i - na)) = make_uint4(0, 0, 0, 0);
  if (i0 < (a_bytes & 15)) a[(na << 4) + i0] = 0;
  if (i0 < (b_bytes & 15)) b[(b_bytes & ~(size_t)15) + i0] = 0;
}

// Clears up to ZERO_LIST buffers, 16 bytes per store, each from a 16-byte boundary: the gradients of a whole stack of layers in one
// launch.  A block clears parts of ZERO_PART bytes of the buffers laid end to end, so that many small ones cost no more than one.
constexpr int ZERO_LIST = 64;
constexpr unsigned ZERO_PART = 16384;
struct ZeroList {
  uint8_t* at[ZERO_LIST];
  size_t bytes[ZERO_LIST];
  unsigned first_part[ZERO_LIST + 1];  // parts before a buffer
  int n;
};
__global__ void __launch_bounds__(256) zero_list_kernel(const __grid_constant__ ZeroList z) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int i = 0;
  for (unsigned part = blockIdx.x; part < z.first_part[z.n]; part += gridDim.x) {
    while (part >= z.first_part[i + 1]) ++i;
    const size_t from = (size_t)(part - z.first_part[i]) * ZERO_PART, bytes = min((size_t)ZERO_PART, z.bytes[i] - from);
    uint8_t* at = z.at[i] + from;
    for (unsigned b = threadIdx.x * 16; b + 16 <= bytes; b += 256 * 16) *reinterpret_cast<uint4*>(at + b) = make_uint4(0, 0, 0, 0);
    if (threadIdx.x < (bytes & 15)) at[(bytes & ~(size_t)15) + threadIdx.x] = 0;
  }
}

// y += x, in fp16 each sum rounded once: the skip connections of a stack and their gradients.  Both start on 16-byte boundaries.
template <bool F16>
__global__ void __launch_bounds__(256) add_kernel(uint8_t* y, const uint8_t* x, long long count) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  constexpr int PER = F16 ? 8 : 4;
  const long long n = count / PER, step = (long long)gridDim.x * blockDim.x, i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long i = i0; i < n; i += step) {
    uint4 a = reinterpret_cast<uint4*>(y)[i];
    const uint4 b = reinterpret_cast<const uint4*>(x)[i];
    auto sum = [](uint32_t u, uint32_t v) {
      if (F16) {
        const __half2 s = __hadd2(*reinterpret_cast<__half2*>(&u), *reinterpret_cast<__half2*>(&v));
        return *reinterpret_cast<const uint32_t*>(&s);
      }
      return __float_as_uint(__uint_as_float(u) + __uint_as_float(v));
    };
    a = make_uint4(sum(a.x, b.x), sum(a.y, b.y), sum(a.z, b.z), sum(a.w, b.w));
    reinterpret_cast<uint4*>(y)[i] = a;
  }
  const long long rest = n * PER + i0;
  if (rest < count) {
    if (F16) reinterpret_cast<__half*>(y)[rest] = __hadd(reinterpret_cast<__half*>(y)[rest], reinterpret_cast<const __half*>(x)[rest]);
    else reinterpret_cast<float*>(y)[rest] += reinterpret_cast<const float*>(x)[rest];
  }
}

// The first `len` values of `rows` rows from one pitch to another, fp32 rounded to fp16 on the way where the types differ: rows padded
// to a width that the tensor-core kernels take, and gradients without the padding.
template <typename From>
__global__ void __launch_bounds__(256) copy_rows_kernel(const From* src, long long src_pitch, __half* dst, long long dst_pitch, long long rows, int len) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const long long count = rows * len, step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += step) {
    const long long r = i / len, c = i - r * len;
    dst[r * dst_pitch + c] = __float2half_rn((float)src[r * src_pitch + c]);
  }
}

}  // namespace fgms
