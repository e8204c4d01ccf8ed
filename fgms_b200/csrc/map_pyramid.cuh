// Kernel maps of a whole pyramid of resolutions at once: for every level the 3x3x3 submanifold map, and between two levels
// the 2x2x2 stride-2 map and its transpose.  Same canonical form, bit for bit, as map_builder.cuh.
//
// One map after the other (hash table, dense table of k_vol x voxels, scan, sort of the parents, and the host waiting for
// a count after each) took 1.1 ms for the 13 maps of a 120 k-voxel scene: 170 launches, nine waits, 580 us of kernels.
// A scene's voxels fill a box of a few hundred cells a side, so here every level is a BITMAP of that box:
//
//   * setting a bit inserts a voxel and all its ancestors, and removes duplicates among the ancestors;
//   * the number of set bits before a cell is the voxel's rank in lexicographic order: what the sort was for;
//   * the neighbours of a voxel along z are three bits side by side, so the 27 hash probes are 9 words.
//
// A row's neighbours become one mask of k_vol bits; counting the bits per (offset, block of rows), scanning those counts
// and writing the pairs needs no dense table.  The host waits once, for the sizes of the maps.
//
// The box is limited by the workspace (cells / 8 bytes; the plan says what a larger box needs): a cloud whose box exceeds
// the builder's own limit, a voxel met twice or a coordinate beyond the packable range is left to map_builder.cuh.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "map_builder.cuh"  // COORD_BIAS, align256
#include "umma.cuh"         // launch_pdl, griddep_*

namespace fgms {
namespace pyramid {

constexpr int MAX_LEVELS = 8;             // resolutions
constexpr int MAX_JOBS = 3 * MAX_LEVELS;  // maps
constexpr int THREADS = 256, ROWS = 256;  // rows of a map a block of the last kernel works on
constexpr int WARPS = THREADS / 32;
constexpr int PLAN_THREADS = 1024, PLAN_WARPS = PLAN_THREADS / 32;
constexpr int MAX_BLOCKS = 1024;          // of the planning kernel
enum { SUBM = 1, DOWN = 2, UP = 4 };      // which maps
enum { TOO_LARGE = 1, DUPLICATE = 2, OUT_OF_RANGE = 4 };

struct Level {
  int ox, oy, oz;  // coordinate of cell 0: one below the smallest, so that a neighbour of a voxel is always a cell
  int dy, dzw;     // rows of z per x, words per row of z
  int word0;       // first word of the level (a multiple of 4)
};
// Lives in the workspace, written by the first block.
struct Header {
  int flags;       // what makes the cloud unfit
  int groups;      // groups of 4 words, all levels
  int need;        // words the levels' boxes take, 0x7fffffff where it is more
  int first_group[MAX_LEVELS + 1];
  Level level[MAX_LEVELS];
};
struct Job { int kind, level, k_vol; };  // DOWN / UP: between level and level + 1
// Where the blocks of the jobs begin, and the levels' sizes and ranks.
struct Jobs {
  int base[MAX_LEVELS + 1];       // rank before the level
  int first_block[MAX_JOBS + 1];  // blocks of ROWS rows, job after job
  int rows[MAX_JOBS];
  int first_count[MAX_JOBS];      // of the job's [k_vol][blocks] in counts
};
struct Args {
  const int32_t* coords;       // [n, 3]
  int n, levels, n_jobs;
  Job job[MAX_JOBS];
  Header* head;
  uint32_t* bits;
  int* prefix;                 // [groups + 1] set bits before a group
  int* boxes;                  // [blocks][8] of the planning kernel: smallest coordinates, negated largest ones, whether one is out of range
  int* block_sums;             // [blocks] of the planning kernel
  Jobs* jobs;                  // written with the positions, read by the last kernel
  int* row_of;                 // [n] input row of the voxel of a rank
  uint32_t* mask;              // [n_jobs][n]
  int* counts;                 // per job [k_vol][blocks], job after job, sized for n rows each
  int32_t* kpos;               // [n_jobs][28]
  int32_t* out_coords[MAX_LEVELS];  // level 1 ..: [n, 3]
  int32_t *in_map[MAX_JOBS], *out_map[MAX_JOBS];
  int cap_words;
};
constexpr int KPOS_STRIDE = 28;

__device__ __forceinline__ const int32_t* coords_of(const Args& a, int level) { return level == 0 ? a.coords : a.out_coords[level]; }

// Three bits from cell z on (a cell of the padded row): bit d is cell z + d.
__device__ __forceinline__ uint32_t window(const uint32_t* row, int z) {
  const int w = z >> 5, b = z & 31;
  uint32_t v = row[w] >> b;
  if (b > 29) v |= row[w + 1] << (32 - b);  // cell z + 2 is inside the padded row
  return v & 7u;
}
// set bits of the level before bit b of word w
__device__ __forceinline__ int rank_before(const Args& a, int w, int b, int level_base) {
  const uint4 v = reinterpret_cast<const uint4*>(a.bits)[w >> 2];
  const int i = w & 3;
  const uint32_t mine = i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
  int r = a.prefix[w >> 2] - level_base + __popc(mine & ((1u << b) - 1u));
  if (i > 0) r += __popc(v.x);
  if (i > 1) r += __popc(v.y);
  if (i > 2) r += __popc(v.z);
  return r;
}
__device__ __forceinline__ int row_word(const Level& L, int x, int y) { return L.word0 + ((x - L.ox) * L.dy + (y - L.oy)) * L.dzw; }
__device__ __forceinline__ int rank_of(const Args& a, const Level& L, int base, int x, int y, int z) {
  const int zz = z - L.oz;
  return rank_before(a, row_word(L, x, y) + (zz >> 5), zz & 31, base);
}

// ---- the planning kernel: one block on every SM, all of them resident (a cooperative launch), a barrier of the grid between its steps.
// Eight kernels in a row did this before, each 3.7 us behind the one before it however little it had to do: 46 us for 120 k voxels
// and their coarser levels, with the memset ahead and the copy of the sizes behind 51; now 35 (LiDAR, 250 k voxels in a box of 48 MB of bits, 98).
// Of these the seven barriers take 1.0 to 2.2 us each, the voxels' bits 2.8, their rows 3.8, the masks and counts 4.7 (instructions; 7.2
// with a vote per offset), the positions 3.7 (one block per map: loads side by side; one after the other 7.1); a step is a few
// dependent trips to memory.  With more than a gigabyte of cells memory itself is the bound.
__device__ __forceinline__ int group_count(const Args& a, int g) {
  const uint4 x = reinterpret_cast<const uint4*>(a.bits)[g];
  return __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
}
__device__ __forceinline__ int block_sum(int v, int* part) {  // every thread gets the sum
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  const int s = __reduce_add_sync(0xffffffffu, part[threadIdx.x & 31]);
  __syncthreads();
  return s;
}
__device__ __forceinline__ int warp_scan(int v, int lane) {  // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  return v;
}

// Lane i's bit k to lane k's bit i.  A row's offsets turned into an offset's rows, whose number is one population count: 30
// instructions where a vote per offset takes 135.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t m = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = lane & j ? (x & ~m) | (y >> j & m) : (x & m) | (y & m) << j;
  }
  return x;
}

// which offsets an output row of a map has
__device__ __forceinline__ uint32_t row_mask(const Args& a, const Level* level, const Job& job, int row) {
  uint32_t m = 0;
  if (job.kind == SUBM) {
    const Level& L = level[job.level];
    const int32_t* c = coords_of(a, job.level) + 3 * (size_t)row;
    const int x = c[0], y = c[1], z = c[2] - L.oz - 1;
#pragma unroll
    for (int d = 0; d < 9; ++d) m |= window(a.bits + row_word(L, x + d / 3 - 1, y + d % 3 - 1), z) << (3 * d);
  } else if (job.kind == DOWN) {
    const Level& L = level[job.level];
    const int32_t* c = coords_of(a, job.level + 1) + 3 * (size_t)row;
    // a parent's children may lie outside the box of the finer level by one cell, the padding
    const int x = 2 * c[0], y = 2 * c[1], z = 2 * c[2] - L.oz;
#pragma unroll
    for (int d = 0; d < 4; ++d) m |= (window(a.bits + row_word(L, x + d / 2, y + d % 2), z) & 3u) << (2 * d);
  } else {
    const int32_t* c = coords_of(a, job.level) + 3 * (size_t)row;
    m = 1u << (((c[0] & 1) * 2 + (c[1] & 1)) * 2 + (c[2] & 1));
  }
  return m;
}

__global__ void __launch_bounds__(PLAN_THREADS, 1) plan_kernel(Args a, int* sizes /* [1 + levels + jobs]: flags, voxels, pairs */) {
  const auto grid = cooperative_groups::this_grid();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, me = blockIdx.x, blocks = gridDim.x;
  const int first = me * PLAN_THREADS + tid, all = blocks * PLAN_THREADS;
  __shared__ int part[PLAN_WARPS][32];
  __shared__ Header head;
  __shared__ Jobs jobs;

  // 1: bounding box of a block's voxels
  {
    int m[7] = {0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff, 0};
    for (int i = first; i < a.n; i += all) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int v = a.coords[3 * (size_t)i + d];
        if (v < -maps::COORD_BIAS || v >= maps::COORD_BIAS) m[6] = -1;
        else { m[d] = min(m[d], v); m[3 + d] = min(m[3 + d], -v); }
      }
    }
#pragma unroll
    for (int d = 0; d < 7; ++d) {
      m[d] = __reduce_min_sync(0xffffffffu, m[d]);
      if (lane == 0) part[d][warp] = m[d];
    }
    __syncthreads();
    if (warp < 7) {
      const int v = __reduce_min_sync(0xffffffffu, part[warp][lane]);
      if (lane == 0) a.boxes[8 * me + warp] = v;
    }
  }
  grid.sync();

  // 2: every block lays out the levels, and clears its part of their bitmaps
  {
    if (warp < 7) {
      int v = 0x7fffffff;
      for (int b = lane; b < blocks; b += 32) v = min(v, a.boxes[8 * b + warp]);
      v = __reduce_min_sync(0xffffffffu, v);
      if (lane == 0) part[0][warp] = v;
    }
    __syncthreads();
    if (tid == 0) {
      int flags = part[0][6] < 0 ? OUT_OF_RANGE : 0;
      long long word = 0, need = 0;
      for (int l = 0; l < a.levels; ++l) {
        Level L;
        const int lx = part[0][0] >> l, ly = part[0][1] >> l, lz = part[0][2] >> l;
        const int hx = -part[0][3] >> l, hy = -part[0][4] >> l, hz = -part[0][5] >> l;
        L.ox = lx - 1; L.oy = ly - 1; L.oz = lz - 1;
        L.dy = hy - ly + 3;
        L.dzw = (hz - lz + 3 + 31) / 32;
        L.word0 = (int)word;
        const long long words = ((long long)(hx - lx + 3) * L.dy * L.dzw + 3) & ~3ll;
        need += words;
        word += words;
        if (flags || word > a.cap_words) { flags |= TOO_LARGE; word = 0; }
        head.level[l] = L;
        head.first_group[l + 1] = (int)(word >> 2);
      }
      head.first_group[0] = 0;
      head.groups = (int)(word >> 2);
      head.need = (int)min(need, 0x7fffffffll);
      head.flags = flags;
      if (me == 0) *a.head = head;
    }
    __syncthreads();
    uint4* p = reinterpret_cast<uint4*>(a.bits);
    for (int i = first; i < head.groups; i += all) p[i] = make_uint4(0, 0, 0, 0);
  }
  if (head.flags) {  // the same in every block
    if (first == 0) { sizes[0] = head.flags; sizes[1] = head.need; }
    return;
  }
  grid.sync();

  // 3: voxels and their ancestors
  for (int i0 = first - lane; i0 < a.n; i0 += all) {
    const int i = i0 + lane;
    const uint32_t active = __ballot_sync(0xffffffffu, i < a.n);
    if (i < a.n) {
      const int x = a.coords[3 * (size_t)i], y = a.coords[3 * (size_t)i + 1], z = a.coords[3 * (size_t)i + 2];
      for (int l = 0; l < a.levels; ++l) {
        const Level L = head.level[l];
        const int zz = (z >> l) - L.oz, w = row_word(L, x >> l, y >> l) + (zz >> 5);
        const uint32_t bit = 1u << (zz & 31);
        if (l == 0) {
          if (atomicOr(a.bits + w, bit) & bit) atomicOr(&a.head->flags, DUPLICATE);
        } else {
          // neighbouring rows mostly share an ancestor's word: one atomic for those of a warp (the few hundred words of a
          // coarse level took one per voxel before, 37 us on 120 k voxels)
          const uint32_t same = __match_any_sync(active, w);
          const uint32_t bits = __reduce_or_sync(same, bit);
          if (lane == __ffs(same) - 1 && (*(volatile uint32_t*)(a.bits + w) & bits) != bits) atomicOr(a.bits + w, bits);
        }
      }
    }
  }
  grid.sync();
  {
    const int flags = *(volatile int*)&a.head->flags;
    if (flags) {
      if (first == 0) { sizes[0] = flags; sizes[1] = head.need; }
      return;
    }
  }

  // 4: set bits before every group of 4 words: a block's sum, then its groups from the sum of the blocks before
  const int groups = head.groups, per = (groups + blocks - 1) / blocks;
  const int g0 = min(groups, me * per), g1 = min(groups, g0 + per);
  {
    int c = 0;
    for (int g = g0 + tid; g < g1; g += PLAN_THREADS) c += group_count(a, g);
    const int s = block_sum(c, part[0]);
    if (tid == 0) a.block_sums[me] = s;
  }
  grid.sync();
  {
    int before = 0;
    for (int b = tid; b < me; b += PLAN_THREADS) before += a.block_sums[b];
    before = block_sum(before, part[0]);
    for (int g = g0; g < g1; g += PLAN_THREADS) {
      const int c = g + tid < g1 ? group_count(a, g + tid) : 0;
      const int incl = warp_scan(c, lane);
      if (lane == 31) part[0][warp] = incl;
      __syncthreads();
      const int sums = part[0][lane];
      const int ahead = __reduce_add_sync(0xffffffffu, lane < warp ? sums : 0);
      if (g + tid < g1) a.prefix[g + tid] = before + ahead + incl - c;
      before += __reduce_add_sync(0xffffffffu, sums);
      __syncthreads();
    }
    if (g1 == groups && g0 < g1 && tid == 0) a.prefix[groups] = before;
  }
  grid.sync();

  // 5: rows of every level
  for (int i = first; i < a.n; i += all) {
    const int x = a.coords[3 * (size_t)i], y = a.coords[3 * (size_t)i + 1], z = a.coords[3 * (size_t)i + 2];
    a.row_of[rank_of(a, head.level[0], 0, x, y, z)] = i;
    for (int l = 1; l < a.levels; ++l) {
      const int px = x >> l, py = y >> l, pz = z >> l;
      const int r = rank_of(a, head.level[l], a.prefix[head.first_group[l]], px, py, pz);
      int32_t* o = a.out_coords[l] + 3 * (size_t)r;  // the same value from every voxel below this one
      o[0] = px; o[1] = py; o[2] = pz;
    }
  }
  if (tid <= a.levels) jobs.base[tid] = a.prefix[head.first_group[tid]];
  __syncthreads();
  if (tid == 0) {
    int b = 0, c = 0;
    for (int j = 0; j < a.n_jobs; ++j) {
      const int l = a.job[j].level + (a.job[j].kind == DOWN ? 1 : 0);  // the level of the map's output rows
      jobs.first_block[j] = b;
      jobs.first_count[j] = c;
      jobs.rows[j] = jobs.base[l + 1] - jobs.base[l];
      const int nb = (jobs.rows[j] + ROWS - 1) / ROWS;
      b += nb;
      c += nb * a.job[j].k_vol;
    }
    jobs.first_block[a.n_jobs] = b;
  }
  grid.sync();

  // 6: which offsets a row has, and how many rows of ROWS consecutive ones have each; PLAN_THREADS / ROWS such blocks side by side
  {
    constexpr int SIDE = PLAN_THREADS / ROWS;
    const int side = tid / ROWS, t = tid % ROWS, total = jobs.first_block[a.n_jobs];
    for (int b0 = me * SIDE; b0 < total; b0 += blocks * SIDE) {
      const int blk = b0 + side;
      int j = 0, b = 0, k_vol = 0, mine = 0;
      if (blk < total) {
        while (blk >= jobs.first_block[j + 1]) ++j;
        b = blk - jobs.first_block[j];
        k_vol = a.job[j].k_vol;
        const int row = b * ROWS + t;
        uint32_t m = 0;
        if (row < jobs.rows[j]) {
          m = row_mask(a, head.level, a.job[j], row);
          a.mask[(size_t)j * a.n + row] = m;
        }
        mine = __popc(transpose_bits(m, lane));  // lane k: rows of the warp with offset k
      }
      part[warp][lane] = mine;
      __syncthreads();
      if (blk < total && t < k_vol) {
        int c = 0;
#pragma unroll
        for (int w = 0; w < ROWS / 32; ++w) c += part[side * (ROWS / 32) + w][t];
        a.counts[jobs.first_count[j] + t * (jobs.first_block[j + 1] - jobs.first_block[j]) + b] = c;
      }
      __syncthreads();
    }
  }
  grid.sync();

  // 7: position of every (offset, block of rows) in its map: a block takes a map, a warp an offset
  if (me == 0) {
    if (tid == 0) sizes[0] = 0;
    if (tid < a.levels) sizes[1 + tid] = jobs.base[tid + 1] - jobs.base[tid];
    for (int i = tid; i < (int)(sizeof(Jobs) / 4); i += PLAN_THREADS) reinterpret_cast<int*>(a.jobs)[i] = reinterpret_cast<const int*>(&jobs)[i];
  }
  for (int j = me; j < a.n_jobs; j += blocks) {
    const int nb = jobs.first_block[j + 1] - jobs.first_block[j], k_vol = a.job[j].k_vol;
    int* c = a.counts + jobs.first_count[j] + warp * nb;
    constexpr int BATCH = 16;  // times 32 counts asked for together
    int v[BATCH], sum = 0;
    auto load = [&](int i0) {
#pragma unroll
      for (int u = 0; u < BATCH; ++u) v[u] = i0 + 32 * u + lane < nb ? c[i0 + 32 * u + lane] : 0;
    };
    if (warp < k_vol)
      for (int i0 = 0; i0 < nb; i0 += 32 * BATCH) {
        load(i0);
#pragma unroll
        for (int u = 0; u < BATCH; ++u) sum += v[u];
      }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) part[0][warp] = sum;
    __syncthreads();
    int at = __reduce_add_sync(0xffffffffu, lane < warp ? part[0][lane] : 0);
    if (lane == 0 && warp <= k_vol) a.kpos[j * KPOS_STRIDE + warp] = at;
    if (lane == 0 && warp == k_vol) sizes[1 + a.levels + j] = at;
    if (warp < k_vol)
      for (int i0 = 0; i0 < nb; i0 += 32 * BATCH) {
        if (nb > 32 * BATCH) load(i0);
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
          const int incl = warp_scan(v[u], lane);
          if (i0 + 32 * u + lane < nb) c[i0 + 32 * u + lane] = at + incl - v[u];
          at += __shfl_sync(0xffffffffu, incl, 31);
        }
      }
    __syncthreads();
  }
}

// ---- the pairs ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(THREADS, 4) emit_kernel(Args a) {
  umma::griddep_wait();
  umma::griddep_launch_dependents();
  __shared__ Jobs s;
  __shared__ int part[WARPS][32];  // pairs of the warp per offset, then where they go
  for (int i = threadIdx.x; i < (int)(sizeof(Jobs) / 4); i += THREADS) reinterpret_cast<int*>(&s)[i] = reinterpret_cast<const int*>(a.jobs)[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int blk = blockIdx.x; blk < s.first_block[a.n_jobs]; blk += gridDim.x) {
    int j = 0;
    while (blk >= s.first_block[j + 1]) ++j;
    const Job job = a.job[j];
    const int b = blk - s.first_block[j], row = b * ROWS + (int)threadIdx.x, k_vol = job.k_vol;
    const bool there = row < s.rows[j];
    const uint32_t m = there ? a.mask[(size_t)j * a.n + row] : 0u;
    part[warp][lane] = __popc(transpose_bits(m, lane));
    // input rows: the rank before the first of a column's cells; the cells after it follow in rank
    int first[9];
    if (there) {
      const int32_t* c = coords_of(a, job.level + (job.kind == DOWN ? 1 : 0)) + 3 * (size_t)row;
      if (job.kind == SUBM) {
        const Level L = a.head->level[job.level];
        const int z = c[2] - L.oz - 1;
#pragma unroll
        for (int d = 0; d < 9; ++d)
          if (m >> (3 * d) & 7u) first[d] = rank_before(a, row_word(L, c[0] + d / 3 - 1, c[1] + d % 3 - 1) + (z >> 5), z & 31, s.base[job.level]);
      } else if (job.kind == DOWN) {
        const Level L = a.head->level[job.level];
        const int z = 2 * c[2] - L.oz;
#pragma unroll
        for (int d = 0; d < 4; ++d)
          if (m >> (2 * d) & 3u) first[d] = rank_before(a, row_word(L, 2 * c[0] + d / 2, 2 * c[1] + d % 2) + (z >> 5), z & 31, s.base[job.level]);
      } else {
        first[0] = rank_of(a, a.head->level[job.level + 1], s.base[job.level + 1], c[0] >> 1, c[1] >> 1, c[2] >> 1);
      }
    }
    __syncthreads();
    if ((int)threadIdx.x < k_vol) {
      int at = a.counts[s.first_count[j] + (int)threadIdx.x * (s.first_block[j + 1] - s.first_block[j]) + b];
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const int c = part[w][threadIdx.x];
        part[w][threadIdx.x] = at;
        at += c;
      }
    }
    __syncthreads();
    int32_t *in_map = a.in_map[j], *out_map = a.out_map[j];
    const uint32_t below = (1u << lane) - 1u;
    auto put = [&](int k, int src) {  // the whole warp calls it
      const uint32_t who = __ballot_sync(0xffffffffu, m >> k & 1u);
      if (m >> k & 1u) {
        const int at = part[warp][k] + __popc(who & below);
        in_map[at] = src;
        out_map[at] = row;
      }
    };
    // all of a row's input rows are asked for before the first pair is written: one trip to memory instead of one per offset
    if (job.kind == SUBM) {
      int src[27];
#pragma unroll
      for (int d = 0; d < 9; ++d) {
        int r = first[d];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          const bool on = m >> (3 * d + u) & 1u;
          src[3 * d + u] = on && job.level == 0 ? a.row_of[r] : r;
          r += on ? 1 : 0;
        }
      }
#pragma unroll
      for (int k = 0; k < 27; ++k) put(k, src[k]);
    } else if (job.kind == DOWN) {
      int src[8];
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        int r = first[d];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const bool on = m >> (2 * d + u) & 1u;
          src[2 * d + u] = on && job.level == 0 ? a.row_of[r] : r;
          r += on ? 1 : 0;
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) put(k, src[k]);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) put(k, first[0]);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
struct Plan {
  size_t sizes, jobs, bits, prefix, boxes, block_sums, row_of, mask, counts, total;  // offsets into the workspace (the header is at 0)
  int n_jobs, cap_words;
  Job job[MAX_JOBS];
};
// Words of bitmaps a cloud may have: 64 MB (a 2000 x 2000 x 80 scan and its coarser levels take 55 MB), more for clouds of
// more than 200 k voxels, at most 400 MB.
inline int most_words(int n) {
  const long long want = 80ll * n, least = 16ll << 20, most = 100ll << 20;
  return (int)(want < least ? least : (want > most ? most : want));
}
// What a first attempt makes room for: all of that from 16 k voxels on, in proportion below (300 voxels: 1.2 MB).
inline int first_words(int n) { return (int)(1024ll * n < most_words(n) ? 1024ll * n : most_words(n)); }
// Layout of a workspace with room for `words` words of bitmaps.
inline bool plan(int n, int levels, int what, int words, Plan* p) {
  if (n < 1 || levels < 1 || levels > MAX_LEVELS || (what & ~(SUBM | DOWN | UP)) || !what) return false;
  p->n_jobs = 0;
  for (int kind : {SUBM, DOWN, UP})
    if (what & kind)
      for (int l = 0; l < levels - (kind == SUBM ? 0 : 1); ++l) p->job[p->n_jobs++] = Job{kind, l, kind == SUBM ? 27 : 8};
  if (p->n_jobs == 0) return false;
  p->cap_words = words;
  size_t off = maps::align256(sizeof(Header));
  auto take = [&](size_t bytes) { const size_t at = off; off += maps::align256(bytes); return at; };
  p->sizes = take((1 + MAX_LEVELS + MAX_JOBS) * 4);
  p->jobs = take(sizeof(Jobs));
  p->boxes = take(MAX_BLOCKS * 8 * 4);
  p->block_sums = take(MAX_BLOCKS * 4);
  p->row_of = take((size_t)n * 4);
  p->mask = take((size_t)p->n_jobs * n * 4);
  size_t counts = 0;
  for (int j = 0; j < p->n_jobs; ++j) counts += (size_t)p->job[j].k_vol * (((size_t)n + ROWS - 1) / ROWS);
  p->counts = take(counts * 4);
  p->bits = take(((size_t)words + 64) * 4);
  p->prefix = take(((size_t)words / 4 + 1) * 4);
  p->total = off;
  return true;
}
// The layout of a workspace of `bytes`: as many words as fit (each takes 5 bytes, its share of the prefix included).
// False if that is less than the first attempt's.
inline bool plan_in(int n, int levels, int what, size_t bytes, Plan* p) {
  if (!plan(n, levels, what, 0, p) || bytes < p->total) return false;
  const size_t room = (bytes - p->total) / 5;
  const int words = room < (size_t)most_words(n) ? (int)room & ~63 : most_words(n);
  return words >= (first_words(n) & ~63) && plan(n, levels, what, words, p);
}
// Bytes with which plan_in has room for `words` words: 2 x 256 for the alignment of both arrays, 64 words for the rounding.
inline size_t bytes_for(int n, int levels, int what, int words) {
  Plan p;
  return plan(n, levels, what, 0, &p) ? p.total + ((size_t)words + 64) * 5 + 512 : 0;
}
inline Args arguments(const Plan& p, const int32_t* coords, int n, int levels, int32_t* kpos, int32_t* const* out_coords, uint8_t* ws) {
  Args a = {};
  a.coords = coords; a.n = n; a.levels = levels; a.n_jobs = p.n_jobs;
  for (int j = 0; j < p.n_jobs; ++j) a.job[j] = p.job[j];
  a.head = reinterpret_cast<Header*>(ws);
  a.bits = reinterpret_cast<uint32_t*>(ws + p.bits);
  a.prefix = reinterpret_cast<int*>(ws + p.prefix);
  a.boxes = reinterpret_cast<int*>(ws + p.boxes);
  a.block_sums = reinterpret_cast<int*>(ws + p.block_sums);
  a.jobs = reinterpret_cast<Jobs*>(ws + p.jobs);
  a.row_of = reinterpret_cast<int*>(ws + p.row_of);
  a.mask = reinterpret_cast<uint32_t*>(ws + p.mask);
  a.counts = reinterpret_cast<int*>(ws + p.counts);
  a.kpos = kpos;
  for (int l = 1; l < levels; ++l) a.out_coords[l] = out_coords[l - 1];
  a.cap_words = p.cap_words;
  return a;
}
inline int map_blocks(const Plan& p, int n, int sms) {
  const long long most = (long long)p.n_jobs * ((n + ROWS - 1) / ROWS);
  return (int)(most < 4ll * sms ? most : 4ll * sms);
}
// everything up to the sizes of the maps, which go to `sizes` (device memory, or host memory that the device can write); false on a launch error
inline bool launch_plan(const Args& a, int* sizes, int sms, cudaStream_t st) {
  // a block per SM, and no more than the cloud has work for
  const int want = (a.n + PLAN_THREADS / 4 - 1) / (PLAN_THREADS / 4), most = sms < MAX_BLOCKS ? sms : MAX_BLOCKS;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)(want < most ? want : most));
  lc.blockDim = dim3(PLAN_THREADS);
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, plan_kernel, a, sizes) == cudaSuccess;
}

}  // namespace pyramid
}  // namespace fgms
