// Output-stationary forward on tcgen05: every output row is produced by ONE accumulator and written once.
//
//   out[r] (=, +=) act( sum_k in[nbr[k][r]] * W[k]  (+ bias) )        for the output rows r of a tile
//
// The scatter form (umma_gms3.cuh, the reference's scheme, backend/fwd_kernels.cuh:130-141) walks the pair list
// offset by offset and adds every pair's product to its output row with an atomic, so an output row receives up
// to k_vol atomics in an order that changes from run to run, and nothing can be applied to the finished row
// inside the kernel.  Here the map is a neighbour table nbr[k][r] (input row of output row r under offset k, -1
// for none; built from the pair list by os_fill_nbr_kernel): a tile is 128 consecutive output rows, its
// accumulator stays in tensor memory while the CTA walks all k_vol offsets, and the epilogue adds the bias, applies ReLU
// and stores the rows — plain stores, the same bits on every run.  Up to eight tiles (as many accumulators as the 512
// tensor-memory columns hold) are walked together, offset by offset, so that a weight matrix is staged once per group of
// tiles and offset.
//
// The price is one 128-row stage per (tile, offset) however few of the tile's rows have a neighbour there: k_vol stages per
// 128 output rows against pairs / 128 stages in the scatter form.  Rows without a neighbour are not copied, and
// tcgen05.mma's output-lane mask leaves their accumulator rows alone: whatever their place in shared memory holds does not
// matter (the accumulators are cleared by the epilogue before the first MMA).
//
// Roles (20 warps): 12 producers, each filling whole stages (16-byte cp.async gathers into the K-major 128-byte-swizzled
// ring), up to three MMA warps, one warp that loads weights by TMA, 4 epilogue warps.  All waits are bounded; all but the MMA
// lanes' are parked (85 -> 79 us on the layer below).
//
// An MMA lane's stage is some 130 instructions one after the other, 540-650 cycles, of which it waits for rows during 95; its four
// MMAs of 128 x 64 x 16 are 192.  So where rows are short enough for it (os_split) the work is dealt to up to three pipelines, each an
// MMA lane with ring slots and producers of its own: tiles of a group, or, where a CTA has fewer than three tiles, offsets, whose
// partial accumulators the epilogue adds in the pipelines' order.  Against one pipeline: 64 -> 64 on a full block of 48^3 (2.9 M
// pairs, 27 stages for each of 864 tiles) 55.8 -> 39.9 us, 390 cycles a stage, of which shared memory needs 320 (rows written, rows
// and weights read by the MMAs); 32 -> 32 52.5 -> 35.1; 64 -> 64 on a surface of 100 k voxels 54.4 -> 38.3, on 30^3 26.5 -> 20.0, on 1000
// voxels 15.0 -> 12.6 (by offsets); 128 -> 128 on 48^3 95 -> 92; 256 -> 256 on 512 voxels, which has one pipeline, 72.2 -> 72.2.
// (With eight warps that each filled 16 rows of every stage and copied zeros the block took 141 us.)
#pragma once
#include "common.cuh"
#include "umma.cuh"
#include "umma_gms3.cuh"  // G3Config / g3_plan (operand and stage sizes), g3_wait, G3_STAGE_BYTES

namespace fgms {

constexpr int OS_EPI_WARPS = 4;
constexpr int OS_MMA_WARP = 4;   // and 12 and 16: one per pipeline, all on one scheduler
constexpr int OS_MAX_PIPES = 3;
// pipeline of an MMA warp (< 0: none)
__device__ __forceinline__ int os_mma_pipe(int warp) { return warp == 4 ? 0 : warp == 12 ? 1 : warp == 16 ? 2 : -1; }
constexpr int OS_W_WARP = 8;
constexpr int OS_PROD_WARPS = 12;
constexpr int OS_THREADS = 640;
// producer of a warp (< 0: none): the warps from 5 on that do not share a scheduler with the MMA warp
__device__ __forceinline__ int os_producer(int warp) { return (warp & 3) && warp > OS_MMA_WARP ? ((warp >> 2) - 1) * 3 + (warp & 3) - 1 : -1; }
constexpr int OS_UNROLL = 4;
constexpr int OS_TILE = 128;
constexpr int OS_MAX_STAGES = 12;
constexpr int OS_MAX_GROUP = 8;  // tiles walked together, an accumulator each

struct OsConfig {
  int n_stage, n_wbuf, w_bytes;
  int n_pipe;  // pipelines: each an MMA warp with producers and n_stage / n_pipe ring slots of its own
  int by_offset;  // 0: the tiles of a group are dealt to the pipelines; 1: the offsets are, every pipeline has an accumulator of
                  // its own for each of the CTA's tiles (which are one group), and the epilogue adds them up
  int n_prod;  // producer warps of a pipeline that work: no more than it has slots (see the producers)
  int kch;     // 128-byte chunks of an input row (= stages of a tile and offset)
  int n_acc;   // tensor-memory columns of an accumulator: whole 128-byte blocks of the output row
  int group;   // tiles walked together
  int smem;
  long long w_limit;  // cycles the MMA lane waits for a weight matrix before it gives up (for anything else: about a second)
};

struct OsParams {
  const void* src;       // [n_in , c_in ]
  const void* weights;   // [k_vol, c_in, c_out]
  void* dst;             // [n_out, c_out]
  const int32_t* nbr;    // [k_vol][nbr_stride]: input row of output row r under offset k, -1 for none
  const void* bias;      // [c_out] in the storage type, or null
  long long nbr_stride;  // entries per offset: n_tiles * 128
  int n_in, n_out, n_tiles;
  int c_in, c_out, k_vol;
  int relu;        // 1: max(x, 0) after the bias
  int accumulate;  // 1: out += result (what the reference's forward does); 0: out = result
  int alone = 0;   // see GmsParams
};

struct OsShared {
  uint64_t full[OS_MAX_STAGES];   // stage landed: 32 hardware arrivals and one after the mask was written
  uint64_t empty[OS_MAX_STAGES];  // stage consumed (tcgen05.commit)
  uint64_t tmem_full[OS_MAX_GROUP];
  uint64_t tmem_empty[OS_MAX_GROUP];  // accumulator read and cleared (one arrival per epilogue warp)
  uint64_t w_full[2 * OS_MAX_PIPES];
  uint64_t w_free[2 * OS_MAX_PIPES];
  uint4 on[OS_MAX_STAGES];  // rows a stage holds, a bit each
  uint64_t drained[OS_MAX_PIPES];  // every MMA of the pipeline has finished
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int OS_SHARED_BYTES = (sizeof(OsShared) + 15) & ~15;

// nbr[k][out_map[j]] = in_map[j] for every pair j of offset k (the table is filled with -1 beforehand).  Every kpos
// entry is clamped to [0, map_len]; a pair with an entry outside the tensors is skipped and counted.
__global__ void os_fill_nbr_kernel(const int32_t* __restrict__ kpos, const int32_t* __restrict__ in_map,
                                   const int32_t* __restrict__ out_map, long long map_len, int n_in, int n_out, int k_vol,
                                   long long stride, int32_t* __restrict__ nbr) {
  extern __shared__ int kp[];  // [k_vol + 1], clamped
  for (int i = threadIdx.x; i <= k_vol; i += blockDim.x) {
    long long v = kpos[i];
    kp[i] = (int)(v < 0 ? 0 : (v > map_len ? map_len : v));
  }
  __syncthreads();
  const long long total = kp[k_vol];
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += (long long)gridDim.x * blockDim.x) {
    int lo = 0, hi = k_vol;  // the offset k with kp[k] <= j < kp[k + 1]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (kp[mid] <= j) lo = mid; else hi = mid;
    }
    const int i = in_map[j], o = out_map[j];
    if ((unsigned)i < (unsigned)n_in && (unsigned)o < (unsigned)n_out) nbr[(long long)lo * stride + o] = i;
    else report_problem();
  }
}

// What is dealt out to the pipelines, known at compile time: by_offset asked at run time cost every stage of the other forms 2-6 %, the
// number of pipelines asked where there is one 2-4 %.  (The offsets' form spills 24 bytes in fp16 and 48 in tf32 at the 96 registers that
// 640 threads leave, the other two none; it is the faster one where it is chosen all the same, see os_split.)
enum { OS_ONE_PIPE, OS_DEAL_TILES, OS_DEAL_OFFSETS };
template <bool TF32, int DEAL = OS_ONE_PIPE>
__global__ void __launch_bounds__(OS_THREADS, 1) umma_osfwd_kernel(OsParams p, OsConfig cfg, const __grid_constant__ CUtensorMap w_map) {
  using namespace umma;
  constexpr int ES = TF32 ? 4 : 2;
  constexpr int EPR = 128 / ES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sW = smem;
  uint8_t* sStage = sW + (size_t)cfg.n_wbuf * cfg.w_bytes;
  uint8_t* sPatch = sStage + (size_t)cfg.n_stage * G3_STAGE_BYTES;
  OsShared* sh = reinterpret_cast<OsShared*>(sPatch + OS_EPI_WARPS * 4096);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kch = cfg.kch, n_pipe = DEAL == OS_ONE_PIPE ? 1 : cfg.n_pipe, n_slot = cfg.n_stage / n_pipe, gsz = cfg.group;  // ring slots of a pipeline
  constexpr bool by_offset = DEAL == OS_DEAL_OFFSETS;
  const int n_part = by_offset ? n_pipe : 1;  // accumulators of a tile
  const int k_bytes = p.c_in * ES;
  volatile int* abort_flag = &sh->abort_flag;

  if (tid == 0) {
    for (int s = 0; s < cfg.n_stage; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 33);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int b = 0; b < OS_MAX_GROUP; ++b) {
      mbar_init(smem_u32(&sh->tmem_full[b]), 1);
      mbar_init(smem_u32(&sh->tmem_empty[b]), OS_EPI_WARPS);
    }
    for (int b = 0; b < 2 * OS_MAX_PIPES; ++b) {
      mbar_init(smem_u32(&sh->w_full[b]), 1);
      mbar_init(smem_u32(&sh->w_free[b]), by_offset ? 1 : n_pipe);
    }
    for (int b = 0; b < OS_MAX_PIPES; ++b) mbar_init(smem_u32(&sh->drained[b]), 1);
    sh->abort_flag = 0;
    mbar_fence_init();
  }
  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)(gsz * n_part * cfg.n_acc)) tmem_cols <<= 1;
  if (warp == OS_MMA_WARP) {
    tmem_alloc(smem_u32(&sh->tmem_base), tmem_cols);
    tmem_relinquish();
  }
  griddep_begin(0, p.alone);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;

  // this CTA's tiles
  int t0, t1;
  cta_tile_range(p.n_tiles, &t0, &t1);
  bool ok = true;
  // Pipeline m has tiles m, m + n_pipe, ... of a group, or offsets m, m + n_pipe, ...; its stages come offset by offset, tile by tile,
  // chunk by chunk.
  auto tiles_of = [&](int tb, int pipe) { return by_offset ? min(gsz, t1 - tb) : (min(gsz, t1 - tb) - pipe + n_pipe - 1) / n_pipe; };
  auto offsets_of = [&](int pipe) { return by_offset ? (p.k_vol - pipe + n_pipe - 1) / n_pipe : p.k_vol; };

  if (t0 >= t1) {
    // nothing for this CTA
  } else if (os_producer(warp) >= n_pipe * cfg.n_prod || os_mma_pipe(warp) >= n_pipe) {
    // more warps than slots, or than pipelines
  } else if (os_producer(warp) >= 0) {
    // ------------------------------------------------------------------ producers
    // Warp w of a pipeline fills its stages w, w + nw, ...  With nw <= n_slot a wait for a ring slot by parity is safe: the warp's stage
    // before, q - nw, was let in after stage q - nw - n_slot had been consumed, stages are consumed in order, and so the slot's
    // barrier is at most one phase behind the one that stage q waits for.  (With more warps than slots it may be two behind,
    // which looks the same, and two warps fill one slot.)  Lane l holds the neighbour entries of the tile's rows l, l + 32,
    // l + 64, l + 96, and copies 16-byte chunk l % 8 of the rows l / 8, l / 8 + 4, ...
    const int pipe = DEAL == OS_ONE_PIPE ? 0 : os_producer(warp) % n_pipe, w = os_producer(warp) / n_pipe, nw = cfg.n_prod;
    const int rs = lane >> 3, pc = lane & 7;
    const uint8_t* src = static_cast<const uint8_t*>(p.src) + pc * 16;
    uint32_t a_dst[2];  // rows rs, rs + 4 of a group of eight
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t r = (uint32_t)(rs + 4 * j);
      a_dst[j] = r * 128u + (((uint32_t)pc ^ r) << 4);
    }
    const uint32_t kch_recip = (65536u + (uint32_t)kch - 1u) / (uint32_t)kch;  // x / kch = x * kch_recip >> 16 for x < 64, kch <= 8
    int s = w, base = 0;  // the warp's next ring slot, stages of the groups before
    uint32_t ph = 0;
    for (int tb = t0; tb < t1 && ok; tb += gsz) {
      // the pipeline's stages of the group: offset k, then r = tile of the pipeline * kch + chunk
      const int per_k = tiles_of(tb, pipe) * kch, n = per_k * offsets_of(pipe);
      if (n == 0) continue;
      const int first = (w + nw - base % nw) % nw;
      const int step_k = nw / per_k, step_r = nw % per_k;
      int k = first / per_k, r = first % per_k;
      auto load_entries = [&](int (&e)[4]) {
        const int g = (int)((uint32_t)r * kch_recip >> 16);
        const int tile = tb + (by_offset ? g : pipe + n_pipe * g), offset = by_offset ? pipe + n_pipe * k : k;
        const int32_t* at = p.nbr + (long long)offset * p.nbr_stride + (long long)tile * OS_TILE + lane;
#pragma unroll
        for (int x = 0; x < 4; ++x) e[x] = __ldg(at + 32 * x);
      };
      int e[4];
      if (first < n) load_entries(e);
      for (int i = first; i < n; i += nw) {
        const int kc = r - (int)((uint32_t)r * kch_recip >> 16) * kch;
        const int slot = pipe * n_slot + s;
        ok = g3_wait(&sh->empty[slot], ph ^ 1u, abort_flag);
        if (!ok) break;
        int ent[4];
        uint32_t on[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const bool good = (unsigned)e[x] < (unsigned)p.n_in;
          if (!good && e[x] != -1 && kc == 0) report_problem();  // outside the tensor: treated as no neighbour, counted
          on[x] = __ballot_sync(0xffffffffu, good);
          ent[x] = good ? e[x] : -1;
        }
        k += step_k; r += step_r;
        if (r >= per_k) { r -= per_k; ++k; }
        const uint32_t st = smem_u32(sStage) + (uint32_t)slot * G3_STAGE_BYTES;
        const uint8_t* from = src + kc * 128;
        // a place whose row has no neighbour keeps what it held: the MMA leaves that accumulator row alone
        const bool pc_ok = kc * 128 + pc * 16 < k_bytes;
#pragma unroll
        for (int x = 0; x < 32; ++x) {
          const int g = __shfl_sync(0xffffffffu, ent[x / 8], (4 * x & 31) + rs);
          if (g >= 0 && pc_ok) cp_async16(st + a_dst[x & 1] + (uint32_t)(x >> 1) * 1024u, from + (size_t)(unsigned)g * (uint32_t)k_bytes, true);
        }
        if (lane == 0) {
          sh->on[slot] = make_uint4(on[0], on[1], on[2], on[3]);
          mbar_arrive(smem_u32(&sh->full[slot]));
        }
        cp_async_arrive_noinc(smem_u32(&sh->full[slot]));
        // behind the copies: asked for ahead of them, the entries were waited for in front of the copies (10-18 % where rows or entries
        // come from memory: tf32 160 -> 96 on 110 k voxels 273 -> 225 us, fp16 192 -> 192 217 -> 195; 64 -> 64 on 30 k 20.0 -> 19.5)
        if (i + nw < n) load_entries(e);
        s += nw;
        if (s >= n_slot) { s -= n_slot; ph ^= 1u; }
      }
      base += n;
    }
  } else if (warp == OS_W_WARP) {
    // ------------------------------------------------------------------ weights: W_k, once per group and offset, a TMA box per
    // 128-byte column block (by one warp with cp.async it bounded wide layers: 128 -> 128 on a full block of 48^3 270 us)
    if (elect_one()) {
      int wb = 0, loads = 0;
      uint32_t w_ph = 0;
      for (int tb = t0; tb < t1 && ok; tb += gsz)
        for (int k = 0; k < p.k_vol; ++k) {
          ok = mbar_parked_wait(smem_u32(&sh->w_free[wb]), w_ph ^ 1u, abort_flag);
          if (!ok) break;
          const uint32_t bar = smem_u32(&sh->w_full[wb]), sw = smem_u32(sW + (size_t)wb * cfg.w_bytes);
          mbar_expect_tx(bar, (uint32_t)cfg.w_bytes);
          for (int b = 0; b * EPR < cfg.n_acc; ++b) tma_load_2d(sw + (uint32_t)(b * p.c_in) * 128u, &w_map, bar, b * EPR, k * p.c_in);
          if (loads < cfg.n_wbuf) ++loads;
          if (++wb == cfg.n_wbuf) { wb = 0; w_ph ^= 1u; }
        }
      // the CTA's shared memory outlives its copies, also after a wait that ran out: the last load of every buffer
      for (; loads > 0; --loads) {
        if (--wb < 0) { wb = cfg.n_wbuf - 1; w_ph ^= 1u; }
        mbar_parked_wait(smem_u32(&sh->w_full[wb]), w_ph, nullptr);
      }
    }
    __syncwarp();
    ok = __all_sync(0xffffffffu, ok) != 0;
  } else if (os_mma_pipe(warp) >= 0) {
    // ------------------------------------------------------------------ MMA issuers
    const uint32_t idesc = make_idesc(TF32, false, true, OS_TILE, cfg.n_acc);
    const int pipe = DEAL == OS_ONE_PIPE ? 0 : os_mma_pipe(warp);
    const uint64_t a_desc0 = make_sdesc(smem_u32(sStage) + (uint32_t)(pipe * n_slot) * G3_STAGE_BYTES, 16u, 1024u);
    const uint64_t b_desc0 = make_sdesc(smem_u32(sW), (uint32_t)p.c_in * 128u, TF32 ? 512u : 1024u, TF32 ? 1u : 2u);
    constexpr uint32_t B_KC = (uint32_t)EPR * 8u, B_KS = (32u / ES) * 8u;  // one 128-byte K chunk / 32-byte MMA step further, in 16-byte units
    // One lane, named by elect.sync (see elect_one), runs the whole loop (waits, issue, commits); the other lanes wait at the
    // end.  A loop over tiles around one over chunks takes 77 us for 64 -> 64 on a full block of 48^3, a flat one 58, with four
    // stages unrolled 56.  A wait that runs out leaves at once and by itself: nothing is issued or committed behind it, so no
    // accumulator whose rows or weights did not land reaches the epilogue, none that it may still be reading is written, and no
    // stage or buffer is handed back that is still being filled (one test of all waits behind a stage's last: 57.5 us).
    if (elect_one()) {
      // accumulators: the tiles' of the pipeline, or every tile's part of it
      const int g_step = n_pipe, w_step = by_offset ? n_pipe : 1;  // (weight buffers are a multiple of the pipelines then)
      int s = 0, wb = by_offset ? pipe : 0, grp = 0, g = pipe, kc = 0;  // ring slot, weight buffer, group; accumulator, chunk of the row
      const int off = pipe * n_slot;
      uint32_t ph = 0, w_ph = 0;
      auto take_weights = [&]() { return mbar_wait(smem_u32(&sh->w_full[wb]), w_ph, abort_flag, cfg.w_limit); };
      auto free_weights = [&]() {
        mma_commit(smem_u32(&sh->w_free[wb]));
        if (by_offset) {
          wb += w_step;
          if (wb >= cfg.n_wbuf) { wb -= cfg.n_wbuf; w_ph ^= 1u; }
        } else if (++wb == cfg.n_wbuf) {
          wb = 0; w_ph ^= 1u;
        }
        g = pipe;
      };
      auto stage = [&](bool first_k, bool last_k) -> bool {
        // first offset of the group: the accumulator must have been read and cleared
        if (first_k && kc == 0 && !mbar_wait(smem_u32(&sh->tmem_empty[g]), (uint32_t)grp & 1u, abort_flag)) return false;
        if (!mbar_wait(smem_u32(&sh->full[off + s]), ph, abort_flag)) return false;
        const uint4 on = sh->on[off + s];
        fence_proxy_async();  // the stage was written through cp.async; the MMA reads it through the async proxy
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(g * cfg.n_acc);
        const uint64_t a_desc = a_desc0 + (uint64_t)((uint32_t)s * (G3_STAGE_BYTES >> 4));
        const uint64_t b_desc = b_desc0 + (uint64_t)((uint32_t)wb * ((uint32_t)cfg.w_bytes >> 4) + (uint32_t)kc * B_KC);
        const int n_ks = min(4, (k_bytes - kc * 128) >> 5);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          if (ks < n_ks)
            mma_ss_masked<TF32>(d_tmem, a_desc + (uint64_t)(ks * 2), b_desc + (uint64_t)((uint32_t)ks * B_KS), idesc, ~on.x, ~on.y, ~on.z, ~on.w);
        mma_commit(smem_u32(&sh->empty[off + s]));
        if (++s == n_slot) { s = 0; ph ^= 1u; }
        if (++kc == kch) {
          if (last_k) mma_commit(smem_u32(&sh->tmem_full[g]));
          kc = 0; g += g_step;
        }
        return true;
      };
      auto all_stages = [&]() -> bool {
        for (int tb = t0; tb < t1; tb += gsz, ++grp) {
          const int per_k = tiles_of(tb, pipe) * kch, n_k = offsets_of(pipe);
          if (per_k == 1) {
            // a single stage per offset: one loop over the offsets (1000 voxels 64 -> 64 15.0 us, 17.7 with a loop inside it)
            for (int k0 = 0; k0 < n_k; k0 += OS_UNROLL) {
#pragma unroll
              for (int u = 0; u < OS_UNROLL; ++u) {
                if (k0 + u >= n_k) break;
                if (!take_weights()) return false;
                if (!stage(k0 + u == 0, k0 + u + 1 == n_k)) return false;
                free_weights();
              }
            }
          } else {
            for (int k = 0; k < n_k; ++k) {
              if (!take_weights()) return false;
              for (int r0 = 0; r0 < per_k; r0 += OS_UNROLL) {
#pragma unroll
                for (int u = 0; u < OS_UNROLL; ++u) {
                  if (r0 + u >= per_k) break;
                  if (!stage(k == 0, k + 1 == n_k)) return false;
                }
              }
              free_weights();
            }
          }
        }
        return true;
      };
      ok = all_stages();
      mma_drain(smem_u32(&sh->drained[pipe]));
    }
    __syncwarp();
    ok = __all_sync(0xffffffffu, ok) != 0;
  } else if (warp < OS_EPI_WARPS) {
    // ------------------------------------------------------------------ epilogue (warps 0-3)
    // Warp q owns TMEM lanes 32 q .. 32 q + 31 = tile rows 32 q + lane.  16 accumulator columns at a time:
    // tcgen05.ld -> bias, ReLU, conversion -> the warp's patch -> eight consecutive lanes write 128 consecutive
    // bytes of one output row.
    const uint32_t row_bytes = (uint32_t)p.c_out * ES;
    constexpr uint32_t BLK_COLS = 128 / ES;
    uint8_t* dst = static_cast<uint8_t*>(p.dst);
    uint8_t* patch = sPatch + warp * 4096;
    const uint32_t sw7 = (uint32_t)(lane & 7);
    const uint32_t ch = (uint32_t)(lane & 7), rsub = (uint32_t)(lane >> 3);
    for (int g = 0; g < min(gsz, t1 - t0) * n_part; ++g)
      for (int c = 0; c < cfg.n_acc; c += 16) tmem_zero16(tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(g * cfg.n_acc + c));
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane < OS_MAX_GROUP) mbar_arrive(smem_u32(&sh->tmem_empty[lane]));
    int grp_i = 0;
    for (int tb = t0; tb < t1 && ok; tb += gsz, ++grp_i) {
      const int gv = min(gsz, t1 - tb);
      for (int g = 0; g < gv && ok; ++g) {
        for (int q = 0; q < n_part && ok; ++q) ok = g3_wait(&sh->tmem_full[g * n_part + q], (uint32_t)grp_i & 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const int row0 = (tb + g) * OS_TILE + 32 * warp;  // output row of this warp's lane 0
        const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(g * n_part * cfg.n_acc);
        for (uint32_t cb = 0; cb < row_bytes; cb += 128) {
          const uint32_t vb = min(128u, row_bytes - cb);  // bytes of this block that belong to the row
          const uint32_t col0 = cb / ES;
#pragma unroll
          for (uint32_t c0 = 0; c0 < BLK_COLS; c0 += 16) {
            if (c0 * ES >= vb) break;  // columns beyond the row (n_acc is the row rounded up to a whole block)
            uint32_t v[16];
            tmem_ld16(taddr + col0 + c0, v);
            tmem_ld_wait();
            tmem_zero16(taddr + col0 + c0);
            float f[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) f[k] = __uint_as_float(v[k]);
            for (int q = 1; q < n_part; ++q) {  // (one group: these accumulators are not used again)
              tmem_ld16(taddr + (uint32_t)(q * cfg.n_acc) + col0 + c0, v);
              tmem_ld_wait();
#pragma unroll
              for (int k = 0; k < 16; ++k) f[k] += __uint_as_float(v[k]);
            }
            if (p.bias != nullptr) {
              if (TF32) {
                const float4* b4 = reinterpret_cast<const float4*>(static_cast<const float*>(p.bias) + col0 + c0);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  const float4 b = __ldg(b4 + k);
                  f[4 * k] += b.x; f[4 * k + 1] += b.y; f[4 * k + 2] += b.z; f[4 * k + 3] += b.w;
                }
              } else {
                const uint4* b4 = reinterpret_cast<const uint4*>(static_cast<const __half*>(p.bias) + col0 + c0);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  const uint4 b = __ldg(b4 + k);
                  const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
                    f[8 * k + 2 * j] += t.x; f[8 * k + 2 * j + 1] += t.y;
                  }
                }
              }
            }
            if (p.relu) {
#pragma unroll
              for (int k = 0; k < 16; ++k) f[k] = fmaxf(f[k], 0.f);
            }
            if (TF32) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                *reinterpret_cast<uint4*>(patch + lane * 128 + (((uint32_t)(c0 / 4 + k) ^ sw7) << 4)) =
                    make_uint4(__float_as_uint(f[4 * k]), __float_as_uint(f[4 * k + 1]), __float_as_uint(f[4 * k + 2]), __float_as_uint(f[4 * k + 3]));
            } else {
              uint32_t h[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) h[k] = pack_half2(f[2 * k], f[2 * k + 1]);
              *reinterpret_cast<uint4*>(patch + lane * 128 + (((c0 / 8) ^ sw7) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
              *reinterpret_cast<uint4*>(patch + lane * 128 + (((c0 / 8 + 1) ^ sw7) << 4)) = make_uint4(h[4], h[5], h[6], h[7]);
            }
          }
          if (cb + 128 >= row_bytes) {
            // accumulator read and cleared: hand it back before the last rows go out
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sh->tmem_empty[g]));
          }
          __syncwarp();
          const bool ch_ok = (ch << 4) < vb;
#pragma unroll
          for (uint32_t u = 0; u < 8; ++u) {
            const uint32_t r = rsub + 4 * u;
            const int orow = row0 + (int)r;
            const uint4 v = *reinterpret_cast<const uint4*>(patch + r * 128 + ((ch ^ (r & 7)) << 4));
            if (orow < p.n_out && ch_ok) {
              uint8_t* o = dst + (size_t)orow * row_bytes + cb + (ch << 4);
              if (!p.accumulate) *reinterpret_cast<uint4*>(o) = v;
              else if (TF32) red_add_v4(reinterpret_cast<float*>(o), __uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
              else red_add_h8(reinterpret_cast<__half*>(o), v.x, v.y, v.z, v.w);
            }
          }
          __syncwarp();
        }
      }
    }
  }

  if (!ok && lane == 0) report_problem();
  cp_async_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == OS_MMA_WARP) tmem_dealloc(tmem_base, tmem_cols);
}

// Shared memory and accumulators of a launch; false: not a shape of this kernel.
inline bool os_plan(int c_in, int c_out, int es, int max_smem, OsConfig* cfg) {
  if (!umma_supported(c_in, c_out, es)) return false;
  const int epr = 128 / es;
  cfg->kch = (c_in * es + 127) / 128;
  cfg->n_acc = (c_out + epr - 1) / epr * epr;
  cfg->w_bytes = c_in * 128 * (cfg->n_acc / epr);
  cfg->group = 512 / cfg->n_acc < OS_MAX_GROUP ? 512 / cfg->n_acc : OS_MAX_GROUP;
  const int fixed = 1024 + OS_EPI_WARPS * 4096 + OS_SHARED_BYTES;
  // two weight buffers if at least four stages still fit beside them
  cfg->n_wbuf = fixed + 2 * cfg->w_bytes + 4 * G3_STAGE_BYTES <= max_smem ? 2 : 1;
  cfg->n_stage = (max_smem - fixed - cfg->n_wbuf * cfg->w_bytes) / G3_STAGE_BYTES;
  if (cfg->n_stage > OS_MAX_STAGES) cfg->n_stage = OS_MAX_STAGES;
  if (cfg->n_stage < 2) return false;
  cfg->n_pipe = 1;
  cfg->by_offset = 0;
  cfg->n_prod = cfg->n_stage < OS_PROD_WARPS ? cfg->n_stage : OS_PROD_WARPS;
  cfg->smem = fixed + cfg->n_wbuf * cfg->w_bytes + cfg->n_stage * G3_STAGE_BYTES;
  cfg->w_limit = umma::WAIT_LIMIT_CYCLES;
  return true;
}

// Cycles between two stages of a CTA's pipelines: what an MMA lane's stage takes, what it takes from asking for a stage's rows to its
// slot being free again (more where a row is long), shared out over the slots of a ring, and what shared memory takes for a stage of every
// pipeline.
inline int os_stage_cycles(int pipes, int n_stage, int kch) {
  const int rows = (kch > 3 ? 3300 : 3100) / (n_stage / pipes), shared = 360 * pipes, lane = 550;
  return rows > shared ? (rows > lane ? rows : lane) : (shared > lane ? shared : lane);
}

// Pipelines for CTAs of up to `tiles` tiles.
//
// A CTA of one tile has its offsets dealt out to three pipelines, if their accumulators fit tensor memory, each has a weight
// buffer, and the rings together hold three rows of the input or nine stages.  (fp16 128 -> 128 on 1000 voxels 22.8 -> 21.2 us, 160 -> 48 25.2 ->
// 20.7, tf32 64 -> 64 22.0 -> 17.5, 128 -> 16 29.0 -> 25.5.  With smaller rings a pipeline waits for its one buffer of weights, or for
// rows: 160 -> 160 30.6 -> 44.8, 256 -> 128 33.4 -> 44.1, 208 -> 64 28.6 -> 30.1, tf32 80 -> 80 26.2 -> 29.9.)  Two weight buffers each, where that takes no slots
// (80 -> 64 16.3 -> 15.0) or the rings then hold six rows: 64 -> 128 16.0 -> 14.8, but tf32 48 -> 48 17.6 -> 18.3; with six rows a CTA of two tiles
// has its offsets dealt out as well (16 -> 16 on 30 k voxels 15.5, by tiles 16.3; 128 -> 64 30.6 / 28.6).  Where the accumulators of two fit, two
// with two buffers each, if rings hold three rows and weights are what it waits for: 48 -> 240 22.0 -> 19.6, 64 -> 208 23.2 -> 21.5, 32 -> 208 (16 KB of
// weights) 19.6 -> 18.9, but 16 -> 208 (8 KB) 18.5 -> 19.0 and with one buffer each 64 -> 208 26.4.
//
// Otherwise tiles are dealt out so that the most loaded pipeline ends first; equally good, three for rows of one 128-byte chunk (fp16
// 16 -> 16 on 100 k voxels, six tiles, with one / two / three 48.5 / 35.2 / 31.6 us), fewer for longer ones (96 -> 96 88.3 / 72.5 / 78.1).  With three
// slots and an odd number of tiles two pipelines lose what they gain: 144 -> 144 on 52 k voxels, three tiles, 75.2 / 83.4, on 100 k 145 / 135; 224 -> 112
// 80.3 / 101.4, on 30 k (two tiles) 56.6 / 58.2; with two slots always (160 -> 160 on 100 k 166 / 190).
inline void os_split(OsConfig* cfg, int tiles, int k_vol, int max_smem) {
  const int other = cfg->smem - cfg->n_wbuf * cfg->w_bytes - cfg->n_stage * G3_STAGE_BYTES;
  auto set = [&](int pipes) {
    const int most = OS_PROD_WARPS / pipes, slots = cfg->n_stage / pipes;
    cfg->n_pipe = pipes;
    cfg->n_prod = slots < most ? slots : most;
  };
  auto stages = [&](int wbufs) {  // that fit beside so many weight buffers
    const int fit = (max_smem - other - wbufs * cfg->w_bytes) / G3_STAGE_BYTES;
    return max_smem - other < wbufs * cfg->w_bytes ? 0 : fit < OS_MAX_STAGES ? fit : OS_MAX_STAGES;
  };
  auto fits = [&](int pipes) { return pipes <= k_vol && tiles * pipes <= OS_MAX_GROUP && tiles * pipes * cfg->n_acc <= 512; };
  int m = 0, each = 0;  // pipelines that offsets are dealt out to, weight buffers of each
  if (tiles < 3 && fits(3)) {
    const int one = stages(3) / 3 * 3, two = stages(6) / 3 * 3;
    if (two >= 6 && two >= 6 * cfg->kch) m = 3, each = 2;
    else if (tiles == 1 && one >= 6 && (one >= 9 || one >= 3 * cfg->kch)) m = 3, each = two == one ? 2 : 1;
  } else if (tiles == 1 && fits(2)) {
    const int two = stages(4) / 2 * 2;
    if (two >= 4 && two >= 3 * cfg->kch && cfg->w_bytes >= 16384) m = 2, each = 2;
  }
  if (m > 0) {
    cfg->by_offset = 1;
    cfg->n_wbuf = each * m;
    cfg->n_stage = stages(cfg->n_wbuf);
    cfg->group = tiles;
    cfg->smem = other + cfg->n_wbuf * cfg->w_bytes + cfg->n_stage * G3_STAGE_BYTES;
    set(m);
    return;
  }
  int pipes = 1;
  long long least = 0;
  for (int n = 1; n <= OS_MAX_PIPES && n <= tiles && n <= cfg->group && cfg->n_stage >= 2 * n; ++n) {
    const int group = cfg->group / n * n, last = tiles % group;
    const long long turns = (long long)(tiles / group) * (group / n) + (last + n - 1) / n, cycles = turns * os_stage_cycles(n, cfg->n_stage, cfg->kch);
    if (n == 1 || cycles < least || (cycles == least && cfg->kch == 1)) pipes = n, least = cycles;
  }
  cfg->group = cfg->group / pipes * pipes;
  set(pipes);
}

template <bool TF32, int DEAL>
inline int os_launch_as(const OsParams& p, const OsConfig& cfg, const CUtensorMap& w_map, int grid, cudaStream_t st, int max_smem) {
  static std::atomic<int> granted[64];
  if (int rc = ensure_smem(umma_osfwd_kernel<TF32, DEAL>, max_smem, granted)) return rc;
  return launch_pdl(umma_osfwd_kernel<TF32, DEAL>, grid, OS_THREADS, (size_t)cfg.smem, st, p, cfg, w_map) == cudaSuccess ? 0 : -1;
}

template <bool TF32>
inline int os_launch(const OsParams& p, const OsConfig& cfg, const CUtensorMap& w_map, int grid, cudaStream_t st, int max_smem) {
  if (cfg.by_offset) return os_launch_as<TF32, OS_DEAL_OFFSETS>(p, cfg, w_map, grid, st, max_smem);
  if (cfg.n_pipe > 1) return os_launch_as<TF32, OS_DEAL_TILES>(p, cfg, w_map, grid, st, max_smem);
  return os_launch_as<TF32, OS_ONE_PIPE>(p, cfg, w_map, grid, st, max_smem);
}

// 0 launched, 1 the shape has no plan or a pointer is not 16-byte aligned (there is no CUDA-core form of this
// kernel: the caller reports it), < 0 CUDA error
inline int launch_umma_osfwd(const OsParams& p, bool f16, cudaStream_t st, int sms, int max_smem) {
  if ((reinterpret_cast<uintptr_t>(p.src) | reinterpret_cast<uintptr_t>(p.weights) | reinterpret_cast<uintptr_t>(p.dst) |
       reinterpret_cast<uintptr_t>(p.bias)) & 15)
    return 1;
  OsConfig cfg;
  G3Config scatter;  // the shapes of the scatter form, no more
  if (!g3_plan(p.c_in, p.c_out, f16 ? 2 : 4, p.k_vol, max_smem, false, &scatter) || !os_plan(p.c_in, p.c_out, f16 ? 2 : 4, max_smem, &cfg)) return 1;
  const int grid = p.n_tiles < sms ? p.n_tiles : sms;
  if (grid <= 0) return 0;
  os_split(&cfg, (p.n_tiles + grid - 1) / grid, p.k_vol, max_smem);
  CUtensorMap w_map;
  if (int rc = weight_tensor_map(&w_map, p.weights, p.k_vol, p.c_in, p.c_out, f16, true)) return rc;
  return f16 ? os_launch<false>(p, cfg, w_map, grid, st, max_smem) : os_launch<true>(p, cfg, w_map, grid, st, max_smem);
}

}  // namespace fgms
