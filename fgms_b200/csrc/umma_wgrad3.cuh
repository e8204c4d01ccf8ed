// Weight gradient on tcgen05, warp-specialised with private hand-offs only.
//
//   dw[k] (c_in x c_out, fp32) += sum over the pairs j of offset k of feats[in_map[j]]^T (x) out_grad[out_map[j]]
//
// The pair index is the contraction index: both operands are gathered rows used MN-major.
//   A = feats rows     [pb pairs x c_in ]   M = c_in  (tiles of 128 rows; the last tile has 64 when at most 64 rows remain)
//   B = out_grad rows  [pb pairs x c_out]   N = c_out rounded up to a whole 128-byte piece
// Rows are staged in 128-byte pieces.  A piece that a short row fills only in part, or that exists only to
// complete the last row tile, holds stale shared memory beyond the row: those values reach accumulator rows
// >= c_in and columns >= c_out only, which are never written out.
// One persistent CTA per SM walks a contiguous range of pb-pair stages.  The accumulator stays in TMEM
// while consecutive stages belong to the same offset and is flushed with 16-byte vector reds to the
// fp32 gradient when the offset changes (split-K across CTAs).
//
//   producers (2 teams   the teams take the stages in turn; warp w of a team of four owns rows [w pb/4, (w+1) pb/4) of its team's
//   of 4 warps, or 8)    stages: it fetches those rows' map entries two of them ahead into a ring of its own and gathers both
//                        operands with 16-byte cp.async;
//   MMA warp             one lane issues tcgen05.mma per stage and commits the stage back to the producers;
//                        on a change of offset it commits the accumulator to the epilogue;
//   epilogue (4 warps)   tcgen05.ld -> private 4 KB patch -> reds with consecutive lanes on consecutive
//                        addresses of one gradient row.
// All waits are bounded; a wait that runs out sets the CTA's abort flag and every role leaves its loop; in-flight copies and MMAs
// are awaited before tensor memory is freed.
//
// What bounded it were the producers' instructions: with every copy left out it took as long.  Eight warps went through all
// stages together, tested for each of eight possible pieces of a row whether the row has it, and waited in every stage for
// the map entries they had just asked for.  Straight code for the usual numbers of pieces: 128 -> 128 on 303 k pairs 26.9 -> 20.2
// us in a row of launches; two teams of four that are in different phases of a stage (one copies while the other is at its
// entries and barriers) 18.4, two teams of eight with fewer registers 20.8; the MMA lane's loops 18.0; a commit for every stage
// instead of groups of stages that no shape had more than one in 17.7.  Also 96 -> 160
// on 358 k pairs 43.6 -> 27.7, tf32 64 -> 64 on 296 k 25.6 -> 17.2, tf32 48 -> 64 on 208 k 23.0 -> 13.6, 160 -> 160 on 296 k 40.3 -> 28.5, 64 -> 128 stride 2
// on 9 k 6.9 -> 6.4; 256 -> 256, where a stage is 64 pairs, a CTA has three and the sums' reds are the larger part, 15.1 -> 15.1 (28 k pairs).
// Now a stage of 128 pairs at 128 -> 128 is about 1500 cycles, of which shared memory needs 1024 (64 KB written, read by the MMAs).
#pragma once
#include <type_traits>

#include "common.cuh"
#include "umma.cuh"
#include "umma_gms3.cuh"  // G3Walk, g3_wait

namespace fgms {

constexpr int W3_EPI_WARPS = 4;
constexpr int W3_MMA_WARP = 4;
constexpr int W3_PROD_WARP0 = 5;
constexpr int W3_PROD_WARPS = 4;  // of a team where there are as many as can be: they share a stage
constexpr int W3_PROD_TEAMS = 2;  // at most; they take the stages in turn
// CTAs of up to this many stages have one team of all producers: there the first stage's copies are part of the time.  Two teams /
// one: 256 -> 208 on 12 k pairs, one or two stages a CTA, 14.8 / 14.1 us, 128 -> 128 on 12 k 6.3 / 5.8, tf32 208 -> 144 on 2.9 k 10.0 / 9.6, 224 -> 208 on 6.8 k
// 19.4 / 19.1; two or three: 128 -> 128 on 39 k 8.5 / 8.6, tf32 160 -> 160 on 11 k 14.6 / 14.8, 256 -> 256 on 28 k 15.3 / 15.2; six: 256 -> 256 on 55 k 17.9 / 18.0;
// more: 128 -> 128 on 303 k 18.1 / 21.0.
constexpr int W3_ONE_TEAM_STAGES = 2;
constexpr int W3_THREADS = (W3_PROD_WARP0 + W3_PROD_TEAMS * W3_PROD_WARPS) * 32;
constexpr int W3_MAX_STAGES = 8;
constexpr int W3_MAX_PB = 128;
constexpr int W3_PATCH_BYTES = W3_EPI_WARPS * 4096;
constexpr int W3_PREFETCH = 2;  // map entries are fetched this many of the team's stages ahead
// the producers' rings of map entries: W3_PREFETCH + 1 slots of both entries of every pair of a stage
__host__ __device__ constexpr int w3_ring_bytes(int pb) { return W3_PROD_TEAMS * (W3_PREFETCH + 1) * 2 * 4 * pb; }

struct W3Shared {
  uint64_t full[W3_MAX_STAGES];
  uint64_t empty[W3_MAX_STAGES];
  uint64_t tmem_full[4];
  uint64_t tmem_empty[4];
  uint64_t drained;  // every MMA has finished
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int W3_SHARED_BYTES = (sizeof(W3Shared) + 15) & ~15;

struct W3Config {
  int pb;         // pairs per stage: 32, 64 or 128
  int pack;       // pairs that share one staged row (their rows side by side): 1 or 2
  int slot_a, slot_b;  // packed stages: bytes a pair's row takes in the staged row of A / of B
  int n_mtile;    // 1 or 2 accumulator row tiles: all of 128 rows but possibly the last
  int last_m;     // rows of the last tile's MMA: 128, or 64 when at most 64 rows remain
  int alias;      // 1: the last tile's second piece is its first one read again (descriptor LBO = 0) instead of a
                  //    piece of its own — tf32 with at most 32 rows left: an M = 64 MMA reads two 32-row pieces, only
                  //    one is real, and the rows it repeats land in accumulator rows that are never written out
  int pa, pbp;    // 128-byte pieces per staged row of A (enough for every row tile) and of B (n_acc columns)
  int n_acc;      // TMEM columns of one row tile: c_out rounded up to a whole piece
  int parts_a, parts_b;  // blocks of dW_k, one CTA's each: of c_a input by c_b output channels
  int c_a, c_b;
  int smem;       // dynamic shared memory of the launch
  int n_buf;      // TMEM accumulator sets: 1, 2 or 4
  int buf_shift;  // log2(n_buf)
  int n_stage;
};

// stage t of the table: first pair and number of pairs
__device__ __forceinline__ void w3_stage(const G3Walk& w, int pb, const int* kpos_s, int* base, int* cnt) {
  const int lt = w.t - w.seg_first;
  const int seg_base = kpos_s[w.seg];
  *base = seg_base + lt * pb;
  *cnt = min(pb, kpos_s[w.seg + 1] - seg_base - lt * pb);
}

// FULL: both row lengths are whole 128-byte pieces; the producers' copy loops then carry no per-chunk test.
// PACKED: several pairs share a staged row (cfg.pack > 1); the unpacked instantiations carry none of its arithmetic.
// TEAMS: of producers.  PARTS: several CTAs share dW_k; with one for all of it a row's part is the row, and a kernel that distinguished them all the
// same was 1.5 to 3 % slower for every whole gradient (417 k pairs 128 -> 128 23.1 / 23.4 us, 128 -> 64 19.8 / 20.4, packed with 72 bytes of spills).
template <bool TF32, bool FULL, bool PACKED, int TEAMS, bool PARTS>
__global__ void __launch_bounds__(W3_THREADS, 1) umma_wgrad3_kernel(WgradParams p, W3Config cfg) {
  using namespace umma;
  constexpr int TEAM_WARPS = W3_PROD_TEAMS * W3_PROD_WARPS / TEAMS;
  constexpr int ES = TF32 ? 4 : 2;
  constexpr int UK = 32 / ES;  // contraction length of one MMA
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int pb = cfg.pb, n_stage = cfg.n_stage;
  const int kr = PACKED ? pb / cfg.pack : pb;  // staged rows (contraction steps) per stage
  const uint32_t a_bytes = (uint32_t)kr * 128u * cfg.pa;
  const uint32_t stage_bytes = (uint32_t)kr * 128u * (cfg.pa + cfg.pbp);
  uint8_t* sStage = smem;
  uint8_t* sPatch = sStage + (size_t)n_stage * stage_bytes;
  uint8_t* sRing = sPatch + W3_PATCH_BYTES;
  W3Shared* sh = reinterpret_cast<W3Shared*>(sRing + w3_ring_bytes(pb));
  int* tile_start = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(sh) + W3_SHARED_BYTES);  // [k_vol + 2]
  int* kpos_s = tile_start + p.k_vol + 2;                                                        // [k_vol + 1]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_seg = p.k_vol + 1;
  volatile int* abort_flag = &sh->abort_flag;
  // this CTA's channels of dW_k, and the first ones
  const int c_a = PARTS ? cfg.c_a : p.c_in, c_b = PARTS ? cfg.c_b : p.c_out;
  const int part_a = PARTS ? (int)blockIdx.y % cfg.parts_a : 0;
  const int a0 = part_a * c_a, b0 = PARTS ? ((int)blockIdx.y - part_a) / cfg.parts_a * c_b : 0;
  const uint32_t lbo = (uint32_t)kr * 128u;  // next 128 bytes of every staged row
  const uint32_t buf_cols = (uint32_t)(cfg.n_mtile * cfg.n_acc);

  if (tid == 0) {
    for (int s = 0; s < n_stage; ++s) {
      mbar_init(smem_u32(&sh->full[s]), TEAM_WARPS * 32);  // one hardware arrival per producer thread
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int b = 0; b < 4; ++b) {
      mbar_init(smem_u32(&sh->tmem_full[b]), 1);
      mbar_init(smem_u32(&sh->tmem_empty[b]), W3_EPI_WARPS);
    }
    mbar_init(smem_u32(&sh->drained), 1);
    sh->abort_flag = 0;
    mbar_fence_init();
  }
  // TMEM allocation overlaps the first global loads below
  uint32_t tmem_cols = 32;
  while (tmem_cols < buf_cols * (uint32_t)cfg.n_buf) tmem_cols <<= 1;
  if (warp == W3_MMA_WARP) {
    tmem_alloc(smem_u32(&sh->tmem_base), tmem_cols);
    tmem_relinquish();
  }
  // everything above touches no global memory; from here on the previous kernel's results may be needed
  griddep_begin(0, p.alone);
  build_tile_table(pb, p.kpos, p.pairs, p.k_vol, 0, kpos_s, tile_start);  // syncs the CTA
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;

  int t0, t1;
  cta_tile_range(tile_start[n_seg], &t0, &t1);
  bool ok = true;

  if (t0 >= t1) {
    // nothing for this CTA
  } else if (warp >= W3_PROD_WARP0) {
    // ------------------------------------------------------------------ producers
    const int team = (warp - W3_PROD_WARP0) / TEAM_WARPS, pw = (warp - W3_PROD_WARP0) % TEAM_WARPS;
    const int rpw = pb / TEAM_WARPS;  // rows of a stage owned by this warp: 4, 8, 16 or 32
    const uint8_t* feats = static_cast<const uint8_t*>(p.feats);
    const uint8_t* og = static_cast<const uint8_t*>(p.out_grad);
    const uint32_t a_row_bytes = (uint32_t)c_a * ES, b_row_bytes = (uint32_t)c_b * ES;  // of a row's part
    const uint32_t a_pitch = (uint32_t)p.c_in * ES, b_pitch = (uint32_t)p.c_out * ES;
    // Lane (rs, cc) = (lane / 8, lane % 8) copies 16-byte chunk cc of every 128-byte piece of the rows rs, rs + 4, ... of the warp's
    // block: one shuffle and one address per row, then one cp.async per piece at a fixed distance (128 bytes in global memory,
    // `lbo` in shared memory).
    constexpr int rpp = 4;         // rows per round
    const int n_pass = rpw / rpp;  // rounds per stage: 1 .. 8
    const int rs = lane >> 3, cc = lane & 7;
    const int np_a = ((int)a_row_bytes + 127) / 128, np_b = ((int)b_row_bytes + 127) / 128;  // pieces of a row
    // this lane's chunk exists in the last piece, which a row that is no whole number of pieces fills in part
    const bool tail_a = FULL || (np_a - 1) * 128 + cc * 16 < (int)a_row_bytes;
    const bool tail_b = FULL || (np_b - 1) * 128 + cc * 16 < (int)b_row_bytes;
    // Where the chunk of round u = 0 .. 3 lies in the operand's stage.  Packed stages: pair j sits in staged row j / pack,
    // its rows at byte (j % pack) * slot_a of A and (j % pack) * slot_b of B (a position beyond 128 bytes is a further
    // piece).  Rows 8 apart are 1024 bytes apart in both layouts, so four more rounds are a fixed distance further on.
    const int pack = PACKED ? cfg.pack : 1;
    const uint32_t row0 = (uint32_t)(pw * rpw + rs) / (uint32_t)pack, row_step = (uint32_t)(rpp / pack);
    const uint32_t slot = (uint32_t)((pw * rpw + rs) % pack);
    const uint32_t byte_a = (PACKED ? slot * (uint32_t)cfg.slot_a : 0u) + (uint32_t)cc * 16u;
    const uint32_t byte_b = (PACKED ? slot * (uint32_t)cfg.slot_b : 0u) + (uint32_t)cc * 16u;
    uint32_t rel_a[4], rel_b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t row = row0 + (uint32_t)u * row_step;
      rel_a[u] = TF32 ? mnmajor32_offset(row, byte_a, lbo, 512u) : mnmajor_offset(row, byte_a, lbo, 1024u);
      rel_b[u] = TF32 ? mnmajor32_offset(row, byte_b, lbo, 512u) : mnmajor_offset(row, byte_b, lbo, 1024u);
    }
    const uint32_t four_rounds = row_step * 512u;
    const uint8_t* feats_c = feats + a0 * ES + cc * 16;
    const uint8_t* og_c = og + b0 * ES + cc * 16;
    // The pieces of R rows of one operand.  What this role spends its time on are instructions (with the copies left out
    // the kernel took as long: tests of every one of eight possible pieces and address arithmetic, 400 instructions a
    // warp and stage), so the usual numbers of pieces have their own straight code.  (tf32 rows of 5 to 8 pieces with eight tests / in a loop /
    // so: 240 -> 240 on 268 k pairs 65 / 69 / 57 us, 160 -> 208 on 754 k 138 / 133 / 103, 80 -> 224 stride 2 on 5.8 k 8.5 / 8.9 / 8.4.)
    auto copy_pieces = [&](auto rounds, auto pieces, const uint8_t* const (&from)[4], const uint32_t (&rel)[4], uint32_t to, const uint32_t (&n)[4],
                           bool tail) {
      constexpr int R = decltype(rounds)::value, NP = decltype(pieces)::value;
#pragma unroll
      for (int h = 0; h < NP; ++h)
#pragma unroll
        for (int u = 0; u < R; ++u)
          if (FULL || h + 1 < NP || tail) cp_async16_n(to + (uint32_t)h * lbo + rel[u], from[u] + h * 128, n[u]);
    };
    // rows rs + rpp u of rounds u0 .. u0 + R - 1 of one operand; their entries are in lanes rs + rpp u of `cur`, -1 zero-fills
    auto copy_rows = [&](auto rounds, int u0, int cur, const uint8_t* base, uint32_t row_bytes, const uint32_t (&rel)[4], uint32_t to, int np, bool tail) {
      constexpr int R = decltype(rounds)::value;
      const uint8_t* from[4];
      uint32_t n[4];
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int i = __shfl_sync(0xffffffffu, cur, rs + rpp * (u0 + u));
        n[u] = i >= 0 ? 16u : 0u;  // 0 bytes read: the chunk is zero-filled
        from[u] = base + (size_t)max(i, 0) * row_bytes;
      }
      if (np == 2) copy_pieces(rounds, std::integral_constant<int, 2>(), from, rel, to, n, tail);
      else if (np == 1) copy_pieces(rounds, std::integral_constant<int, 1>(), from, rel, to, n, tail);
      else if (np == 3) copy_pieces(rounds, std::integral_constant<int, 3>(), from, rel, to, n, tail);
      else if (np == 4) copy_pieces(rounds, std::integral_constant<int, 4>(), from, rel, to, n, tail);
      else if constexpr (TF32) {
        if (np == 8) copy_pieces(rounds, std::integral_constant<int, 8>(), from, rel, to, n, tail);
        else if (np == 7) copy_pieces(rounds, std::integral_constant<int, 7>(), from, rel, to, n, tail);
        else if (np == 6) copy_pieces(rounds, std::integral_constant<int, 6>(), from, rel, to, n, tail);
        else copy_pieces(rounds, std::integral_constant<int, 5>(), from, rel, to, n, tail);
      } else {
        // any other number (no fp16 row has one); with nothing here the compiler lays the others out worse: 128 -> 64 on 591 k 23.9 -> 26.9 us,
        // 128 -> 128 on 303 k 17.7 -> 18.7
#pragma unroll 1
        for (int h = 0; h < np; ++h)
#pragma unroll
          for (int u = 0; u < R; ++u)
            if (FULL || h + 1 < np || tail) cp_async16_n(to + (uint32_t)h * lbo + rel[u], from[u] + h * 128, n[u]);
      }
    };
    auto copy_rounds = [&](auto rounds, int u0, int cur_a, int cur_b, uint32_t sa, uint32_t sb) {
      copy_rows(rounds, u0, cur_a, feats_c, a_pitch, rel_a, sa, np_a, tail_a);
      copy_rows(rounds, u0, cur_b, og_c, b_pitch, rel_b, sb, np_b, tail_b);
    };
    // lane r < rpw fetches both map entries of the warp's row r (-1 beyond the stage) into its words of a ring slot: copied
    // there, they are waited for when they are used, where entries handed on through registers were waited for a stage after
    // they had been asked for
    const uint32_t ring = smem_u32(sRing) + (uint32_t)(team * (W3_PREFETCH + 1) * pb + pw * rpw + min(lane, rpw - 1)) * 8u;
    const uint32_t ring_step = (uint32_t)pb * 8u;
    auto fetch_entry = [&](const G3Walk& w, uint32_t slot) {
      int base, cnt;
      w3_stage(w, pb, kpos_s, &base, &cnt);
      const int row = pw * rpw + lane;
      if (lane >= rpw) return;
      if (row < cnt) {
        cp_async4(slot, p.in_map + base + row);
        cp_async4(slot + 4, p.out_map + base + row);
      } else {
        st_shared_i32(slot, -1);
        st_shared_i32(slot + 4, -1);
      }
    };
    G3Walk pf;
    if (t0 + team < t1) pf.init(tile_start, n_seg, t0 + team);
    else pf.t = t1;
    uint32_t put = 0, get = 0;  // slots, in bytes from the ring's start
    auto fetch_next = [&]() {
      if (pf.t < t1) fetch_entry(pf, ring + put);
      cp_async_commit();  // also closes the group of the stage before
#pragma unroll
      for (int i = 0; i < TEAMS; ++i)
        if (pf.t < t1) pf.next(tile_start, n_seg);
      put = put == W3_PREFETCH * ring_step ? 0 : put + ring_step;
    };
    for (int d = 0; d < W3_PREFETCH; ++d) fetch_next();
    // Ring slot and its phase.  Waiting by parity is safe with two teams: a team's stage before, two back, was let in after the one a
    // ring before that had been consumed, and stages are consumed in order, so the barrier is at most one phase behind the one
    // waited for (a ring has at least two slots).
    int s = team;
    uint32_t ph = 0;
    for (int t = t0 + team; t < t1 && ok; t += TEAMS) {
      fetch_next();
      cp_async_wait<W3_PREFETCH>();  // this stage's entries have landed
      int cur_a = -1, cur_b = -1;
      if (lane < rpw) { cur_a = ld_shared_i32(ring + get); cur_b = ld_shared_i32(ring + get + 4); }
      get = get == W3_PREFETCH * ring_step ? 0 : get + ring_step;
      // a pair is used only if both its entries are inside the tensors
      if (!((unsigned)cur_a < (unsigned)p.n_in && (unsigned)cur_b < (unsigned)p.n_out)) {
        if ((!PARTS || blockIdx.y == 0) && (cur_a != -1 || cur_b != -1)) report_problem();  // counted once per skipped pair
        cur_a = cur_b = -1;
      }
      ok = g3_wait(&sh->empty[s], ph ^ 1u, abort_flag);
      if (!ok) break;
      const uint32_t sa = smem_u32(sStage + (size_t)s * stage_bytes);
      const uint32_t sb = sa + a_bytes;
      if (n_pass >= 4) {
        for (int u0 = 0; u0 < n_pass; u0 += 4) copy_rounds(std::integral_constant<int, 4>(), u0, cur_a, cur_b, sa + (uint32_t)(u0 >> 2) * four_rounds, sb + (uint32_t)(u0 >> 2) * four_rounds);
      } else if (n_pass == 2) {
        copy_rounds(std::integral_constant<int, 2>(), 0, cur_a, cur_b, sa, sb);
      } else {
        copy_rounds(std::integral_constant<int, 1>(), 0, cur_a, cur_b, sa, sb);
      }
      // the stage's barrier hears from this thread when everything it has issued so far has landed
      cp_async_arrive_noinc(smem_u32(&sh->full[s]));
      s += TEAMS;
      if (s >= n_stage) { s -= n_stage; ph ^= 1u; }
    }
  } else if (warp == W3_MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t idesc_full = make_idesc(TF32, true, true, 128, cfg.n_acc);
    const uint32_t idesc_last = make_idesc(TF32, true, true, cfg.last_m, cfg.n_acc);
    const uint32_t sbo = TF32 ? 512u : 1024u, ltype = TF32 ? 1u : 2u;
    const uint32_t mtile_stride = (uint32_t)ES * lbo;  // a 128-row tile spans 128 * ES / 128 pieces
    const uint32_t last_lbo = cfg.alias ? 0u : lbo;
    // Descriptors of stage 0 at K step 0 (A: one per row tile); all others differ only in the start-address field
    // (address >> 4, no carry out of it), so the issue loop adds small integers instead of rebuilding them
    const uint32_t stage0 = smem_u32(sStage);
    const uint64_t b_desc0 = make_sdesc(stage0 + a_bytes, lbo, sbo, ltype);
    uint64_t a_desc0[2];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
      a_desc0[mt] = make_sdesc(stage0 + (uint32_t)mt * mtile_stride, mt + 1 == cfg.n_mtile ? last_lbo : lbo, sbo, ltype);
    const int n_ks = kr / UK;  // 2, 4, 8 or 16
    const uint32_t ks_step = (uint32_t)UK * 8u;  // UK contraction rows of 128 bytes, in 16-byte units
    // One lane, named by elect.sync (see elect_one), runs the whole loop — waits, issue, commits — so that no warp-wide
    // hand-shake sits between a stage landing and its MMAs; the other lanes wait at the end.  A loop over the CTA's offsets
    // around one over an offset's stages, whose body has its row tiles and (eight, four or two at a time) its steps written
    // out: tests and branches are what this lane spends its time on.
    auto issue = [&](auto row_tiles, auto steps) -> bool {
      constexpr int MT = decltype(row_tiles)::value, N = decltype(steps)::value;
      const uint32_t idesc0 = MT == 1 ? idesc_last : idesc_full;
      int s = 0, buf = 0;
      uint32_t ph = 0, buf_ph = 1;
      int t = t0, seg = find_segment(tile_start, n_seg, t0);
      while (t < t1) {
        while (t >= tile_start[seg + 1]) ++seg;
        const int run_end = min(t1, tile_start[seg + 1]);
        if (!mbar_wait(smem_u32(&sh->tmem_empty[buf]), buf_ph, abort_flag)) return false;
        tc_fence_after();
        const uint32_t d0 = tmem_base + (uint32_t)buf * buf_cols;
        bool more = false;  // the accumulator holds something
        for (; t < run_end; ++t) {
          if (!mbar_wait(smem_u32(&sh->full[s]), ph, abort_flag)) return false;
          fence_proxy_async();  // the stage was written through cp.async; the MMA reads it through the async proxy
          tc_fence_after();
          uint64_t off = (uint64_t)((uint32_t)s * (stage_bytes >> 4));
          for (int ks = 0; ks < n_ks; ks += N) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
              mma_ss<TF32>(d0, a_desc0[0] + off, b_desc0 + off, idesc0, more || i > 0);
              if (MT == 2) mma_ss<TF32>(d0 + (uint32_t)cfg.n_acc, a_desc0[1] + off, b_desc0 + off, idesc_last, more || i > 0);
              off += ks_step;
            }
            more = true;
          }
          mma_commit(smem_u32(&sh->empty[s]));
          if (++s == n_stage) { s = 0; ph ^= 1u; }
        }
        mma_commit(smem_u32(&sh->tmem_full[buf]));
        if (++buf == cfg.n_buf) { buf = 0; buf_ph ^= 1u; }
      }
      return true;
    };
    if (elect_one()) {
      using One = std::integral_constant<int, 1>;
      using Two = std::integral_constant<int, 2>;
      if (n_ks >= 8) ok = cfg.n_mtile == 1 ? issue(One(), std::integral_constant<int, 8>()) : issue(Two(), std::integral_constant<int, 8>());
      else if (n_ks == 4) ok = cfg.n_mtile == 1 ? issue(One(), std::integral_constant<int, 4>()) : issue(Two(), std::integral_constant<int, 4>());
      else ok = cfg.n_mtile == 1 ? issue(One(), Two()) : issue(Two(), Two());
      mma_drain(smem_u32(&sh->drained));
    }
    __syncwarp();
    ok = __all_sync(0xffffffffu, ok) != 0;
  } else if (warp < W3_EPI_WARPS) {
    // ------------------------------------------------------------------ epilogue (warps 0-3)
    // Thread (warp, lane) holds accumulator row m in its TMEM lane.  32 columns of the warp's 32 rows
    // go through the warp's patch so that eight consecutive lanes add 128 consecutive bytes of one row.
    uint8_t* patch = sPatch + warp * 4096;
    const uint32_t sw7 = (uint32_t)(lane & 7);
    const uint32_t ch = (uint32_t)(lane & 7), rsub = (uint32_t)(lane >> 3);
    // Packed stages: staged row k holds `pack` pairs side by side, in A and in B, so the accumulator is pack x pack
    // blocks of slot_m x slot_n elements of which the diagonal ones are sums over pairs (block (s, s): the pairs in
    // position s) and the others mix two pairs' rows and are dropped.  A warp's rows (32 of a 128-row accumulator,
    // 16 of a 64-row one) lie in one block row; it adds columns [col_base, col_base + c_b) of its rows to gradient
    // rows (row - row_base).  (tf32 with at most 32 staged elements: the 64-row MMA reads them twice, rows 32 .. 63
    // repeat rows 0 .. 31 and are dropped.)
    const int slot_m = PACKED ? cfg.slot_a / ES : 0, slot_n = PACKED ? cfg.slot_b / ES : 0;
    const int warp_row0 = (cfg.last_m == 128 ? 32 : 16) * warp;  // packed stages have one row tile
    const bool blk_ok = !PACKED || warp_row0 < cfg.pack * slot_m;
    const int blk = (PACKED && blk_ok) ? warp_row0 / slot_m : 0;
    const int row_base = blk * slot_m, col_base = blk * slot_n;
    int run_i = 0;
    int t = t0;
    while (t < t1 && ok) {
      const int seg = find_segment(tile_start, n_seg, t);
      t = min(t1, tile_start[seg + 1]);  // this CTA's stages of the offset end here
      const int buf = run_i & (cfg.n_buf - 1);
      const uint32_t use = (uint32_t)run_i >> cfg.buf_shift;
      ok = g3_wait(&sh->tmem_full[buf], use & 1u, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const size_t first = ((size_t)seg * p.c_in + a0) * p.c_out + b0;
      float* dwk = p.dw + first;
      if (!TF32 && p.dw_f16 != nullptr) {
        // fp16 destination: 64 columns (128 bytes of fp16) of the warp's 32 rows per round
        __half* dwk16 = p.dw_f16 + first;
        for (int mt = 0; mt < cfg.n_mtile; ++mt) {
          const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)buf * buf_cols + (uint32_t)(mt * cfg.n_acc);
          const bool m128 = mt + 1 < cfg.n_mtile || cfg.last_m == 128;
          for (int c0 = 0; c0 < c_b; c0 += 64) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // 16 columns at a time: few registers in flight
              uint32_t v[16], h[8];
              if (PACKED && c0 + 16 * q >= slot_n) break;  // the block's columns end here
              tmem_ld16(taddr + col_base + c0 + 16 * q, v);
              tmem_ld_wait();
#pragma unroll
              for (int k = 0; k < 8; ++k) h[k] = pack_half2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
              *reinterpret_cast<uint4*>(patch + lane * 128 + (((uint32_t)(2 * q) ^ sw7) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
              *reinterpret_cast<uint4*>(patch + lane * 128 + (((uint32_t)(2 * q + 1) ^ sw7) << 4)) = make_uint4(h[4], h[5], h[6], h[7]);
            }
            __syncwarp();
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) {
              const uint32_t r = rsub + 4 * u;
              int m;
              if (m128) m = blk_ok ? mt * 128 + warp * 32 + (int)r - row_base : -1;
              else m = (r < 16 && blk_ok) ? mt * 128 + warp * 16 + (int)r - row_base : -1;
              const uint4 v = *reinterpret_cast<const uint4*>(patch + r * 128 + ((ch ^ (r & 7)) << 4));
              if (m >= 0 && m < c_a && c0 + (int)(ch << 3) < c_b) red_add_h8(dwk16 + (size_t)m * p.c_out + c0 + (ch << 3), v.x, v.y, v.z, v.w);
            }
            __syncwarp();
          }
        }
      } else
      for (int mt = 0; mt < cfg.n_mtile; ++mt) {
        const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)buf * buf_cols + (uint32_t)(mt * cfg.n_acc);
        const bool m128 = mt + 1 < cfg.n_mtile || cfg.last_m == 128;
        for (int c0 = 0; c0 < c_b; c0 += 32) {
          uint32_t v0[16], v1[16];
          tmem_ld16(taddr + col_base + c0, v0);
          if (!PACKED || slot_n - c0 > 16) {
            tmem_ld16(taddr + col_base + c0 + 16, v1);
          } else {  // the block has 16 columns: the next ones belong to another block (or to no accumulator at all)
#pragma unroll
            for (int k = 0; k < 16; ++k) v1[k] = 0u;
          }
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            *reinterpret_cast<uint4*>(patch + lane * 128 + (((uint32_t)k ^ sw7) << 4)) = make_uint4(v0[4 * k], v0[4 * k + 1], v0[4 * k + 2], v0[4 * k + 3]);
            *reinterpret_cast<uint4*>(patch + lane * 128 + (((uint32_t)(4 + k) ^ sw7) << 4)) = make_uint4(v1[4 * k], v1[4 * k + 1], v1[4 * k + 2], v1[4 * k + 3]);
          }
          __syncwarp();
#pragma unroll
          for (uint32_t u = 0; u < 8; ++u) {
            const uint32_t r = rsub + 4 * u;  // TMEM lane (within the warp's quarter) whose row this is
            // M = 128: lane r of warp w is row 32 w + r; M = 64: row i lives in lane (i / 16) * 32 + i % 16
            int m;
            if (m128) m = blk_ok ? mt * 128 + warp * 32 + (int)r - row_base : -1;
            else m = (r < 16 && blk_ok) ? mt * 128 + warp * 16 + (int)r - row_base : -1;
            const uint4 v = *reinterpret_cast<const uint4*>(patch + r * 128 + ((ch ^ (r & 7)) << 4));
            if (m >= 0 && m < c_a && c0 + (int)(ch << 2) < c_b)
              red_add_v4(dwk + (size_t)m * p.c_out + c0 + (ch << 2), __uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
          }
          __syncwarp();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->tmem_empty[buf]));
      ++run_i;
    }
  }

  if (!ok && lane == 0) report_problem();
  cp_async_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == W3_MMA_WARP) tmem_dealloc(tmem_base, tmem_cols);
}

// Plan of a launch: accumulator row tiling for c_in, pieces per staged row, stage size and count.  Returns
// false for shapes the kernel does not take or that do not fit `max_smem`; used by the launcher and by the
// kernel-family query alike.
inline bool w3_plan(int c_in, int c_out, int es, int k_vol, int max_smem, W3Config* cfg) {
  if (!umma_supported(c_in, c_out, es)) return false;
  const int epr = 128 / es;  // elements per 128-byte piece
  cfg->parts_a = cfg->parts_b = 1; cfg->c_a = c_in; cfg->c_b = c_out;
  // Packed stages: two pairs share a staged row, their rows side by side in A and in B, so one MMA contracts
  // twice as many pairs — an MMA of 64 x 64 x 16 costs what one of 128 x 128 x 16 does, and with rows of up to
  // 256 bytes the issue loop is what bounds the kernel.  The accumulator then holds 2 x 2 blocks; the epilogue
  // keeps the diagonal.  For rows of more than 64 bytes whose lengths are powers of two, each its own slot, while both fit one
  // 128-row, 256-column accumulator (twice, so that two accumulators alternate) and three packed stages of 128 pairs fit shared
  // memory — else the shape is planned unpacked (second pass of the loop).  (Shorter rows come here only with more pairs
  // than the short-row kernel's positions hold.)
  const int a_row = c_in * es, b_row = c_out * es, max_row = a_row > b_row ? a_row : b_row;
  const bool pow2 = (a_row & (a_row - 1)) == 0 && (b_row & (b_row - 1)) == 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
  cfg->pack = 1; cfg->slot_a = cfg->slot_b = 0;
  if (attempt == 0) {
    if (max_row > 64 && pow2 && 2 * c_in <= 128 && 2 * c_out <= 256) { cfg->pack = 2; cfg->slot_a = a_row; cfg->slot_b = b_row; }
    else continue;
  }
  // rows and columns of the accumulator
  const int m_eff = cfg->pack > 1 ? cfg->pack * cfg->slot_a / es : c_in;
  const int n_eff = cfg->pack > 1 ? cfg->pack * cfg->slot_b / es : c_out;
  cfg->n_mtile = (m_eff + 127) / 128;
  const int rem = m_eff - 128 * (cfg->n_mtile - 1);
  cfg->last_m = rem <= 64 ? 64 : 128;
  cfg->alias = (es == 4 && rem <= 32) ? 1 : 0;
  cfg->pa = (cfg->n_mtile - 1) * es + (cfg->last_m == 128 ? es : es / 2) - cfg->alias;  // a 128-row tile reads 128 / epr = es pieces
  cfg->n_acc = (n_eff + epr - 1) / epr * epr;
  cfg->pbp = cfg->n_acc / epr;
  const int buf_cols = cfg->n_mtile * cfg->n_acc;
  if (buf_cols > 512) { if (cfg->pack > 1) continue; return false; }
  cfg->n_buf = 4 * buf_cols <= 512 ? 4 : (2 * buf_cols <= 512 ? 2 : 1);
  cfg->buf_shift = cfg->n_buf == 4 ? 2 : (cfg->n_buf == 2 ? 1 : 0);
  // pairs per stage: 8, 16 or 32 rows per producer warp (packed stages: always 32, the stage is small)
  int pb = W3_MAX_PB;
  const int fixed = 1024 + W3_PATCH_BYTES + W3_SHARED_BYTES + (((2 * k_vol + 3) * 4 + 15) & ~15);
  const int row_bytes = 128 * (cfg->pa + cfg->pbp) / cfg->pack;  // staged bytes per pair
  // keep at least three stages in flight; a packed stage keeps the producers' round a whole number of staged rows
  while (pb > (cfg->pack > 1 ? 128 : 32) && (max_smem - fixed - w3_ring_bytes(pb)) / (pb * row_bytes) < 3) pb >>= 1;
  int n_stage = (max_smem - fixed - w3_ring_bytes(pb)) / (pb * row_bytes);
  if (n_stage > W3_MAX_STAGES) n_stage = W3_MAX_STAGES;
  if (cfg->pack > 1 && n_stage < 3) continue;  // too large packed: plan it unpacked
  if (n_stage < 2) return false;
  cfg->pb = pb;
  cfg->n_stage = n_stage;
  cfg->smem = fixed + w3_ring_bytes(pb) + n_stage * pb * row_bytes;
  return true;
  }
  return false;
}

// Sides of dW_k longer than 128 channels are halved, each block a CTA's, where a CTA would have few stages: what such a CTA takes its time
// for is the way of the sums of 256 x 256 products, 128 KB of reds behind one another (with one set of accumulators, which fills tensor
// memory, nothing overlaps them), and the halves of rows that are then gathered twice cost less.  Whole / halved, by stages of 128 pairs a CTA
// (t): both sides, fp16 256 x 256 t = 0.4 / 1 / 1.6 / 3 9.0 / 13.9 / 15.8 / 17.8 -> 7.4 / 9.1 / 11.1 / 14.6 us, 160 x 160 t = 1 11.3 -> 9.4, t = 3 14.1 -> 15.4, one
// side only 13.3; t = 9 20.8 -> 24.8; 256 x 256 t = 5.3, one side, 21.2 -> 18.9, t = 11 29.5 -> 30.6; tf32 256 x 256 t = 1 / 3 22.3 / 28.0 -> 12.4 / 20.9.
// One long side: fp16 256 x 64 t = 1 / 3 7.2 / 9.6 -> 6.3 / 9.1, t = 9 15.0 -> 15.9, 128 x 192 (rows of the output side are the longer part of a
// stage) t = 1 7.9 -> 7.5, t = 3 10.1 -> 10.9; tf32 128 x 256 t = 1 / 3 13.2 / 16.9 -> 10.2 / 14.9.  Shorter sides, fp16, where the halves have a CTA each: 128 x
// 128 on 65 stages 5.8 -> 5.2, 96 x 96 on 29 5.8 -> 5.2, tf32 128 x 128 on 65 6.8 -> 7.0.
// The whole plan stays where a half is no multiple of 16 channels.
struct W3Parts {
  int a, b;
  bool operator==(const W3Parts& o) const { return a == o.a && b == o.b; }
};
inline W3Parts w3_parts(int c_in, int c_out, int es, int k_vol, long long pairs, int sms) {
  const double stages = (double)pairs / 128 + 0.5 * k_vol, t = stages / sms;  // (an offset's last stage is half empty on average)
  int a = 1, b = 1;
  if (c_in > 128 && c_out > 128) {
    if (t <= 2.2) a = b = 2;
    else if (t <= (c_in * c_out >= 224 * 256 ? 5.5 : 3.3)) a = 2;
  } else if (c_in > 128) {
    if (t <= 3) a = 2;
  } else if (c_out > 128) {
    if (t <= (es == 2 ? 1.2 : 3)) b = 2;
  } else if (es == 2 && c_in >= 96 && c_out >= 96 && t <= 0.5) {
    b = 2;
  }
  if (c_in % (16 * a)) a = 1;
  if (c_out % (16 * b)) b = 1;
  return {a, b};
}
// the plan of such a block in place of the whole one
inline void w3_split(int c_in, int c_out, int es, int k_vol, long long pairs, int sms, int max_smem, W3Config* cfg) {
  const W3Parts n = w3_parts(c_in, c_out, es, k_vol, pairs, sms);
  W3Config part;
  if (n.a * n.b == 1 || sms < n.a * n.b || !w3_plan(c_in / n.a, c_out / n.b, es, k_vol, max_smem, &part)) return;
  *cfg = part;
  cfg->parts_a = n.a;
  cfg->parts_b = n.b;
}

template <bool TF32, bool FULL, bool PACKED, int TEAMS, bool PARTS>
inline int w3_launch_as(const WgradParams& p, const W3Config& cfg, cudaStream_t st, int sms, int max_smem) {
  static std::atomic<int> granted[64];
  if (int rc = ensure_smem(umma_wgrad3_kernel<TF32, FULL, PACKED, TEAMS, PARTS>, max_smem, granted)) return rc;
  const int parts = cfg.parts_a * cfg.parts_b;
  return launch_pdl(umma_wgrad3_kernel<TF32, FULL, PACKED, TEAMS, PARTS>, dim3((unsigned)(sms / parts), (unsigned)parts), W3_THREADS, (size_t)cfg.smem, st, p, cfg) == cudaSuccess ? 0 : -1;
}
template <bool TF32, bool FULL, bool PACKED, int TEAMS>
inline int w3_launch_parts(const WgradParams& p, const W3Config& cfg, cudaStream_t st, int sms, int max_smem) {
  return cfg.parts_a * cfg.parts_b > 1 ? w3_launch_as<TF32, FULL, PACKED, TEAMS, true>(p, cfg, st, sms, max_smem)
                                       : w3_launch_as<TF32, FULL, PACKED, TEAMS, false>(p, cfg, st, sms, max_smem);
}
template <bool TF32, bool FULL, bool PACKED>
inline int w3_launch_teams(const WgradParams& p, const W3Config& cfg, cudaStream_t st, int sms, int max_smem) {
  const bool few = p.pairs / cfg.pb + p.k_vol / 2 <= W3_ONE_TEAM_STAGES * (sms / (cfg.parts_a * cfg.parts_b));  // (an offset's last stage is half empty on average)
  return few ? w3_launch_parts<TF32, FULL, PACKED, 1>(p, cfg, st, sms, max_smem)
             : w3_launch_parts<TF32, FULL, PACKED, W3_PROD_TEAMS>(p, cfg, st, sms, max_smem);
}
template <bool TF32>
inline int w3_launch(const WgradParams& p, const W3Config& cfg, cudaStream_t st, int sms, int max_smem) {
  const int es = TF32 ? 4 : 2;
  const bool full = (cfg.c_a * es) % 128 == 0 && (cfg.c_b * es) % 128 == 0;
  if (cfg.pack > 1)
    return full ? w3_launch_teams<TF32, true, true>(p, cfg, st, sms, max_smem) : w3_launch_teams<TF32, false, true>(p, cfg, st, sms, max_smem);
  return full ? w3_launch_teams<TF32, true, false>(p, cfg, st, sms, max_smem) : w3_launch_teams<TF32, false, false>(p, cfg, st, sms, max_smem);
}

// 0 launched, 1 the pointers are not 16-byte aligned or the shape has no plan (the caller takes the CUDA-core
// path and counts it), < 0 CUDA error
inline int launch_umma_wgrad3(const WgradParams& p, bool f16, cudaStream_t st, int sms, int max_smem) {
  if ((reinterpret_cast<uintptr_t>(p.feats) | reinterpret_cast<uintptr_t>(p.out_grad) | reinterpret_cast<uintptr_t>(p.dw) | reinterpret_cast<uintptr_t>(p.dw_f16)) & 15) return 1;
  W3Config cfg;
  if (!w3_plan(p.c_in, p.c_out, f16 ? 2 : 4, p.k_vol, max_smem, &cfg)) return 1;
  w3_split(p.c_in, p.c_out, f16 ? 2 : 4, p.k_vol, p.pairs, sms, max_smem, &cfg);
  return f16 ? w3_launch<false>(p, cfg, st, sms, max_smem) : w3_launch<true>(p, cfg, st, sms, max_smem);
}

}  // namespace fgms
