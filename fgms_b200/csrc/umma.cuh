// Thin wrappers over the sm_100a PTX this library uses: mbarriers, cp.async, the async-proxy
// fence, and tcgen05 (tensor-memory allocation, UMMA issue/commit, tensor-memory loads), plus the
// shared-memory and instruction descriptors of tcgen05.mma and the 128-byte-swizzled canonical
// operand layouts.  All waits are bounded: a wait that runs out returns false and the caller
// reports it instead of spinning forever.
#pragma once
#include <atomic>
#include <mutex>

#include <cuda.h>  // CUtensorMap; its encoder is looked up at run time
#include <cuda_runtime.h>
#include <stdint.h>

namespace fgms {
namespace umma {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// one arrival, and `bytes` more for TMA copies to report
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// box of a 2-D tensor map at (x, y), into shared memory; reports its bytes to `bar`
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
               "l"(map), "r"(bar), "r"(x), "r"(y)
               : "memory");
}
// One non-blocking probe of the barrier.  The MMA lanes poll with it: every stage passes through them, and a thread that
// mbarrier.try_wait has parked wakes up late.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same, but the thread may be parked until the phase completes or a time limit of the hardware's own runs out.  All other
// roles wait with it: they are ahead of the MMA lane or wide, and parked they leave it its issue slots.
__device__ __forceinline__ bool mbar_park(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after about one second of SM clock, or `limit` cycles of it.  `abort_flag` (shared memory) lets one
// role tell the others to stop waiting once something has gone wrong.
constexpr long long WAIT_LIMIT_CYCLES = 2000000000ll;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, long long limit = WAIT_LIMIT_CYCLES) {
  if (mbar_test(bar, parity)) return true;
  const long long start = clock64();
  for (uint32_t it = 1;; ++it) {
    if (mbar_test(bar, parity)) return true;
    if ((it & 255u) == 0) {
      if (abort_flag && *abort_flag) return false;
      if (clock64() - start > limit) break;
    }
  }
  if (abort_flag) *abort_flag = 1;
  return false;
}

// The bounded wait that parks.
__device__ __forceinline__ bool mbar_parked_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_test(bar, parity)) return true;
  const long long start = clock64();
  while (!mbar_park(bar, parity)) {
    if (abort_flag && *abort_flag) return false;
    if (clock64() - start > WAIT_LIMIT_CYCLES) {
      if (abort_flag) *abort_flag = 1;
      return false;
    }
  }
  return true;
}

// ------------------------------------------------------------------ programmatic dependent launch
// A kernel launched with the programmatic-stream-serialization attribute may start while the kernel before
// it in the stream is still running.  griddep_wait() returns once that kernel has finished and its writes
// are visible: nothing it may have written (or may still read and this kernel overwrites) is touched
// before the call.  griddep_launch_dependents() lets the next such kernel in the stream start its own
// preamble as soon as this grid's CTAs make room, also on SMs that this grid has left free: where those are meant for a kernel
// of another stream it is left out (`alone`).  Both do nothing in a kernel launched the plain way.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// A kernel that neither reads nor overwrites what the kernel ahead of it in the stream writes or reads may run beside it: instead of
// waiting at its start it waits before it ends.  The one ahead lets it go (griddep_launch_dependents) behind its own wait in every
// CTA, so all that came earlier has finished and is in memory; the fence keeps this SM from answering out of what it held before
// that.  It orders the thread's own loads only: a thread that has TMA read global memory puts fence_proxy_async_global() ahead.
// Whoever waits for this kernel thereby waits for both.  All threads call griddep_begin and griddep_end.  (The input
// gradient alone pays for asking: 40 ns a launch.  The forward does not ask: by asking it lost as much, 16 -> 16 on 14 k pairs 3.04 -> 3.08 us.)
__device__ __forceinline__ void griddep_begin(bool beside, bool alone) {
  if (beside) asm volatile("fence.acq_rel.gpu;" ::: "memory");
  else griddep_wait();
  if (!alone) griddep_launch_dependents();
}
__device__ __forceinline__ void griddep_end(bool beside) {
  if (beside) griddep_wait();
}
// what this thread may read of global memory, its TMA copies behind the fence may read too
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// ------------------------------------------------------------------ cp.async (16-byte, zero fill)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const uint32_t n = valid ? 16u : 0u;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
// same with the number of bytes to read (16, or 0 for a zero-filled chunk) already in a register
__device__ __forceinline__ void cp_async16_n(uint32_t dst, const void* src, uint32_t n) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
// 4-byte copy (goes through L1): used to prefetch map entries into shared memory without tying up a register
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void st_shared_i32(uint32_t dst, int v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst), "r"(v) : "memory"); }
__device__ __forceinline__ int ld_shared_i32(uint32_t src) {
  int v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(src) : "memory");
  return v;
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// the mbarrier receives one arrival from this thread once all cp.async it has issued so far have landed
// (.noinc: the arrival counts against the barrier's expected count like an ordinary arrive)
__device__ __forceinline__ void cp_async_arrive_noinc(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// make generic-proxy / cp.async writes to shared memory visible to the async proxy (tcgen05.mma)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ------------------------------------------------------------------ tcgen05
// whole warp; ncols a power of two in [32, 512]; the base address lands in *smem_dst
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// True in one lane of the (converged) warp.  tcgen05 instructions are issued by the lane that elect.sync names: the compiler
// then knows that one thread runs the code.  Behind a plain `lane == 0` it does not, and every tcgen05.mma and commit costs
// more issue slots: 128 x 64 x 16 back to back 56.8 cycles each against 48 (N = 32: 56.8 / 40, the tensor pipe's own time),
// with a commit after every four 87 against 49; in a kernel whose other warps compete for those slots it was 144 an MMA.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
  return ok != 0;
}

// D[tmem] (+)= A[smem] * B[smem]; one thread issues
template <bool TF32>
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  if (TF32) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc)
        : "memory");
  }
}
// accumulating, except into the accumulator rows whose bit of off0 .. off3 is set (row = tensor-memory lane)
template <bool TF32>
__device__ __forceinline__ void mma_ss_masked(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t off0, uint32_t off1,
                                              uint32_t off2, uint32_t off3) {
  if (TF32) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%4, %5, %6, %7}, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(off0), "r"(off1), "r"(off2), "r"(off3)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%4, %5, %6, %7}, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(off0), "r"(off1), "r"(off2), "r"(off3)
        : "memory");
  }
}
// arrive on an mbarrier once every tcgen05.mma issued so far by this thread has finished
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 lanes x 32-bit, 16 consecutive columns: thread t of the warp reads lane (warp%4)*32 + t
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
// zeros to 16 consecutive columns of the warp's 32 lanes
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(0u) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// the issuing lane, behind its last MMA: returns when the tensor cores are done with shared and tensor memory, whatever became
// of the roles that would have waited for it (a barrier of its own, in its first phase)
__device__ __forceinline__ void mma_drain(uint32_t bar) {
  mma_commit(bar);
  mbar_wait(bar, 0u, nullptr);
}

// ------------------------------------------------------------------ descriptors
// Instruction descriptor of tcgen05.mma kind::f16 / kind::tf32 with fp32 accumulation:
//   [4,6) D format (1 = f32)   [7,10) A format   [10,13) B format  (0 = f16, 2 = tf32)
//   [15] A major  [16] B major (0 = K-major, 1 = MN-major)   [17,23) N >> 3   [24,29) M >> 4
__host__ __device__ constexpr uint32_t make_idesc(bool tf32, bool a_mn_major, bool b_mn_major, int m, int n) {
  return (1u << 4) | ((tf32 ? 2u : 0u) << 7) | ((tf32 ? 2u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Shared-memory matrix descriptor, 128-byte swizzle:
//   [0,14) start address >> 4   [16,30) leading byte offset >> 4   [32,46) stride byte offset >> 4
//   [46,48) version = 1 (sm_100)   [61,64) layout type = 2 (SWIZZLE_128B)
__device__ __forceinline__ uint64_t make_sdesc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes,
                                              uint32_t layout_type = 2) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)layout_type << 61;
  return d;
}

// Canonical 128-byte-swizzled operand layouts (tile bases are 1024-byte aligned).
//
// K-major (the contraction index is contiguous in a row): a tile of R rows is stored as sub-tiles of
// [R rows x 128 bytes]; inside a sub-tile rows are 128 bytes apart, groups of 8 rows 1024 bytes apart
// (the stride byte offset), and the 16-byte chunk c of row r sits at chunk position c ^ (r % 8).
// One MMA consumes 32 bytes of every row: advancing the start address by 32 selects the next K step.
//
// MN-major (the M or N index is contiguous in a row, one row per contraction index k): rows of
// [128 bytes] are grouped in atoms of 8 consecutive k (1024 bytes); atoms that follow each other in k
// are `sbo` bytes apart, atoms that follow each other along M/N (the next 128 bytes of every row) are
// `lbo` bytes apart; chunk c of row k sits at c ^ (k % 8).
__host__ __device__ constexpr uint32_t mnmajor_offset(uint32_t k, uint32_t byte_in_row, uint32_t lbo, uint32_t sbo) {
  return (byte_in_row >> 7) * lbo + (k >> 3) * sbo + (k & 7u) * 128u +
         ((((byte_in_row >> 4) & 7u) ^ (k & 7u)) << 4) + (byte_in_row & 15u);
}

// MN-major for 32-bit elements (tf32) has its own layout, "128-byte swizzle with 32-byte atomicity"
// (descriptor layout type 1): atoms are 4 consecutive k (512 bytes), and the 32-byte chunk q of row k
// sits at chunk position q ^ (k % 4).  `sbo` is the distance between atoms that follow each other in k.
__host__ __device__ constexpr uint32_t mnmajor32_offset(uint32_t k, uint32_t byte_in_row, uint32_t lbo, uint32_t sbo) {
  return (byte_in_row >> 7) * lbo + (k >> 2) * sbo + (k & 3u) * 128u +
         ((((byte_in_row >> 5) & 3u) ^ (k & 3u)) << 5) + (byte_in_row & 31u);
}

}  // namespace umma

// Tensor map over weights [k_vol, c_in, c_out] whose box is `box_rows` rows of one 128-byte column block (0: all c_in of a matrix): what tma_load_2d writes, block after block box_rows * 128 bytes apart, is the 128-byte-swizzled operand: MN-major (forward: rows = contraction index) or
// K-major (input gradient: rows = output index), which differ only for 32-bit elements.  Columns beyond c_out come as zeros.
// Made for every call (42 ns): nothing is kept by an address.  The encoder wants a context, which a host thread has after its first
// launch and not after cudaGetDevice: where it finds none, the current device's is made the thread's and the encoder asked again.
// Returns 0, or -1000 less the driver's status.  An encoder that was not found is looked up again by the next call.
inline int weight_tensor_map(CUtensorMap* map, const void* weights, int k_vol, int c_in, int c_out, bool f16, bool mn_major, int box_rows = 0) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static std::atomic<Encode> known{nullptr};
  Encode encode = known.load(std::memory_order_acquire);
  if (encode == nullptr) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found);
    if (e != cudaSuccess || found != cudaDriverEntryPointSuccess || fn == nullptr) return -1000 - (int)CUDA_ERROR_NOT_FOUND;
    encode = reinterpret_cast<Encode>(fn);
    known.store(encode, std::memory_order_release);
  }
  const int es = f16 ? 2 : 4;
  const cuuint64_t dims[2] = {(cuuint64_t)c_out, (cuuint64_t)k_vol * c_in}, pitch[1] = {(cuuint64_t)c_out * es};
  const cuuint32_t box[2] = {(cuuint32_t)(128 / es), (cuuint32_t)(box_rows > 0 ? box_rows : c_in)}, steps[2] = {1, 1};
  auto made = [&] {
    return encode(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(weights), dims, pitch, box, steps,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, f16 || !mn_major ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult rc = made();
  if (rc == CUDA_ERROR_INVALID_CONTEXT) {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) rc = made();
  }
  return rc == CUDA_SUCCESS ? 0 : -1000 - (int)rc;
}

// Launch with the programmatic-stream-serialization attribute.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = grid;
  lc.blockDim = dim3((unsigned)block);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, kernel, static_cast<KArgs>(args)...);
}

// The dynamic shared memory a kernel may be launched with, raised when a launch needs more than any before it on its
// device; `granted` remembers it (any thread may call).  Looking, setting and writing down are one step: of two threads
// that ask for different sizes the smaller would otherwise be set last and the larger written down, and every later
// launch of the larger size would fail.
template <typename K>
inline int ensure_smem(K kernel, int bytes, std::atomic<int>* granted /* [64], by device */) {
  static std::mutex raising;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (granted[dev].load(std::memory_order_acquire) >= bytes) return 0;
  std::lock_guard<std::mutex> lock(raising);
  if (granted[dev].load(std::memory_order_relaxed) >= bytes) return 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return -1;
  granted[dev].store(bytes, std::memory_order_release);
  return 0;
}
}  // namespace fgms
