// Shared helpers for the sm_100a kernels of axonn_b200: error reporting to the
// ctypes caller, bounded waits, and thin wrappers over the PTX used by several
// kernels (mbarrier, TMA, tcgen05, peer-memory loads/stores).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "axonn_b200.h"

namespace axb {

// ----------------------------------------------------------------------------- host error state
void set_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);
// Cap on the CTAs of GEMM launches (axb_gemm_set_max_ctas), 0: none.
int max_ctas();
// Per-device word that kernels set when a bounded wait expires (0 = clean).
// Lives in mapped pinned host memory so the host can read it without a sync.
volatile unsigned int* device_status_word(int device, unsigned int** dev_ptr);
// Deadline of every device-side wait in nanoseconds (default 120 s; axb_set_wait_timeout_ms changes it).
unsigned long long wait_timeout_ns();
// Number of SMs of `device` (cached); sm_count_current() asks for the calling thread's current device.
int sm_count(int device);
int sm_count_current();

// Ablation switches of the kernels (timing experiments) exist only in builds with -DAXB_ABLATION; in the
// shipped library AXB_DBG is the constant 0, so the branches and the probe words vanish at compile time.
#ifdef AXB_ABLATION
#define AXB_DBG(p, bit) (((p).debug & (bit)) != 0)
#else
#define AXB_DBG(p, bit) (false)
#endif

#define AXB_CUDA(call)                                   \
  do {                                                   \
    if (::axb::check_cuda((call), #call)) return -1;     \
  } while (0)

// ----------------------------------------------------------------------------- device PTX wrappers
#ifdef __CUDACC__

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}

// Bounded wait on an mbarrier phase.  Returns false when `abort_flag` (shared
// memory) is raised by another thread or the deadline passes; in the latter
// case it raises `abort_flag` itself.  No wait in this library is unbounded.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          uint64_t timeout_ns) {
  uint32_t ok;
  uint64_t start = 0;
  for (uint32_t it = 0;; ++it) {
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if ((it & 0xff) == 0xff) {
      if (*abort_flag) return false;
      uint64_t now = globaltimer_ns();
      if (start == 0) start = now;
      else if (now - start > timeout_ns) { *abort_flag = 1; return false; }
    }
  }
}

// Record why a bounded wait gave up.  The first reason stays: later writers (warps that only notice the
// abort flag of the first one) do not overwrite it.
__device__ __forceinline__ void report_status(unsigned int* status, unsigned int code) {
  volatile unsigned int* w = reinterpret_cast<volatile unsigned int*>(status);
  if (*w == 0u) *w = code;
}

// Debug builds (-DAXB_DEBUG_BOUNDS, `python axonn_b200/utils/build.py --debug-bounds`): every store that a kernel
// makes into peer memory or through a computed index is checked against the extent of its target first; a
// violation is recorded (status code + the offending byte offset in diagnostic words 14 / 15) and the access is
// skipped instead of being made.  In the shipped library the check is the constant `true`.
#ifdef AXB_DEBUG_BOUNDS
__device__ __forceinline__ bool in_range_or_report(unsigned int* status, unsigned long long offset, unsigned long long bytes,
                                                   unsigned long long extent, unsigned int code) {
  if (offset + bytes <= extent) return true;
  report_status(status, code);
  volatile unsigned int* w = reinterpret_cast<volatile unsigned int*>(status);
  w[14] = static_cast<unsigned int>(offset); w[15] = static_cast<unsigned int>(offset >> 32);
  return false;
}
#define AXB_IN_RANGE(status, offset, bytes, extent, code) (::axb::in_range_or_report((status), (offset), (bytes), (extent), (code)))
#else
#define AXB_IN_RANGE(status, offset, bytes, extent, code) (true)
#endif

// 2-D tiled TMA load (no multicast) into CTA shared memory.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* tmap, uint64_t* bar,
                                            int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      : : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
// The same for a 3-D map (columns, rows, batch): rows past the end of a batch element read zeros.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* tmap, uint64_t* bar,
                                            int32_t c0, int32_t c1, int32_t c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      : : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// Fetches a tile into the L2.  The L2 is where every writer's data is, so a tile may be fetched before its writer has finished.
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* tmap, int32_t c0, int32_t c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}

// --- programmatic dependent launch.  A kernel launched with the attribute may start before its predecessor in the stream has
// ended, once all of that one's CTAs have called pdl_launch_next or ended (at its end, if it never calls it); pdl_wait returns when
// the predecessor has ended and its writes are visible.  Every thread that reads or writes global memory calls pdl_wait first, and a
// CTA calls pdl_launch_next after its tensor memory is allocated: a CTA of the next kernel may be given what is left.  Bounded waits
// start after pdl_wait too: their deadline does not include the predecessor's run.
// Two kernels touch global memory before pdl_wait.  Split-K products fetch weights into the L2, where every writer's data is.  The later
// pruning passes load the gradient: all passes before them only read it, and the first one is an ordinary launch, which starts when
// whatever wrote the gradient has ended.
// One B200: attention layer of 777 tokens (four launches) 96 -> 90 us, residual LayerNorm forward and backward 104.6 -> 102.7, loss
// head of 4096 tokens 2057 -> 2016.  The attention backward's kernels are launched without: 1 % slower with (803 / 795 us).
// While GEMMs are capped nothing is launched ahead: the SMs that the cap leaves are for another stream's kernel, not for blocks that
// wait there for the end of the capped one.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... Params, typename... Args>
static inline cudaError_t pdl_launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = max_ctas() == 0 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// --- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tcgen05_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc], issued by one thread.
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      : : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// mbarrier arrives once all MMAs issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// --- CTA pairs (cta_group::2): two CTAs of a cluster of two share one MMA of 256 rows.  In the cluster
// shared-memory window bit 24 of an address selects the CTA of the pair; clearing it names the same
// offset in the even ("leader") CTA.
constexpr uint32_t PAIR_LEADER_MASK = 0xFEFFFFFFu;
__device__ __forceinline__ uint32_t cluster_cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 2-D tiled TMA load into this CTA's shared memory whose bytes are counted on the leader CTA's mbarrier
// at the same offset (no multicast: every CTA fetches its own tile).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tmap, uint64_t* bar,
                                                 int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      : : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar) & PAIR_LEADER_MASK),
          "r"(c0), "r"(c1)
      : "memory");
}
// arrive on the leader CTA's mbarrier at this offset (from either CTA of the pair)
__device__ __forceinline__ void mbar_arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & PAIR_LEADER_MASK) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem of both CTAs] (+)= A[256 rows: 128 in each CTA's smem] * B[N columns: N/2 in each CTA's smem]
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      : : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// the mbarrier at this offset in BOTH CTAs of the pair gets an arrival once all MMAs issued so far completed
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3)) : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns -> 32 registers per thread.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// The same wait with the registers of one load as operands: nothing that uses them can move before it.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
        "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
        "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
        "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
      : : "memory");
}
// 16 tensor-memory lanes x 32 columns: thread t gets, of columns 8 g + 2 (t % 4) and the next one, lanes t / 4 (r[4 g], r[4 g + 1])
// and t / 4 + 8 (r[4 g + 2], r[4 g + 3]).
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// 4 x 4 transpose among the four lanes of a quad: lane j gives w[i] to lane i, which gets it as w[j].
__device__ __forceinline__ void quad_transpose(uint32_t& w0, uint32_t& w1, uint32_t& w2, uint32_t& w3) {
  const bool odd = (threadIdx.x & 1) != 0, upper = (threadIdx.x & 2) != 0;
  uint32_t a = __shfl_xor_sync(0xffffffffu, odd ? w0 : w1, 1), b = __shfl_xor_sync(0xffffffffu, odd ? w2 : w3, 1);
  if (odd) { w0 = a; w2 = b; } else { w1 = a; w3 = b; }
  a = __shfl_xor_sync(0xffffffffu, upper ? w0 : w2, 2); b = __shfl_xor_sync(0xffffffffu, upper ? w1 : w3, 2);
  if (upper) { w0 = a; w1 = b; } else { w2 = a; w3 = b; }
}

// 32 accumulator rows x 32 columns of a warp as bf16: `dst` is where column 0 of row 0 goes, rows lie `pitch` elements apart, the
// first `rows` of them exist; row lane / 4 + 8 e is multiplied by scale[e].  A store instruction writes 64 consecutive bytes of eight
// rows: with a row per lane it touched 32 lines with 16 bytes each, and the 64 KB of dK and dV of 128 keys took 6900 cycles, now
// 3400.  One B200, before / after: dK / dV with the delta kernel, 8 x 2048, 16 heads, head_dim 128 331 / 297 us, head_dim 64
// 217 / 208, dQ 264 / 252; forward of 8 x 2048 143 / 139, of 4 x 1531, 32 heads over 8, 97 / 93.
__device__ __forceinline__ void store_rows_bf16(__nv_bfloat16* dst, size_t pitch, int rows, uint32_t taddr, const float (&scale)[4]) {
  const int lane = threadIdx.x & 31;
  dst += static_cast<size_t>(lane >> 2) * pitch + (lane & 3) * 8;
  uint32_t v[32];
  tmem_ld_16x32(taddr, v);
  tmem_ld_16x32(taddr + (16u << 16), v + 16);
  tmem_ld_wait(v);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    uint32_t w[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int i = (e >> 1) * 16 + g * 4 + (e & 1) * 2;
      const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[i]) * scale[e], __uint_as_float(v[i + 1]) * scale[e]);
      w[g] = *reinterpret_cast<const uint32_t*>(&h);
    }
    quad_transpose(w[0], w[1], w[2], w[3]);
    if ((lane >> 2) + 8 * e < rows) *reinterpret_cast<uint4*>(dst + 8 * e * pitch) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// 32 registers per thread -> 32 lanes x 32 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      : : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]: the A operand (128 rows = TMEM lanes, 16-bit elements packed two per
// 32-bit column, even element in the low half) is read from tensor memory.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      : : "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// Shared-memory matrix descriptor for tcgen05.mma, 128-byte swizzle.
// start address, leading/stride byte offsets in 16-byte units, descriptor
// version 1 (bit 46), layout type SWIZZLE_128B = 2 (bits 61-63).
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}

// Instruction descriptor for kind::f16: fp32 accumulate, A/B format
// (0 = fp16, 1 = bf16), A/B majorness (0 = K-major, 1 = MN-major), N>>3, M>>4.
__host__ __device__ constexpr uint32_t umma_idesc(int ab_format, int a_mn_major, int b_mn_major, int M, int N) {
  return (1u << 4) | (static_cast<uint32_t>(ab_format) << 7) | (static_cast<uint32_t>(ab_format) << 10) |
         (static_cast<uint32_t>(a_mn_major) << 15) | (static_cast<uint32_t>(b_mn_major) << 16) |
         (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  return 0.5f * x * (1.f + tanhf(u));
}
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  float t = tanhf(u);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k0 * (1.f + 3.f * k1 * x * x);
}

#endif  // __CUDACC__

}  // namespace axb
