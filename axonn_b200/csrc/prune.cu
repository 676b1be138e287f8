// Gradient pruning: keep the k largest-magnitude entries of a tensor, zero the rest.
//
// The threshold (k-th largest |g|) comes from a radix select on the magnitude bits instead of a sort: one histogram
// pass over the top 15 magnitude bits (block-private shared-memory histograms, flushed with atomics; the last block to
// finish scans the bins for the one that holds the k-th element), for fp32 a second histogram over the next 16 bits
// restricted to that bin, then one masking pass.  bf16 tensors (15 magnitude bits in total) need exactly two passes
// over the data.  Ties at the threshold are all kept (|g| >= threshold), the same rule as thresholding with the k-th
// value of a sort.
//
// Scratch: 32768 + 65536 + 8 32-bit words, supplied by the caller.
#include <mutex>

#include "common.cuh"

namespace axb {

constexpr int PR_BINS1 = 32768;
constexpr int PR_BINS2 = 65536;
constexpr int PR_THREADS = 1024;
constexpr int PR_WORK_WORDS = PR_BINS1 + PR_BINS2 + 8;
// dtype codes are the library-wide ones of axonn_b200.h: 0 bf16, 1 fp16, 2 fp32
constexpr int PR_F32 = 2;

__device__ __forceinline__ uint32_t mag_bits(const void* g, long long i, int dtype) {
  if (dtype == PR_F32) return reinterpret_cast<const uint32_t*>(g)[i] & 0x7FFFFFFFu;
  return (static_cast<uint32_t>(reinterpret_cast<const uint16_t*>(g)[i]) & 0x7FFFu) << 16;
}

// the last 8 words of the scratch
struct PruneMeta {
  long long bin1, rank1;      // bin of the threshold's top 15 bits, rank of the threshold inside it
  long long bin2;             // fp32: the next 16 bits
  unsigned int blocks_done;   // zero between kernels
  unsigned int pad;
};
static_assert(sizeof(PruneMeta) == 32, "scratch layout");

// Called by all threads of the block that finishes last: the largest bin b with count(bins > b) < k <= count(bins >= b).
// Every thread sums its bins with 16-byte loads (8-byte ones if the caller's scratch is aligned to no more: 4 us longer)
// and the block scans the sums in registers: a one-block kernel of its own with a word-wise sum and a log-step scan in
// shared memory took 21 us per tensor.
template <int BINS>
__device__ void prune_select(const unsigned int* __restrict__ hist, long long k, long long* bin, long long* rank) {
  __shared__ unsigned long long warp_sum[PR_THREADS / 32];
  __shared__ unsigned long long found_above;
  __shared__ int found_hi;
  constexpr int PER = BINS / PR_THREADS;
  // thread t owns bins [BINS - (t+1)*PER, BINS - t*PER): thread 0 holds the largest magnitudes
  const int hi = BINS - threadIdx.x * PER, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long mine = 0;
  if ((reinterpret_cast<uintptr_t>(hist) & 15) == 0) {
#pragma unroll 8
    for (int i = 0; i < PER / 4; ++i) {
      const uint4 u = __ldcg(reinterpret_cast<const uint4*>(hist + hi - PER) + i);
      mine += static_cast<unsigned long long>(u.x) + u.y + u.z + u.w;
    }
  } else {
#pragma unroll 8
    for (int i = 0; i < PER / 2; ++i) {
      const uint2 u = __ldcg(reinterpret_cast<const uint2*>(hist + hi - PER) + i);
      mine += static_cast<unsigned long long>(u.x) + u.y;
    }
  }
  unsigned long long incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
  if (lane == 31) warp_sum[w] = incl;
  __syncthreads();
  if (w == 0) {
    const unsigned long long v = warp_sum[lane];
    unsigned long long pre = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const unsigned long long u = __shfl_up_sync(0xffffffffu, pre, o); if (lane >= o) pre += u; }
    warp_sum[lane] = pre - v;
  }
  __syncthreads();
  incl += warp_sum[w];
  const unsigned long long excl = incl - mine;
  if (threadIdx.x == 0) found_hi = 0;
  __syncthreads();
  if (excl < (unsigned long long)k && (unsigned long long)k <= incl) { found_hi = hi; found_above = excl; }
  __syncthreads();
  if (w != 0) return;
  if (found_hi == 0) {                                     // k > n: keep all
    if (lane == 0) { *bin = 0; if (rank) *rank = 1; }
    return;
  }
  // one warp looks through that thread's bins, 32 at a time from the top
  unsigned long long above = found_above;
  for (int top = found_hi; top > found_hi - PER; top -= 32) {
    const unsigned long long c = __ldcg(hist + top - 1 - lane);
    unsigned long long upto = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const unsigned long long u = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += u; }
    const unsigned hit = __ballot_sync(0xffffffffu, above + upto >= (unsigned long long)k);
    if (hit) {
      if (lane == __ffs(hit) - 1) { *bin = top - 1 - lane; if (rank) *rank = k - (long long)(above + upto - c); }
      return;
    }
    above += __shfl_sync(0xffffffffu, upto, 31);
  }
}

// True in every thread of the block that arrives last (its predecessors' histogram updates are visible to it).
__device__ __forceinline__ bool prune_last_block(unsigned int* counter) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
    if (last) { *counter = 0; __threadfence(); }
  }
  __syncthreads();
  return last;
}

// level 1: histogram of the top 15 magnitude bits, then (last block) the threshold's bin.  Four 16-byte loads per thread
// are in flight; they are ordinary loads, so that a tensor that fits the L2 is still there for the masking pass.  LONG, for
// tensors that do not fit: the passes go through them in turn from the end (whose gradients were written last) and from the
// beginning, so that the next one first reads what the L2 has kept, and the next vectors are fetched before the current ones
// are counted.  Shorter ones gain nothing from either (25 M fp16 56.9 -> 58.3 us, 4 M fp32 48.1 -> 49.4).
// The pass is not bound by its atomics alone: the writes of whatever filled the tensor still go to memory meanwhile, and
// counters without atomics or without bank conflicts took as long.  One B200, with the refill of the tensor: 117 M bf16 221 ->
// 215 us, 67 M 133 -> 127, 67 M fp32 294 -> 280, 25 M fp32 128 -> 120.
// The three passes of fp32 gain from 64 MB to some 400 MB only: 100 M 423 -> 421, but 117 M 483 -> 487, 400 M 1531 -> 1543; 16-bit
// tensors at any length (800 M 1394 -> 1372).
constexpr long long PR_LONG_BYTES = 64ll << 20, PR_LONG_F32_BYTES = 400ll << 20;
template <bool LONG>
__global__ void __launch_bounds__(PR_THREADS)
prune_hist1_kernel(const void* __restrict__ g, long long n, int dtype, long long k, unsigned int* __restrict__ hist,
                   PruneMeta* __restrict__ meta) {
  extern __shared__ unsigned int sh[];
  for (int i = threadIdx.x; i < PR_BINS1; i += PR_THREADS) sh[i] = 0;
  __syncthreads();
  auto count = [&](uint32_t key) { atomicAdd(&sh[key], 1u); };
  long long tail = 0;
  const long long first = blockIdx.x * (long long)PR_THREADS + threadIdx.x, step = (long long)gridDim.x * PR_THREADS;
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
    const int per_vec = dtype == PR_F32 ? 4 : 8;
    const long long nv = n / per_vec;
    const uint4* q = reinterpret_cast<const uint4*>(g);
    uint4 next[4];
    auto fetch = [&](long long i) {
#pragma unroll
      for (int v = 0; v < 4; ++v) if (i + v * step < nv) next[v] = q[LONG ? nv - 1 - (i + v * step) : i + v * step];
    };
    if (LONG) fetch(first);
    for (long long i = first; i < nv; i += 4 * step) {
      uint4 u[4];
      if (!LONG) fetch(i);
#pragma unroll
      for (int v = 0; v < 4; ++v) u[v] = next[v];
      if (LONG) fetch(i + 4 * step);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        if (i + v * step >= nv) break;
        const uint32_t w[4] = {u[v].x, u[v].y, u[v].z, u[v].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          count((w[j] >> 16) & 0x7FFFu);
          if (dtype != PR_F32) count(w[j] & 0x7FFFu);
        }
      }
    }
    tail = nv * per_vec;
  }
  for (long long i = tail + first; i < n; i += step) count(mag_bits(g, i, dtype) >> 16);
  __syncthreads();
  pdl_launch_next();             // its blocks fetch their first vectors while the bins are added up and searched
  for (int i = threadIdx.x; i < PR_BINS1; i += PR_THREADS)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
  if (!prune_last_block(&meta->blocks_done)) return;
  prune_select<PR_BINS1>(hist, k, &meta->bin1, &meta->rank1);
}

// level 2 (fp32 only): histogram of the next 16 bits among elements whose top bits equal the threshold's, and its bin
__global__ void __launch_bounds__(PR_THREADS)
prune_hist2_kernel(const void* __restrict__ g, long long n, PruneMeta* __restrict__ meta, unsigned int* __restrict__ hist2) {
  uint32_t top = 0;
  auto count = [&](uint32_t w) { if (((w >> 16) & 0x7FFFu) == top) atomicAdd(&hist2[w & 0xFFFFu], 1u); };
  const uint32_t* f = reinterpret_cast<const uint32_t*>(g);
  const long long first = blockIdx.x * (long long)PR_THREADS + threadIdx.x, step = (long long)gridDim.x * PR_THREADS;
  long long tail = 0;
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
    const long long nv = n / 4;
    const uint4* q = reinterpret_cast<const uint4*>(g);
    uint4 u[4];
    auto fetch = [&](long long i) {
#pragma unroll
      for (int v = 0; v < 4; ++v) if (i + v * step < nv) u[v] = q[i + v * step];
    };
    fetch(first);                // nothing since the launch before the first pass has written the tensor
    pdl_wait();
    top = static_cast<uint32_t>(__ldcg(&meta->bin1));
    for (long long i = first; i < nv; i += 4 * step) {
      if (i != first) fetch(i);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        if (i + v * step >= nv) break;
        count(u[v].x); count(u[v].y); count(u[v].z); count(u[v].w);
      }
    }
    tail = nv * 4;
  } else {
    pdl_wait();
    top = static_cast<uint32_t>(__ldcg(&meta->bin1));
  }
  for (long long i = tail + first; i < n; i += step) count(f[i]);
  pdl_launch_next();
  if (!prune_last_block(&meta->blocks_done)) return;
  prune_select<PR_BINS2>(hist2, meta->rank1, &meta->bin2, nullptr);
}

// thr = 31-bit magnitude threshold: keep |g| bits >= thr.  Bound by one read and one write of the tensor.
template <bool REVERSE>
__global__ void __launch_bounds__(512)
prune_mask_kernel(void* __restrict__ g, long long n, int dtype, const PruneMeta* __restrict__ meta) {
  uint32_t thr = 0;
  auto threshold = [&] {
    pdl_wait();
    thr = ((uint32_t)__ldcg(&meta->bin1) << 16) | (dtype == PR_F32 ? (uint32_t)__ldcg(&meta->bin2) : 0u);
  };
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  long long tail = 0;
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
    const int per_vec = dtype == PR_F32 ? 4 : 8;
    const long long nv = n / per_vec;
    uint4* const q = reinterpret_cast<uint4*>(g);
    // vector j of the traversal: from the end that the pass before this one read last
    auto at = [&](long long j) { return REVERSE ? nv - 1 - j : j; };
    uint4 u[4];
    auto fetch = [&](long long i) {
#pragma unroll
      for (int v = 0; v < 4; ++v) if (i + v * step < nv) u[v] = q[at(i + v * step)];
    };
    fetch(first);                // the passes before this one only read the tensor
    threshold();
    const uint32_t t16 = thr >> 16;
    for (long long i = first; i < nv; i += 4 * step) {
      if (i != first) fetch(i);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        if (i + v * step >= nv) break;
        uint32_t w[4] = {u[v].x, u[v].y, u[v].z, u[v].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (dtype == PR_F32) {
            if ((w[j] & 0x7FFFFFFFu) < thr) w[j] = 0u;
          } else {
            if ((w[j] & 0x7FFFu) < t16) w[j] &= 0xFFFF0000u;
            if (((w[j] >> 16) & 0x7FFFu) < t16) w[j] &= 0x0000FFFFu;
          }
        }
        q[at(i + v * step)] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    tail = nv * per_vec;
  } else {
    threshold();
  }
  for (long long i = tail + first; i < n; i += step) {
    if (mag_bits(g, i, dtype) < thr) {
      if (dtype == PR_F32) reinterpret_cast<uint32_t*>(g)[i] = 0; else reinterpret_cast<uint16_t*>(g)[i] = 0;
    }
  }
}

int sm_count(int device);

// Shared by the allocating and the static-scratch entry points.
int prune_topk_launch(void* g, long long n, int dtype, long long k, unsigned int* work, int device, cudaStream_t s) {
  if (n <= 0) return 0;
  if (k <= 0) { AXB_CUDA(cudaMemsetAsync(g, 0, (size_t)n * (dtype == PR_F32 ? 4 : 2), s)); return 0; }
  if (k >= n) return 0;
  unsigned int* hist1 = work;
  unsigned int* hist2 = work + PR_BINS1;
  PruneMeta* meta = reinterpret_cast<PruneMeta*>(work + PR_BINS1 + PR_BINS2);
  // one memset: for 16-bit tensors it covers the second level's bins too, which costs less than a second launch
  AXB_CUDA(cudaMemsetAsync(work, 0, sizeof(unsigned int) * PR_WORK_WORDS, s));
  static bool configured[64] = {false};
  if (!configured[device & 63]) {
    AXB_CUDA(cudaFuncSetAttribute(prune_hist1_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_BINS1 * 4));
    AXB_CUDA(cudaFuncSetAttribute(prune_hist1_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_BINS1 * 4));
    configured[device & 63] = true;
  }
  const int sms = sm_count(device);
  const long long bytes = n * (dtype == PR_F32 ? 4 : 2);
  const bool is_long = bytes >= PR_LONG_BYTES && (dtype != PR_F32 || bytes <= PR_LONG_F32_BYTES);
  auto hist = is_long ? prune_hist1_kernel<true> : prune_hist1_kernel<false>;
  // An ordinary launch, and it has to stay one: the passes after it load the gradient before they wait for their predecessor, and mask
  // what they have loaded.  Launched ahead itself, this pass could let them do so while the gradient is still being written.
  hist<<<sms, PR_THREADS, PR_BINS1 * 4, s>>>(g, n, dtype, k, hist1, meta);
  AXB_CUDA(cudaGetLastError());
  if (dtype == PR_F32) {
    AXB_CUDA(pdl_launch(prune_hist2_kernel, dim3(sms * 2), dim3(PR_THREADS), 0, s, g, n, meta, hist2));
  }
  auto mask = is_long && dtype == PR_F32 ? prune_mask_kernel<true> : prune_mask_kernel<false>;   // after two passes or one
  // The passes after the first are launched while the one before them still looks for its bin, and have their first vectors by then
  // (the first pass itself follows a memset and starts when all before it has ended).  One B200, with the refill of the
  // tensors: four of a Llama-8B block 430 -> 425 us, four of hidden 256 90 -> 80.
  AXB_CUDA(pdl_launch(mask, dim3(sms * 4), dim3(512), 0, s, g, n, dtype, meta));
  return 0;
}

}  // namespace axb

extern "C" int axb_prune_workspace_words(void) { return axb::PR_WORK_WORDS; }

// g: gradient tensor (dtype 0 bf16, 1 fp16, 2 fp32: the library-wide codes), modified in place; keeps the k largest |g|.
// work: device scratch of axb_prune_workspace_words() 32-bit words (8-byte aligned).
extern "C" int axb_prune_topk(void* g, long long n, int dtype, long long k, void* work, int device, void* stream) {
  if (!work) { axb::set_error("prune: workspace is null"); return -1; }
  if (reinterpret_cast<uintptr_t>(work) & 7) { axb::set_error("prune: the workspace must be 8-byte aligned"); return -1; }
  if (dtype < 0 || dtype > 2) { axb::set_error("prune: bad dtype %d (0 bf16, 1 fp16, 2 fp32)", dtype); return -1; }
  return axb::prune_topk_launch(g, n, dtype, k, static_cast<unsigned int*>(work), device, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------
// Entry point for callers that must not allocate.
//
// Some programs that embed this library own every byte of device memory themselves (a serving
// process that hands the whole GPU to its own pool at start-up, or one that runs under a
// "nothing is allocated after initialisation" rule): asking the driver for a workspace in the
// middle of their step can fail or fragment their pool, so they cannot supply freshly allocated
// scratch and do not want this library to allocate it behind their back.  For them the
// radix-select scratch lives in the library image itself, in the array below.
//
// The array takes PR_WORK_WORDS * 4 bytes (32768 + 65536 + 8 words = 393,248 bytes) of every
// GPU that loads the library, from load until the process exits.
static __device__ __align__(256) unsigned int g_prune_static_scratch[axb::PR_WORK_WORDS];

namespace axb {
// Largest tensor the static entry point accepts: the histogram counters are 32-bit.
constexpr long long PR_STATIC_MAX_NUMEL = 2147483647LL;
// Device address of g_prune_static_scratch per device.  In host code the array's name is only a
// handle for the runtime, not an address a kernel can use, so the address is looked up once per
// device with cudaGetSymbolAddress while that device is current.
static unsigned int* g_prune_static_ptr[64] = {nullptr};
static std::mutex g_prune_static_mu;   // first-use lookup may race between host threads
}  // namespace axb

// Keep the k largest-magnitude entries of g (dtype 0 bf16, 1 fp16, 2 fp32), zero the rest, in place,
// like axb_prune_topk, but with no workspace argument and without allocating anything: no cudaMalloc,
// no cudaFree, no allocating library call.
//
// * `device` must be the calling thread's current device on every call (checked; the launches and the
//   clearing of the scratch go to the current device).  The first call on a device also looks up the
//   scratch array's device address: make that first call before starting any stream capture on the device.
// * n must not exceed 2,147,483,647 elements; larger tensors are rejected with an error.
// * All calls on a device share one scratch array.  It is cleared at the start of each call, so
//   nothing needs to be reset between calls, but two calls whose kernels may overlap on the GPU
//   (different streams without an ordering between them) race on it: serialise them.
extern "C" int axb_prune_topk_static(void* g, long long n, int dtype, long long k, int device, void* stream) {
  using namespace axb;
  if (n > PR_STATIC_MAX_NUMEL) {
    set_error("axb_prune_topk_static: %lld elements exceed the supported maximum of %lld", n, PR_STATIC_MAX_NUMEL);
    return -1;
  }
  if (device < 0 || device >= 64) { set_error("axb_prune_topk_static: bad device index %d", device); return -1; }
  if (dtype < 0 || dtype > 2) { set_error("axb_prune_topk_static: bad dtype %d", dtype); return -1; }
  int current = -1;
  AXB_CUDA(cudaGetDevice(&current));
  if (current != device) {
    set_error("axb_prune_topk_static: device %d must be the current device (current is %d)", device, current);
    return -1;
  }
  std::lock_guard<std::mutex> lock(g_prune_static_mu);
  if (g_prune_static_ptr[device] == nullptr) {
    unsigned int* p = nullptr;
    AXB_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_prune_static_scratch));
    if (p == nullptr) { set_error("axb_prune_topk_static: scratch symbol has no device address"); return -1; }
    g_prune_static_ptr[device] = p;
  }
  return prune_topk_launch(g, n, dtype, k, g_prune_static_ptr[device], device, (cudaStream_t)stream);
}
