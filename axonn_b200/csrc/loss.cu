// Softmax cross-entropy over (possibly vocabulary-sharded) logits.
//
// forward statistics, one block per row:  m = max_j z_j, s = sum_j exp(z_j - m),
// t = z_target when the target lies in this shard (else 0), in one pass over the row (running maximum per thread).
// With the whole vocabulary on this GPU the kernel also writes lse = m + log s, and a one-block kernel turns the rows
// into the mean loss; otherwise the caller all-reduces (m, s, t) over the vocabulary shards first.
// backward, in place: z_j <- (exp(z_j - lse) - [j == target]) * scale.
#include "common.cuh"

namespace axb {

constexpr int CE_THREADS = 512;

__device__ __forceinline__ float block_max(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  v = l < nw ? red[l] : -INFINITY;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  v = l < nw ? red[l] : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void ld8bf(const __nv_bfloat16* p, float (&f)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}

// stats: [rows, 3] = (max, sumexp, target logit); lse: [rows] or null.  The row is read once: every thread keeps its own
// running maximum and rescales its sum when the maximum of the next CE_UNROLL vectors raises it.  The next vectors are
// loaded before the current ones are used, and many small blocks (one row each) share an SM, so that the reductions at
// the end of one row run under the loads of others.
constexpr int CE_FWD_THREADS = 256, CE_UNROLL = 4;
__global__ void __launch_bounds__(CE_FWD_THREADS)
ce_fwd_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets,
              float* __restrict__ stats, float* __restrict__ lse, int rows, int V, int vocab_start) {
  __shared__ float red[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const __nv_bfloat16* z = logits + (size_t)row * V;
    const int nchunk = V / 8;
    uint4 next[CE_UNROLL];
    auto fetch = [&](int c) {
#pragma unroll
      for (int k = 0; k < CE_UNROLL; ++k) {
        const int cc = c + k * CE_FWD_THREADS;
        // vectors past the row: -inf, which adds exactly nothing
        next[k] = cc < nchunk ? __ldg(reinterpret_cast<const uint4*>(z) + cc)
                              : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);
      }
    };
    float m = -INFINITY, s = 0.f;
    fetch(threadIdx.x);
    for (int c = threadIdx.x; c < nchunk; c += CE_FWD_THREADS * CE_UNROLL) {
      uint4 u[CE_UNROLL];
#pragma unroll
      for (int k = 0; k < CE_UNROLL; ++k) u[k] = next[k];
      if (c + CE_FWD_THREADS * CE_UNROLL < nchunk) fetch(c + CE_FWD_THREADS * CE_UNROLL);
      __nv_bfloat162 m2 = *reinterpret_cast<const __nv_bfloat162*>(&u[0].x);
#pragma unroll
      for (int k = 0; k < CE_UNROLL; ++k) {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u[k]);
#pragma unroll
        for (int i = 0; i < 4; ++i) m2 = __hmax2(m2, h[i]);
      }
      const float2 mf = __bfloat1622float2(m2);
      const float mx = fmaxf(m, fmaxf(mf.x, mf.y));
      // nothing but -inf so far: keep the sum at zero (a NaN among them must still reach it)
      const float ref = mx == -INFINITY ? 0.f : mx;
      s *= __expf((m == -INFINITY ? ref : m) - ref);
      m = mx;
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < CE_UNROLL; ++k) {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u[k]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 d = __fadd2_rn(__bfloat1622float2(h[i]), make_float2(-ref, -ref));
          acc = __fadd2_rn(acc, make_float2(__expf(d.x), __expf(d.y)));
        }
      }
      s += acc.x + acc.y;
    }
    const float mrow = block_max(m, red);
    s *= __expf((m == -INFINITY && mrow != -INFINITY ? mrow : m) - mrow);   // a row of -inf only: NaN, as its softmax is
    s = block_sum(s, red);
    if (threadIdx.x == 0) {
      const long long t = targets[row] - vocab_start;
      stats[3 * row] = mrow;
      stats[3 * row + 1] = s;
      stats[3 * row + 2] = (t >= 0 && t < V) ? __bfloat162float(z[t]) : 0.f;
      if (lse) lse[row] = mrow + logf(s);
    }
  }
}

// The same statistics from those of 256 columns each that the GEMM left (axb_gemm_ce): part float2 [parts][rows].  A block has
// 32 rows, a warp every eighth part of them.
__global__ void __launch_bounds__(256)
ce_parts_kernel(const float2* __restrict__ part, int parts, const __nv_bfloat16* __restrict__ logits,
                const long long* __restrict__ targets, float* __restrict__ stats, float* __restrict__ lse, int rows, int V) {
  __shared__ float2 red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + lane;
  auto join = [](float2& a, const float2 b) {
    const float m = fmaxf(a.x, b.x), ref = m == -INFINITY ? 0.f : m;
    a = make_float2(m, a.y * __expf((a.x == -INFINITY ? ref : a.x) - ref) + b.y * __expf((b.x == -INFINITY ? ref : b.x) - ref));
  };
  float2 a = make_float2(-INFINITY, 0.f);
  if (row < rows) {
#pragma unroll 8
    for (int i = w; i < parts; i += 8) join(a, __ldg(part + static_cast<size_t>(i) * rows + row));
  }
  red[w][lane] = a;
  __syncthreads();
  if (w != 0 || row >= rows) return;
#pragma unroll
  for (int i = 1; i < 8; ++i) join(a, red[i][lane]);
  const long long t = targets[row];
  stats[3 * static_cast<size_t>(row)] = a.x;
  stats[3 * static_cast<size_t>(row) + 1] = a.y;
  stats[3 * static_cast<size_t>(row) + 2] = (t >= 0 && t < V) ? __bfloat162float(logits[static_cast<size_t>(row) * V + t]) : 0.f;
  // a row of -inf only: NaN, as its softmax is
  lse[row] = a.x == -INFINITY && a.y == 0.f ? __int_as_float(0x7fffffff) : a.x + logf(a.y);
}

// mean = mean over the rows whose target is not ignore_index of lse - target logit, kept = max(number of them, 1).
// One block: the rows' losses are a few hundred KB at most, and the fixed order keeps the result reproducible.
__global__ void __launch_bounds__(1024)
ce_mean_kernel(const float* __restrict__ stats, const float* __restrict__ lse, const long long* __restrict__ targets,
               float* __restrict__ mean, float* __restrict__ kept, int rows, long long ignore_index) {
  __shared__ float red[32];
  float loss = 0.f, count = 0.f;                     // counts stay below 2^24 per thread
#pragma unroll 4
  for (int r = threadIdx.x; r < rows; r += 1024) {
    const float valid = targets[r] != ignore_index ? 1.f : 0.f;
    loss += (lse[r] - stats[3 * (size_t)r + 2]) * valid;
    count += valid;
  }
  loss = block_sum(loss, red);
  count = block_sum(count, red);
  if (threadIdx.x == 0) {
    count = fmaxf(count, 1.f);
    *mean = loss / count;
    *kept = count;
  }
}

// In place: logits <- dlogits.  scale_ptr: device scalar (upstream gradient x 1/num_tokens).
__global__ void __launch_bounds__(CE_THREADS)
ce_bwd_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets,
              const float* __restrict__ lse, const float* __restrict__ scale_ptr, int rows, int V, int vocab_start,
              long long ignore_index) {
  const float scale = *scale_ptr;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    __nv_bfloat16* z = logits + (size_t)row * V;
    const long long tgt = targets[row];
    const long long t = tgt - vocab_start;
    const float l = lse[row];
    const float rs = (tgt == ignore_index) ? 0.f : scale;
    const int nchunk = V / 8;
    for (int c = threadIdx.x; c < nchunk; c += blockDim.x) {
      float f[8]; ld8bf(z + c * 8, f);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float p = __expf(f[i] - l);
        if (c * 8 + i == t) p -= 1.f;
        f[i] = p * rs;
      }
      uint4 u;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
      for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      *reinterpret_cast<uint4*>(z + c * 8) = u;
    }
  }
}

}  // namespace axb

using namespace axb;

// lse null: statistics of a vocabulary shard only; otherwise also lse [rows], the mean loss and the rows that count
static int ce_fwd(const void* logits, const long long* targets, float* stats, float* lse, float* mean, float* kept,
                  int rows, int V, int vocab_start, long long ignore_index, void* stream) {
  if (V % 8) { set_error("cross entropy: vocab shard %d must be a multiple of 8", V); return -1; }
  // one block per row (a block that walked several rows would leave the last round of a capped grid half empty)
  ce_fwd_kernel<<<rows, CE_FWD_THREADS, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, targets, stats, lse, rows, V,
                                                             vocab_start);
  AXB_CUDA(cudaGetLastError());
  if (mean) {
    ce_mean_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(stats, lse, targets, mean, kept, rows, ignore_index);
    AXB_CUDA(cudaGetLastError());
  }
  return 0;
}
extern "C" int axb_ce_fwd(const void* logits, const long long* targets, float* stats, int rows, int V, int vocab_start,
                          void* stream) {
  return ce_fwd(logits, targets, stats, nullptr, nullptr, nullptr, rows, V, vocab_start, 0, stream);
}
extern "C" int axb_ce_fwd_mean(const void* logits, const long long* targets, float* stats, float* lse, float* mean,
                               float* kept, int rows, int V, long long ignore_index, void* stream) {
  return ce_fwd(logits, targets, stats, lse, mean, kept, rows, V, 0, ignore_index, stream);
}
// axb_ce_fwd_mean with the statistics of every 256 columns at hand
extern "C" int axb_ce_fwd_parts(const void* part, const void* logits, const long long* targets, float* stats, float* lse,
                                float* mean, float* kept, int rows, int V, long long ignore_index, void* stream) {
  ce_parts_kernel<<<(rows + 31) / 32, 256, 0, (cudaStream_t)stream>>>((const float2*)part, (V + 255) / 256, (const __nv_bfloat16*)logits,
                                                                    targets, stats, lse, rows, V);
  AXB_CUDA(cudaGetLastError());
  ce_mean_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(stats, lse, targets, mean, kept, rows, ignore_index);
  AXB_CUDA(cudaGetLastError());
  return 0;
}
extern "C" int axb_ce_bwd(void* logits, const long long* targets, const float* lse, const float* scale, int rows, int V,
                          int vocab_start, long long ignore_index, void* stream) {
  if (V % 8) { set_error("cross entropy: vocab shard %d must be a multiple of 8", V); return -1; }
  const int cap = sm_count_current() * 8;
  const int grid = rows < cap ? rows : cap;
  ce_bwd_kernel<<<grid, CE_THREADS, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)logits, targets, lse, scale, rows, V,
                                                             vocab_start, ignore_index);
  AXB_CUDA(cudaGetLastError());
  return 0;
}
