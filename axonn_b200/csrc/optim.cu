// Multi-tensor kernels: fused AdamW step, squared L2 norm, in-place scale.
//
// A launch covers a whole list of tensors through a device table; work is cut
// into fixed-size chunks (the table holds their prefix sums), and a grid-stride
// loop maps units of work -> (tensor, offset), so one launch replaces hundreds
// of per-parameter launches.  A unit is a quarter to a sixteenth of a chunk for
// the optimizers, whose 28 bytes per element make a whole chunk too long a last
// unit (the table's c: quarters); squared norm and scale take whole chunks for tables of small tensors,
// where three of four quarters would be empty.  One B200, us, inputs warm in
// the L2 where they fit; a: whole chunks found by binary search, b: quarters
// found by a linear search, c: now
//                                       AdamW            scale          norm
//                                       a    b    c      a    b   c    a    b   c
//   12 tensors of 4 M (bf16)            288  238  237    130  29  30   20   19  20
//   a 300-tensor model, 315 M           1650 1409 1409   671  190 188  110  135 96
//   1500 tensors of 32768               282  261  239    110  90  32   22   91  18
//   3000 tensors of 4096                109  328  80     29   272 20   19   279 18
//   300 tensors of 2048                 13   12   10     5.3  8.3 4.3  5.8  9.5 5.1
// (the scale used 2-byte accesses in a)
#include <mutex>

#include "common.cuh"

namespace axb {

constexpr int MT_CHUNK = 1 << 16;
constexpr int MT_PARTS = 4;                      // units per chunk of the optimizer kernels (and of the scale of long tensors)
constexpr int MT_THREADS = 512;
constexpr int ADAM_THREADS = 256;
constexpr int ADAM_UNROLL = 2;


// table row for norm/scale: {ptr, numel, dtype (0 fp32, 1 bf16, 2 fp16), chunk_prefix}
// table row for adamw:      {master fp32, model bf16 or 0, grad, exp_avg, exp_avg_sq, numel, grad dtype, chunk_prefix}
// Row of the tensor that holds `chunk`: the last one whose prefix is <= chunk (tensors without elements share the prefix of
// their successor).  Whole warps call it; every round the 32 lanes look at 32 evenly spaced rows of what is left, so
// 32 tensors take one load latency, 1024 two.
__device__ __forceinline__ int find_tensor(const long long* table, int width, int prefix_col, int n, long long chunk) {
  const int lane = threadIdx.x & 31;
  int lo = 0, len = n;
  while (len > 1) {
    const int step = (len + 31) / 32, at = lane * step;
    const bool le = at < len && (at == 0 || __ldg(table + static_cast<size_t>(lo + at) * width + prefix_col) <= chunk);
    const int c = __popc(__ballot_sync(0xffffffffu, le)) - 1;      // prefixes are sorted, and the first is taken
    lo += c * step;
    len = min(step, len - c * step);
  }
  return lo;
}

__device__ __forceinline__ float load_as_f32(const void* p, long long i, int dtype) {
  if (dtype == 0) return reinterpret_cast<const float*>(p)[i];
  if (dtype == 1) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  return __half2float(reinterpret_cast<const __half*>(p)[i]);
}
__device__ __forceinline__ void store_from_f32(void* p, long long i, int dtype, float v) {
  if (dtype == 0) reinterpret_cast<float*>(p)[i] = v;
  else if (dtype == 1) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else reinterpret_cast<__half*>(p)[i] = __float2half_rn(v);
}

// Clipping by the norm of one table (CLIP): with `blocks_done` zero on entry, the block that arrives last has the whole sum and
// writes the norm and the factor min(1, max_norm / (norm + 1e-6)) itself.  As tensor operations after the kernel (square
// root, sum, reciprocal, ...) that was seven launches of 2 us each: clipping and AdamW of 50 M parameters 305 -> 277 us.
struct ClipOut {
  unsigned int* blocks_done;
  float* norm;
  float* factor;
  float max_norm;
};

template <int PARTS, bool CLIP>      // units per chunk
__global__ void __launch_bounds__(MT_THREADS)
multi_l2norm_sq_kernel(const long long* __restrict__ table, int n, long long total_chunks, float* __restrict__ out,
                       const ClipOut clip) {
  pdl_launch_next();
  pdl_wait();
  __shared__ float red[32];
  float acc = 0.f;
  constexpr int UNIT = MT_CHUNK / PARTS;
  for (long long unit = blockIdx.x; unit < total_chunks * PARTS; unit += gridDim.x) {
    const long long chunk = unit / PARTS;
    const int t = find_tensor(table, 4, 3, n, chunk);
    const long long* row = table + (size_t)t * 4;
    const void* p = reinterpret_cast<const void*>(row[0]);
    const long long numel = row[1];
    const int dtype = (int)row[2];
    const long long begin = (chunk - row[3]) * MT_CHUNK + (unit % PARTS) * UNIT;
    const long long end = begin + UNIT < numel ? begin + UNIT : numel;
    if (begin >= numel) continue;
    const bool vec = (reinterpret_cast<uintptr_t>(p) & 15) == 0;
    if (vec && dtype == 1) {
      const long long nv = (end - begin) / 8;
      const uint4* q = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p) + begin);
#pragma unroll 4
      for (long long i = threadIdx.x; i < nv; i += blockDim.x) {
        const uint4 u = q[i];
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int k = 0; k < 4; ++k) { float2 f = __bfloat1622float2(h[k]); acc += f.x * f.x + f.y * f.y; }
      }
      for (long long i = begin + nv * 8 + threadIdx.x; i < end; i += blockDim.x) {
        float v = load_as_f32(p, i, dtype); acc += v * v;
      }
    } else if (vec && dtype == 0) {
      const long long nv = (end - begin) / 4;
      const float4* q = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + begin);
#pragma unroll 4
      for (long long i = threadIdx.x; i < nv; i += blockDim.x) {
        const float4 f = q[i]; acc += f.x * f.x + f.y * f.y + f.z * f.z + f.w * f.w;
      }
      for (long long i = begin + nv * 4 + threadIdx.x; i < end; i += blockDim.x) {
        float v = load_as_f32(p, i, dtype); acc += v * v;
      }
    } else {
      for (long long i = begin + threadIdx.x; i < end; i += blockDim.x) {
        float v = load_as_f32(p, i, dtype); acc += v * v;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    acc = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (threadIdx.x == 0) {
      atomicAdd(out, acc);
      if (CLIP) {
        __threadfence();
        if (atomicAdd(clip.blocks_done, 1u) == gridDim.x - 1) {
          __threadfence();
          const float norm = __fsqrt_rn(__ldcg(out));
          const float f = __fdiv_rn(clip.max_norm, norm + 1e-6f);
          *clip.norm = norm;
          *clip.factor = f > 1.f ? 1.f : f;      // a NaN stays one
        }
      }
    }
  }
}

// one 32-bit word (one fp32 or two 16-bit values) times s, each product rounded once
__device__ __forceinline__ uint32_t scale_word(uint32_t w, int dtype, float s) {
  if (dtype == 0) return __float_as_uint(__uint_as_float(w) * s);
  if (dtype == 1) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
    const __nv_bfloat162 h = __floats2bfloat162_rn(f.x * s, f.y * s);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  const __half2 h = __floats2half2_rn(f.x * s, f.y * s);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// In-place scale, bound by one read and one write of the tensors: 16-byte accesses with SCALE_UNROLL of them in flight
// per thread.  A factor of exactly one (a gradient norm below the clipping limit) leaves every value as it is.
constexpr int SCALE_UNROLL = 4;
template <int PARTS>      // units per chunk
__global__ void __launch_bounds__(MT_THREADS)
multi_scale_kernel(const long long* __restrict__ table, int n, long long total_chunks, const float* __restrict__ scale_ptr) {
  pdl_launch_next();
  pdl_wait();
  const float s = *scale_ptr;
  if (s == 1.f) return;
  constexpr int UNIT = MT_CHUNK / PARTS;
  // from the last unit to the first: the norm that the factor comes from has just read the list to its end, and the optimizer
  // will start where this ends (100 MB of gradients on a B200: scale 28.2 -> 26.5 us, AdamW after it 236 -> 233)
  for (long long left = total_chunks * PARTS - 1 - blockIdx.x; left >= 0; left -= gridDim.x) {
    const long long unit = left, chunk = unit / PARTS;
    const int t = find_tensor(table, 4, 3, n, chunk);
    const long long* row = table + (size_t)t * 4;
    void* p = reinterpret_cast<void*>(row[0]);
    const long long numel = row[1];
    const int dtype = (int)row[2];
    const long long begin = (chunk - row[3]) * MT_CHUNK + (unit % PARTS) * UNIT;
    const long long end = begin + UNIT < numel ? begin + UNIT : numel;
    if (begin >= numel) continue;
    long long scalar_from = begin;
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {      // chunks start at multiples of 65536 elements
      const int per_vec = dtype == 0 ? 4 : 8;
      const long long nv = (end - begin) / per_vec;
      uint4* q = reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p) + begin * (dtype == 0 ? 4 : 2));
      for (long long i0 = threadIdx.x; i0 < nv; i0 += blockDim.x * SCALE_UNROLL) {
        uint4 u[SCALE_UNROLL];
#pragma unroll
        for (int k = 0; k < SCALE_UNROLL; ++k)
          if (i0 + k * blockDim.x < nv) u[k] = q[i0 + k * blockDim.x];
#pragma unroll
        for (int k = 0; k < SCALE_UNROLL; ++k) {
          if (i0 + k * blockDim.x >= nv) continue;
          uint32_t w[4] = {u[k].x, u[k].y, u[k].z, u[k].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) w[j] = scale_word(w[j], dtype, s);
          q[i0 + k * blockDim.x] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      scalar_from = begin + nv * per_vec;
    }
    for (long long i = scalar_from + threadIdx.x; i < end; i += blockDim.x)
      store_from_f32(p, i, dtype, load_as_f32(p, i, dtype) * s);
  }
}

// SGD with momentum (torch.optim.SGD semantics without dampening / Nesterov): g' = g * grad_scale + wd * p,
// buf = mu * buf + g', p -= lr * buf.  Table rows: {param, grad, momentum buffer (fp32), numel, param dtype,
// grad dtype, chunk prefix, -}.
template <int PARTS>      // units per chunk
__global__ void __launch_bounds__(MT_THREADS)
multi_sgd_kernel(const long long* __restrict__ table, int n, long long total_chunks, float lr, float momentum,
                 float weight_decay, const float* __restrict__ grad_scale, const unsigned int* __restrict__ status) {
  if (status && *reinterpret_cast<const volatile unsigned int*>(status) != 0u) return;
  const float gs = grad_scale ? *grad_scale : 1.f;
  constexpr int UNIT = MT_CHUNK / PARTS;
  for (long long unit = blockIdx.x; unit < total_chunks * PARTS; unit += gridDim.x) {
    const long long chunk = unit / PARTS;
    const int t = find_tensor(table, 8, 6, n, chunk);
    const long long* row = table + (size_t)t * 8;
    void* p = reinterpret_cast<void*>(row[0]);
    const void* g = reinterpret_cast<const void*>(row[1]);
    float* buf = reinterpret_cast<float*>(row[2]);
    const long long numel = row[3];
    const int pdtype = (int)row[4], gdtype = (int)row[5];
    const long long begin = (chunk - row[6]) * MT_CHUNK + (unit % PARTS) * UNIT;
    const long long end = begin + UNIT < numel ? begin + UNIT : numel;
    if (begin >= numel) continue;
    for (long long i = begin + threadIdx.x; i < end; i += blockDim.x) {
      const float w = load_as_f32(p, i, pdtype);
      const float gi = load_as_f32(g, i, gdtype) * gs + weight_decay * w;
      const float b = momentum * buf[i] + gi;
      buf[i] = b;
      store_from_f32(p, i, pdtype, w - lr * b);
    }
  }
}

struct AdamArgs {
  float lr, beta1, beta2, eps, weight_decay, bias_c1, bias_c2;
  const float* grad_scale;       // device scalar multiplied into every gradient (may be null)
  const float* found_inf;        // device scalar; non-zero => skip the whole step (may be null)
  const unsigned int* status;    // copy, in device memory, of the device status word taken just before this launch;
                                 // non-zero (a bounded wait of an earlier kernel expired: gradients may be
                                 // incomplete) => skip the whole step (may be null)
};

template <int PARTS>      // units per chunk
__global__ void __launch_bounds__(ADAM_THREADS, 4)
multi_adamw_kernel(const long long* __restrict__ table, int n, long long total_chunks, AdamArgs a) {
  pdl_launch_next();
  pdl_wait();
  if (a.found_inf && *a.found_inf != 0.f) return;
  if (a.status && *reinterpret_cast<const volatile unsigned int*>(a.status) != 0u) return;
  const float gs = a.grad_scale ? *a.grad_scale : 1.f;
  const float decay = 1.f - a.lr * a.weight_decay;
  const float step = a.lr / a.bias_c1;
  const float inv_sqrt_c2 = rsqrtf(a.bias_c2);
  constexpr int UNIT = MT_CHUNK / PARTS;
  for (long long unit = blockIdx.x; unit < total_chunks * PARTS; unit += gridDim.x) {
    const long long chunk = unit / PARTS;
    const int t = find_tensor(table, 8, 7, n, chunk);
    const long long* row = table + (size_t)t * 8;
    float* master = reinterpret_cast<float*>(row[0]);
    __nv_bfloat16* model = reinterpret_cast<__nv_bfloat16*>(row[1]);
    const void* grad = reinterpret_cast<const void*>(row[2]);
    float* m = reinterpret_cast<float*>(row[3]);
    float* v = reinterpret_cast<float*>(row[4]);
    const long long numel = row[5];
    const int gdtype = (int)row[6];
    const long long begin = (chunk - row[7]) * MT_CHUNK + (unit % PARTS) * UNIT;
    const long long end = begin + UNIT < numel ? begin + UNIT : numel;
    if (begin >= numel) continue;
    const bool aligned = ((reinterpret_cast<uintptr_t>(master) | reinterpret_cast<uintptr_t>(m) |
                           reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(grad) |
                           reinterpret_cast<uintptr_t>(model)) & 15) == 0;
    long long scalar_from = begin;
    if (aligned && gdtype != 2) {
      // 4 elements per vector: 16-byte accesses to the fp32 state, 8-byte to bf16 tensors.  Every thread loads
      // ADAM_UNROLL vectors of all four streams before it computes; the loads of one block run under the arithmetic
      // and the stores of the three others on its SM.  50 M parameters on a B200: four vectors, two blocks and
      // streaming hints 280 us, two vectors and four blocks 250 us, the same without the hints 241 us.
      const long long nv = (end - begin) / 4;
      for (long long q0 = threadIdx.x; q0 < nv; q0 += (long long)blockDim.x * ADAM_UNROLL) {
        float4 p4[ADAM_UNROLL], m4[ADAM_UNROLL], v4[ADAM_UNROLL];
        float g4[ADAM_UNROLL][4];
#pragma unroll
        for (int u = 0; u < ADAM_UNROLL; ++u) {
          const long long q = q0 + (long long)u * blockDim.x;
          if (q < nv) {
            const long long i = begin + q * 4;
            p4[u] = *reinterpret_cast<const float4*>(master + i);
            m4[u] = *reinterpret_cast<const float4*>(m + i);
            v4[u] = *reinterpret_cast<const float4*>(v + i);
            if (gdtype == 0) {
              const float4 t = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(grad) + i);
              g4[u][0] = t.x; g4[u][1] = t.y; g4[u][2] = t.z; g4[u][3] = t.w;
            } else {
              const uint2 t = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(grad) + i);
              const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&t.x);
              const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&t.y);
              g4[u][0] = __bfloat162float(lo.x); g4[u][1] = __bfloat162float(lo.y);
              g4[u][2] = __bfloat162float(hi.x); g4[u][3] = __bfloat162float(hi.y);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < ADAM_UNROLL; ++u) {
          const long long q = q0 + (long long)u * blockDim.x;
          if (q >= nv) continue;
          const long long i = begin + q * 4;
          float pp[4] = {p4[u].x, p4[u].y, p4[u].z, p4[u].w}, mm[4] = {m4[u].x, m4[u].y, m4[u].z, m4[u].w},
                vv[4] = {v4[u].x, v4[u].y, v4[u].z, v4[u].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float g = g4[u][k] * gs;
            mm[k] = a.beta1 * mm[k] + (1.f - a.beta1) * g;
            vv[k] = a.beta2 * vv[k] + (1.f - a.beta2) * g * g;
            const float denom = sqrtf(vv[k]) * inv_sqrt_c2 + a.eps;
            pp[k] = pp[k] * decay - step * mm[k] / denom;
          }
          *reinterpret_cast<float4*>(master + i) = (make_float4(pp[0], pp[1], pp[2], pp[3]));
          *reinterpret_cast<float4*>(m + i) = (make_float4(mm[0], mm[1], mm[2], mm[3]));
          *reinterpret_cast<float4*>(v + i) = (make_float4(vv[0], vv[1], vv[2], vv[3]));
          if (model) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(pp[0], pp[1]), hi = __floats2bfloat162_rn(pp[2], pp[3]);
            uint2 o;
            o.x = *reinterpret_cast<const uint32_t*>(&lo); o.y = *reinterpret_cast<const uint32_t*>(&hi);
            *reinterpret_cast<uint2*>(model + i) = o;
          }
        }
      }
      scalar_from = begin + nv * 4;
    }
    for (long long i = scalar_from + threadIdx.x; i < end; i += blockDim.x) {
      const float g = load_as_f32(grad, i, gdtype) * gs;
      const float mi = a.beta1 * m[i] + (1.f - a.beta1) * g;
      const float vi = a.beta2 * v[i] + (1.f - a.beta2) * g * g;
      m[i] = mi; v[i] = vi;
      const float denom = sqrtf(vi) * inv_sqrt_c2 + a.eps;
      const float p = master[i] * decay - step * mi / denom;
      master[i] = p;
      if (model) model[i] = __float2bfloat16_rn(p);
    }
  }
}

// The status word itself lives in mapped host memory (the host polls it without synchronising); a read of it
// costs a PCIe round trip per warp, which serialises to milliseconds when every warp of a large grid does it.
// One thread copies it into device memory first and the optimizer's blocks read that copy.
__global__ void status_gate_kernel(const unsigned int* __restrict__ status, unsigned int* __restrict__ gate) {
  pdl_launch_next();
  pdl_wait();
  *gate = *reinterpret_cast<const volatile unsigned int*>(status);
}

int sm_count(int device);
// blocks for `units` of work: at most `per_sm` per SM
static inline int mt_grid(long long units, int per_sm = 64) {
  const long long cap = static_cast<long long>(sm_count_current()) * per_sm;
  return (int)(units < cap ? (units < 1 ? 1 : units) : cap);
}
// at least 8 chunks per tensor on average: few quarters of a chunk are empty
static inline bool mt_long_tensors(int n, long long total_chunks) { return total_chunks >= 8ll * n; }

}  // namespace axb

using namespace axb;

template <bool CLIP>
static int l2norm_sq(const long long* table, int n, long long total_chunks, float* out, const ClipOut& clip, void* stream) {
  // Every block ends with an atomic: few blocks.  Whole chunks, unless there are so few of them that the last wave counts
  // and the tensors are long and found in one round of the search.  From DRAM, whole / quarters: 12 tensors of 64 chunks
  // 30.8 / 28.7 us, 8 of 10 12.3 / 10.2; 33 of 16 22.6 / 22.6, 300 of 16 121 / 127, 1500 of one half 31 / 45.
  if (n <= 32 && mt_long_tensors(n, total_chunks) && total_chunks < 16ll * sm_count_current())
    AXB_CUDA(pdl_launch(multi_l2norm_sq_kernel<MT_PARTS, CLIP>, dim3(mt_grid(total_chunks * MT_PARTS, 4)), dim3(MT_THREADS), 0, (cudaStream_t)stream, table, n, total_chunks, out, clip));
  else
    AXB_CUDA(pdl_launch(multi_l2norm_sq_kernel<1, CLIP>, dim3(mt_grid(total_chunks, 8)), dim3(MT_THREADS), 0, (cudaStream_t)stream, table, n, total_chunks, out, clip));
  return 0;
}
extern "C" int axb_multi_l2norm_sq(const long long* table, int n, long long total_chunks, float* out, void* stream) {
  return l2norm_sq<false>(table, n, total_chunks, out, ClipOut{}, stream);
}
// words: four 32-bit words, the first two zero on entry: squared norm, block counter, norm, min(1, max_norm / (norm + 1e-6)).
extern "C" int axb_multi_clip_factor(const long long* table, int n, long long total_chunks, float max_norm, float* words,
                                     void* stream) {
  return l2norm_sq<true>(table, n, total_chunks, words,
                   ClipOut{reinterpret_cast<unsigned int*>(words + 1), words + 2, words + 3, max_norm}, stream);
}
extern "C" int axb_multi_scale(const long long* table, int n, long long total_chunks, const float* scale, void* stream) {
  // quarters of a chunk where tensors are long: 29 against 30 us for 12 tensors of 64 chunks, 188 against 194 for 300 of 16,
  // but 104 against 96 for 1500 of 2
  if (mt_long_tensors(n, total_chunks))
    AXB_CUDA(pdl_launch(multi_scale_kernel<MT_PARTS>, dim3(mt_grid(total_chunks * MT_PARTS)), dim3(MT_THREADS), 0, (cudaStream_t)stream, table, n, total_chunks, scale));
  else
    AXB_CUDA(pdl_launch(multi_scale_kernel<1>, dim3(mt_grid(total_chunks)), dim3(MT_THREADS), 0, (cudaStream_t)stream, table, n, total_chunks, scale));
  return 0;
}
// Device-memory copy of the status word of the current device, refreshed on `stream` (see status_gate_kernel);
// null when the device has no status word.
static unsigned int* refreshed_status_gate(cudaStream_t stream) {
  int dev = 0;
  unsigned int* status = nullptr;
  unsigned int* gate = nullptr;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
    device_status_word(dev, &status);
    static unsigned int* gates[64] = {nullptr};
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (status && !gates[dev]) {
      if (cudaMalloc(&gates[dev], sizeof(unsigned int)) != cudaSuccess) { gates[dev] = nullptr; cudaGetLastError(); }
    }
    gate = status ? gates[dev] : nullptr;
  }
  if (gate) pdl_launch(status_gate_kernel, dim3(1), dim3(1), 0, stream, status, gate);
  return gate;
}

extern "C" int axb_multi_sgd(const long long* table, int n, long long total_chunks, float lr, float momentum,
                             float weight_decay, const float* grad_scale, void* stream) {
  unsigned int* gate = refreshed_status_gate((cudaStream_t)stream);
  AXB_CUDA(cudaGetLastError());
  const bool parts = mt_long_tensors(n, total_chunks);
  auto kern = parts ? multi_sgd_kernel<MT_PARTS> : multi_sgd_kernel<1>;
  kern<<<mt_grid(total_chunks * (parts ? MT_PARTS : 1)), MT_THREADS, 0, (cudaStream_t)stream>>>(table, n, total_chunks, lr, momentum, weight_decay, grad_scale, gate);
  AXB_CUDA(cudaGetLastError());
  return 0;
}

extern "C" int axb_multi_adamw(const long long* table, int n, long long total_chunks, float lr, float beta1, float beta2,
                               float eps, float weight_decay, float bias_c1, float bias_c2, const float* grad_scale,
                               const float* found_inf, void* stream) {
  // The step is also skipped when a kernel that ran before it on this device reported an expired wait:
  // its output (activations or gradients) is incomplete, and the host learns of it at its next check_status.
  unsigned int* gate = refreshed_status_gate((cudaStream_t)stream);
  AXB_CUDA(cudaGetLastError());
  AdamArgs a{lr, beta1, beta2, eps, weight_decay, bias_c1, bias_c2, grad_scale, found_inf, gate};
  // Many small units: the blocks of the last wave are soon done.  One B200, quarters / eighths / sixteenths of a chunk: 12 tensors of 64
  // chunks 239.0 / 225.5 / 224.5 us, 33 of 16 167 / 161 / 159, 10 of half a chunk 16.4 / 11.6 / 9.3; 300 of 16 1389 / 1372 / 1381.
  // Quarters for many tensors of one chunk: most of the others would be empty, 3000 of 4096 elements 78 / 98, 300 of 2048 8 / 16.
  const int parts = total_chunks < 2ll * n && n > 32 ? MT_PARTS : (total_chunks < 1024 ? 16 : 8);
  const auto kern = parts == MT_PARTS ? multi_adamw_kernel<MT_PARTS> : parts == 8 ? multi_adamw_kernel<8> : multi_adamw_kernel<16>;
  AXB_CUDA(pdl_launch(kern, dim3(mt_grid(total_chunks * parts)), dim3(ADAM_THREADS), 0, (cudaStream_t)stream, table, n, total_chunks, a));
  return 0;
}
