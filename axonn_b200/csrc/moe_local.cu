// Token permutation of a mixture-of-experts layer whose experts all live on this GPU: routing slots, dispatch of the
// token rows into expert-major capacity buffers, combine of the expert outputs, and their adjoints.
//
//   moe_slots    slot of every assignment inside its expert's buffer (order of the assignments, as a running count),
//                the inverse map (buffer row -> assignment) and the per-expert counts
//   moe_rows     one warp per buffer row: the row of its token (optionally scaled by the gate; the dot product with a
//                second buffer is the gate's gradient), zeros for rows without a token
//   moe_tokens   one warp per token: sum of the rows of its kept assignments (optionally weighted by the gate)
//
// All three are bound by memory traffic: every row is read and written once with 16-byte accesses, sums are fp32.
// One B200, 8192 tokens x 2048, 8 experts, top 2: slots 7 us (a running count through torch.cumsum over 16384 x 8 took
// 3454 us, one thread per column), dispatch 17 us, combine 21 us, adjoint with the gate's gradient 35 us.
#include "common.cuh"

namespace axb {

constexpr int MS_THREADS = 1024, MS_PER = 4;

// Block e numbers the assignments to expert e.  Assignment order is preserved by a block-wide scan over chunks of
// MS_THREADS * MS_PER consecutive assignments.  expert index -> slot < C: kept.  Buffers have Cp >= C rows per expert.
__global__ void __launch_bounds__(MS_THREADS)
moe_slots_kernel(const long long* __restrict__ idx, int n, int C, int Cp, int* __restrict__ dest, int* __restrict__ inverse,
                 int* __restrict__ counts, float* __restrict__ assigned) {
  __shared__ int warp_sum[2][32];
  const int e = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int base = 0;
  int it = 0;
  for (int a0 = 0; a0 < n; a0 += MS_THREADS * MS_PER, ++it) {
    const int a = a0 + threadIdx.x * MS_PER;
    bool hit[MS_PER];
    int mine = 0;
#pragma unroll
    for (int i = 0; i < MS_PER; ++i) { hit[i] = a + i < n && idx[a + i] == e; mine += hit[i]; }
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
    int* ws = warp_sum[it & 1];                       // double-buffered: one barrier per chunk
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    const int v = ws[lane];
    int pre = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, pre, o); if (lane >= o) pre += u; }
    const int before = __shfl_sync(0xffffffffu, pre - v, w), total = __shfl_sync(0xffffffffu, pre, 31);
    int slot = base + before + incl - mine;
#pragma unroll
    for (int i = 0; i < MS_PER; ++i)
      if (hit[i]) {
        dest[a + i] = slot < C ? e * Cp + slot : -1;
        if (slot < C) inverse[e * Cp + slot] = a + i;
        ++slot;
      }
    base += total;
  }
  for (int s = min(base, C) + threadIdx.x; s < Cp; s += MS_THREADS) inverse[e * Cp + s] = -1;
  if (threadIdx.x == 0) { counts[e] = min(base, C); assigned[e] = static_cast<float>(base); }
}

__device__ __forceinline__ void bf16x8_to_f32(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ uint4 f32_to_bf16x8(const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// out[row] = gate[a] * x[a / k] for the assignment a of buffer row `row`; zeros without one.  GATE: scaled by gate[a],
// and dgate[a] = sum_h x[a / k][h] * other[row][h].
template <bool GATE>
__global__ void __launch_bounds__(256)
moe_rows_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ inverse, __nv_bfloat16* __restrict__ out,
                const float* __restrict__ gate, const __nv_bfloat16* __restrict__ other, float* __restrict__ dgate,
                int rows, int k, int vecs) {
  const int lane = threadIdx.x & 31;
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8) {
    const int a = inverse[row];
    uint4* dst = reinterpret_cast<uint4*>(out) + static_cast<size_t>(row) * vecs;
    if (a < 0) {
      for (int v = lane; v < vecs; v += 32) dst[v] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const uint4* src = reinterpret_cast<const uint4*>(x) + static_cast<size_t>(a / k) * vecs;
    if (!GATE) {
#pragma unroll 4
      for (int v = lane; v < vecs; v += 32) dst[v] = __ldg(src + v);
    } else {
      const uint4* oth = reinterpret_cast<const uint4*>(other) + static_cast<size_t>(row) * vecs;
      const float gt = gate[a];
      float dot = 0.f;
#pragma unroll 4
      for (int v = lane; v < vecs; v += 32) {
        float f[8], o[8];
        bf16x8_to_f32(__ldg(src + v), f);
        bf16x8_to_f32(__ldg(oth + v), o);
#pragma unroll
        for (int i = 0; i < 8; ++i) { dot += f[i] * o[i]; f[i] *= gt; }
        dst[v] = f32_to_bf16x8(f);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (lane == 0) dgate[a] = dot;
    }
  }
}

// out[t] = sum over the choices j of token t that were kept of gate[t, j] * buf[dest[t, j]]  (gate null: weight 1)
__global__ void __launch_bounds__(256)
moe_tokens_kernel(const __nv_bfloat16* __restrict__ buf, const int* __restrict__ dest, const float* __restrict__ gate,
                  __nv_bfloat16* __restrict__ out, int T, int k, int vecs) {
  const int lane = threadIdx.x & 31;
  for (int t = blockIdx.x * 8 + (threadIdx.x >> 5); t < T; t += gridDim.x * 8) {
    uint4* dst = reinterpret_cast<uint4*>(out) + static_cast<size_t>(t) * vecs;
#pragma unroll 2
    for (int v = lane; v < vecs; v += 32) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int j = 0; j < k; ++j) {
        const int d = __ldg(dest + static_cast<size_t>(t) * k + j);
        if (d < 0) continue;
        const float w = gate ? __ldg(gate + static_cast<size_t>(t) * k + j) : 1.f;
        float f[8];
        bf16x8_to_f32(__ldg(reinterpret_cast<const uint4*>(buf) + static_cast<size_t>(d) * vecs + v), f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += w * f[i];
      }
      dst[v] = f32_to_bf16x8(acc);
    }
  }
}

static int warp_rows_grid(int rows) {
  const int want = (rows + 7) / 8, cap = sm_count_current() * 8;
  return want < cap ? (want < 1 ? 1 : want) : cap;
}

}  // namespace axb

using namespace axb;

// idx: [n] int64 expert of every assignment; dest: [n] int32 buffer row or -1; inverse: [E * Cp] int32 assignment or -1;
// counts: [E] int32 rows in use (<= C); assigned: [E] fp32 assignments before the capacity cut.
extern "C" int axb_moe_slots(const long long* idx, long long n, int E, int C, int Cp, int* dest, int* inverse, int* counts,
                             float* assigned, void* stream) {
  if (n <= 0 || n > 0x7ffffff0ll || E <= 0 || C <= 0 || Cp < C || static_cast<long long>(E) * Cp > 0x7fffffffll) {
    set_error("moe_slots: bad sizes");
    return -1;
  }
  moe_slots_kernel<<<E, MS_THREADS, 0, (cudaStream_t)stream>>>(idx, static_cast<int>(n), C, Cp, dest, inverse, counts, assigned);
  AXB_CUDA(cudaGetLastError());
  return 0;
}

// gate null: out[row] = x[token of row]; otherwise scaled, with dgate (zero on entry for dropped assignments)
extern "C" int axb_moe_rows(const void* x, const int* inverse, void* out, const float* gate, const void* other, float* dgate,
                            int rows, int k, int H, void* stream) {
  if (H % 8 || rows <= 0 || k <= 0) { set_error("moe_rows: hidden must be a multiple of 8"); return -1; }
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(other)) & 15) {
    set_error("moe_rows: tensors must be 16-byte aligned");
    return -1;
  }
  const int grid = warp_rows_grid(rows);
  if (gate)
    moe_rows_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, inverse, (__nv_bfloat16*)out, gate,
                                                                 (const __nv_bfloat16*)other, dgate, rows, k, H / 8);
  else
    moe_rows_kernel<false><<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, inverse, (__nv_bfloat16*)out, nullptr,
                                                                  nullptr, nullptr, rows, k, H / 8);
  AXB_CUDA(cudaGetLastError());
  return 0;
}

extern "C" int axb_moe_tokens(const void* buf, const int* dest, const float* gate, void* out, int T, int k, int H, void* stream) {
  if (H % 8 || T <= 0 || k <= 0) { set_error("moe_tokens: hidden must be a multiple of 8"); return -1; }
  if ((reinterpret_cast<uintptr_t>(buf) | reinterpret_cast<uintptr_t>(out)) & 15) {
    set_error("moe_tokens: tensors must be 16-byte aligned");
    return -1;
  }
  moe_tokens_kernel<<<warp_rows_grid(T), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)buf, dest, gate,
                                                                        (__nv_bfloat16*)out, T, k, H / 8);
  AXB_CUDA(cudaGetLastError());
  return 0;
}
