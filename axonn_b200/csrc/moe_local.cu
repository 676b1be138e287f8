// Token permutation of a mixture-of-experts layer whose experts all live on this GPU: routing slots, dispatch of the
// token rows into expert-major capacity buffers, combine of the expert outputs, and their adjoints.
//
//   moe_route    softmax over the experts, the k largest, their gates and the sums for the balance loss; its adjoint
//   moe_slots    slot of every assignment inside its expert's buffer (order of the assignments, as a running count),
//                the inverse map (buffer row -> assignment) and the per-expert counts
//   moe_rows     one warp per buffer row: the row of its token (optionally scaled by the gate; the dot product with a
//                second buffer is the gate's gradient), zeros for rows without a token
//   moe_tokens   one warp per token: sum of the rows of its kept assignments (optionally weighted by the gate)
//
// All three are bound by memory traffic: every row is read and written once with 16-byte accesses, sums are fp32.
// One B200, 8192 tokens x 2048, 8 experts, top 2: routing 4 us, slots 9 us, adjoint of the routing 7 us (as thirty torch
// operations 170 us; layer forward and backward 5117 -> 4944 us, 1289 -> 892 us of host time); dispatch 17 us, combine
// 21 us, adjoint with the gate's gradient 35 us.
#include "common.cuh"

namespace axb {

constexpr int MS_THREADS = 1024, MS_PER = 4;

// What the layer reports about its routing, written by the slot kernel when it follows the routing kernel.
struct RouteStats {
  const float* prob_part;        // [parts, E] sums of the probabilities; null: slots and counts only
  int parts;
  float inv_tokens, inv_assignments;
  unsigned int* blocks_done;     // zero on entry
  float* prob_sum;               // [E] scratch
  float* assigned;               // [E] a second copy of the assignments
  float* dropped;                // [E]
  float* aux;                    // E * sum_e (share of the assignments) * (mean probability)
  float* drop_fraction;
};

// Block e numbers the assignments to expert e.  Assignment order is preserved by a block-wide scan over chunks of
// MS_THREADS * MS_PER consecutive assignments.  expert index -> slot < C: kept.  Buffers have Cp >= C rows per expert.
template <typename Index>
__global__ void __launch_bounds__(MS_THREADS)
moe_slots_kernel(const Index* __restrict__ idx, int n, int C, int Cp, int* __restrict__ dest, int* __restrict__ inverse,
                 int* __restrict__ counts, float* __restrict__ assigned, const RouteStats st) {
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
  if (st.prob_part == nullptr || w != 0) return;
  // one warp: this expert's probabilities in the order of the parts, then (last block) the sums over the experts
  const int E = gridDim.x;
  float p = 0.f;
  for (int i = lane; i < st.parts; i += 32) p += st.prob_part[static_cast<size_t>(i) * E + e];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
  if (lane != 0) return;
  st.prob_sum[e] = p;
  st.assigned[e] = static_cast<float>(base);
  st.dropped[e] = static_cast<float>(max(base - C, 0));
  __threadfence();
  if (atomicAdd(st.blocks_done, 1u) != gridDim.x - 1) return;
  __threadfence();
  float aux = 0.f, kept = 0.f;
  for (int i = 0; i < E; ++i) {
    const float a = __ldcg(assigned + i);
    aux += a * st.inv_assignments * (__ldcg(st.prob_sum + i) * st.inv_tokens);
    kept += a - __ldcg(st.dropped + i);
  }
  *st.aux = E * aux;
  *st.drop_fraction = 1.f - kept * st.inv_assignments;
}

// ---------------------------------------------------------------------------------------------- top-k softmax router
// One thread per token, its E <= EM logits in registers.  The k largest probabilities are taken with equal ones in the order
// of the experts (what torch.topk does for the set that it returns); a row with a NaN has only NaN probabilities and takes
// the first k experts.  Everything is fp32 from the bf16 logits on.
constexpr int MR_THREADS = 128;

template <int EM>
__device__ __forceinline__ void route_softmax(const __nv_bfloat16* __restrict__ z, int E, float (&p)[EM]) {
  if ((E & 7) == 0 && (reinterpret_cast<uintptr_t>(z) & 15) == 0) {
#pragma unroll
    for (int v = 0; v < EM / 8; ++v) {
      const uint4 u = v * 8 < E ? __ldg(reinterpret_cast<const uint4*>(z) + v) : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int i = 0; i < 4; ++i) { const float2 t = __bfloat1622float2(h[i]); p[v * 8 + 2 * i] = t.x; p[v * 8 + 2 * i + 1] = t.y; }
    }
  } else {
#pragma unroll
    for (int i = 0; i < EM; ++i) p[i] = i < E ? __bfloat162float(z[i]) : -INFINITY;
  }
  float m = -INFINITY, s = 0.f;
#pragma unroll
  for (int i = 0; i < EM; ++i) m = fmaxf(m, p[i]);
  // the double-precision exponential is correct to the last fp32 bit, which the fast one is not; it is a few per token
#pragma unroll
  for (int i = 0; i < EM; ++i) { p[i] = i < E ? static_cast<float>(exp(static_cast<double>(p[i] - m))) : 0.f; s += p[i]; }
#pragma unroll
  for (int i = 0; i < EM; ++i) p[i] = __fdiv_rn(p[i], s);
}

template <int EM>
__global__ void __launch_bounds__(MR_THREADS)
moe_route_kernel(const __nv_bfloat16* __restrict__ logits, int T, int E, int k, int* __restrict__ idx, float* __restrict__ gate,
                 float* __restrict__ prob_part, unsigned int* __restrict__ blocks_done) {
  __shared__ float part[MR_THREADS / 32][EM];
  const int t = blockIdx.x * MR_THREADS + threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (t == 0) *blocks_done = 0;                       // of the slot kernel that follows
  float p[EM];
  if (t < T) route_softmax<EM>(logits + static_cast<size_t>(t) * E, E, p);
  else {
#pragma unroll
    for (int i = 0; i < EM; ++i) p[i] = 0.f;
  }
#pragma unroll
  for (int i = 0; i < EM; ++i) {
    float v = p[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) part[w][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < E) {
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < MR_THREADS / 32; ++i) v += part[i][threadIdx.x];
    prob_part[static_cast<size_t>(blockIdx.x) * E + threadIdx.x] = v;
  }
  if (t >= T) return;
  float sum = 0.f;
  unsigned int taken = 0u;
  for (int j = 0; j < k; ++j) {
    int best = -1;
    float top = 0.f;
#pragma unroll
    for (int i = 0; i < EM; ++i)
      if (i < E && !((taken >> i) & 1u) && (best < 0 || p[i] > top)) { best = i; top = p[i]; }
    taken |= 1u << best;
    idx[static_cast<size_t>(t) * k + j] = best;
    gate[static_cast<size_t>(t) * k + j] = top;
    sum += top;
  }
  for (int j = 0; j < k; ++j) gate[static_cast<size_t>(t) * k + j] = __fdiv_rn(gate[static_cast<size_t>(t) * k + j], sum);
}

// dlogits of (gate, aux) by their gradients; either may be null.  With s the sum of the chosen probabilities:
// dp_e = [e chosen] (dgate_e - sum_j dgate_j gate_j) / s + daux * E * (share of e) / T,   dlogit = p (dp - sum p dp).
template <int EM>
__global__ void __launch_bounds__(MR_THREADS)
moe_route_bwd_kernel(const __nv_bfloat16* __restrict__ logits, int T, int E, int k, const int* __restrict__ idx,
                     const float* __restrict__ gate, const float* __restrict__ dgate, const float* __restrict__ daux,
                     const float* __restrict__ assigned, float aux_scale, __nv_bfloat16* __restrict__ dlogits) {
  const int t = blockIdx.x * MR_THREADS + threadIdx.x;
  if (t >= T) return;
  float p[EM], dp[EM];
  route_softmax<EM>(logits + static_cast<size_t>(t) * E, E, p);
  const float da = daux ? *daux * aux_scale : 0.f;
#pragma unroll
  for (int i = 0; i < EM; ++i) dp[i] = daux && i < E ? da * __ldg(assigned + i) : 0.f;
  if (dgate) {
    const size_t at = static_cast<size_t>(t) * k;
    float s = 0.f, mean = 0.f;
    for (int j = 0; j < k; ++j) {
      const int e = idx[at + j];
      mean += dgate[at + j] * gate[at + j];
#pragma unroll
      for (int i = 0; i < EM; ++i) if (i == e) s += p[i];
    }
    for (int j = 0; j < k; ++j) {
      const int e = idx[at + j];
      const float d = __fdiv_rn(dgate[at + j] - mean, s);
#pragma unroll
      for (int i = 0; i < EM; ++i) if (i == e) dp[i] += d;
    }
  }
  float dot = 0.f;
#pragma unroll
  for (int i = 0; i < EM; ++i) dot += p[i] * dp[i];
#pragma unroll
  for (int i = 0; i < EM; ++i)
    if (i < E) dlogits[static_cast<size_t>(t) * E + i] = __float2bfloat16_rn(p[i] * (dp[i] - dot));
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
  moe_slots_kernel<long long><<<E, MS_THREADS, 0, (cudaStream_t)stream>>>(idx, static_cast<int>(n), C, Cp, dest, inverse, counts,
                                                                          assigned, RouteStats{});
  AXB_CUDA(cudaGetLastError());
  return 0;
}

// Router and slots of T tokens over E <= AXB_MOE_MAX_EXPERTS experts, two launches.  logits [T, E] bf16; idx [T, k] int32 chosen
// experts; gate [T, k] their renormalised probabilities; dest, inverse, counts, assigned as in axb_moe_slots; assigned_too [E] the
// same as assigned (for a caller who keeps one and hands on the other); dropped [E]; aux and drop_fraction scalars.  scratch: (ceil(T / 128) + 1) * E + 1 words.
extern "C" int axb_moe_route(const void* logits, int T, int E, int k, int C, int Cp, int* idx, float* gate, int* dest,
                             int* inverse, int* counts, float* assigned, float* assigned_too, float* dropped, float* aux,
                             float* drop_fraction, float* scratch, void* stream) {
  const long long n = static_cast<long long>(T) * k;
  if (T <= 0 || k <= 0 || k > E || E > AXB_MOE_MAX_EXPERTS || n > 0x7ffffff0ll || C <= 0 || Cp < C ||
      static_cast<long long>(E) * Cp > 0x7fffffffll) {
    set_error("moe_route: bad sizes");
    return -1;
  }
  const int grid = (T + MR_THREADS - 1) / MR_THREADS;
  float* prob_sum = scratch + static_cast<size_t>(grid) * E;
  unsigned int* done = reinterpret_cast<unsigned int*>(prob_sum + E);
  auto kern = E <= 8 ? moe_route_kernel<8> : (E <= 16 ? moe_route_kernel<16> : moe_route_kernel<AXB_MOE_MAX_EXPERTS>);
  kern<<<grid, MR_THREADS, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, T, E, k, idx, gate, scratch, done);
  AXB_CUDA(cudaGetLastError());
  const RouteStats st{scratch, grid, 1.f / T, 1.f / static_cast<float>(n), done, prob_sum, assigned_too, dropped, aux, drop_fraction};
  moe_slots_kernel<int><<<E, MS_THREADS, 0, (cudaStream_t)stream>>>(idx, static_cast<int>(n), C, Cp, dest, inverse, counts, assigned, st);
  AXB_CUDA(cudaGetLastError());
  return 0;
}

// dlogits [T, E] bf16 by dgate [T, k] and daux (a scalar on the device); either may be null
extern "C" int axb_moe_route_bwd(const void* logits, int T, int E, int k, const int* idx, const float* gate, const float* dgate,
                                 const float* daux, const float* assigned, void* dlogits, void* stream) {
  if (T <= 0 || k <= 0 || k > E || E > AXB_MOE_MAX_EXPERTS) { set_error("moe_route_bwd: bad sizes"); return -1; }
  const float aux_scale = static_cast<float>(static_cast<double>(E) / (static_cast<double>(T) * k) / T);
  auto kern = E <= 8 ? moe_route_bwd_kernel<8> : (E <= 16 ? moe_route_bwd_kernel<16> : moe_route_bwd_kernel<AXB_MOE_MAX_EXPERTS>);
  kern<<<(T + MR_THREADS - 1) / MR_THREADS, MR_THREADS, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)logits, T, E, k, idx, gate, dgate, daux, assigned, aux_scale, (__nv_bfloat16*)dlogits);
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
