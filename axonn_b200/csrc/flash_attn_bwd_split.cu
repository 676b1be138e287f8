// Causal flash attention backward as two tcgen05 kernels without atomics (sm_100a), grouped-query aware.
//
// The one-kernel backward (flash_attn.cu) keeps dK and dV in tensor memory and has to push dQ partials through
// the score columns and a global fp32 accumulator, which serialises every step.  Here the work is split the way
// the forward kernel is organised - persistent CTAs, every probability / score-gradient tile goes from the
// softmax threads back into tensor memory as the A operand of the next MMA, nothing is staged in shared memory:
//
//   fa_bwd_dq_kernel   one 128-row query tile per work item, walks the key tiles up to the diagonal:
//                      S = Q K^T and dP = dO V^T (128 x 128 each) into tensor memory, the softmax threads read
//                      them into registers (the MMA warp then already issues the next tile's S and dP),
//                      dS = P (dP - delta) goes back as bf16 and dQ += dS K accumulates in tensor memory.
//                      dQ is scaled and written once, as bf16, into the packed gradient tensor.
//   fa_bwd_dkv_kernel  one 128-row key tile per work item, walks the query tiles from the diagonal down (and the
//                      query heads of the group) in steps of 64 queries: S^T = K Q^T and dP^T = V dO^T into
//                      double-buffered 64-column score buffers (a thread has 4 keys x 8 queries), P^T and dS^T go back
//                      as bf16, dV += P^T dO and dK += dS^T Q accumulate in tensor memory; one MMA warp per
//                      accumulator.
//
// Both recompute S, so the pair does 7 MMA units per tile against 5 of the one-kernel form, but neither has a
// serial chain through shared memory, global reductions or the fp32 accumulator (no zero fill, no conversion).
// delta = rowsum(dO * O) comes from a small pre-kernel.  All waits are bounded.
#include <cstdlib>

#include "common.cuh"

namespace axb {

int make_tmap_3d_bf16(CUtensorMap* out, const void* ptr, uint64_t batch, uint64_t rows, uint64_t cols, uint32_t box_rows);
int sm_count(int device);

struct FaSplitParams {
  // per query row, [B, heads, Sp] with Sp = S rounded up to 128: -lse in units of log2 and -delta.  Rows past S have
  // -inf there, so that their probabilities (and with them every contribution to dK, dV and dQ) are exact zeros.
  const float* neg_lse2;
  const float* neg_delta;
  __nv_bfloat16* dqkv;   // [B, S, G, qpk + 2, D]
  int B, S, Sp, G, qpk;
  float scale, scale_log2;
  unsigned int* status;
  unsigned long long timeout_ns;
  int debug;   // ablation builds only (-DAXB_ABLATION, read once from AXB_FA_DEBUG; otherwise 0 and compiled out): 4 phase timers
};

// TMA warp, two MMA warps and an idle one (first warpgroup), 16 softmax warps.  The probabilities are what bounds both
// kernels (one exponential, one conversion and two multiply-adds per score, behind tensor-memory loads); four warps
// per scheduler with 32 scores per thread hide that latency, two warps with 64 do not.  Registers: 640 threads get 96
// each at launch, 128 * 64 + 512 * 104 after the split are exactly those.
// Measured on a B200, 8 x 2048, 16 heads, head_dim 128, back to back in one graph: dQ, dK / dV and delta kernel together 660 -
// 700 us with two warps per scheduler, 584 - 599 us with four, 502 - 516 us now (the library's backward 434 us in the same run).
constexpr int FS_THREADS = 640;
constexpr int FS_SOFTMAX_WARPS = 16;
#define FS_REGS_CONTROL "setmaxnreg.dec.sync.aligned.u32 64;"
#define FS_REGS_SOFTMAX "setmaxnreg.inc.sync.aligned.u32 104;"

__device__ __forceinline__ uint32_t fs_pack(float2 v) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// neg_delta[b, h, s] = -sum_d dO[b, s, h, d] * O[b, s, h, d] and neg_lse2 = -lse * log2(e); HD / 8 threads per row, four
// rows per thread with all their 16-byte loads in flight.  Rows S .. Sp - 1 get -inf / 0 (see FaSplitParams).  The grid's
// y dimension is the batch, so that a row's data lies at its index and the only division is by the head count.  One B200,
// 262144 rows: head_dim 128 (134 MB) 35 -> 31 us, head_dim 64 20 -> 11 us (64-bit divisions for every 16 bytes before).
constexpr int FS_DELTA_ROWS = 4;
template <int HD>
__global__ void __launch_bounds__(256)
fa_split_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                      const float* __restrict__ lse, float* __restrict__ neg_lse2, float* __restrict__ neg_delta,
                      int B, int S, int Sp, unsigned H) {
  constexpr unsigned TPR = HD / 8, RPT = 256 / TPR;          // threads per row, rows per step of the block
  const unsigned rows = static_cast<unsigned>(Sp) * H, live_rows = static_cast<unsigned>(S) * H, sub = threadIdx.x % TPR;
  for (unsigned b = blockIdx.y; b < static_cast<unsigned>(B); b += gridDim.y) {
  const size_t base = static_cast<size_t>(b) * live_rows * HD, vec = static_cast<size_t>(b) * H;
  // all threads of a warp run the same number of rounds: the row's lanes are reduced with full-warp shuffles
  for (unsigned r0 = blockIdx.x * (RPT * FS_DELTA_ROWS); r0 < rows; r0 += gridDim.x * (RPT * FS_DELTA_ROWS)) {
    uint4 a[FS_DELTA_ROWS], c[FS_DELTA_ROWS];
#pragma unroll
    for (int u = 0; u < FS_DELTA_ROWS; ++u) {
      const unsigned row = r0 + u * RPT + threadIdx.x / TPR;
      a[u] = c[u] = make_uint4(0u, 0u, 0u, 0u);
      if (row < live_rows) {
        a[u] = __ldg(reinterpret_cast<const uint4*>(o + base + static_cast<size_t>(row) * HD + sub * 8));
        c[u] = __ldg(reinterpret_cast<const uint4*>(d_o + base + static_cast<size_t>(row) * HD + sub * 8));
      }
    }
#pragma unroll
    for (int u = 0; u < FS_DELTA_ROWS; ++u) {
      const unsigned row = r0 + u * RPT + threadIdx.x / TPR;
      const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a[u]);
      const __nv_bfloat162* c2 = reinterpret_cast<const __nv_bfloat162*>(&c[u]);
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = __bfloat1622float2(a2[i]), y = __bfloat1622float2(c2[i]);
        acc += x.x * y.x + x.y * y.y;
      }
#pragma unroll
      for (unsigned off = TPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      if (sub == 0 && row < rows) {
        const unsigned s = row / H, h = row - s * H;
        const size_t dst = (vec + h) * Sp + s;
        neg_delta[dst] = -acc;
        neg_lse2[dst] = row < live_rows ? -lse[(vec + h) * S + s] * 1.4426950408889634f : -INFINITY;
      }
    }
  }
  }
}

// ------------------------------------------------------------------------------------------------ dQ
template <int HD>
struct DqSmem {
  static constexpr int TILE = 128 * HD * 2;
  static constexpr int Q_OFF = 0, DO_OFF = TILE;
  // K is held from the step's S MMA until its dQ MMA, a whole step later, so it gets three stages; V is released
  // as soon as dP has completed and gets two (7 tiles = 224 KB at head_dim 128).
  static constexpr int K_OFF = 2 * TILE;           // 3 stages
  static constexpr int V_OFF = 5 * TILE;           // 2 stages
  static constexpr int BAR_OFF = 7 * TILE;
  static constexpr int NBARS = 2 + 6 + 4 + 4;
  static constexpr int TOTAL = BAR_OFF + NBARS * 8 + 16 + 1024;
};

__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      : : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// Counterpart of tmem_ld_16x32 for pairs of columns packed into one of 32 bits.
__device__ __forceinline__ void tmem_st_16x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
      : : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
      : "memory");
}

// Work item k of this CTA: query tiles sorted by decreasing length (tile i walks i + 1 key tiles), dealt to the
// persistent CTAs in a snake.
struct DqItem { int i, head, b; };
__device__ __forceinline__ bool dq_item(const FaSplitParams& p, int k, DqItem& w) {
  const int G = gridDim.x, c = blockIdx.x;
  const int heads = p.G * p.qpk, bh = p.B * heads, nq = p.Sp / 128;
  const int idx = k * G + ((k & 1) ? G - 1 - c : c);
  if (idx >= bh * nq) return false;
  w.i = nq - 1 - idx / bh;
  const int rem = idx % bh;
  w.head = rem % heads;
  w.b = rem / heads;
  return true;
}

template <int HD>
__global__ void __launch_bounds__(FS_THREADS, 1)
fa_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO, const FaSplitParams p) {
  using S_ = DqSmem<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S_::BAR_OFF);
  uint64_t* q_full = bars;          // Q and dO of the item
  uint64_t* q_empty = bars + 1;
  uint64_t* k_full = bars + 2;      // [3]
  uint64_t* k_empty = bars + 5;     // [3]
  uint64_t* v_full = bars + 8;      // [2]
  uint64_t* v_empty = bars + 10;    // [2]
  uint64_t* sdp_full = bars + 12;   // S and dP of a step are complete
  uint64_t* sdp_free = bars + 13;   // ... and held in registers: their columns may be overwritten
  uint64_t* ds_full = bars + 14;    // dS of a step is in tensor memory
  uint64_t* dq_done = bars + 15;    // the step's dQ MMA has completed (dS may be overwritten; at the end: dQ final)
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + S_::NBARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t timeout = p.timeout_ns;
  const int heads = p.G * p.qpk;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1); mbar_init(q_empty, 1);
    for (int i = 0; i < 3; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 2); }   // released by both MMA warps
    for (int i = 0; i < 2; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    mbar_init(sdp_full, 1); mbar_init(sdp_free, FS_SOFTMAX_WARPS); mbar_init(ds_full, FS_SOFTMAX_WARPS); mbar_init(dq_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tmQKV); tma_prefetch_desc(&tmDO); }
  if (warp == 1) { tmem_alloc(tmem_ptr_smem, 512); tmem_relinquish(); }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  // columns: S [0,128), dP [128,256), dS (bf16, 128 keys) [256,320), dQ [384,384+HD)
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 128, tm_ds = tmem_base + 256, tm_dq = tmem_base + 384;

  if (warp < 4) {
   asm volatile(FS_REGS_CONTROL);
   if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      uint32_t kvc = 0;
      DqItem w;
      for (int it = 0; ok && dq_item(p, it, w); ++it) {
        const int g = w.head / p.qpk, jq = w.head % p.qpk;
        const int col_q = (g * (p.qpk + 2) + jq) * HD;
        const int col_k = (g * (p.qpk + 2) + p.qpk) * HD;
        const int col_v = col_k + HD;
        const int row0 = w.i * 128;
        if (!mbar_wait(q_empty, (it & 1) ^ 1, abort_flag, timeout)) { ok = false; break; }
        mbar_expect_tx(q_full, 2 * S_::TILE);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) {
          tma_load_3d(smem + S_::Q_OFF + c * 16384, &tmQKV, q_full, col_q + 64 * c, row0, w.b);
          tma_load_3d(smem + S_::DO_OFF + c * 16384, &tmDO, q_full, w.head * HD + 64 * c, row0, w.b);
        }
        for (int j = 0; j <= w.i && ok; ++j, ++kvc) {
          const int st = kvc % 3;
          const uint32_t ph = (kvc / 3) & 1;
          const int krow = j * 128;
          if (!mbar_wait(&k_empty[st], ph ^ 1, abort_flag, timeout)) { ok = false; break; }
          mbar_expect_tx(&k_full[st], S_::TILE);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c)
            tma_load_3d(smem + S_::K_OFF + st * S_::TILE + c * 16384, &tmQKV, &k_full[st], col_k + 64 * c, krow, w.b);
          if (!mbar_wait(&v_empty[kvc & 1], ((kvc >> 1) & 1) ^ 1, abort_flag, timeout)) { ok = false; break; }
          mbar_expect_tx(&v_full[kvc & 1], S_::TILE);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c)
            tma_load_3d(smem + S_::V_OFF + (kvc & 1) * S_::TILE + c * 16384, &tmQKV, &v_full[kvc & 1], col_v + 64 * c, krow, w.b);
        }
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();     // give in-flight copies time to land before the CTA exits
        while (globaltimer_ns() - t0 < 200000ull) {}
        report_status(p.status, 0x421u);
      }
    }
   } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA warp 1: S = Q K^T and dP = dO V^T
    if (elect_one()) {
      bool ok = true;
      const uint32_t idesc_s = umma_idesc(1, 0, 0, 128, 128);
      const uint64_t qd = umma_smem_desc(smem_u32(smem + S_::Q_OFF), 16, 1024);
      const uint64_t dod = umma_smem_desc(smem_u32(smem + S_::DO_OFF), 16, 1024);
      auto issue_sdp = [&](uint32_t kv) {
        const uint64_t kd = umma_smem_desc(smem_u32(smem + S_::K_OFF + (kv % 3) * S_::TILE), 16, 1024);
        const uint64_t vd = umma_smem_desc(smem_u32(smem + S_::V_OFF + (kv & 1) * S_::TILE), 16, 1024);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          umma_f16(tm_s, qd + off, kd + off, idesc_s, kk != 0 ? 1u : 0u);
        }
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          umma_f16(tm_dp, dod + off, vd + off, idesc_s, kk != 0 ? 1u : 0u);
        }
      };
      uint32_t kvc = 0, c = 0;     // key tiles and steps of earlier items (ring stages, barrier phases)
      const bool probe = AXB_DBG(p, 4) && blockIdx.x == 0;
      long long pw_free = 0, pw_kv = 0, p_mark = 0, p_t0 = probe ? clock64() : 0;
      DqItem w;
      for (int it = 0; ok && dq_item(p, it, w); ++it) {
        const int n = w.i + 1;
        if (!mbar_wait(q_full, it & 1, abort_flag, timeout)) { ok = false; break; }
        for (int j = 0; j < n && ok; ++j, ++c) {
          const uint32_t kv = kvc + j;
          // S and dP columns are free once the softmax threads hold the previous step's tile in registers
          if (probe) p_mark = clock64();
          if (c >= 1 && !mbar_wait(sdp_free, (c - 1) & 1, abort_flag, timeout)) { ok = false; break; }
          if (probe) { const long long now = clock64(); pw_free += now - p_mark; p_mark = now; }
          if (!mbar_wait(&k_full[kv % 3], (kv / 3) & 1, abort_flag, timeout) ||
              !mbar_wait(&v_full[kv & 1], (kv >> 1) & 1, abort_flag, timeout)) { ok = false; break; }
          if (probe) pw_kv += clock64() - p_mark;
          tcgen05_fence_after();
          issue_sdp(kv);
          umma_commit(sdp_full);
          umma_commit(&v_empty[kv & 1]);
          umma_commit(&k_empty[kv % 3]);              // first of the two releases of this K tile
          if (j + 1 == n) umma_commit(q_empty);       // the item's last reads of Q and dO
        }
        kvc += n;
      }
      if (probe) {
        volatile unsigned int* wd = reinterpret_cast<volatile unsigned int*>(p.status);
        wd[12] = static_cast<unsigned>(pw_free); wd[13] = static_cast<unsigned>(pw_kv);
        wd[15] = static_cast<unsigned>(clock64() - p_t0);
      }
      if (!ok) report_status(p.status, 0x422u);
    }
   } else if (warp == 2) {
    // ------------------------------------------------------------------ MMA warp 2: dQ += dS K
    if (elect_one()) {
      bool ok = true;
      const uint32_t idesc_dq = umma_idesc(1, 0, 1, 128, HD);
      uint32_t kvc = 0, c = 0;
      const bool probe = AXB_DBG(p, 4) && blockIdx.x == 0;
      long long pw_ds = 0, p_mark = 0;
      DqItem w;
      for (int it = 0; ok && dq_item(p, it, w); ++it) {
        const int n = w.i + 1;
        for (int j = 0; j < n && ok; ++j, ++c) {
          const uint32_t kv = kvc + j;
          if (probe) p_mark = clock64();
          // dS of the step is in tensor memory (the softmax threads saw S of this K tile, so the tile is loaded)
          if (!mbar_wait(ds_full, c & 1, abort_flag, timeout)) { ok = false; break; }
          if (probe) pw_ds += clock64() - p_mark;
          tcgen05_fence_after();
          // K as the B operand of dQ = dS K: keys are the reduction dimension, head_dim is contiguous (MN-major):
          // 64-wide column chunks 16 KB apart (leading), 8-row groups 1 KB apart (stride)
          const uint64_t kmn = umma_smem_desc(smem_u32(smem + S_::K_OFF + (kv % 3) * S_::TILE), 16384, 1024);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16_ts(tm_dq, tm_ds + kk * 8, kmn + ((kk * 2048) >> 4), idesc_dq, (j == 0 && kk == 0) ? 0u : 1u);
          umma_commit(dq_done);
          umma_commit(&k_empty[kv % 3]);              // second release of this K tile
        }
        kvc += n;
      }
      if (probe) reinterpret_cast<volatile unsigned int*>(p.status)[14] = static_cast<unsigned>(pw_ds);
      if (!ok) report_status(p.status, 0x424u);
    }
   }
  } else {
    // ------------------------------------------------------------------ P, dS: thread = (query row, quarter of the keys)
    asm volatile(FS_REGS_SOFTMAX);
    const int q4 = warp & 3;
    const int quarter = (warp - 4) >> 2;
    const int r = q4 * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(q4 * 32) << 16;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    bool ok = true;
    uint32_t c = 0;
    const bool probe = AXB_DBG(p, 4) && blockIdx.x == 0 && warp == 4 && lane == 0;
    long long pw_s = 0, pt_ld = 0, pt_cmp = 0, pw_dq = 0, pt_st = 0, p_mark = 0;
    DqItem w;
    for (int it = 0; ok && dq_item(p, it, w); ++it) {
      const int n = w.i + 1;
      const int srow = w.i * 128 + r;
      const size_t vec = (static_cast<size_t>(w.b) * heads + w.head) * p.Sp + srow;
      const float nl = p.neg_lse2[vec], nd = p.neg_delta[vec];
      const float2 nl2 = make_float2(nl, nl), nd2 = make_float2(nd, nd);
      for (int j = 0; j < n; ++j, ++c) {
        if (probe) p_mark = clock64();
        if (!mbar_wait(sdp_full, c & 1, abort_flag, timeout)) { ok = false; break; }
        if (probe) { const long long now = clock64(); pw_s += now - p_mark; p_mark = now; }
        tcgen05_fence_after();
        uint32_t sv[32], dv[32];
        tmem_ld_32x32(tm_s + lane_base + quarter * 32, sv);
        tmem_ld_32x32(tm_dp + lane_base + quarter * 32, dv);
        tmem_ld_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(sdp_free);          // the MMA warp may issue the next tile's S and dP
        if (probe) { const long long now = clock64(); pt_ld += now - p_mark; p_mark = now; }
        if (j == w.i) {                                // keys to the right of the query: probability 0
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (quarter * 32 + i > r) sv[i] = 0xff800000u;
        }
        // dS = P (dP - delta); the softmax scale is applied once to the finished dQ and dK
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sc2, nl2);
          const float2 t = __fadd2_rn(make_float2(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])), nd2);
          packed[i] = fs_pack(__fmul2_rn(make_float2(exp2f(x.x), exp2f(x.y)), t));
        }
        // the previous step's dQ MMA (of this or of the previous item) has read its dS: every phase is observed
        if (probe) { const long long now = clock64(); pt_cmp += now - p_mark; p_mark = now; }
        if (c >= 1 && !mbar_wait(dq_done, (c - 1) & 1, abort_flag, timeout)) { ok = false; break; }
        if (probe) { const long long now = clock64(); pw_dq += now - p_mark; p_mark = now; }
        tmem_st_32x16(tm_ds + lane_base + quarter * 16, packed);
        tmem_st_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full);
        if (probe) { const long long now = clock64(); pt_st += now - p_mark; p_mark = now; }
      }
      if (!ok || !mbar_wait(dq_done, (c - 1) & 1, abort_flag, timeout)) { ok = false; break; }
      tcgen05_fence_after();
      // dQ row r, 32 columns per quarter -> packed gradient tensor, query slot of this head
      const int g = w.head / p.qpk, jq = w.head % p.qpk;
      if (quarter < HD / 32) {
        const int row0 = w.i * 128 + q4 * 32;           // the warp's first query
        const size_t pos = static_cast<size_t>(w.b) * p.S + row0;
        const float scale[4] = {p.scale, p.scale, p.scale, p.scale};
        store_rows_bf16(p.dqkv + ((pos * p.G + g) * (p.qpk + 2) + jq) * HD + quarter * 32, static_cast<size_t>(p.G) * (p.qpk + 2) * HD,
                        p.S - row0, tm_dq + lane_base + quarter * 32, scale);
      }
      // the next item's first dQ MMA overwrites these columns; it waits for ds_full, which this thread arrives on
      // after these reads
      tcgen05_fence_before();
    }
    if (probe) {
      volatile unsigned int* wd = reinterpret_cast<volatile unsigned int*>(p.status);
      wd[6] = c; wd[7] = static_cast<unsigned>(pw_s); wd[8] = static_cast<unsigned>(pt_ld); wd[9] = static_cast<unsigned>(pt_cmp);
      wd[10] = static_cast<unsigned>(pw_dq); wd[11] = static_cast<unsigned>(pt_st);
    }
    if (!ok && lane == 0) report_status(p.status, 0x423u);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) { __syncwarp(); tcgen05_fence_after(); tmem_dealloc(tmem_base, 512); }
}

template <int HD>
static int dq_launch(const CUtensorMap& tq, const CUtensorMap& td, const FaSplitParams& p, int device, cudaStream_t s) {
  using S_ = DqSmem<HD>;
  static bool configured[64] = {false};
  auto kern = fa_bwd_dq_kernel<HD>;
  if (!configured[device & 63]) {
    AXB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S_::TOTAL));
    configured[device & 63] = true;
  }
  const long long items = static_cast<long long>(p.B) * p.G * p.qpk * (p.Sp / 128);
  const int sms = sm_count(device);
  kern<<<static_cast<int>(items < sms ? items : sms), FS_THREADS, S_::TOTAL, s>>>(tq, td, p);
  AXB_CUDA(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------------------------------------------ dK, dV
template <int HD>
struct DkvSmem {
  static constexpr int TILE = 128 * HD * 2;
  static constexpr int K_OFF = 0, V_OFF = TILE;
  // Q / dO: two query tiles of two halves (64 queries) each.  A half is loaded and released by itself: its step's
  // accumulator MMAs free it a whole tile before its successor is needed, which hides the load; a ring of whole tiles
  // got half a tile's time for that and the MMA warps waited for it in every tile.
  // dK / dV kernel by itself on a B200: 8 x 2048, 16 heads, head_dim 128 338 -> 318 us; head_dim 64 285 -> 244 us.
  static constexpr int Q_OFF = 2 * TILE;           // 2 stages
  static constexpr int DO_OFF = 4 * TILE;          // 2 stages
  static constexpr int LSE_OFF = 6 * TILE;         // [2 stages][lse, delta][128] fp32
  static constexpr int BAR_OFF = LSE_OFF + 2048;
  static constexpr int NBARS = 2 + 8 + 4 + 4 + 2;
  static constexpr int TOTAL = BAR_OFF + NBARS * 8 + 16 + 1024;
};

// Work item k of this CTA: key tiles sorted by decreasing length (tile jt is visited by (nq - jt) * qpk query
// tiles), dealt to the persistent CTAs in a snake.
struct DkvItem { int jt, g, b; };
__device__ __forceinline__ bool dkv_item(const FaSplitParams& p, int k, DkvItem& w) {
  const int G = gridDim.x, c = blockIdx.x;
  const int bg = p.B * p.G, nq = p.Sp / 128;
  const int idx = k * G + ((k & 1) ? G - 1 - c : c);
  if (idx >= bg * nq) return false;
  w.jt = idx / bg;
  const int rem = idx % bg;
  w.g = rem % p.G;
  w.b = rem / p.G;
  return true;
}

// global -> shared bulk copy (16-byte aligned, size a multiple of 16) that completes on an mbarrier
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

template <int HD>
__global__ void __launch_bounds__(FS_THREADS, 1)
fa_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO, const FaSplitParams p) {
  using S_ = DkvSmem<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S_::BAR_OFF);
  uint64_t* kv_full = bars;          // K and V of the item
  uint64_t* kv_empty = bars + 1;     // both MMA warps are done with them
  uint64_t* qdo_full = bars + 2;     // [stage][half]: Q, dO, lse, delta of 64 queries
  uint64_t* qdo_empty = bars + 6;    // [stage][half]: 2 MMA warps + the half's 8 softmax warps
  uint64_t* t_full = bars + 10;      // [S^T, dP^T][score buffer]: complete
  uint64_t* a_full = bars + 14;      // [P^T, dS^T][score buffer]: in tensor memory
  uint64_t* acc_done = bars + 18;    // dK and dV of the item are final (one arrival per MMA warp)
  uint64_t* acc_free = bars + 19;    // ... and have been read: the next item may overwrite them
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + S_::NBARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  float* lse_s = reinterpret_cast<float*>(smem + S_::LSE_OFF);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t timeout = p.timeout_ns;
  const int heads = p.G * p.qpk, nq = p.Sp / 128;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1); mbar_init(kv_empty, 2); mbar_init(acc_done, 2);
    mbar_init(acc_free, FS_SOFTMAX_WARPS);
    for (int i = 0; i < 4; ++i) { mbar_init(&qdo_full[i], 1); mbar_init(&qdo_empty[i], 2 + FS_SOFTMAX_WARPS / 2); }
    for (int i = 0; i < 4; ++i) { mbar_init(&t_full[i], 1); mbar_init(&a_full[i], FS_SOFTMAX_WARPS / 2); }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tmQKV); tma_prefetch_desc(&tmDO); }
  if (warp == 1) { tmem_alloc(tmem_ptr_smem, 512); tmem_relinquish(); }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  // columns: S^T buffers [0,64) [64,128), dP^T buffers [128,192) [192,256) (P^T / dS^T of a buffer's queries
  // [0,32) in its columns [0,16), of queries [32,64) in [32,48)), dK [256,256+HD), dV [384,384+HD)

  if (warp < 4) {
   asm volatile(FS_REGS_CONTROL);
   if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      uint32_t tq = 0;                 // query tiles loaded so far: ring stage and phase
      DkvItem w;
      for (int it = 0; ok && dkv_item(p, it, w); ++it) {
        const int col_k = (w.g * (p.qpk + 2) + p.qpk) * HD;
        const int krow = w.jt * 128;
        if (!mbar_wait(kv_empty, (it & 1) ^ 1, abort_flag, timeout)) { ok = false; break; }
        mbar_expect_tx(kv_full, 2 * S_::TILE);
#pragma unroll
        for (int c = 0; c < 2 * (HD / 64); ++c) {            // boxes of 64 rows x 64 columns
          const int at = (c >> 1) * 16384 + (c & 1) * 8192, col = col_k + 64 * (c >> 1), row = krow + (c & 1) * 64;
          tma_load_3d(smem + S_::K_OFF + at, &tmQKV, kv_full, col, row, w.b);
          tma_load_3d(smem + S_::V_OFF + at, &tmQKV, kv_full, col + HD, row, w.b);
        }
        const int per_head = nq - w.jt;
        for (int t = 0; t < per_head * p.qpk && ok; ++t, ++tq) {
          const int jq = t / per_head, i = w.jt + t % per_head;
          const int head = w.g * p.qpk + jq;
          const int st = tq & 1;
          const size_t vec = (static_cast<size_t>(w.b) * heads + head) * p.Sp + static_cast<size_t>(i) * 128;
          for (int hq = 0; hq < 2; ++hq) {
            uint64_t* full = &qdo_full[st * 2 + hq];
            const int row0 = i * 128 + hq * 64;
            if (!mbar_wait(&qdo_empty[st * 2 + hq], ((tq >> 1) & 1) ^ 1, abort_flag, timeout)) { ok = false; break; }
            mbar_expect_tx(full, S_::TILE + 512);
#pragma unroll
            for (int c = 0; c < HD / 64; ++c) {
              const int at = st * S_::TILE + c * 16384 + hq * 8192;
              tma_load_3d(smem + S_::Q_OFF + at, &tmQKV, full, (w.g * (p.qpk + 2) + jq) * HD + 64 * c, row0, w.b);
              tma_load_3d(smem + S_::DO_OFF + at, &tmDO, full, head * HD + 64 * c, row0, w.b);
            }
            bulk_load_1d(lse_s + st * 256 + hq * 64, p.neg_lse2 + vec + hq * 64, 256, full);
            bulk_load_1d(lse_s + st * 256 + 128 + hq * 64, p.neg_delta + vec + hq * 64, 256, full);
          }
        }
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();     // give in-flight copies time to land before the CTA exits
        while (globaltimer_ns() - t0 < 200000ull) {}
        report_status(p.status, 0x431u);
      }
    }
   } else if (warp <= 2) {
    // ------------------------------------------------------------------ MMA: warp 1 = S^T and dV, warp 2 = dP^T and dK
    if (elect_one()) {
      bool ok = true;
      const int which = warp - 1;                              // 0: scores / dV (operands K, Q | P^T, dO); 1: dP^T / dK (V, dO | dS^T, Q)
      const uint32_t idesc_t = umma_idesc(1, 0, 0, 128, 64);
      const uint32_t idesc_acc = umma_idesc(1, 0, 1, 128, HD);
      const uint32_t t_buf = tmem_base + which * 128;          // this warp's two 64-column buffers
      const uint32_t t_acc = tmem_base + (which ? 256 : 384);  // dK | dV
      const uint64_t ad = umma_smem_desc(smem_u32(smem + (which ? S_::V_OFF : S_::K_OFF)), 16, 1024);
      const int b_off = which ? S_::DO_OFF : S_::Q_OFF;        // B operand of the transposed score MMA
      const int m_off = which ? S_::Q_OFF : S_::DO_OFF;        // B operand (MN-major) of the accumulator MMA
      // scores of step s = (query tile, half hq): 64 query rows of the tile in ring stage st, into buffer hq
      auto issue_t = [&](int st, int hq) {
        const uint64_t bd = umma_smem_desc(smem_u32(smem + b_off + st * S_::TILE) + hq * 8192, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          umma_f16(t_buf + hq * 64, ad + off, bd + off, idesc_t, kk != 0 ? 1u : 0u);
        }
      };
      auto issue_acc = [&](int st, int hq, bool first) {
        // dO (or Q) as an MN-major B operand: the 64 queries of the half step are the reduction dimension
        const uint64_t md = umma_smem_desc(smem_u32(smem + m_off + st * S_::TILE) + hq * 8192, 16384, 1024);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          // P^T / dS^T of queries [32 h, 32 h + 32) sit in the first 16 of the 32 columns that thread half h read
          umma_f16_ts(t_acc, t_buf + hq * 64 + (kk >> 1) * 32 + (kk & 1) * 8, md + ((kk * 2048) >> 4), idesc_acc,
                      (first && kk == 0) ? 0u : 1u);
      };
      uint32_t tq = 0, c = 0;          // query tiles and steps of earlier items
      DkvItem w;
      for (int it = 0; ok && dkv_item(p, it, w); ++it) {
        const int ns = 2 * (nq - w.jt) * p.qpk;
        if (!mbar_wait(kv_full, it & 1, abort_flag, timeout)) { ok = false; break; }
        // both buffers are free: the previous item's accumulator MMAs, which read them, were issued earlier
        for (int hq = 0; hq < 2 && ok; ++hq) {
          if (!mbar_wait(&qdo_full[(tq & 1) * 2 + hq], (tq >> 1) & 1, abort_flag, timeout)) { ok = false; break; }
          tcgen05_fence_after();
          issue_t(tq & 1, hq); umma_commit(&t_full[which * 2 + hq]);
        }
        for (int s = 0; s < ns && ok; ++s, ++c) {
          const uint32_t tile = tq + (s >> 1);
          const int hq = s & 1;
          if (!mbar_wait(&a_full[which * 2 + hq], (c >> 1) & 1, abort_flag, timeout)) { ok = false; break; }
          // the warps of either score buffer read dK / dV of the previous item; only those of buffer 0 are known to be done
          if (s == 0 && it > 0 && !mbar_wait(acc_free, (it - 1) & 1, abort_flag, timeout)) { ok = false; break; }
          tcgen05_fence_after();
          issue_acc(tile & 1, hq, s == 0);
          umma_commit(&qdo_empty[(tile & 1) * 2 + hq]);          // this warp's last read of the half
          if (s + 2 < ns) {
            const uint32_t tn = tile + 1;
            if (!mbar_wait(&qdo_full[(tn & 1) * 2 + hq], (tn >> 1) & 1, abort_flag, timeout)) { ok = false; break; }
            tcgen05_fence_after();
            issue_t(tn & 1, hq);
            umma_commit(&t_full[which * 2 + hq]);
          }
        }
        umma_commit(acc_done);
        umma_commit(kv_empty);
        tq += ns >> 1;
      }
      if (!ok) report_status(p.status, 0x432u);
    }
   }
  } else {
    // ------------------------------------------------------------------ P^T, dS^T: warp = 32 keys x 32 of the step's 64 queries
    // Warps 4-11 take the steps of score buffer 0 (first 64 queries of every tile), warps 12-19 those of buffer 1.
    // P^T is handed on before dP^T is waited for: the first MMA warp then issues dV and the next scores while the threads
    // still work on dS^T, and each warp's chain (scores -> P -> dV, dP -> dS -> dK) is its own.  One B200, this kernel with the
    // delta kernel, both handed on together / one by one: 1 x 4096, 32 heads over 8, head_dim 128 258 / 229 us, 1 x 777 62.3 /
    // 55, 8 x 2048, 16 heads, head_dim 64 252 / 244.  The dQ kernel gains nothing from the same split (22.0 / 21.9, 176 / 176).
    // A thread has 4 keys x 8 queries of the block (tmem_ld_16x32) and reads 8 + 8 values of -lse and -delta: with a key and all 32
    // queries per thread it read 64, and their broadcasts took 1000 of the 3600 cycles of shared-memory bandwidth that a tile
    // needs, which is what bounds this kernel.  8 x 2048, 16 heads, head_dim 128 350 / 335 us, head_dim 64 247 / 217.
    asm volatile(FS_REGS_SOFTMAX);
    const int q4 = warp & 3;
    const int hq = (warp - 4) >> 3;
    const int half = ((warp - 4) >> 2) & 1;
    const uint32_t lane_base = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t t_s = tmem_base + lane_base + hq * 64 + half * 32, t_dp = t_s + 128;
    // first key row and query column of this thread's scores inside the tile (tmem_ld_16x32)
    const int r0 = q4 * 32 + (lane >> 2), qc = hq * 64 + half * 32 + (lane & 3) * 2;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    bool ok = true;
    uint32_t tq = 0;                                  // query tiles so far: this buffer's steps, ring stage and phases
    DkvItem w;
    for (int it = 0; ok && dkv_item(p, it, w); ++it) {
      const int per_head = nq - w.jt;
      const int nt = per_head * p.qpk;
      for (int t = 0; t < nt; ++t, ++tq) {
        const int st = tq & 1;
        const bool diag = t % per_head == 0;
        // -lse and -delta of the tile arrive with its Q and dO
        if (!mbar_wait(&qdo_full[st * 2 + hq], (tq >> 1) & 1, abort_flag, timeout) ||
            !mbar_wait(&t_full[hq], tq & 1, abort_flag, timeout)) { ok = false; break; }
        tcgen05_fence_after();
        uint32_t sv[32];
        tmem_ld_16x32(t_s, sv);
        tmem_ld_16x32(t_s + (16u << 16), sv + 16);
        tmem_ld_wait(sv);
        if (diag) {                                   // the key lies after the query: probability 0
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (r0 + (i >> 4) * 16 + ((i >> 1) & 1) * 8 > qc + ((i >> 2) & 3) * 8 + (i & 1)) sv[i] = 0xff800000u;
        }
        const float* lv = lse_s + st * 256 + qc;
        float2 pr[16];
        uint32_t pk[16];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float2 nl2 = *reinterpret_cast<const float2*>(lv + g * 8);
#pragma unroll
          for (int e = 0; e < 4; ++e) {               // 16 lanes each e >> 1, 8 lanes each e & 1
            const int i = (e >> 1) * 8 + g * 2 + (e & 1);
            const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sc2, nl2);
            pr[i] = make_float2(exp2f(x.x), exp2f(x.y));
            pk[i] = fs_pack(pr[i]);
          }
        }
        // into this warp's own score columns: the other half's warp may not have read its scores yet
        tmem_st_16x16(t_s, pk);
        tmem_st_16x16(t_s + (16u << 16), pk + 8);
        tmem_st_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[hq]);      // dV and the next scores need not wait for dS
        if (!mbar_wait(&t_full[2 + hq], tq & 1, abort_flag, timeout)) { ok = false; break; }
        tcgen05_fence_after();
        uint32_t dv[32];
        tmem_ld_16x32(t_dp, dv);
        tmem_ld_16x32(t_dp + (16u << 16), dv + 16);
        tmem_ld_wait(dv);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float2 nd2 = *reinterpret_cast<const float2*>(lv + 128 + g * 8);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = (e >> 1) * 8 + g * 2 + (e & 1);
            const float2 t2 = __fadd2_rn(make_float2(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])), nd2);
            pk[i] = fs_pack(__fmul2_rn(pr[i], t2));   // the softmax scale is applied to the finished dK
          }
        }
        tmem_st_16x16(t_dp, pk);
        tmem_st_16x16(t_dp + (16u << 16), pk + 8);
        tmem_st_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&a_full[2 + hq]);
          mbar_arrive(&qdo_empty[st * 2 + hq]);       // this warp has read its share of -lse / -delta
        }
      }
      if (!ok || !mbar_wait(acc_done, it & 1, abort_flag, timeout)) { ok = false; break; }
      tcgen05_fence_after();
      // half 0 stores dK, half 1 stores dV, each warp 32 rows, into the key / value slots of the packed gradient tensor; the
      // warps of buffer 0 take the even, those of buffer 1 the odd 32-column blocks
      const int row0 = w.jt * 128 + q4 * 32;            // the warp's first key
      const size_t kvpos = static_cast<size_t>(w.b) * p.S + row0;
      __nv_bfloat16* dst = p.dqkv + ((kvpos * p.G + w.g) * (p.qpk + 2) + p.qpk + half) * HD;
      const uint32_t src = tmem_base + lane_base + (half ? 384 : 256);
      const float sc = half ? 1.f : p.scale, scale[4] = {sc, sc, sc, sc};
#pragma unroll
      for (int cc = hq; cc < HD / 32; cc += 2)
        store_rows_bf16(dst + cc * 32, static_cast<size_t>(p.G) * (p.qpk + 2) * HD, p.S - row0, src + cc * 32, scale);
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free);
    }
    if (!ok && lane == 0) report_status(p.status, 0x433u);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) { __syncwarp(); tcgen05_fence_after(); tmem_dealloc(tmem_base, 512); }
}

template <int HD>
static int dkv_launch(const CUtensorMap& tq, const CUtensorMap& td, const FaSplitParams& p, int device, cudaStream_t s) {
  using S_ = DkvSmem<HD>;
  static bool configured[64] = {false};
  auto kern = fa_bwd_dkv_kernel<HD>;
  if (!configured[device & 63]) {
    AXB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S_::TOTAL));
    configured[device & 63] = true;
  }
  const long long items = static_cast<long long>(p.B) * p.G * (p.Sp / 128);
  const int sms = sm_count(device);
  kern<<<static_cast<int>(items < sms ? items : sms), FS_THREADS, S_::TOTAL, s>>>(tq, td, p);
  AXB_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace axb

// fp32 words of scratch that axb_flash_attn_bwd_split needs: -lse and -delta of every query row, rows padded to 128
extern "C" long long axb_flash_attn_bwd_scratch(int B, int S, int heads) {
  return 2ll * B * heads * ((static_cast<long long>(S) + 127) / 128 * 128);
}

// which: bit 0 = dQ kernel (writes the query slots of dqkv), bit 1 = dK / dV kernel (writes the key and value slots).
// qkv [B,S,G,qpk+2,D], out / d_out [B,S,G*qpk,D] bf16; lse [B,G*qpk,S]; scratch: axb_flash_attn_bwd_scratch fp32 words.
extern "C" int axb_flash_attn_bwd_split(const void* qkv, const void* out, const void* d_out, const float* lse,
                                        float* scratch, void* dqkv, int B, int S, int G, int qpk, int D, float scale,
                                        int which, int device, void* stream) {
  using namespace axb;
  if (D != 64 && D != 128) { set_error("flash attention: head_dim must be 64 or 128"); return -1; }
  if (B <= 0 || S <= 0 || G <= 0 || qpk <= 0) { set_error("flash attention: empty problem"); return -1; }
  if (!(scale > 0.f)) { set_error("flash attention: the scale must be positive"); return -1; }   // masked scores are -inf before it
  if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(d_out) | reinterpret_cast<uintptr_t>(dqkv) |
       reinterpret_cast<uintptr_t>(scratch)) & 15) {
    set_error("flash attention: tensors must be 16-byte aligned");
    return -1;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int H = G * qpk, Sp = (S + 127) / 128 * 128;
  const int rows_per_block = 256 / (D / 8) * FS_DELTA_ROWS;
  const long long rows = static_cast<long long>(Sp) * H;
  if (rows > 0x7fffffffll) { set_error("flash attention: too many rows"); return -1; }
  const dim3 dgrid(static_cast<unsigned>((rows + rows_per_block - 1) / rows_per_block), B < 65535 ? B : 65535);
  float* neg_delta = scratch + static_cast<size_t>(B) * H * Sp;
  if (D == 128)
    fa_split_delta_kernel<128><<<dgrid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(d_out),
                                                     lse, scratch, neg_delta, B, S, Sp, H);
  else
    fa_split_delta_kernel<64><<<dgrid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(d_out),
                                                    lse, scratch, neg_delta, B, S, Sp, H);
  AXB_CUDA(cudaGetLastError());
  CUtensorMap tq, td, tq64, td64;                     // dQ kernel: 128-row boxes, dK / dV kernel: 64-row boxes
  const uint64_t cols = static_cast<uint64_t>(G) * (qpk + 2) * D, do_cols = static_cast<uint64_t>(H) * D;
  if (make_tmap_3d_bf16(&tq, qkv, B, S, cols, 128) || make_tmap_3d_bf16(&td, d_out, B, S, do_cols, 128) ||
      make_tmap_3d_bf16(&tq64, qkv, B, S, cols, 64) || make_tmap_3d_bf16(&td64, d_out, B, S, do_cols, 64))
    return -1;
  FaSplitParams p;
  p.neg_lse2 = scratch; p.neg_delta = scratch + static_cast<size_t>(B) * H * Sp; p.dqkv = static_cast<__nv_bfloat16*>(dqkv);
  p.B = B; p.S = S; p.Sp = Sp; p.G = G; p.qpk = qpk; p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  unsigned int* st = nullptr;
  if (!device_status_word(device, &st)) { set_error("flash attention: no status word"); return -1; }
  p.status = st; p.timeout_ns = wait_timeout_ns();
  p.debug = 0;
#ifdef AXB_ABLATION
  { static int dbg = -1; if (dbg < 0) { const char* e = getenv("AXB_FA_DEBUG"); dbg = e ? atoi(e) : 0; } p.debug = dbg; }
#endif
  if (which & 2) {
    if (D == 128) { if (dkv_launch<128>(tq64, td64, p, device, s)) return -1; }
    else          { if (dkv_launch<64>(tq64, td64, p, device, s)) return -1; }
  }
  if (which & 1) {
    if (D == 128) { if (dq_launch<128>(tq, td, p, device, s)) return -1; }
    else          { if (dq_launch<64>(tq, td, p, device, s)) return -1; }
  }
  return 0;
}
