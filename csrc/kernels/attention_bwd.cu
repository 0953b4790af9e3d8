// Flash attention backward on tcgen05 (no counterpart in the reference, which has no
// attention backward at all: lua/luatorch/nn/flash_attention.lua:52-108 never records one).
//
// Three launches, no floating-point atomics, bitwise reproducible:
//   1. per query: lse * log2(e) and delta * scale, delta = sum_d dO[i,d] * O[i,d]
//   2. dK/dV kernel: one CTA per 128-key tile, loops over the queries that see it.
//   3. dQ kernel: one CTA per 128-query tile, loops over its keys.
// Both rebuild P = exp(scale*S - lse) and dS = P * (dP - delta) * scale from S = Q K^T and
// dP = dO V^T.
#include "attention.h"
#include "sm100_ptx.cuh"
#include "common.cuh"

#include <cuda.h>
#include <stdio.h>
#include <atomic>

namespace lt {

using namespace ptx;

extern std::atomic<uint64_t> g_attn_launches;
// Status word of the backward kernels (device symbols are per translation unit).
static __device__ int g_attn_error = 0;
int attention_bwd_device_error() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_attn_error, sizeof(int));
  return v;
}

namespace attn_detail {
bool make_qkv_map(CUtensorMap* map, const void* base, int D, int S, int H, int B, int64_t ss,
                  int64_t sh, int64_t sb, int box_rows);
}

namespace {

constexpr int BT = 128;                  // tile edge (queries and keys)
constexpr int CHUNK_BYTES = 128 * 128;   // 128 rows x 64 bf16
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct BwdParams {
  int S, Sp, H, causal;     // Sp: S rounded up to a multiple of BT
  float scale, scale_log2;
  const float* lse2;        // [B, H, Sp]: lse * log2(e), +inf beyond S
  const float* dsc;         // [B, H, Sp]: delta * scale
  __nv_bfloat16* out0;  // dK (kernel 2) or dQ (kernel 3)
  long long o0_sb, o0_ss, o0_sh;
  __nv_bfloat16* out1;  // dV (kernel 2)
  long long o1_sb, o1_ss, o1_sh;
  int late_wait = 0;      // independent of the previous kernel: wait for it before exit (common.cuh)
};

// ------------------------------------------------------------------ row statistics
// delta[i] = sum_d dO[i, d] O[i, d], and the two numbers per query that the main kernels want:
// lse * log2(e) and delta * scale, in rows padded to a multiple of 128 queries so that any length
// can be fetched by bulk copies (16-byte aligned, never past the end).  A padded query gets
// lse = +inf: its probabilities are exp2(-inf) = 0 and nothing else has to mask it.
// D / 8 lanes share a query (16-byte loads, whole lines), 32 queries of one head per CTA.
// Bound by memory; [8, 1024, 12, 64] takes 7.1 us (8.8 with a thread per query and strided loads),
// [4, 2048, 16, 128] 13.1 us (21.7).
constexpr int STAT_ROWS = 32;
template <int D>
__global__ void __launch_bounds__(STAT_ROWS * 8)
attn_stats_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                  const float* __restrict__ lse, float* __restrict__ lse2, float* __restrict__ dsc,
                  int H, int S, int Sp, float scale, long long o_sb, long long o_ss, long long o_sh,
                  long long do_sb, long long do_ss, long long do_sh) {
  pdl_enter();
  constexpr int PARTS = D / 64;              // 16-byte loads per lane: 8 lanes per query
  const int h = blockIdx.x % H, b = blockIdx.y;   // tiles in x: the other dimensions end at 65535
  const int s = (int)(blockIdx.x / H) * STAT_ROWS + (threadIdx.x >> 3), v = threadIdx.x & 7;
  float t[PARTS][4] = {};
  if (s < S) {
    const __nv_bfloat16* op = o + b * o_sb + s * o_ss + h * o_sh + v * 8;
    const __nv_bfloat16* dp = d_o + b * do_sb + s * do_ss + h * do_sh + v * 8;
    uint4 x[PARTS], y[PARTS];
#pragma unroll
    for (int i = 0; i < PARTS; ++i) {
      x[i] = *reinterpret_cast<const uint4*>(op + 64 * i);
      y[i] = *reinterpret_cast<const uint4*>(dp + 64 * i);
    }
#pragma unroll
    for (int i = 0; i < PARTS; ++i) {
      const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&x[i]);
      const __nv_bfloat162* yh = reinterpret_cast<const __nv_bfloat162*>(&y[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = __bfloat1622float2(xh[j]), c = __bfloat1622float2(yh[j]);
        t[i][j] = a.x * c.x + a.y * c.y;
      }
    }
  }
  // added in the order of d, the sum handed from lane to lane
  float acc = 0.0f;
#pragma unroll
  for (int i = 0; i < PARTS; ++i)
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float sum = __shfl_sync(0xffffffffu, acc, (q + 7) & 7, 8);
      if (v == q) acc = sum + t[i][0] + t[i][1] + t[i][2] + t[i][3];
    }
  acc = __shfl_sync(0xffffffffu, acc, 7, 8);
  if (v == 0) {
    const long long bh = (long long)b * H + h, at = bh * Sp + s;
    lse2[at] = s < S ? lse[bh * S + s] * LOG2E : INFINITY;
    dsc[at] = acc * scale;
  }
}

// Stores one accumulator row (D fp32 columns in TMEM) as bf16; the PARTS warps that share a lane
// quadrant take its 32-column chunks in turn.
template <int D, int PARTS>
__device__ __forceinline__ void store_acc_row(uint32_t taddr, __nv_bfloat16* dst, int first) {
#pragma unroll 1
  for (int c32 = first; c32 < D / 32; c32 += PARTS) {
    uint32_t r[32];
    tmem_ld_32x32(taddr + c32 * 32, r);
    tmem_ld_wait();
    if (dst) {
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint4 u;
        __nv_bfloat162* hb = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
        for (int t = 0; t < 4; ++t)
          hb[t] = __floats2bfloat162_rn(__uint_as_float(r[i + 2 * t]),
                                        __uint_as_float(r[i + 2 * t + 1]));
        *reinterpret_cast<uint4*>(dst + c32 * 32 + i) = u;
      }
    }
  }
}

// =====================================================================================
// Main kernels, any length, head dim 64 and 128.
//
// The row index of the STATIONARY operand sits on the TMEM lanes, the streamed operand arrives
// in sub-tiles of 64 rows that become the columns:
//   DKDV = true : lanes = 128 keys of this CTA, columns = 64 queries per step
//                 S^T = K Q^T, dP^T = V dO^T; thread (key) rebuilds P^T and dS^T for its row;
//                 dV += P^T dO and dK += dS^T Q
//   DKDV = false: lanes = 128 queries of this CTA, columns = 64 keys per step
//                 S = Q K^T, dP = dO V^T; thread (query) rebuilds dS; dQ += dS K
// In both cases the rebuilt P / dS tile is exactly the A operand (M = lanes, K = the 64
// streamed rows) of the accumulating MMAs, so it is written back to tensor memory as packed
// bf16 (over the columns its fp32 source occupied) and read from there by tcgen05.mma: no
// shared-memory staging of P or dS, no proxy fences.
//
// What runs under what: at head dim 64 a CTA needs 128 + 2 x 64 TMEM columns and 83 KB of shared
// memory, so two CTAs share an SM and one CTA's exponentials run under the other's MMAs.  At head
// dim 128 only one CTA fits; there S and dP have two buffers (2 x 128 + 2 x 128 = all 512 columns)
// and the MMAs of step i + 1 are issued before the exponentials of step i have come back.
// Bound by the chain MMA -> barrier -> TMEM load -> exponentials -> TMEM store -> barrier -> MMA (about
// 2500 cycles per step; issue slots, tensor pipe and MUFU are all below a third).  Tiles of 128
// streamed rows with a barrier each for S, P, dP and dS, so that P dO and dS Q alternate with the
// exponentials of one CTA, took the same time at head dim 128 and 5 % more at 64.
// All three launches, causal: [4, 1000, 12, 64] 83 -> 61 us, [4, 2048, 16, 128] 426 -> 299 us, against
// kernels that staged P and dS through shared memory (and dS through 0.5 GB of device memory).
//
// Lengths that are no multiple of a tile: TMA fills the missing rows with zeros, a missing query has
// lse = +inf (attn_stats_kernel), missing keys are masked where they are columns, and missing
// rows of the outputs are not stored.
// =====================================================================================
constexpr int SUB = 64;                         // streamed rows per step
constexpr int SUB_CHUNK = SUB * 128;            // 64 rows x 64 bf16

template <int D>
struct BwdCfg {
  static constexpr int DC = D / 64;
  static constexpr int FIX = DC * CHUNK_BYTES;            // one [128 x D] stationary operand
  static constexpr int STR = DC * SUB_CHUNK;              // one [64 x D] streamed operand
  static constexpr int STAGES = 3;
  static constexpr int OFF_FIX0 = 0;
  static constexpr int OFF_FIX1 = FIX;
  static constexpr int OFF_STR = 2 * FIX;                 // [stage][2][STR]
  static constexpr int OFF_SCAL = OFF_STR + STAGES * 2 * STR;   // [stage][2][64] floats: lse, delta
  static constexpr int OFF_BAR = OFF_SCAL + STAGES * 2 * SUB * 4;
  static constexpr int TOTAL = OFF_BAR + 256 + 1024;
  static constexpr int NBUF = D == 64 ? 1 : 2;            // S / dP buffers in TMEM
  static constexpr int TMEM_COLS = NBUF * 2 * SUB + 2 * D;
  static constexpr int CTAS = D == 64 ? 2 : 1;            // per SM
  static constexpr int WARPS = D == 64 ? 8 : 16;          // that rebuild P and dS: 16 on an SM
  static constexpr int PARTS = WARPS / 4;                 // warps that share a TMEM lane quadrant
  static constexpr int PW = SUB / PARTS;                  // columns of a step per thread
  static constexpr int THREADS = 64 + 32 * WARPS;
};

// 16 columns of one lane's row: scores s and dp (fp32 from TMEM) -> packed bf16 P and dS.
// lse2 / dsc: log2-domain log-sum-exp and delta * scale, per column (COLV) or for the lane.
template <bool COLV, bool MASKED>
__device__ __forceinline__ void rebuild16(const uint32_t (&s)[16], const uint32_t (&dp)[16],
                                          const float* lse2_c, const float* dsc_c, float lse2_l,
                                          float dsc_l, float c, float scale, int lo, int hi,
                                          uint32_t (&pp)[8], uint32_t (&dd)[8]) {
  // columns j with lo <= j < hi are inside the causal / sequence bounds (only when MASKED)
  const float2 cc = make_float2(c, c), ss = make_float2(scale, scale);
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const float2 ll = COLV ? make_float2(-lse2_c[i], -lse2_c[i + 1]) : make_float2(-lse2_l, -lse2_l);
    const float2 dl = COLV ? make_float2(-dsc_c[i], -dsc_c[i + 1]) : make_float2(-dsc_l, -dsc_l);
    const float2 x = ffma2(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), cc, ll);
    float2 pv = make_float2(ex2(x.x), ex2(x.y));
    if (MASKED) {
      pv.x = (i >= lo && i < hi) ? pv.x : 0.0f;
      pv.y = (i + 1 >= lo && i + 1 < hi) ? pv.y : 0.0f;
    }
    const float2 g = ffma2(make_float2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), ss, dl);
    const float2 dv = fmul2(pv, g);
    __nv_bfloat162 hp = __floats2bfloat162_rn(pv.x, pv.y), hd = __floats2bfloat162_rn(dv.x, dv.y);
    pp[i >> 1] = *reinterpret_cast<uint32_t*>(&hp);
    dd[i >> 1] = *reinterpret_cast<uint32_t*>(&hd);
  }
}

template <int D, bool DKDV>
__global__ void __launch_bounds__(BwdCfg<D>::THREADS, BwdCfg<D>::CTAS)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tm_fix0, const __grid_constant__ CUtensorMap tm_fix1,
                 const __grid_constant__ CUtensorMap tm_str0, const __grid_constant__ CUtensorMap tm_str1,
                 const BwdParams p) {
  // DKDV: fix0 = K, fix1 = V (128-row boxes), str0 = Q, str1 = dO (64-row boxes)
  // dQ  : fix0 = Q, fix1 = dO,                 str0 = K, str1 = V
  using L = BwdCfg<D>;
  constexpr int DC = L::DC, ST = L::STAGES, NBUF = L::NBUF, PARTS = L::PARTS, PW = L::PW;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* fix_full = bars;           // 1
  uint64_t* str_full = bars + 1;       // ST
  uint64_t* str_empty = bars + 1 + ST; // ST
  uint64_t* s_full = bars + 1 + 2 * ST;           // [NBUF] S and dP of a step are in TMEM
  uint64_t* pds_full = s_full + NBUF;             // [NBUF] P / dS of a step are back in TMEM
  uint64_t* acc_full = pds_full + NBUF;           // final accumulators
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp_idx = warp_index(), lane = threadIdx.x & 31;
  const int h = blockIdx.x, b = blockIdx.y;
  const int n_sub = (p.S + SUB - 1) / SUB;
  const int own = DKDV ? (int)blockIdx.z : (int)gridDim.z - 1 - (int)blockIdx.z;  // longest first
  const int it_begin = DKDV ? (p.causal ? 2 * own : 0) : 0;
  const int it_end = DKDV ? n_sub : (p.causal ? min(2 * own + 2, n_sub) : n_sub);
  const int n_it = it_end - it_begin;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(smem_u32(fix_full), 1);
    for (int i = 0; i < ST; ++i) {
      mbar_init(smem_u32(&str_full[i]), 1);
      mbar_init(smem_u32(&str_empty[i]), 1);
    }
    for (int i = 0; i < NBUF; ++i) {
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&pds_full[i]), 32 * L::WARPS);
    }
    mbar_init(smem_u32(acc_full), 1);
    fence_mbar_init();
    tma_prefetch_desc(&tm_fix0);
    tma_prefetch_desc(&tm_fix1);
    tma_prefetch_desc(&tm_str0);
    tma_prefetch_desc(&tm_str1);
  }
  if (warp_idx == 1) {
    tmem_alloc(smem_u32(tmem_holder), L::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;
  // operands come from kernels before the previous one when `late_wait` is set (the dQ kernel
  // after the dK / dV kernel: both read q, k, v, dO, lse, delta and write disjoint outputs)
  pdl_enter(p.late_wait != 0);
  // buffer `i`: 64 fp32 score columns, then 64 fp32 dP columns; packed P and dS land in them
  auto tmem_s = [&](int i) { return tmem_base + (uint32_t)(i * 2 * SUB); };
  auto tmem_dp = [&](int i) { return tmem_base + (uint32_t)(i * 2 * SUB + SUB); };
  const uint32_t tmem_acc0 = tmem_base + NBUF * 2 * SUB;   // dK (DKDV) or dQ: from dS
  const uint32_t tmem_acc1 = tmem_acc0 + D;                // dV (DKDV only): from P
  // packed bf16 operand columns: the PW columns of a compute warp keep PW / 2 packed columns at the
  // start of their own fp32 range (so no warp touches another's); 16 rows of K per step
  auto packed_col = [](int ks) { return (ks * 16 / PW) * PW + (ks * 16 % PW) / 2; };

  auto str0 = [&](int st) { return smem + L::OFF_STR + st * 2 * L::STR; };
  auto str1 = [&](int st) { return smem + L::OFF_STR + st * 2 * L::STR + L::STR; };

  if (warp_idx == 0) {
    if (elect_one()) {
      const uint32_t fb = smem_u32(fix_full);
      mbar_arrive_expect_tx(fb, 2 * L::FIX);
#pragma unroll
      for (int c = 0; c < DC; ++c) {
        tma_load_4d(smem_u32(smem + L::OFF_FIX0 + c * CHUNK_BYTES), &tm_fix0, fb, 64 * c, own * BT, h, b);
        tma_load_4d(smem_u32(smem + L::OFF_FIX1 + c * CHUNK_BYTES), &tm_fix1, fb, 64 * c, own * BT, h, b);
      }
      for (int it = 0; it < n_it; ++it) {
        const int st = it % ST, use = it / ST, t = it_begin + it;
        if (!mbar_wait_bounded(smem_u32(&str_empty[st]), (use & 1) ^ 1, abort_flag, &g_attn_error, 71))
          break;
        const uint32_t sb = smem_u32(&str_full[st]);
        mbar_arrive_expect_tx(sb, 2 * L::STR + (DKDV ? 2 * SUB * 4 : 0));
#pragma unroll
        for (int c = 0; c < DC; ++c) {
          tma_load_4d(smem_u32(str0(st) + c * SUB_CHUNK), &tm_str0, sb, 64 * c, t * SUB, h, b);
          tma_load_4d(smem_u32(str1(st) + c * SUB_CHUNK), &tm_str1, sb, 64 * c, t * SUB, h, b);
        }
        if (DKDV) {
          // the 64 streamed queries' log-sum-exp and delta ride on the same barrier: every
          // compute thread needs all of them, and reads them as shared-memory broadcasts
          const long long row0 = ((long long)b * p.H + h) * p.Sp + (long long)t * SUB;
          float* sc = reinterpret_cast<float*>(smem + L::OFF_SCAL) + st * 2 * SUB;
          bulk_load(smem_u32(sc), p.lse2 + row0, SUB * 4, sb);
          bulk_load(smem_u32(sc + SUB), p.dsc + row0, SUB * 4, sb);
        }
      }
    }
  } else if (warp_idx == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = make_idesc_bf16(BT, SUB, 0, 0);   // [128 lanes] x [64 streamed rows]
      const uint32_t idesc_acc = make_idesc_bf16(BT, D, 0, 1);   // A from TMEM, B = streamed tile, rows as K
      bool ok = mbar_wait_bounded(smem_u32(fix_full), 0, abort_flag, &g_attn_error, 72);
      // S and dP of a step: lanes x streamed rows, contraction over the head dim.  They overwrite
      // the packed operands of the step before (NBUF = 1) or before that (NBUF = 2), which the
      // in-order tensor pipe has consumed by then: those accumulating MMAs were issued earlier.
      auto issue_scores = [&](int it) {
        const int st = it % ST, use = it / ST, buf = it % NBUF;
        if (!mbar_wait_bounded(smem_u32(&str_full[st]), use & 1, abort_flag, &g_attn_error, 73)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < DC; ++c) {
          const uint64_t f0 = make_smem_desc_sw128(smem_u32(smem + L::OFF_FIX0 + c * CHUNK_BYTES), 16, 1024);
          const uint64_t s0 = make_smem_desc_sw128(smem_u32(str0(st) + c * SUB_CHUNK), 16, 1024);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16(tmem_s(buf), f0 + (uint64_t)(ks * 2), s0 + (uint64_t)(ks * 2), idesc_s,
                      (c > 0 || ks > 0) ? 1u : 0u);
        }
#pragma unroll
        for (int c = 0; c < DC; ++c) {
          const uint64_t f1 = make_smem_desc_sw128(smem_u32(smem + L::OFF_FIX1 + c * CHUNK_BYTES), 16, 1024);
          const uint64_t s1 = make_smem_desc_sw128(smem_u32(str1(st) + c * SUB_CHUNK), 16, 1024);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16(tmem_dp(buf), f1 + (uint64_t)(ks * 2), s1 + (uint64_t)(ks * 2), idesc_s,
                      (c > 0 || ks > 0) ? 1u : 0u);
        }
        umma_commit(smem_u32(&s_full[buf]));
        return true;
      };
      if (ok && NBUF > 1) ok = issue_scores(0);
      for (int it = 0; ok && it < n_it; ++it) {
        const int st = it % ST, buf = it % NBUF;
        if (NBUF == 1) ok = issue_scores(it);
        else if (it + 1 < n_it) ok = issue_scores(it + 1);
        if (!ok) break;
        if (!mbar_wait_bounded(smem_u32(&pds_full[buf]), (it / NBUF) & 1, abort_flag, &g_attn_error, 74)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        // accumulate over the 64 streamed rows (K), 16 rows = 2048 bytes of the tile per step
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          // dS-based product: B = streamed operand 0 (Q for dK, K for dQ), its rows as K
          const uint64_t bd = make_smem_desc_sw128(smem_u32(str0(st)) + ks * 2048, SUB_CHUNK, 1024);
          umma_bf16_ts(tmem_acc0, tmem_dp(buf) + packed_col(ks), bd, idesc_acc, (it > 0 || ks > 0) ? 1u : 0u);
        }
        if (DKDV) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint64_t bd = make_smem_desc_sw128(smem_u32(str1(st)) + ks * 2048, SUB_CHUNK, 1024);
            umma_bf16_ts(tmem_acc1, tmem_s(buf) + packed_col(ks), bd, idesc_acc, (it > 0 || ks > 0) ? 1u : 0u);
          }
        }
        umma_commit(smem_u32(&str_empty[st]));
      }
      if (ok) umma_commit(smem_u32(acc_full));
    }
  } else {
    const int quad = warp_idx & 3;
    const int part = (warp_idx - 2) >> 2;        // which PW of the 64 columns
    const int row = quad * 32 + lane;
    const uint32_t lane_base = ((uint32_t)(quad * 32)) << 16;
    const int row_g = own * BT + row;            // key index (DKDV) or query index; < Sp
    float lse2_l = 0.0f, dsc_l = 0.0f;
    if (!DKDV) {
      const long long at = ((long long)b * p.H + h) * p.Sp + row_g;
      lse2_l = p.lse2[at];
      dsc_l = p.dsc[at];
    }
    bool ok = true;
    for (int it = 0; ok && it < n_it; ++it) {
      const int t = it_begin + it, buf = it % NBUF;
      const int c0 = t * SUB + part * PW;        // global index of this thread's first column
      // bounds in units of this thread's columns
      int lo = 0, hi = PW;
      bool masked = false;
      if (p.causal && (t >> 1) == own) {
        masked = true;
        if (DKDV) lo = row_g - c0;               // query >= key
        else hi = row_g - c0 + 1;                // key <= query
      }
      if (!DKDV && (t + 1) * SUB > p.S) {        // keys beyond the sequence
        masked = true;
        hi = min(hi, p.S - c0);
      }
      float lse2_c[16], dsc_c[16];
      const float* sc = reinterpret_cast<const float*>(smem + L::OFF_SCAL) + (it % ST) * 2 * SUB + part * PW;
      auto load_cols = [&](int off) {   // broadcast reads: every lane takes the same 16 columns
        const float4* l4 = reinterpret_cast<const float4*>(sc + off);
        const float4* d4 = reinterpret_cast<const float4*>(sc + SUB + off);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 a = l4[q], d = d4[q];
          lse2_c[4 * q] = a.x; lse2_c[4 * q + 1] = a.y; lse2_c[4 * q + 2] = a.z; lse2_c[4 * q + 3] = a.w;
          dsc_c[4 * q] = d.x; dsc_c[4 * q + 1] = d.y; dsc_c[4 * q + 2] = d.z; dsc_c[4 * q + 3] = d.w;
        }
      };
      if (!mbar_wait_bounded_warp(smem_u32(&s_full[buf]), (it / NBUF) & 1, abort_flag, &g_attn_error, 75)) {
        ok = false;
        break;
      }
      // the stage's barrier completed long ago (the MMAs waited for it); observing it here
      // makes the bulk-copied scalars visible to this thread
      if (DKDV && !mbar_wait_bounded_warp(smem_u32(&str_full[it % ST]), (it / ST) & 1, abort_flag,
                                          &g_attn_error, 77)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const uint32_t s_addr = tmem_s(buf) + lane_base + part * PW;
      const uint32_t d_addr = tmem_dp(buf) + lane_base + part * PW;
      // chunks of 16 columns; the packed bf16 results of chunk k go to columns [8 k, 8 k + 8)
      // of this thread's own range, which holds fp32 values it has already read
#pragma unroll
      for (int k = 0; k < PW / 16; ++k) {
        uint32_t sv[16], dv[16], pp[8], dd[8];
        tmem_ld_32x16(s_addr + 16 * k, sv);
        tmem_ld_32x16(d_addr + 16 * k, dv);
        if (DKDV) load_cols(16 * k);      // the stage (s_full follows str_full) is complete
        tmem_ld_wait();
        if (masked)
          rebuild16<DKDV, true>(sv, dv, lse2_c, dsc_c, lse2_l, dsc_l, p.scale_log2, p.scale,
                                lo - 16 * k, hi - 16 * k, pp, dd);
        else
          rebuild16<DKDV, false>(sv, dv, lse2_c, dsc_c, lse2_l, dsc_l, p.scale_log2, p.scale, 0, 16, pp, dd);
        if (DKDV) tmem_st_32x8(s_addr + 8 * k, pp);
        tmem_st_32x8(d_addr + 8 * k, dd);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(smem_u32(&pds_full[buf]));
    }
    if (ok && n_it > 0 &&
        mbar_wait_bounded_warp(smem_u32(acc_full), 0, abort_flag, &g_attn_error, 76)) {
      tc_fence_after_sync();
      const bool in_range = row_g < p.S;
      __nv_bfloat16* d0p = in_range ? p.out0 + (long long)b * p.o0_sb + (long long)row_g * p.o0_ss +
                                          (long long)h * p.o0_sh
                                    : nullptr;
      store_acc_row<D, PARTS>(tmem_acc0 + lane_base, d0p, part);
      if (DKDV) {
        __nv_bfloat16* d1p = in_range ? p.out1 + (long long)b * p.o1_sb + (long long)row_g * p.o1_ss +
                                            (long long)h * p.o1_sh
                                      : nullptr;
        store_acc_row<D, PARTS>(tmem_acc1 + lane_base, d1p, part);
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp_idx == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
  pdl_leave(p.late_wait != 0);
}

template <int D, bool DKDV>
cudaError_t launch_bwd(const CUtensorMap& f0, const CUtensorMap& f1, const CUtensorMap& s0,
                       const CUtensorMap& s1, const BwdParams& p, dim3 grid, cudaStream_t s) {
  using L = BwdCfg<D>;
  static const cudaError_t attr = cudaFuncSetAttribute(
      flash_bwd_kernel<D, DKDV>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
  if (attr != cudaSuccess) return attr;
  cudaError_t le = launch_pdl(flash_bwd_kernel<D, DKDV>, grid, dim3(L::THREADS), L::TOTAL, s, f0, f1, s0, s1, p);
  if (le != cudaSuccess) return le;
  g_attn_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

bool ok8(int64_t a, int64_t b, int64_t c) { return a % 8 == 0 && b % 8 == 0 && c % 8 == 0; }

}  // namespace

cudaError_t flash_attention_backward(const AttnArgs& a, const AttnBwdArgs& g, cudaStream_t stream) {
  if (a.B <= 0 || a.H <= 0 || a.S <= 0) return cudaSuccess;
  if (a.D != 64 && a.D != 128) return cudaErrorInvalidValue;
  if (!ok8(a.q_ss, a.q_sh, a.q_sb) || !ok8(a.k_ss, a.k_sh, a.k_sb) || !ok8(a.v_ss, a.v_sh, a.v_sb) ||
      !ok8(g.do_ss, g.do_sh, g.do_sb) || !ok8(g.dq_ss, g.dq_sh, g.dq_sb) ||
      !ok8(g.dk_ss, g.dk_sh, g.dk_sb) || !ok8(g.dv_ss, g.dv_sh, g.dv_sb))
    return cudaErrorInvalidValue;

  const int Sp = (a.S + BT - 1) / BT * BT;
  BwdParams p;
  p.S = a.S; p.Sp = Sp; p.H = a.H; p.causal = a.causal;
  p.scale = a.scale; p.scale_log2 = a.scale * LOG2E;
  float* lse2 = g.stats;
  float* dsc = g.stats + (long long)a.B * a.H * Sp;
  p.lse2 = lse2; p.dsc = dsc;
  if ((reinterpret_cast<uintptr_t>(lse2) & 15) != 0) return cudaErrorInvalidValue;   // bulk copies

  CUtensorMap q128, k128, v128, do128, q64, k64, v64, do64;
  if (!attn_detail::make_qkv_map(&q128, a.q, a.D, a.S, a.H, a.B, a.q_ss, a.q_sh, a.q_sb, BT) ||
      !attn_detail::make_qkv_map(&k128, a.k, a.D, a.S, a.H, a.B, a.k_ss, a.k_sh, a.k_sb, BT) ||
      !attn_detail::make_qkv_map(&v128, a.v, a.D, a.S, a.H, a.B, a.v_ss, a.v_sh, a.v_sb, BT) ||
      !attn_detail::make_qkv_map(&do128, g.d_o, a.D, a.S, a.H, a.B, g.do_ss, g.do_sh, g.do_sb, BT) ||
      !attn_detail::make_qkv_map(&q64, a.q, a.D, a.S, a.H, a.B, a.q_ss, a.q_sh, a.q_sb, SUB) ||
      !attn_detail::make_qkv_map(&k64, a.k, a.D, a.S, a.H, a.B, a.k_ss, a.k_sh, a.k_sb, SUB) ||
      !attn_detail::make_qkv_map(&v64, a.v, a.D, a.S, a.H, a.B, a.v_ss, a.v_sh, a.v_sb, SUB) ||
      !attn_detail::make_qkv_map(&do64, g.d_o, a.D, a.S, a.H, a.B, g.do_ss, g.do_sh, g.do_sb, SUB))
    return cudaErrorInvalidValue;

  const auto stats = a.D == 64 ? attn_stats_kernel<64> : attn_stats_kernel<128>;
  cudaError_t e = launch_pdl(stats, dim3((unsigned)a.H * (Sp / STAT_ROWS), a.B), dim3(STAT_ROWS * 8), 0, stream,
                             (const __nv_bfloat16*)a.o, (const __nv_bfloat16*)g.d_o, (const float*)a.lse, lse2,
                             dsc, a.H, a.S, Sp, a.scale, (long long)a.o_sb, (long long)a.o_ss, (long long)a.o_sh,
                             (long long)g.do_sb, (long long)g.do_ss, (long long)g.do_sh);
  if (e != cudaSuccess) return e;
  g_attn_launches.fetch_add(1, std::memory_order_relaxed);

  const dim3 grid(a.H, a.B, Sp / BT);   // tile index slowest: longest CTAs of every head go first
  p.out0 = (__nv_bfloat16*)g.dk; p.o0_sb = g.dk_sb; p.o0_ss = g.dk_ss; p.o0_sh = g.dk_sh;
  p.out1 = (__nv_bfloat16*)g.dv; p.o1_sb = g.dv_sb; p.o1_ss = g.dv_ss; p.o1_sh = g.dv_sh;
  e = a.D == 64 ? launch_bwd<64, true>(k128, v128, q64, do64, p, grid, stream)
                : launch_bwd<128, true>(k128, v128, q64, do64, p, grid, stream);
  if (e != cudaSuccess) return e;
  p.out0 = (__nv_bfloat16*)g.dq; p.o0_sb = g.dq_sb; p.o0_ss = g.dq_ss; p.o0_sh = g.dq_sh;
  p.out1 = nullptr; p.o1_sb = p.o1_ss = p.o1_sh = 0;
  const LateWait lw = late_wait_begin(1);   // independent of the dK / dV kernel: runs in its tail
  p.late_wait = lw.on;
  e = a.D == 64 ? launch_bwd<64, false>(q128, do128, k64, v64, p, grid, stream)
                : launch_bwd<128, false>(q128, do128, k64, v64, p, grid, stream);
  late_wait_commit(lw);
  return e;
}

size_t flash_attention_backward_stats(int B, int H, int S) {
  return 2 * (size_t)B * H * ((S + BT - 1) / BT * BT);
}

}  // namespace lt
