// Tensor-core GEMM whose operand tiles are fetched by the CUDA cores instead of TMA.
//
// TMA wants bf16 matrices with 16-byte row strides.  What does not come that way - fp32 operands,
// odd row lengths, a [256, 10] classifier head - used to be split, concatenated and padded by
// separate kernels or to fall back to a scalar kernel ([1021,777] x [777,1333] in fp32: 632 us).
// Here sixteen warps read the tiles with plain loads of whatever alignment there is, convert in
// registers and write the 128-byte-swizzled rows that tcgen05.mma reads; one more warp issues
// the MMAs into a TMEM accumulator.
//
// fp32 operands are split as x = hi + lo in bf16 and hi*hi + hi*lo + lo*hi is accumulated in
// fp32 (what the concatenated form computed, about 16 mantissa bits of each operand); the parts
// exist in shared memory only.
//
// What bounds it: a 128 x 128 x 64 step is 768 cycles of MMA (three products) against 16384
// values to load, split and store by 512 threads, about 13 instructions per pair of values,
// i.e. some 850 issue cycles: the two are balanced, and loads of the next step are issued into a
// second register set before the current one is converted so that neither waits for memory.
//
// Few tiles: the k loop of one tile is shared by a cluster of S CTAs (S <= 8).  Each CTA leaves
// its partial tile in its own shared memory and sums, for its 128 / S rows, the S partial rows
// through distributed shared memory in CTA order (deterministic, no second launch).
#include "gemm_direct.h"
#include "gemm_epilogue.cuh"
#include "sm100_ptx.cuh"
#include "common.cuh"

#include <atomic>

namespace lt {

extern std::atomic<uint64_t> g_gemm_launches;
KernelParams make_gemm_params(const GemmArgs& a);

namespace {

constexpr int BM = 128, BK = 64;
constexpr int LOAD_WARPS = 16;
constexpr int THREADS = 32 * (LOAD_WARPS + 1);

__device__ int g_direct_error = 0;

struct DirectParams {
  const void *A, *B;
  long long lda, ldb;
  long long a_si, a_so, b_si, b_so;   // batch strides (elements)
  int a_vec, b_vec;                   // rows allow paired (8-byte fp32, 4-byte bf16) loads
  int splits;                         // CTAs of a cluster that share one tile's k loop
};

// ------------------------------------------------------------------------------ operand tiles
// Two neighbouring values of a row as loaded.
template <typename T> struct Pair;
template <> struct Pair<float> {
  float x, y;
  __device__ static __forceinline__ Pair load2(const float* p) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    return {v.x, v.y};
  }
  __device__ static __forceinline__ Pair load(const float* p, bool v0, bool v1) {
    return {v0 ? p[0] : 0.0f, v1 ? p[1] : 0.0f};
  }
  __device__ __forceinline__ uint32_t hi() const {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  // bf16 of what `hi` leaves over
  __device__ __forceinline__ uint32_t lo(uint32_t h) const {
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - __uint_as_float(h << 16),
                                                   y - __uint_as_float(h & 0xffff0000u));
    return *reinterpret_cast<const uint32_t*>(&l);
  }
};
template <> struct Pair<__nv_bfloat16> {
  uint32_t v;
  __device__ static __forceinline__ Pair load2(const __nv_bfloat16* p) {
    return {*reinterpret_cast<const uint32_t*>(p)};
  }
  __device__ static __forceinline__ Pair load(const __nv_bfloat16* p, bool v0, bool v1) {
    const unsigned short* s = reinterpret_cast<const unsigned short*>(p);
    const uint32_t a = v0 ? s[0] : 0u, b = v1 ? s[1] : 0u;
    return {a | (b << 16)};
  }
  __device__ __forceinline__ uint32_t hi() const { return v; }
  __device__ __forceinline__ uint32_t lo(uint32_t) const { return 0u; }
};

// A tile of ROWS (m or n) x 64 (k) values as "row blocks" of 64 values that are contiguous in
// memory, one warp per block, a lane per pair of values:
//   K-major (MN = false): block j is row j, 64 values of k;
//   MN-major (MN = true): block j is row k = j % 64 of the 64-wide column chunk j / 64.
// Either way block j is one 128-byte row of the swizzled shared-memory tile.
template <typename T, int ROWS, bool MN>
struct Tile {
  static constexpr int N = ROWS / LOAD_WARPS;      // blocks per warp
  const T* p;            // first value of this lane's block 0 at the current k step
  long long ld;
  int warp, lane, outer_left, K;

  __device__ __forceinline__ void init(const void* base, long long ld_, int outer0, int outer, int k0,
                                       int K_, int warp_, int lane_) {
    warp = warp_; lane = lane_; ld = ld_; K = K_;
    outer_left = outer - outer0;
    const T* b = reinterpret_cast<const T*>(base);
    p = MN ? b + (long long)(k0 + warp) * ld + outer0 + 2 * lane
           : b + (long long)(outer0 + warp) * ld + k0 + 2 * lane;
  }
  __device__ __forceinline__ const T* block(int i) const {
    return MN ? p + (i % 4) * 16 * ld + (i / 4) * 64 : p + i * 16 * ld;
  }
  // loads the pairs of the step that starts at k0, then moves on to the next step
  __device__ __forceinline__ void load(Pair<T> (&r)[N], int k0, bool vec) {
    const int k_left = K - k0;
    if (k_left >= BK && outer_left >= ROWS) {
      if (vec) {
#pragma unroll
        for (int i = 0; i < N; ++i) r[i] = Pair<T>::load2(block(i));
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i) r[i] = Pair<T>::load(block(i), true, true);
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        bool v0, v1;
        if (MN) {
          const int c = (i / 4) * 64 + 2 * lane;
          const bool row = warp + (i % 4) * 16 < k_left;
          v0 = row && c < outer_left;
          v1 = row && c + 1 < outer_left;
        } else {
          const bool row = warp + i * 16 < outer_left;
          v0 = row && 2 * lane < k_left;
          v1 = row && 2 * lane + 1 < k_left;
        }
        r[i] = Pair<T>::load(block(i), v0, v1);
      }
    }
    p += MN ? (long long)BK * ld : (long long)BK;
  }
  // converts and writes the pairs into the swizzled tile(s) at `hi` (and `lo`)
  template <bool SPLIT>
  __device__ __forceinline__ void store(const Pair<T> (&r)[N], uint32_t hi, uint32_t lo) const {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int b = warp + i * 16;
      const uint32_t off = (uint32_t)b * 128u + (((uint32_t)lane * 4u) ^ (((uint32_t)b & 7u) << 4));
      const uint32_t h = r[i].hi();
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(hi + off), "r"(h) : "memory");
      if (SPLIT) asm volatile("st.shared.b32 [%0], %1;" ::"r"(lo + off), "r"(r[i].lo(h)) : "memory");
    }
  }
};

template <int BN, bool SPLIT>
struct Cfg {
  static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
  static constexpr int STAGE = (SPLIT ? 2 : 1) * (A_BYTES + B_BYTES);
  static constexpr int FIT = 200 * 1024 / STAGE;
  static constexpr int STAGES = FIT > 4 ? 4 : FIT;
  static constexpr int LD = BN + 1;                                 // staged result rows: odd, no bank conflicts
  static constexpr int RESULT = BM * LD * 4;
  static constexpr int BODY = STAGES * STAGE > RESULT ? STAGES * STAGE : RESULT;
  static constexpr int SMEM = BODY + 1024 /*align*/ + 256 /*barriers*/;
};

// ------------------------------------------------------------------------------ kernel
template <int BN, typename T, bool SPLIT, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_direct_kernel(const DirectParams d, const KernelParams p) {
  using C = Cfg<BN, SPLIT>;
  constexpr int STAGES = C::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::BODY);
  uint64_t* full_bar = bars;             // [STAGES]: one arrival per load warp
  uint64_t* empty_bar = bars + STAGES;   // [STAGES]: the MMAs that read the stage have retired
  uint64_t* done_bar = bars + 2 * STAGES;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int S = d.splits;
  const int rank = S > 1 ? (int)cluster_cta_rank() : 0;
  // one grid dimension for clusters, tiles and batch: the others end at 65535
  const int tiles = p.tiles_m * p.tiles_n, unit = (int)(blockIdx.x / S), b = unit / tiles, tile = unit % tiles;
  const int m0 = (tile % p.tiles_m) * BM, n0 = (tile / p.tiles_m) * BN;
  const int bi = b % p.batch_inner, bo = b / p.batch_inner;
  const int steps = (p.K + BK - 1) / BK;
  const int it0 = (int)((long long)steps * rank / S), it1 = (int)((long long)steps * (rank + 1) / S);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), LOAD_WARPS);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(done_bar), 1);
    fence_mbar_init();
  }
  if (warp == LOAD_WARPS) {
    tmem_alloc(smem_u32(tmem_holder), BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  pdl_enter();

  // stage layout: A hi | B hi | A lo | B lo
  const uint32_t ring = smem_u32(smem);
  bool ok = true;
  if (warp < LOAD_WARPS) {
    Tile<T, BM, A_MN> ta;
    Tile<T, BN, B_MN> tb;
    ta.init(reinterpret_cast<const T*>(d.A) + bi * d.a_si + bo * d.a_so, d.lda, m0, p.M, it0 * BK, p.K, warp, lane);
    tb.init(reinterpret_cast<const T*>(d.B) + bi * d.b_si + bo * d.b_so, d.ldb, n0, p.N, it0 * BK, p.K, warp, lane);
    Pair<T> ra[2][Tile<T, BM, A_MN>::N], rb[2][Tile<T, BN, B_MN>::N];
    ta.load(ra[0], it0 * BK, d.a_vec);
    tb.load(rb[0], it0 * BK, d.b_vec);
    int stage = 0;
    uint32_t phase = 0;
    // two steps per turn, so that both register sets are indexed statically
    for (int it = it0; ok && it < it1; it += 2) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (it + h >= it1) break;
        if (it + h + 1 < it1) {
          ta.load(ra[h ^ 1], (it + h + 1) * BK, d.a_vec);
          tb.load(rb[h ^ 1], (it + h + 1) * BK, d.b_vec);
        }
        if (!mbar_wait_bounded_warp(smem_u32(&empty_bar[stage]), phase ^ 1, abort_flag, &g_direct_error, 31)) {
          ok = false;
          break;
        }
        const uint32_t sa = ring + stage * C::STAGE, sb = sa + C::A_BYTES;
        ta.template store<SPLIT>(ra[h], sa, sa + C::A_BYTES + C::B_BYTES);
        tb.template store<SPLIT>(rb[h], sb, sb + C::A_BYTES + C::B_BYTES);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&full_bar[stage]));
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
    // the accumulator is complete, and with it every MMA that reads the ring
    if (!mbar_wait_bounded_warp(smem_u32(done_bar), 0, abort_flag, &g_direct_error, 32)) ok = false;
    tc_fence_after_sync();
    if (ok) {
      // TMEM lane = tile row: this warp's 32 rows, its quarter of the columns
      float* dst = reinterpret_cast<float*>(smem) + ((warp & 3) * 32 + lane) * C::LD + (warp >> 2) * (BN / 4);
      const uint32_t src = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * (BN / 4);
      if constexpr (BN == 128) {
        uint32_t r[32];
        tmem_ld_32x32(src, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) dst[i] = __uint_as_float(r[i]);
      } else {
        uint32_t r[16];
        tmem_ld_32x16(src, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) dst[i] = __uint_as_float(r[i]);
      }
      tc_fence_before_sync();
    }
  } else if (elect_one()) {
    const uint32_t idesc = make_idesc_bf16(BM, BN, A_MN, B_MN);
    constexpr uint32_t a_lbo = A_MN ? 64 * BK * 2 : 16, b_lbo = B_MN ? 64 * BK * 2 : 16;
    constexpr uint32_t a_step = A_MN ? (2048 >> 4) : (32 >> 4), b_step = B_MN ? (2048 >> 4) : (32 >> 4);
    int stage = 0;
    uint32_t phase = 0;
    for (int it = it0; it < it1; ++it) {
      if (!mbar_wait_bounded(smem_u32(&full_bar[stage]), phase, abort_flag, &g_direct_error, 33)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const uint32_t sa = ring + stage * C::STAGE;
      const uint64_t a_hi = make_smem_desc_sw128(sa, a_lbo, 1024);
      const uint64_t b_hi = make_smem_desc_sw128(sa + C::A_BYTES, b_lbo, 1024);
#pragma unroll
      for (int j = 0; j < BK / 16; ++j)
        umma_bf16(tmem, a_hi + (uint64_t)(j * a_step), b_hi + (uint64_t)(j * b_step), idesc, (it > it0 || j > 0) ? 1u : 0u);
      if (SPLIT) {
        const uint64_t a_lo = make_smem_desc_sw128(sa + C::A_BYTES + C::B_BYTES, a_lbo, 1024);
        const uint64_t b_lo = make_smem_desc_sw128(sa + 2 * C::A_BYTES + C::B_BYTES, b_lbo, 1024);
#pragma unroll
        for (int j = 0; j < BK / 16; ++j)
          umma_bf16(tmem, a_hi + (uint64_t)(j * a_step), b_lo + (uint64_t)(j * b_step), idesc, 1u);
#pragma unroll
        for (int j = 0; j < BK / 16; ++j)
          umma_bf16(tmem, a_lo + (uint64_t)(j * a_step), b_hi + (uint64_t)(j * b_step), idesc, 1u);
      }
      umma_commit(smem_u32(&empty_bar[stage]));
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (ok) umma_commit(smem_u32(done_bar));
    // nothing may still be on its way to a barrier when the CTA exits
    if (ok) mbar_wait_bounded(smem_u32(done_bar), 0, abort_flag, &g_direct_error, 34);
  }
  __syncthreads();
  if (S > 1) {   // every partial tile of the cluster is staged
    cluster_arrive();
    cluster_wait();
  }
  if (warp < LOAD_WARPS && ok) {
    const size_t esz = p.c_fp32 ? 4 : 2;
    char* c_base = (char*)p.C + (size_t)(bi * p.c_stride_inner + bo * p.c_stride_outer) * esz;
    const int rows = BM / S;
    for (int r = rank * rows + warp; r < (rank + 1) * rows; r += LOAD_WARPS) {
      if (m0 + r >= p.M) break;
      float v[BN / 32];
      if (S == 1) {
        const float* src = reinterpret_cast<const float*>(smem) + r * C::LD + lane;
#pragma unroll
        for (int i = 0; i < BN / 32; ++i) v[i] = src[32 * i];
      } else {
        const uint32_t a = ring + (uint32_t)(r * C::LD + lane) * 4u;
#pragma unroll
        for (int i = 0; i < BN / 32; ++i) v[i] = 0.0f;
        for (int s = 0; s < S; ++s) {
          const uint32_t q = map_to_cta(a, (uint32_t)s);
#pragma unroll
          for (int i = 0; i < BN / 32; ++i) {
            float x;
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(q + 128u * i) : "memory");
            v[i] += x;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < BN / 32; ++i) {
        const int col = n0 + lane + 32 * i;
        if (col < p.N) epilogue_store_scalar(p, c_base, m0 + r, col, v[i]);
      }
    }
  }
  if (S > 1) {   // no CTA leaves while another may read its shared memory
    cluster_arrive();
    cluster_wait();
  }
  if (warp == LOAD_WARPS) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem, BN);
  }
}

// ------------------------------------------------------------------------------ host side
int sms() { return sm_count(); }

struct Plan { int bn, splits; double us; };

// Time of one 64-wide k step of a CTA (us), measured on B200: it is the shared-memory / L1 pipe's
// (operand loads, swizzled stores and the MMAs' own reads share it), and a row that does not start
// on a pair boundary costs a second load per pair.
double step_us(int bn, bool split, bool paired) {
  if (bn == 128) return split ? (paired ? 1.25 : 1.7) : (paired ? 0.8 : 1.4);
  return split ? (paired ? 0.9 : 1.15) : (paired ? 0.6 : 0.95);
}

bool rows_paired(const GemmArgs& a, const void* q, int64_t ld, int64_t si, int64_t so) {
  return reinterpret_cast<uintptr_t>(q) % (a.ab_fp32 ? 8 : 4) == 0 && ld % 2 == 0 && si % 2 == 0 && so % 2 == 0;
}
bool a_paired(const GemmArgs& a) { return rows_paired(a, a.A, a.lda, a.a_stride_inner, a.a_stride_outer); }
bool b_paired(const GemmArgs& a) { return rows_paired(a, a.B, a.ldb, a.b_stride_inner, a.b_stride_outer); }

// Width of the tile and CTAs per tile: the cheapest of waves x (k steps of a CTA + fixed cost).
Plan choose_plan(const GemmArgs& a, bool split, long long batch) {
  const long long tm = (a.M + BM - 1) / BM, steps = (a.K + BK - 1) / BK;
  const bool paired = a_paired(a) && b_paired(a);
  Plan best{64, 1, 1e30};
  for (int bn = 64; bn <= 128; bn += 64) {
    if (bn == 128 && a.N <= 64) continue;
    const long long tiles = tm * ((a.N + bn - 1) / bn) * batch;
    for (int s = 1; s <= 8; s *= 2) {
      if (s > steps) break;
      const long long waves = (tiles * s + sms() - 1) / sms();
      const double cost = (double)waves * ((double)((steps + s - 1) / s) * step_us(bn, split, paired) + 4.0 + (s > 1 ? 1.0 : 0.0));
      if (cost < best.us) best = {bn, s, cost};
    }
  }
  return best;
}

template <int BN, typename T, bool SPLIT, bool A_MN, bool B_MN>
cudaError_t launch(const DirectParams& d, const KernelParams& p, cudaStream_t stream) {
  using C = Cfg<BN, SPLIT>;
  auto* kernel = gemm_direct_kernel<BN, T, SPLIT, A_MN, B_MN>;
  static const cudaError_t attr = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
  if (attr != cudaSuccess) return attr;
  const dim3 grid((unsigned)((long long)p.tiles_m * p.tiles_n * d.splits * p.batch_total));
  const cudaError_t e = launch_pdl_cluster(kernel, grid, dim3(THREADS), C::SMEM, stream, d.splits, d, p);
  if (e != cudaSuccess) return e;
  g_gemm_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaGetLastError();
}

template <int BN, typename T, bool SPLIT>
cudaError_t launch_layout(const GemmArgs& a, const DirectParams& d, const KernelParams& p, cudaStream_t s) {
  if (a.a_mn_major) return a.b_mn_major ? launch<BN, T, SPLIT, true, true>(d, p, s) : launch<BN, T, SPLIT, true, false>(d, p, s);
  return a.b_mn_major ? launch<BN, T, SPLIT, false, true>(d, p, s) : launch<BN, T, SPLIT, false, false>(d, p, s);
}

}  // namespace

cudaError_t gemm_direct(const GemmArgs& a, cudaStream_t stream) {
  const bool f32 = a.ab_fp32 != 0;
  KernelParams p = make_gemm_params(a);
  const Plan plan = choose_plan(a, f32, p.batch_total);
  p.tiles_m = (a.M + BM - 1) / BM;
  p.tiles_n = (a.N + plan.bn - 1) / plan.bn;
  DirectParams d;
  d.A = a.A; d.B = a.B; d.lda = a.lda; d.ldb = a.ldb;
  d.a_si = a.a_stride_inner; d.a_so = a.a_stride_outer;
  d.b_si = a.b_stride_inner; d.b_so = a.b_stride_outer;
  d.splits = plan.splits;
  d.a_vec = a_paired(a);
  d.b_vec = b_paired(a);
  if (f32) return plan.bn == 128 ? launch_layout<128, float, true>(a, d, p, stream) : launch_layout<64, float, true>(a, d, p, stream);
  return plan.bn == 128 ? launch_layout<128, __nv_bfloat16, false>(a, d, p, stream)
                        : launch_layout<64, __nv_bfloat16, false>(a, d, p, stream);
}

double gemm_direct_cost(const GemmArgs& a) {
  const long long batch = (long long)a.batch_inner * a.batch_outer;
  const Plan p = choose_plan(a, a.ab_fp32 != 0, batch);
  const long long tiles = (long long)((a.M + BM - 1) / BM) * ((a.N + p.bn - 1) / p.bn) * batch * p.splits;
  const double waves = (double)((tiles + sms() - 1) / sms()), rows = (a.M < BM ? a.M : BM) / (double)BM;
  const double steps = ((a.K + BK - 1) / BK + p.splits - 1) / p.splits;
  // the plan's own estimate leaves out what the element-wise epilogue takes for its rows; fitted to the
  // same 455 products as the other routes (choose_route)
  const double epilogue = (p.bn == 64 ? 3.5 : 7.2) * rows / p.splits + (p.splits > 1 ? 2.1 : 0.0);
  return 1e-6 * (waves * (0.85 * steps * step_us(p.bn, a.ab_fp32 != 0, a_paired(a) && b_paired(a)) + epilogue + 3.1) - 0.5);
}

// ------------------------------------------------------------------------------ packing
// Copies of the operands that TMA can address.  K-major [R, K] becomes [R, parts x Kp] and MN-major
// [K, C] becomes [parts x Kp, Cp], Kp a multiple of 64, Cp of 8; parts = 2 for fp32 (hi, lo), 1 for
// bf16.  Rows and columns of k beyond K are zero; the matrices of a batch follow one another.  One launch
// for both operands; a thread makes eight values (16-byte stores), a block 2048 of one matrix.
namespace {

struct PackOperand {
  const void* src;
  __nv_bfloat16* dst;
  long long ld, dst_ld, lo;    // lo: distance of the lo part in elements
  long long si, so, dst_matrix;  // batch strides of the source, elements of a copied matrix
  int batch_inner, blocks;     // blocks of one matrix
  int rows, cols;              // of the source
  int drows, dcols;            // of one part
};

// The 16 bytes at `s` from the two aligned 16-byte words around them (rows of odd length start
// anywhere; narrow loads at a 16-byte stride made the pass over two [4095,4095] bf16 matrices 150 us).
__device__ __forceinline__ uint4 load16_any(const void* s) {
  const uintptr_t q = reinterpret_cast<uintptr_t>(s);
  const uint4* a = reinterpret_cast<const uint4*>(q & ~uintptr_t(15));
  const uint4 lo = a[0];
  const unsigned m = (unsigned)(q & 15);
  if (m == 0) return lo;
  const uint4 hi = a[1];
  const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  uint32_t t[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) {   // words m/4 ... m/4 + 4
    const uint32_t e = (m & 8) ? w[i + 2 > 7 ? 7 : i + 2] : w[i];
    const uint32_t o = (m & 8) ? w[i + 3 > 7 ? 7 : i + 3] : w[i + 1];
    t[i] = (m & 4) ? o : e;
  }
  const unsigned sh = (m & 3) * 8;
  return make_uint4(__funnelshift_r(t[0], t[1], sh), __funnelshift_r(t[1], t[2], sh),
                    __funnelshift_r(t[2], t[3], sh), __funnelshift_r(t[3], t[4], sh));
}

template <typename T>
__device__ __forceinline__ void pack_block(const PackOperand& o, unsigned block) {
  const int per_row = o.dcols / 8;
  const int matrix = (int)(block / o.blocks);
  const long long v = (long long)(block % o.blocks) * 256 + threadIdx.x;
  const long long r = v / per_row;
  if (r >= o.drows) return;
  const int c = (int)(v - r * per_row) * 8;
  const T* s = reinterpret_cast<const T*>(o.src) + matrix % o.batch_inner * o.si + matrix / o.batch_inner * o.so +
               r * o.ld + c;
  float x[8];
  const int left = r < o.rows ? o.cols - c : 0;
  if (left >= 8) {
#pragma unroll
    for (int i = 0; i < 8; i += VecIO<T>::N) {
      float t[VecIO<T>::N];
      VecIO<T>::unpack(load16_any(s + i), t);
#pragma unroll
      for (int j = 0; j < VecIO<T>::N; ++j) x[i + j] = t[j];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = i < left ? VecIO<T>::ld(s + i) : 0.0f;
  }
  __nv_bfloat16* d = o.dst + matrix * o.dst_matrix + r * o.dst_ld + c;
  VecIO<__nv_bfloat16>::store(d, x);
  if (sizeof(T) == 4) {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] -= __bfloat162float(__float2bfloat16(x[i]));
    VecIO<__nv_bfloat16>::store(d + o.lo, x);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) pack_kernel(const PackOperand a, const PackOperand b, const unsigned a_blocks) {
  pdl_enter();
  if (blockIdx.x < a_blocks) pack_block<T>(a, blockIdx.x);
  else pack_block<T>(b, blockIdx.x - a_blocks);
}

long long round_up(long long v, long long q) { return (v + q - 1) / q * q; }

long long batch_of(const GemmArgs& a) {
  return (long long)a.batch_inner * a.batch_outer;
}

PackOperand pack_operand(const GemmArgs& g, bool is_a) {
  const int parts = g.ab_fp32 ? 2 : 1, Kp = (int)round_up(g.K, 64);
  const int outer = is_a ? g.M : g.N;
  PackOperand o;
  o.src = is_a ? g.A : g.B; o.dst = nullptr; o.ld = is_a ? g.lda : g.ldb;
  o.si = is_a ? g.a_stride_inner : g.b_stride_inner;
  o.so = is_a ? g.a_stride_outer : g.b_stride_outer;
  o.batch_inner = g.batch_inner;
  if (is_a ? g.a_mn_major : g.b_mn_major) {
    o.rows = g.K; o.cols = outer; o.drows = Kp; o.dcols = (int)round_up(outer, 8);
    o.dst_ld = o.dcols;
    o.lo = (long long)Kp * o.dst_ld;
  } else {
    o.rows = outer; o.cols = g.K; o.drows = outer; o.dcols = Kp;
    o.dst_ld = (long long)parts * Kp;
    o.lo = Kp;
  }
  o.dst_matrix = (long long)parts * o.drows * o.dcols;
  o.blocks = (int)(((long long)o.drows * (o.dcols / 8) + 255) / 256);
  return o;
}
size_t pack_bytes(const PackOperand& o, long long batch) { return (size_t)round_up(batch * o.dst_matrix * 2, 256); }

}  // namespace

size_t gemm_pack_bytes(const GemmArgs& a) {
  return pack_bytes(pack_operand(a, true), batch_of(a)) + pack_bytes(pack_operand(a, false), batch_of(a));
}

bool gemm_pack_fits(const GemmArgs& a) {
  const long long batch = batch_of(a);
  return batch * (pack_operand(a, true).blocks + (long long)pack_operand(a, false).blocks) < (1ll << 31);
}

cudaError_t gemm_pack(GemmArgs& g, void* workspace, cudaStream_t stream) {
  const int parts = g.ab_fp32 ? 2 : 1;
  const long long batch = batch_of(g);
  PackOperand a = pack_operand(g, true), b = pack_operand(g, false);
  a.dst = (__nv_bfloat16*)workspace;
  b.dst = (__nv_bfloat16*)((char*)workspace + pack_bytes(a, batch));
  const unsigned na = (unsigned)(a.blocks * batch), nb = (unsigned)(b.blocks * batch);
  const cudaError_t e = g.ab_fp32
      ? launch_pdl(pack_kernel<float>, dim3(na + nb), dim3(256), 0, stream, a, b, na)
      : launch_pdl(pack_kernel<__nv_bfloat16>, dim3(na + nb), dim3(256), 0, stream, a, b, na);
  if (e != cudaSuccess) return e;
  g_gemm_launches.fetch_add(1, std::memory_order_relaxed);
  const int Kp = (int)round_up(g.K, 64);
  g.A = a.dst; g.lda = a.dst_ld;
  g.B = b.dst; g.ldb = b.dst_ld;
  g.a_stride_inner = a.dst_matrix; g.a_stride_outer = a.dst_matrix * a.batch_inner;
  g.b_stride_inner = b.dst_matrix; g.b_stride_outer = b.dst_matrix * b.batch_inner;
  if (parts == 2) { g.k_seg = Kp; g.K = 3 * Kp; }
  g.ab_fp32 = 0;
  return cudaSuccess;
}

int gemm_direct_last_error() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_direct_error, sizeof(int));
  return v;
}
void gemm_direct_clear_error() {
  int v = 0;
  cudaMemcpyToSymbol(g_direct_error, &v, sizeof(int));
}

}  // namespace lt
