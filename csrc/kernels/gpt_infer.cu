// GPT inference on bf16 weights.
//
// gpt_forward: the launches of a forward pass, issued back to back from C++ (the layer classes
// spend about 15 us of host time per kernel: 1.27 ms for a 124M forward whose kernels take 1 ms).
//
// gpt_decode: one persistent cooperative kernel generates a run of tokens, one position at a
// time against cached keys and values (a full forward per token took 1.8 ms).  A token
// is a chain of matrix-vector products over all weights (247 MB of bf16 at 124M: 38 us of
// memory time), so the kernel is built around the chain's latency:
//   * one CTA per SM; grid-wide barriers of 1.7 us with their skew, four per layer (qkv | attention
//     and out projection | ffn1 | ffn2) and a fifth between those two when there are many keys;
//   * every CTA keeps its own copy of the residual stream in shared memory and redoes the cheap
//     vector work (partial sums, bias, residual, LayerNorm) instead of paying a barrier for it;
//   * a product [K] x [K, N] is cut into units of 8 columns (16-byte loads), 2 to 16 units per
//     CTA, and over K as well where N alone leaves SMs idle; the consumer adds the K partials in
//     fixed order (deterministic);
//   * the next layer's weights are prefetched into L2 while this one's are multiplied, so the
//     products read L2 and memory streams without gaps;
//   * the vocabulary is sampled on the device by every CTA redundantly (no further barrier); the
//     top-k threshold comes from the CTAs' local maxima: the k-th largest of them is a lower
//     bound that leaves a few dozen candidates.
// Intermediate results are rounded to bf16 exactly where the layer kernels round.
#include "gpt_infer.h"
#include "attention.h"
#include "common.cuh"
#include "gemm.h"
#include "ops.h"
#include "sm100_ptx.cuh"

#include <algorithm>

namespace lt {
namespace {

typedef __nv_bfloat16 bf16;

// Threads of the decode kernel.  Its phases are short and made of work that every thread repeats
// (addresses, reductions): with 512 threads the issue slots of that overhead, not memory, took most
// of a phase.
constexpr int DT = 256;
constexpr int WARPS = DT / 32;
constexpr int MAX_CAND = 2048;       // top-k candidates kept in shared memory
constexpr long long BARRIER_BUDGET = 4000000000ll;   // about two seconds of SM clocks

// Where a [K, N] product is cut: `nu` units of 8 columns per CTA, `ks` slices of K.
struct Split { int nu, groups, ks; };   // nu: power of two, at most 16
constexpr int MAX_KS = 16;           // partial sums per element that a consumer adds (out_head: one per head)
constexpr int SPLIT_KS = 4;          // of a product cut over K for its own sake

struct DecodeParams {
  GptWeights w;
  const bf16* x0;                    // residual stream of the prompt's last position
  bf16* cache;                       // [layers, rows, 3 embed]
  long long cache_rows;
  int prompt, first, last;
  float temperature;
  int top_k;
  const float* rnd;
  int* ids_out;
  Split qkv, out, f1, f2, head;
  Split out_head;                    // output projection with a head per K slice; ks = 0: not used
  int fuse_keys;                     // up to here every task of out_head redoes its head's attention
  float* part;                       // [max ks, embed] partial sums
  float* attn;                       // [heads, splits, head_dim + 2]
  bf16* h;                           // [ffn]
  bf16* logits;                      // [vocab padded to 8]
  unsigned* gmax;                    // [grid] largest key of each CTA's logits
  unsigned* bar;
  int* status;
};

__device__ __forceinline__ float rb(float v) { return __bfloat162float(__float2bfloat16(v)); }
__device__ __forceinline__ float ldb(const void* p, int i) { return __bfloat162float(reinterpret_cast<const bf16*>(p)[i]); }
// order-preserving 16-bit key of a bf16
__device__ __forceinline__ unsigned key_of(unsigned short u) { return (u & 0x8000) ? (unsigned)(unsigned short)~u : (u | 0x8000u); }
__device__ __forceinline__ float key_value(unsigned k) {
  const unsigned short u = (k & 0x8000) ? (unsigned short)(k & 0x7fff) : (unsigned short)~k;
  return __uint_as_float((unsigned)u << 16);
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier over all CTAs of the (cooperative) grid, in two halves: what a CTA does between them (asking
// for the next weights: 600 to 2000 cycles of issue per phase) nobody waits for.  `goal` counts
// arrivals over the kernel's life.
__device__ void grid_arrive(unsigned* bar, unsigned& goal) {
  __syncthreads();
  goal += gridDim.x;
  // release at gpu scope: covers what the whole CTA wrote before the __syncthreads
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}
// Returns false, for every thread of the CTA, when the wait ran out of time anywhere.
__device__ bool grid_wait(unsigned* bar, unsigned goal, int* status, int* sh_ok) {
  if (threadIdx.x == 0) {
    const long long t0 = clock64();
    int ok = 1;
    for (unsigned spin = 0; (int)(ld_acquire(bar) - goal) < 0; ++spin) {
      if ((spin & 0x3ff) == 0x3ff) {
        if (*(volatile int*)status != 0) { ok = 0; break; }
        if (clock64() - t0 > BARRIER_BUDGET) { atomicExch(status, 1); ok = 0; break; }
      }
    }
    *sh_ok = ok;
  }
  __syncthreads();
  return *sh_ok != 0;
}

// Asks L2 for a weight array, a line per thread and turn over the whole grid.
__device__ __forceinline__ void prefetch_l2(const void* p, long long bytes) {
  const int lines = (int)((bytes + 127) >> 7), step = gridDim.x * DT;
  for (int i = blockIdx.x * DT + threadIdx.x; i < lines; i += step)
    asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)p + ((long long)i << 7)));
}

// A [K, N] product as a CTA sees it: task t < groups * ks is column group t % groups, K slice
// t / groups; each CTA takes tasks blockIdx.x, + gridDim.x, ...  A thread multiplies unit u (8
// columns) of every RP-th row of the slice.  Lives in shared memory; the geometry of the CTA's
// first task is the same in every layer.
constexpr int FETCH = 24;    // weight slots per thread, see fetch()
struct Product {
  int ldw, K, N, lg, tasks;
  Split sp;
  int k0, n, u0, slice;      // current task: K slice [k0, k0 + n), first unit, index of the slice
  __device__ void init(int ldw_, int K_, int N_, const Split& s) {
    ldw = ldw_; K = K_; N = N_; sp = s;
    lg = 31 - __clz(sp.nu);
    tasks = sp.groups * sp.ks;
    select(blockIdx.x);
  }
  __device__ void select(int t) {
    slice = t / sp.groups;
    u0 = (t - slice * sp.groups) * sp.nu;
    const int len = K / sp.ks;
    k0 = (len * slice) & ~7;
    n = (slice + 1 == sp.ks ? K : (len * (slice + 1)) & ~7) - k0;
  }
  // this thread's first weight and its number of rows
  __device__ __forceinline__ int rows(long long& off) const { return rows_at(off, u0); }
  __device__ __forceinline__ int rows_at(long long& off, int first_unit) const {
    const int u = first_unit + ((int)threadIdx.x & (sp.nu - 1)), r = threadIdx.x >> lg, RP = DT >> lg;
    off = (long long)(k0 + r) * ldw + u * 8;
    return u * 8 < N && r < n ? (n - r + RP - 1) >> (31 - __clz(RP)) : 0;
  }
  // several tasks per CTA, all over the whole of K, whose weights fit half of the slots
  __device__ __forceinline__ bool streamed() const {
    const int RP = DT >> lg;
    return sp.ks == 1 && tasks > (int)gridDim.x && (K + RP - 1) / RP <= FETCH / 2;
  }
};

// The first weights of this CTA's first task, copied into shared memory (a 16-byte slot per thread
// and row) before the barrier that the activations wait for: their latency hides behind it.
__device__ __noinline__ void fetch(const Product& p, const void* W, uint4* slots, int first_unit) {
  long long off;
  int cnt = p.rows_at(off, first_unit);
  if (cnt > FETCH) cnt = FETCH;
  const bf16* q = reinterpret_cast<const bf16*>(W) + off;
  const long long step = (long long)(DT >> p.lg) * p.ldw;
  uint32_t dst = ptx::smem_u32(slots + threadIdx.x);
#pragma unroll 4
  for (int i = 0; i < cnt; ++i, q += step, dst += DT * 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(q) : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void fetch(const Product& p, const void* W, uint4* slots) {
  if ((int)blockIdx.x < p.tasks) fetch(p, W, slots, p.u0);
}

__device__ __forceinline__ void add8(float2 (&acc)[4], const uint4& v, float x) {
  const float2 xx = make_float2(x, x);
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    acc[j] = ptx::ffma2(xx, make_float2(__uint_as_float(u[j] << 16), __uint_as_float(u[j] & 0xffff0000u)), acc[j]);
}

// Sums of the current task: `xs` are the activations of its K slice; column c < 8 nu of the task ends
// up in thread c.  Sums are taken in a fixed order.  `slots`: its first weights, or null; `behind`: one
// more group of copies has been started after them.
__device__ __noinline__ float dot_task(const Product& p, const void* W, const uint4* slots, bool behind,
                                       const float* xs, float* red) {
  float2 acc[4] = {};
  long long off;
  const int cnt = p.rows(off), RP = DT >> p.lg;
  const float* x = xs + (threadIdx.x >> p.lg);
  int i = 0;
  if (slots) {
    // a thread reads the slots it filled itself
    if (behind) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_all;" ::: "memory");
    const uint4* q = slots + threadIdx.x;
    const int m = cnt < FETCH ? cnt : FETCH;
#pragma unroll 4
    for (; i < m; ++i, q += DT) add8(acc, *q, x[i * RP]);
  }
  if (i < cnt) {
    const long long step = (long long)RP * p.ldw;
    const bf16* q = reinterpret_cast<const bf16*>(W) + off + (long long)i * step;
    for (; i + 8 <= cnt; i += 8, q += 8 * step) {
      uint4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __ldg(reinterpret_cast<const uint4*>(q + j * step));
#pragma unroll
      for (int j = 0; j < 8; ++j) add8(acc, v[j], x[(i + j) * RP]);
    }
    for (; i < cnt; ++i, q += step) add8(acc, __ldg(reinterpret_cast<const uint4*>(q)), x[i * RP]);
  }
  // lanes of a warp that share a unit, then the warps
  float a[8] = {acc[0].x, acc[0].y, acc[1].x, acc[1].y, acc[2].x, acc[2].y, acc[3].x, acc[3].y};
  const int nu = p.sp.nu, lane = threadIdx.x & 31;
  for (int o = 16; o >= nu; o >>= 1)
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] += __shfl_xor_sync(0xffffffffu, a[j], o);
  if (lane < nu) {
    float4* d = reinterpret_cast<float4*>(red + (threadIdx.x >> 5) * 132 + lane * 8);
    d[0] = make_float4(a[0], a[1], a[2], a[3]);
    d[1] = make_float4(a[4], a[5], a[6], a[7]);
  }
  __syncthreads();
  float s = 0.0f;
  if ((int)threadIdx.x < nu * 8) {
#pragma unroll
    for (int w = 0; w < WARPS; ++w) s += red[w * 132 + threadIdx.x];
  }
  return s;
}

// Runs this CTA's tasks: `load(k0, n)` gives the activations of a K slice, `emit(slice, column, sum)`
// takes every finished sum.
template <typename Load, typename Emit>
__device__ __forceinline__ void product(Product& p, const void* W, uint4* slots, float* red, Load load,
                                        Emit emit) {
  const int c = threadIdx.x;
  const bool streamed = p.streamed();
  int half = 0;                                // streamed: the half of the slots this task's weights are in
  for (int t = blockIdx.x; t < p.tasks; t += gridDim.x) {
    const bool first = t == (int)blockIdx.x;
    const bool behind = streamed && t + (int)gridDim.x < p.tasks;
    // the next task's weights arrive under this one's sums
    if (behind) fetch(p, W, slots + (half ^ 1) * (FETCH / 2) * DT, (t + (int)gridDim.x) * p.sp.nu);
    if (!first) {
      __syncthreads();
      if (c == 0) p.select(t);
      __syncthreads();
    }
    const float s = dot_task(p, W, first || streamed ? slots + half * (FETCH / 2) * DT : nullptr, behind,
                             load(p.k0, p.n), red);
    half ^= streamed;
    if (c < p.sp.nu * 8 && p.u0 * 8 + c < p.N) emit(p.slice, p.u0 * 8 + c, s);
  }
  if ((int)(blockIdx.x + gridDim.x) < p.tasks) {   // back to the first task
    __syncthreads();
    if (c == 0) p.select(blockIdx.x);
    __syncthreads();
  }
}

// The elements of a vector parameter that this thread handles (e = thread, + DT, ...), loaded
// ahead like the weights; longer vectors load the rest where they are used.
constexpr int EPT = 3;
constexpr int NORM_V = 8;            // 16-byte vectors per lane when a warp norms the whole stream
struct VecSlice {
  const void* p;
  bf16 v[EPT];
  __device__ __forceinline__ void fetch(const void* q, int E) {
    p = q;
#pragma unroll
    for (int i = 0; i < EPT; ++i)
      if ((int)threadIdx.x + i * DT < E) v[i] = reinterpret_cast<const bf16*>(q)[threadIdx.x + i * DT];
  }
  __device__ __forceinline__ float at(int i) const {
    return __bfloat162float(v[i]);
  }
};

constexpr int DECODE_SMEM_MAX = 200 * 1024;   // beside about 17 KB of static shared memory
// Shared memory of the decode kernel (floats): slots | x | n | slice | red.
__host__ __device__ inline int decode_smem_floats(int E, int F) {
  const int wide = E > F ? E : F;
  return FETCH * DT * 4 + 2 * E + wide + WARPS * 132 + 64;
}

// Attention of one head over keys [j0, j1): the unnormalised sum, maximum and denominator.  A group of
// D / 8 lanes takes a key at a time and keeps its own running maximum; the groups are merged at
// the end.
template <int D>
__device__ __noinline__ void attend(const bf16* __restrict__ rows, long long ld, int E, int h, int pos,
                                       int j0, int j1, float scale, float* red, float* out) {
  constexpr int LPK = D / 8;                 // lanes per key: 16 bytes each
  constexpr int KP = DT / LPK;               // keys per pass
  constexpr int B = 4;                       // passes whose loads are in flight together
  const int v = threadIdx.x % LPK, g = threadIdx.x / LPK;
  const bf16* base = rows + h * D + v * 8;
  float q[8];
  VecIO<bf16>::load(base + (long long)pos * ld, q);
  float m = -INFINITY, l = 0.0f, acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int j = j0; j < j1; j += B * KP) {
    uint4 kr[B], vr[B];
#pragma unroll
    for (int b = 0; b < B; ++b)
      if (j + b * KP + g < j1) {
        const bf16* r = base + (long long)(j + b * KP + g) * ld + E;
        kr[b] = VecIO<bf16>::load_raw(r);
        vr[b] = VecIO<bf16>::load_raw(r + E);
      }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const bool in = j + b * KP + g < j1;
      float d = 0.0f, f[8];
      if (in) {
        VecIO<bf16>::unpack(kr[b], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) d += q[i] * f[i];
      }
#pragma unroll
      for (int o = LPK / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if (in) {
        d *= scale;
        const float m2 = fmaxf(m, d), old = __expf(m - m2), w = __expf(d - m2);
        m = m2;
        l = l * old + w;
        VecIO<bf16>::unpack(vr[b], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = acc[i] * old + w * f[i];
      }
    }
  }
  // groups of a warp, then the warps (an empty group has m = -inf and weight 0)
  float M = m;
#pragma unroll
  for (int o = 16; o >= LPK; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  const float w = M == -INFINITY ? 0.0f : __expf(m - M);
  l *= w;
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] *= w;
#pragma unroll
  for (int o = 16; o >= LPK; o >>= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane < LPK) {
#pragma unroll
    for (int i = 0; i < 8; ++i) red[warp * 132 + lane * 8 + i] = acc[i];
    if (lane == 0) { red[warp * 132 + 128] = M; red[warp * 132 + 129] = l; }
  }
  __syncthreads();
  if ((int)threadIdx.x < D + 2) {
    const int d = threadIdx.x;
    float mx = red[128];
#pragma unroll
    for (int k = 1; k < WARPS; ++k) mx = fmaxf(mx, red[k * 132 + 128]);
    const int at = d < D ? d : 129;
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) {
      const float mk = red[k * 132 + 128];
      if (mk > -INFINITY) s += __expf(mk - mx) * red[k * 132 + at];
    }
    out[d] = d == D ? mx : s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(DT, 1) gpt_decode_kernel(const __grid_constant__ DecodeParams p) {
  extern __shared__ __align__(16) float smem[];
  const GptWeights& w = p.w;
  const int E = w.embed, F = w.ffn, D = w.head_dim, H = w.heads, V = w.vocab, G = (int)gridDim.x;
  const int tid = threadIdx.x;
  uint4* slots = reinterpret_cast<uint4*>(smem);
  float* x = smem + FETCH * DT * 4;          // residual stream (bf16 values), the same in every CTA
  float* n = x + E;                          // its LayerNorm
  float* xs = n + E;                         // activations of a product
  float* red = xs + (E > F ? E : F);
  __shared__ float2 sh[32];
  __shared__ int sh_ok, sh_cnt, sh_last;
  __shared__ unsigned sh_key;
  __shared__ unsigned cand[MAX_CAND];        // keys of the logits above the bound
  __shared__ int cand_at[MAX_CAND];          // and their places
  float* shf = reinterpret_cast<float*>(sh);
  unsigned goal = 0;
  const long long ld = 3ll * E;

  VecSlice gamma, beta, bias;
  __shared__ Product qkv, out, out_head, f1, f2, head;
  if (tid == 0) {
    qkv.init(3 * E, E, 3 * E, p.qkv);
    out.init(E, E, E, p.out);
    if (p.out_head.ks) out_head.init(E, E, E, p.out_head);
    f1.init(F, E, F, p.f1);
    f2.init(E, F, E, p.f2);
    head.init((int)w.head_ld, E, V, p.head);
  }
  __syncthreads();
  const float inv_e = 1.0f / E;
  // element e = tid + i DT of the residual stream belongs to this thread
  auto norm = [&]() {
    if (E <= 32 * 4 * NORM_V) {
      // every warp sums the whole vector: two shuffle trees and no block-wide sums
      __syncthreads();
      const int lane = tid & 31;
      float4 t[NORM_V];
      float s = 0.0f, q = 0.0f;
#pragma unroll
      for (int i = 0; i < NORM_V; ++i) {
        const int e = (lane + 32 * i) * 4;
        t[i] = e < E ? *reinterpret_cast<const float4*>(x + e) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        s += (t[i].x + t[i].y) + (t[i].z + t[i].w);
      }
      const float mean = warp_sum(s) * inv_e;
#pragma unroll
      for (int i = 0; i < NORM_V; ++i) {
        const float a = t[i].x - mean, b = t[i].y - mean, c = t[i].z - mean, d = t[i].w - mean;
        if ((lane + 32 * i) * 4 < E) q += (a * a + b * b) + (c * c + d * d);
      }
      const float rstd = rsqrtf(warp_sum(q) * inv_e + w.eps);
#pragma unroll
      for (int i = 0; i < EPT; ++i) {
        const int e = tid + i * DT;
        if (e < E) n[e] = rb((x[e] - mean) * rstd * gamma.at(i) + beta.at(i));
      }
      for (int e = tid + EPT * DT; e < E; e += DT) n[e] = rb((x[e] - mean) * rstd * ldb(gamma.p, e) + ldb(beta.p, e));
      __syncthreads();
      return;
    }
    float s = 0.0f;
    for (int e = tid; e < E; e += DT) s += x[e];
    const float mean = block_sum(s, shf) * inv_e;
    float q = 0.0f;
    for (int e = tid; e < E; e += DT) q += (x[e] - mean) * (x[e] - mean);
    const float rstd = rsqrtf(block_sum(q, shf) * inv_e + w.eps);
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
      const int e = tid + i * DT;
      if (e < E) n[e] = rb((x[e] - mean) * rstd * gamma.at(i) + beta.at(i));
    }
    for (int e = tid + EPT * DT; e < E; e += DT) n[e] = rb((x[e] - mean) * rstd * ldb(gamma.p, e) + ldb(beta.p, e));
    __syncthreads();
  };
  auto add_partials = [&](int ks) {
    float t[EPT][MAX_KS];                    // all loads first
#pragma unroll
    for (int i = 0; i < EPT; ++i)
#pragma unroll
      for (int k = 0; k < MAX_KS; ++k)
        t[i][k] = k < ks && tid + i * DT < E ? p.part[k * E + tid + i * DT] : 0.0f;
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
      const int e = tid + i * DT;
      float s = t[i][0];
#pragma unroll
      for (int k = 1; k < MAX_KS; ++k) s += t[i][k];
      if (e < E) x[e] = rb(s + bias.at(i) + x[e]);
    }
    for (int e = tid + EPT * DT; e < E; e += DT) {
      float s = p.part[e];
      for (int k = 1; k < ks; ++k) s += p.part[k * E + e];
      x[e] = rb(s + ldb(bias.p, e) + x[e]);
    }
  };
  auto whole = [&](int, int) { return n; };
  auto prefetch_layer = [&](int l) {
    const GptLayer& z = w.layer[l];
    prefetch_l2(z.wqkv, 6ll * E * E);
    prefetch_l2(z.wo, 2ll * E * E);
    prefetch_l2(z.w1, 2ll * E * F);
    prefetch_l2(z.w2, 2ll * E * F);
  };
  auto prefetch_head = [&]() { prefetch_l2(w.head, (long long)E * w.head_ld * 2); };
#define GRID_ARRIVE() grid_arrive(p.bar, goal)
#define GRID_WAIT() do { if (!grid_wait(p.bar, goal, p.status, &sh_ok)) return; } while (0)

  int tok = p.first > 0 ? p.ids_out[p.first - 1] : 0;
  for (int i = p.first; i < p.last; ++i) {
    if (i == 0) {
      prefetch_head();
      gamma.fetch(w.lnf_g, E);
      beta.fetch(w.lnf_b, E);
      fetch(head, w.head, slots);
      for (int e = tid; e < E; e += DT) x[e] = __bfloat162float(p.x0[e]);
    } else {
      const int pos = p.prompt + i - 1;
      gamma.fetch(w.layer[0].ln1_g, E);
      beta.fetch(w.layer[0].ln1_b, E);
      fetch(qkv, w.layer[0].wqkv, slots);
      for (int e = tid; e < E; e += DT)
        x[e] = rb(ldb(w.tok, tok * E + e) + ldb(w.pos, pos * E + e));
      const int keys = pos + 1;
      int ns = (keys + 63) / 64;
      if (ns > G / H) ns = G / H > 0 ? G / H : 1;
      const int per = (keys + ns - 1) / ns;
      const int split = D + 2;
      const bool fused = keys <= p.fuse_keys;
      for (int l = 0; l < w.layers; ++l) {
        const GptLayer& y = w.layer[l];
        const bool more = l + 1 < w.layers;
        bf16* rows = p.cache + (long long)l * p.cache_rows * ld;
        // q | k | v of this position, into the cache
        if (l > 0) add_partials(p.f2.ks);
        norm();
        product(qkv, y.wqkv, slots, red, whole,
                [&](int, int c, float v) { rows[(long long)pos * ld + c] = __float2bfloat16(v); });
        GRID_ARRIVE();
        fetch(fused ? out_head : out, y.wo, slots);
        bias.fetch(y.bo, E);
        if (more) prefetch_layer(l + 1); else prefetch_head();
        GRID_WAIT();
        if (fused) {
          // few keys: every task of a head works out the head's attention for itself, which costs
          // less than a barrier
          product(out_head, y.wo, slots, red,
                  [&](int k0, int) {
                    float* o = xs + D;
                    if (D == 64) attend<64>(rows, ld, E, k0 / D, pos, 0, keys, w.scale, red, o);
                    else attend<128>(rows, ld, E, k0 / D, pos, 0, keys, w.scale, red, o);
                    if (tid < D) xs[tid] = rb(__fdividef(o[tid], o[D + 1]));
                    __syncthreads();
                    return xs;
                  },
                  [&](int s, int c, float v) { p.part[s * E + c] = v; });
        } else {
        // attention: a head's keys over ns CTAs
        for (int t = blockIdx.x; t < H * ns; t += G) {
          const int h = t / ns, j0 = (t - h * ns) * per, j1 = j0 + per < keys ? j0 + per : keys;
          float* o = p.attn + (long long)t * split;
          if (D == 64) attend<64>(rows, ld, E, h, pos, j0, j1, w.scale, red, o);
          else attend<128>(rows, ld, E, h, pos, j0, j1, w.scale, red, o);
        }
        GRID_ARRIVE();
        GRID_WAIT();
        // output projection; each task first puts its heads' splits together
        product(out, y.wo, slots, red,
                [&](int k0, int len) {
                  for (int k = tid; k < len; k += DT) {
                    const int h = (k0 + k) / D, d = k0 + k - h * D;
                    const float* a = p.attn + (long long)h * ns * split;
                    float m = a[D], num = a[d], den = a[D + 1];
                    for (int s = 1; s < ns; ++s) {
                      const float* b = a + s * split;
                      const float ms = b[D], m2 = fmaxf(m, ms), f0 = __expf(m - m2), f1 = __expf(ms - m2);
                      num = num * f0 + b[d] * f1;
                      den = den * f0 + b[D + 1] * f1;
                      m = m2;
                    }
                    xs[k] = rb(__fdividef(num, den));
                  }
                  __syncthreads();
                  return xs;
                },
                [&](int s, int c, float v) { p.part[s * E + c] = v; });
        }
        GRID_ARRIVE();
        fetch(f1, y.w1, slots);
        gamma.fetch(y.ln2_g, E);
        beta.fetch(y.ln2_b, E);
        GRID_WAIT();
        add_partials(fused ? p.out_head.ks : p.out.ks);
        norm();
        product(f1, y.w1, slots, red, whole,
                [&](int, int c, float v) {
                  v += ldb(y.b1, c);
                  const float k0 = 0.7978845608f, k0k1 = 0.7978845608f * 0.044715f;
                  float t;
                  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(v * (k0k1 * (v * v) + k0)));
                  p.h[c] = __float2bfloat16(0.5f * v * t + 0.5f * v);
                });
        GRID_ARRIVE();
        fetch(f2, y.w2, slots);
        GRID_WAIT();
        product(f2, y.w2, slots, red,
                [&](int k0, int len) {
                  for (int k = tid * 8; k < len; k += DT * 8) {   // slices start and end at multiples of 8
                    float v[8];
                    VecIO<bf16>::load(p.h + k0 + k, v);
#pragma unroll
                    for (int j = 0; j < 8; ++j) xs[k + j] = v[j];
                  }
                  __syncthreads();
                  return xs;
                },
                [&](int s, int c, float v) { p.part[s * E + c] = v; });
        GRID_ARRIVE();
        const GptLayer& z = w.layer[more ? l + 1 : l];
        if (more) fetch(qkv, z.wqkv, slots); else fetch(head, w.head, slots);
        bias.fetch(y.b2, E);
        gamma.fetch(more ? z.ln1_g : w.lnf_g, E);
        beta.fetch(more ? z.ln1_b : w.lnf_b, E);
        GRID_WAIT();
      }
      add_partials(p.f2.ks);
    }
    norm();
    unsigned kmax = 0;
    product(head, w.head, slots, red, whole,
            [&](int, int c, float v) {
              const bf16 b = __float2bfloat16(v);
              p.logits[c] = b;
              kmax = max(kmax, key_of(__bfloat16_as_ushort(b)));
            });
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    unsigned* shu = reinterpret_cast<unsigned*>(sh);
    if ((tid & 31) == 0) shu[tid >> 5] = kmax;
    __syncthreads();
    if (tid == 0) {
      for (int k = 1; k < WARPS; ++k) kmax = max(kmax, shu[k]);
      p.gmax[blockIdx.x] = kmax;
    }
    GRID_ARRIVE();
    if (i + 1 < p.last) prefetch_layer(0);
    GRID_WAIT();

    // ---- sampling, the same in every CTA
    const unsigned short* lg = reinterpret_cast<const unsigned short*>(p.logits);
    // keys >= k0: how many, and the first MAX_CAND of them with their places
    auto count_from = [&](unsigned k0) {
      if (tid == 0) sh_cnt = 0;
      __syncthreads();
      constexpr int B = 8;                     // loads in flight per thread
      for (int c0 = tid * 8; c0 < V; c0 += B * DT * 8) {
        uint4 q[B];
#pragma unroll
        for (int b = 0; b < B; ++b)
          if (c0 + b * DT * 8 < V) q[b] = *reinterpret_cast<const uint4*>(lg + c0 + b * DT * 8);
#pragma unroll
        for (int b = 0; b < B; ++b) {
          const unsigned u[4] = {q[b].x, q[b].y, q[b].z, q[b].w};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int c = c0 + b * DT * 8 + j;
            const unsigned k = key_of((unsigned short)(u[j / 2] >> (16 * (j & 1))));
            if (c < V && k >= k0) {
              const int at = atomicAdd(&sh_cnt, 1);
              if (at < MAX_CAND) { cand[at] = k; cand_at[at] = c; }
            }
          }
        }
      }
      __syncthreads();
      const int n = sh_cnt;
      __syncthreads();                         // everyone has it before it is reused
      return n;
    };
    // the CTAs' maxima, staged in shared memory
    unsigned* gm = reinterpret_cast<unsigned*>(xs);
    unsigned top = 0;
    for (int c = tid; c < G; c += DT) { gm[c] = p.gmax[c]; top = max(top, gm[c]); }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((tid & 31) == 0) shu[tid >> 5] = top;
    __syncthreads();
    for (int k = 0; k < WARPS; ++k) top = max(top, shu[k]);
    const float mx = p.temperature != 1.0f ? key_value(top) / p.temperature : key_value(top);
    auto weight = [&](unsigned k) {
      const float v = key_value(k);
      return expf((p.temperature != 1.0f ? v / p.temperature : v) - mx);
    };
    unsigned thresh = 0;                       // keys below it are cut off
    int cnt = MAX_CAND + 1;
    if (p.top_k > 0 && p.top_k < V) {
      if (p.top_k <= G) {
        // the k-th largest of the CTAs' maxima: at least k logits reach it
        for (int c = tid; c < G; c += DT) {
          const unsigned mine = gm[c];
          int rank = 0;
          for (int k = 0; k < G; ++k) rank += gm[k] > mine || (gm[k] == mine && k < c);
          if (rank == p.top_k - 1) sh_key = mine;
        }
        __syncthreads();
        cnt = count_from(sh_key);
      }
      if (cnt <= MAX_CAND) {
        for (int c = tid; c < cnt; c += DT) {
          const unsigned mine = cand[c];
          int rank = 0;
          for (int k = 0; k < cnt; ++k) rank += cand[k] > mine || (cand[k] == mine && k < c);
          if (rank == p.top_k - 1) sh_key = mine;
        }
        __syncthreads();
        thresh = sh_key;
      } else {
        // a wide cut: the largest key that still leaves top_k of them
        unsigned lo = 0, hi = top;             // count_from(lo) >= top_k always holds
        while (lo < hi) {
          const unsigned mid = (lo + hi + 1) / 2;
          if (count_from(mid) >= p.top_k) lo = mid; else hi = mid - 1;
        }
        thresh = lo;
      }
    }
    // inverse of the cumulative distribution, in the order of the vocabulary: the candidates that
    // stay, sorted by place, or else all logits, a contiguous run per thread
    float* wt = n;                             // few: weights and places in vocabulary order
    int* at = reinterpret_cast<int*>(wt + DT);
    const bool few = cnt <= DT && 2 * DT <= E + (E > F ? E : F);
    if (few) {
      int rank = 0;
      const bool keep = tid < cnt && cand[tid] >= thresh;
      if (tid < DT) { wt[tid] = 0.0f; at[tid] = V - 1; }
      __syncthreads();
      if (keep) {
        const int mine = cand_at[tid];
        for (int k = 0; k < cnt; ++k) rank += cand[k] >= thresh && cand_at[k] < mine;
        wt[rank] = weight(cand[tid]);
        at[rank] = mine;
      }
      __syncthreads();
    }
    const int per = few ? 1 : ((V + DT - 1) / DT + 7) & ~7;
    const int c0 = tid * per, c1 = few ? c0 + 1 : (c0 + per < V ? c0 + per : V);
    float mine = 0.0f;
    if (few) {
      mine = wt[tid];
    } else {
      for (int c = c0; c < c1; c += 8) {
        const uint4 q = *reinterpret_cast<const uint4*>(lg + c);
        const unsigned u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const unsigned k = key_of((unsigned short)(u[j / 2] >> (16 * (j & 1))));
          if (c + j < c1 && k >= thresh) mine += weight(k);
        }
      }
    }
    float incl = mine;                         // inclusive scan over the block
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    __syncthreads();                           // shu has been read
    if (lane == 31) shf[warp] = incl;
    if (tid == 0) { sh_cnt = V - 1; sh_last = -1; }
    __syncthreads();
    float before = 0.0f, total = 0.0f;
    for (int k = 0; k < WARPS; ++k) {
      if (k < warp) before += shf[k];
      total += shf[k];
    }
    // only threads with weight may draw; the last of them stands in where rounding (a scan's prefixes
    // depend on the place) leaves none that reaches the goal
    const int last = __reduce_max_sync(0xffffffffu, mine > 0.0f ? tid : -1);
    if (lane == 0) atomicMax(&sh_last, last);
    __syncthreads();
    const float goal_w = p.rnd[i] * total;
    if (mine > 0.0f && (before + incl >= goal_w || tid == sh_last)) {   // the first such thread: min over all
      if (few) {
        atomicMin(&sh_cnt, at[tid]);
      } else {
        float run = before + incl - mine;
        int pick = V - 1;                      // a column that the cut has left
        for (int c = c0; c < c1; ++c) {
          const unsigned k = key_of(lg[c]);
          if (k < thresh) continue;
          pick = c;
          run += weight(k);
          if (run >= goal_w) break;
        }
        atomicMin(&sh_cnt, pick);
      }
    }
    __syncthreads();
    tok = sh_cnt;
    if (blockIdx.x == 0 && tid == 0) p.ids_out[i] = tok;
    __syncthreads();
  }
#undef GRID_ARRIVE
#undef GRID_WAIT
}

Split choose_split(int N, int K, int G, int max_ks) {
  const int units = (N + 7) / 8;
  Split best{16, (units + 15) / 16, 1};
  double best_cost = 1e30;
  for (int nu = 2; nu <= 16; nu *= 2)          // 16-byte columns would waste half of each sector
    for (int ks = 1; ks <= max_ks && K / ks >= 64; ++ks) {
      const int groups = (units + nu - 1) / nu;
      const int rounds = (groups * ks + G - 1) / G;
      // 16-byte loads of the busiest CTA, a pass's reduction, the consumers' partial sums
      const double cost = rounds * ((double)nu * K / ks + 100.0) + 40.0 * (ks - 1);
      if (cost < best_cost) { best_cost = cost; best = {nu, groups, ks}; }
    }
  return best;
}

int64_t up(int64_t v) { return (v + 255) & ~int64_t(255); }

// A dense layer's product as the layer classes issue it: [M, K] x [K, N] (+ bias, activation, residual).
GemmArgs dense_args(const void* a, int64_t lda, const void* W, int64_t ldw, const void* bias, int act,
                    const void* residual, void* out, int64_t ldo, int64_t M, int N, int K) {
  GemmArgs g;
  g.M = (int)M; g.N = N; g.K = K;
  g.A = a; g.lda = lda; g.B = W; g.ldb = ldw; g.C = out; g.ldc = ldo;
  g.bias = bias; g.act = act;
  g.residual = residual; g.ldr = ldo;
  return g;
}

// Scratch that the products of a forward over T tokens use (split-K, packed weights), so that they take
// the same route as in the layers.  The activations' buffers are aligned; a layer is looked at again
// where the addresses of its matrices allow less than the first one's.
size_t dense_workspace(const GptWeights& w, int64_t T) {
  const int E = w.embed, F = w.ffn;
  const auto odd = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 != 0; };
  size_t need = gemm_workspace_bytes(dense_args(nullptr, E, w.head, w.head_ld, nullptr, 0, nullptr, nullptr, w.head_ld, T, w.vocab, E));
  const auto at_least = [&](const GemmArgs& g) { need = std::max(need, gemm_workspace_bytes(g)); };
  for (int l = 0; l < w.layers; ++l) {
    const GptLayer &y = w.layer[l], &z = w.layer[0];
    const void* x = w.tok;   // stands for a residual: one is added
    if (l == 0 || odd(y.wqkv) != odd(z.wqkv)) at_least(dense_args(nullptr, E, y.wqkv, 3 * E, nullptr, 0, nullptr, nullptr, 3 * E, T, 3 * E, E));
    if (l == 0 || odd(y.wo) != odd(z.wo)) at_least(dense_args(nullptr, E, y.wo, E, y.bo, 0, x, nullptr, E, T, E, E));
    if (l == 0 || odd(y.w1) != odd(z.w1)) at_least(dense_args(nullptr, E, y.w1, F, y.b1, GEMM_ACT_GELU, nullptr, nullptr, F, T, F, E));
    if (l == 0 || odd(y.w2) != odd(z.w2)) at_least(dense_args(nullptr, F, y.w2, E, y.b2, 0, x, nullptr, E, T, E, F));
  }
  return need;
}

struct FwdBuffers { char *x, *n, *qkv, *att, *h; float* stats; char* gemm; size_t gemm_bytes; };
FwdBuffers carve(const GptWeights& w, int64_t T, void* ws) {
  char* p = (char*)ws;
  FwdBuffers b;
  b.x = p; p += up(T * w.embed * 2);
  b.n = p; p += up(T * w.embed * 2);
  b.qkv = p; p += up(T * w.embed * 6);
  b.att = p; p += up(T * w.embed * 2);
  b.h = p; p += up(T * w.ffn * 2);
  b.stats = (float*)p; p += up(T * 8);
  b.gemm = p;
  b.gemm_bytes = dense_workspace(w, T);
  return b;
}

cudaError_t dense(const FwdBuffers& b, GemmArgs g, cudaStream_t s) {
  g.workspace = b.gemm_bytes ? b.gemm : nullptr;
  g.workspace_bytes = b.gemm_bytes;
  return gemm_bf16(g, s);
}

}  // namespace

size_t gpt_forward_workspace(const GptWeights& w, int64_t T) {
  return (size_t)(up(T * w.embed * 2) * 3 + up(T * w.embed * 6) + up(T * w.ffn * 2) + up(T * 8)) + dense_workspace(w, T);
}

cudaError_t gpt_forward(const GptWeights& w, const void* ids, int id_kind, int64_t batch, int64_t seq,
                        void* workspace, void* cache, int64_t cache_rows, int* err, void** x_out,
                        cudaStream_t s) {
  const int64_t T = batch * seq;
  const int E = w.embed, F = w.ffn;
  const FwdBuffers b = carve(w, T, workspace);
  float *mean = b.stats, *rstd = b.stats + T;
  cudaError_t e = embedding_forward(DT_BF16, w.tok, ids, id_kind, w.pos, seq, b.x, T, E, w.vocab, err, s);
  for (int l = 0; l < w.layers && e == cudaSuccess; ++l) {
    const GptLayer& y = w.layer[l];
    char* qkv = cache ? (char*)cache + (int64_t)l * cache_rows * E * 6 : b.qkv;
    e = layernorm_forward(DT_BF16, b.x, y.ln1_g, y.ln1_b, DT_BF16, w.eps, b.n, mean, rstd, T, E, s);
    if (e == cudaSuccess) e = dense(b, dense_args(b.n, E, y.wqkv, 3 * E, nullptr, 0, nullptr, qkv, 3 * E, T, 3 * E, E), s);
    AttnArgs a;
    a.B = (int)batch; a.H = w.heads; a.S = (int)seq; a.D = w.head_dim;
    a.q = qkv; a.k = qkv + 2 * E; a.v = qkv + 4 * E; a.o = b.att;
    a.q_ss = a.k_ss = a.v_ss = 3 * E; a.q_sb = a.k_sb = a.v_sb = seq * 3 * E;
    a.q_sh = a.k_sh = a.v_sh = a.o_sh = w.head_dim;
    a.o_ss = E; a.o_sb = seq * E;
    a.causal = 1; a.scale = w.scale;
    if (e == cudaSuccess) e = flash_attention_forward(a, s);
    if (e == cudaSuccess) e = dense(b, dense_args(b.att, E, y.wo, E, y.bo, 0, b.x, b.x, E, T, E, E), s);
    if (e == cudaSuccess) e = layernorm_forward(DT_BF16, b.x, y.ln2_g, y.ln2_b, DT_BF16, w.eps, b.n, mean, rstd, T, E, s);
    if (e == cudaSuccess) e = dense(b, dense_args(b.n, E, y.w1, F, y.b1, GEMM_ACT_GELU, nullptr, b.h, F, T, F, E), s);
    if (e == cudaSuccess) e = dense(b, dense_args(b.h, F, y.w2, E, y.b2, 0, b.x, b.x, E, T, E, F), s);
  }
  *x_out = b.x;
  return e;
}

cudaError_t gpt_logits(const GptWeights& w, const void* x, int64_t n, void* workspace, void* logits,
                       cudaStream_t s) {
  const FwdBuffers b = carve(w, n, workspace);
  cudaError_t e = layernorm_forward(DT_BF16, x, w.lnf_g, w.lnf_b, DT_BF16, w.eps, b.n, b.stats, b.stats + n, n, w.embed, s);
  if (e == cudaSuccess)
    e = dense(b, dense_args(b.n, w.embed, w.head, w.head_ld, nullptr, 0, nullptr, logits, w.head_ld, n, w.vocab, w.embed), s);
  return e;
}

bool gpt_decode_fits(int64_t embed, int64_t ffn, int64_t head_dim, int64_t vocab) {
  const int64_t wide = embed > ffn ? embed : ffn;
  if ((head_dim != 64 && head_dim != 128) || wide > (1 << 20) || vocab * embed >= (1ll << 31)) return false;
  // a head's sums and its context vector share the activations' buffer
  return decode_smem_floats((int)embed, (int)ffn) * 4 <= DECODE_SMEM_MAX && 2 * head_dim + 2 <= wide;
}

size_t gpt_decode_scratch(const GptWeights& w) {
  const int G = sm_count();
  return (size_t)(256 + up((int64_t)MAX_KS * w.embed * 4) +
                  up((int64_t)(G + w.heads) * (w.head_dim + 2) * 4) + up(w.ffn * 2) +
                  up((w.vocab + 8 * DT) * 2) + up(G * 4));
}

cudaError_t gpt_decode(const GptWeights& w, const void* x, void* cache, int64_t cache_rows, int prompt,
                       int first, int last, float temperature, int top_k, const float* rnd, int* ids_out,
                       void* scratch, int* status, cudaStream_t s) {
  if (!gpt_decode_fits(w.embed, w.ffn, w.head_dim, w.vocab)) return cudaErrorInvalidValue;
  const int smem = decode_smem_floats(w.embed, w.ffn) * 4;
  static const cudaError_t attr = cudaFuncSetAttribute(gpt_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DECODE_SMEM_MAX);
  if (attr != cudaSuccess) return attr;
  int G = sm_count();
  DecodeParams p;
  p.w = w;
  p.x0 = (const bf16*)x;
  p.cache = (bf16*)cache; p.cache_rows = cache_rows;
  p.prompt = prompt; p.first = first; p.last = last;
  p.temperature = temperature; p.top_k = top_k;
  p.rnd = rnd; p.ids_out = ids_out;
  p.qkv = choose_split(3 * w.embed, w.embed, G, 1);
  p.out = choose_split(w.embed, w.embed, G, SPLIT_KS);
  p.f1 = choose_split(w.ffn, w.embed, G, 1);
  p.f2 = choose_split(w.embed, w.ffn, G, SPLIT_KS);
  p.head = choose_split(w.vocab, w.embed, G, 1);
  // a head per K slice where that fills the grid in one round; 256 keys are 64 KB of a head's rows
  p.out_head = {0, 0, 0};
  p.fuse_keys = 0;
  if (w.heads <= MAX_KS && w.heads * 2 <= G) {
    const int units = w.embed / 8, room = G / w.heads;
    int nu = 2;
    while (nu < 16 && (units + nu - 1) / nu > room) nu *= 2;
    if ((units + nu - 1) / nu <= room) {
      p.out_head = {nu, (units + nu - 1) / nu, w.heads};
      p.fuse_keys = 256 * 64 / w.head_dim;
    }
  }
  char* q = (char*)scratch;
  p.bar = (unsigned*)q; q += 256;
  p.part = (float*)q; q += up((int64_t)MAX_KS * w.embed * 4);
  p.attn = (float*)q; q += up((int64_t)(G + w.heads) * (w.head_dim + 2) * 4);
  p.h = (bf16*)q; q += up(w.ffn * 2);
  p.logits = (bf16*)q; q += up((w.vocab + 8 * DT) * 2);
  p.gmax = (unsigned*)q;
  p.status = status;
  cudaError_t e = cudaMemsetAsync(p.bar, 0, 256, s);
  if (e != cudaSuccess) return e;
  void* args[] = {&p};
  e = cudaLaunchCooperativeKernel((const void*)gpt_decode_kernel, dim3(G), dim3(DT), args, (size_t)smem, s);
  g_late_chain = 0; g_late_side = 0; ++g_pdl_seq;
  LT_COUNT_LAUNCH();
  return e;
}

}  // namespace lt
