// Sampling head over the vocabulary row(s) of logits -- the reference's ms::arch::encode_argmax (greedy, or Gumbel-max =
// exact temperature sampling), encode_topk (k <= 64, with the full-row log-sum-exp for a CPU top-p sampler) and
// encode_log_softmax (src/kernels/arch.hpp:109-122, arch_sample.metal:15-213), and the CPU sampler sample_top_p
// (arch.mm:322-342).  Off the per-token critical path except argmax; written for determinism: every reduction has a
// fixed tree, ties go to the lower index, repeated calls give identical bits.
//
// Each kernel is one launch: grid (groups, rows); a group reduces a contiguous chunk of its row, stores a partial, and
// the group that takes the row's last ticket merges the partials (then resets the ticket for the next call).
#include <algorithm>
#include <cmath>
#include <cooperative_groups.h>
#include "msb_common.cuh"
#include "sample_route.h"

namespace msb {

namespace {
constexpr int kSampT = 1024;          // threads per group
constexpr int kSampK = 64;            // largest k of the top-k
constexpr int kSampMaxGroups = 64;    // groups per row (top-k: 4 logits per thread, chunk <= 4096)
constexpr int kPartWords = kSampMaxGroups * kSampK;   // words per row of each partial array

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x;
}
// Gumbel(0,1) noise of element i under (s0, s1): two rounds of the 32-bit mixer, 24 bits -> u in (0,1), -log(-log u)
// (arch_sample.metal:15-26)
__device__ __forceinline__ float gumbel(uint32_t i, uint32_t s0, uint32_t s1) {
  uint32_t x = hash32(i * 0x9E3779B9u ^ s0);
  x = hash32(x ^ (s1 * 0x85EBCA6Bu + 0x632BE5ABu));
  const float u = ((float)(x >> 8) + 0.5f) * (1.0f / 16777216.0f);
  return -logf(-logf(u));
}
__device__ __forceinline__ bool better(float v, uint32_t i, float w, uint32_t j) { return v > w || (v == w && i < j); }

struct BlockRed {          // shared scratch of the block-wide reductions
  float v[32];
  uint32_t i[32];
  float m[32], s[32];
  int last;
};

// block-wide (value, index) argmax, ties -> lower index; every thread gets the result
__device__ __forceinline__ void block_argmax(float& v, uint32_t& i, BlockRed& r, int tid) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const uint32_t oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (better(ov, oi, v, i)) { v = ov; i = oi; }
  }
  if ((tid & 31) == 0) { r.v[tid >> 5] = v; r.i[tid >> 5] = i; }
  __syncthreads();
  v = r.v[tid & 31]; i = r.i[tid & 31];          // kSampT / 32 = 32 warps: one partial per lane
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const uint32_t oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (better(ov, oi, v, i)) { v = ov; i = oi; }
  }
  __syncthreads();
}
// (max, sum of exp(x - max)) pairs of a warp: the maximum first, then every lane's sum moved to it once
__device__ __forceinline__ void warp_lse(float& m, float& s) {
  const float M = warp_max(m);
  s = warp_sum(s * expf(m - M));
  m = M;
}
// the same over a block of kSampT threads; every thread ends with the block's pair.  m must be finite (-3e38 for none).
__device__ __forceinline__ void block_lse(float& m, float& s, BlockRed& r, int tid) {
  warp_lse(m, s);
  if ((tid & 31) == 0) { r.m[tid >> 5] = m; r.s[tid >> 5] = s; }
  __syncthreads();
  m = r.m[tid & 31]; s = r.s[tid & 31];
  warp_lse(m, s);
}
// the row's last group to arrive (its partial is stored and fenced before the ticket)
__device__ __forceinline__ bool last_group(unsigned* ticket, int groups, BlockRed& r, int tid) {
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    r.last = atomicAdd(ticket, 1u) == (unsigned)groups - 1;
  }
  __syncthreads();
  if (r.last) __threadfence();
  return r.last != 0;
}

struct SampleParams {
  const float* logits;
  int rows, V, groups, chunk, k;
  float inv_temp;
  uint32_t seed_lo, seed_hi;
  int use_gumbel;
  float* part_v;        // argmax: [rows][groups] (value); top-k: [rows][kPartWords] granule maxima (order keys)
  uint32_t* part_i;     // argmax: [rows][groups]
  float2* part_ms;      // top-k: [rows][groups] (max, sum)
  unsigned* ticket;     // [rows]
  int* out_idx;         // argmax [rows]; top-k [rows][64]
  float* out_val;       // argmax [rows] (may be null); top-k [rows][64]
  float* out_lse;       // top-k [rows]
};

__global__ void __launch_bounds__(kSampT) argmax_rows_kernel(const SampleParams p) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ BlockRed r;
  const int tid = threadIdx.x, g = blockIdx.x, row = blockIdx.y;
  const float* l = p.logits + (size_t)row * p.V;
  const int b = g * p.chunk, e = min(p.V, b + p.chunk);
  const uint32_t s0 = p.seed_lo + (uint32_t)row * 0x2545F491u;
  float bv = -INFINITY;
  uint32_t bi = 0xffffffffu;
  for (int i = b + tid; i < e; i += kSampT) {
    const float v = p.use_gumbel ? l[i] * p.inv_temp + gumbel((uint32_t)i, s0, p.seed_hi) : l[i];
    if (better(v, (uint32_t)i, bv, bi)) { bv = v; bi = (uint32_t)i; }
  }
  block_argmax(bv, bi, r, tid);
  if (tid == 0) { p.part_v[row * p.groups + g] = bv; p.part_i[row * p.groups + g] = bi; }
  if (!last_group(p.ticket + row, p.groups, r, tid)) return;
  bv = -INFINITY; bi = 0xffffffffu;
  for (int k = tid; k < p.groups; k += kSampT) {
    const float v = reinterpret_cast<volatile float*>(p.part_v)[row * p.groups + k];
    const uint32_t i = reinterpret_cast<volatile uint32_t*>(p.part_i)[row * p.groups + k];
    if (better(v, i, bv, bi)) { bv = v; bi = i; }
  }
  block_argmax(bv, bi, r, tid);
  if (tid == 0) {
    p.out_idx[row] = (int)bi;
    if (p.out_val) p.out_val[row] = bv;
    p.ticket[row] = 0;
  }
}

// ---- top-k.  A warp reduces a GRANULE of 128 consecutive logits to its maximum; the row's last group then works on the
// granule maxima (at most 2048) alone: with T = the k-th largest of them at least k logits reach T, and every logit above
// T lies in one of the fewer than k granules whose maximum exceeds T.  So the exact top k is among kTkGranules granules
// (those that reach T; with more ties at T than that, the lowest-numbered ones, which hold the lowest indices): 16 logits
// per thread, re-read from L2.  Bound by a chain of latencies (read, ticket, maxima, granules), not by bytes: 64 rounds of
// a block-wide argmax, twice, cost 124 us for 64 of 129280; this takes 16, and 6.7
// for one logit, for which alone such a row still comes here (topk_by_cluster).
// Keys: order-preserving unsigned image of the float (-0 counted as +0, NaN = 0 = never taken).
constexpr int kTkGranule = 128;
constexpr int kTkGranules = 128;                     // granules the finish can hold
constexpr int kTkMaxPerThread = kSampMaxGroups * 4 * kSampT / kTkGranule / kSampT;   // granule maxima per thread: 2
constexpr int kTkList = 256;                         // candidates ranked by counting without a further narrowing
static_assert(kTkGranules * kTkGranule == 16 * kSampT, "16 logits per thread in the finish");

__device__ __forceinline__ uint32_t tk_key(float f) {
  if (f != f) return 0u;
  const uint32_t u = __float_as_uint(f + 0.0f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// sum over the block of one small count per thread; `sh` is one of two alternating 32-word arrays, so that one barrier
// per call is enough
__device__ __forceinline__ unsigned block_count(unsigned c, unsigned* sh, int tid) {
  const unsigned w = __reduce_add_sync(0xffffffffu, c);
  if ((tid & 31) == 0) sh[tid >> 5] = w;
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, sh[tid & 31]);
}
// The largest T with at least `want` of the block's values (N per thread) >= T; stops early at any T that between `want`
// and `enough` values reach (count_out = how many).  T = 0 when fewer than `want` values are non-zero.
template <int N>
__device__ __forceinline__ uint32_t kth_value(const uint32_t (&v)[N], unsigned want, unsigned enough, unsigned (*sh)[32], int tid,
                                              unsigned& count_out) {
  uint32_t T = 0;
  unsigned have = 0xffffffffu;
  for (int b = 31; b >= 0; b--) {
    const uint32_t cand = T | (1u << b);
    unsigned c = 0;
#pragma unroll
    for (int q = 0; q < N; q++) c += v[q] >= cand;
    c = block_count(c, sh[b & 1], tid);
    if (c >= want) {
      T = cand; have = c;
      if (c <= enough) break;
    }
  }
  __syncthreads();                                   // the count arrays are free again
  count_out = have;
  return T;
}

__global__ void __launch_bounds__(kSampT) topk_lse_kernel(const SampleParams p) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ BlockRed r;
  __shared__ unsigned cnt[2][32];
  __shared__ int gran[kTkGranules];
  __shared__ uint32_t list_k[kTkList], list_i[kTkList];
  __shared__ unsigned n_gran, n_list;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = blockIdx.x, row = blockIdx.y;
  const float* l = p.logits + (size_t)row * p.V;
  uint32_t* gmax = reinterpret_cast<uint32_t*>(p.part_v) + (size_t)row * kPartWords;
  const int ngran = (p.V + kTkGranule - 1) / kTkGranule;
  {
    const int i0 = (g * 32 + warp) * kTkGranule + lane;
    float v[4], m = -3.0e38f, s = 0.f;
    uint32_t top = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] = i0 + 32 * q < p.V ? l[i0 + 32 * q] : -INFINITY;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (i0 + 32 * q < p.V) top = max(top, tk_key(v[q]));
      v[q] *= p.inv_temp;
      m = fmaxf(m, v[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) s += i0 + 32 * q < p.V ? expf(v[q] - m) : 0.f;
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0 && g * 32 + warp < ngran) gmax[g * 32 + warp] = top;
    block_lse(m, s, r, tid);
    if (tid == 0) p.part_ms[row * p.groups + g] = make_float2(m, s);
  }
  if (!last_group(p.ticket + row, p.groups, r, tid)) return;
  // ---- the finish: one block per row
  uint32_t km[kTkMaxPerThread];
#pragma unroll
  for (int q = 0; q < kTkMaxPerThread; q++) km[q] = tid + q * kSampT < ngran ? __ldcg(gmax + tid + q * kSampT) : 0u;
  if (warp == 31) {                                  // log-sum-exp of the row from the groups' pairs (at most 64)
    float m = -3.0e38f, s = 0.f, m2 = -3.0e38f, s2 = 0.f;
    const float2* ms = p.part_ms + (size_t)row * p.groups;
    if (lane < p.groups) { const float2 t = __ldcg(ms + lane); m = t.x; s = t.y; }
    if (lane + 32 < p.groups) { const float2 t = __ldcg(ms + lane + 32); m2 = t.x; s2 = t.y; }
    const float M = fmaxf(m, m2);
    s = s * expf(m - M) + s2 * expf(m2 - M);
    m = M;
    warp_lse(m, s);
    if (lane == 0) p.out_lse[row] = m + logf(s);
  }
  if (tid == 0) { n_gran = 0; n_list = 0; p.ticket[row] = 0; }
  // T: the largest maximum when one logit is wanted; 1 (every granule) when all granules fit; else a lower bound of the k-th
  // maximum that few more than k reach, so that the logits that reach it are a short list as well.  (With "as many as fit"
  // for all three, one logit of 32000 took 16.7 us, ten of 1000 25.)
  unsigned reach = 0;
  uint32_t T = 1u;
  if (p.k == 1) {
    uint32_t top = 0;
#pragma unroll
    for (int q = 0; q < kTkMaxPerThread; q++) top = max(top, km[q]);
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) cnt[1][warp] = top;
    __syncthreads();
    T = max(1u, __reduce_max_sync(0xffffffffu, cnt[1][lane]));
    unsigned c = 0;
#pragma unroll
    for (int q = 0; q < kTkMaxPerThread; q++) c += km[q] >= T;
    reach = block_count(c, cnt[0], tid);
    __syncthreads();
  } else if (ngran > kTkGranules) {
    T = max(1u, kth_value<kTkMaxPerThread>(km, (unsigned)p.k, max(32u, 2u * (unsigned)p.k), cnt, tid, reach));
  } else {
    __syncthreads();                                 // n_gran is 0
  }
  if (reach <= kTkGranules || T == 1u) {             // everything that reaches T fits (T == 1: all of them, or fewer than k)
#pragma unroll
    for (int q = 0; q < kTkMaxPerThread; q++)
      if (km[q] >= T) { const unsigned at = atomicAdd(&n_gran, 1u); if (at < kTkGranules) gran[at] = tid + q * kSampT; }
  } else {                                           // T is exact and many granules tie at it: those above, then the first ones
#pragma unroll
    for (int q = 0; q < kTkMaxPerThread; q++)
      if (km[q] > T) gran[atomicAdd(&n_gran, 1u)] = tid + q * kSampT;      // fewer than k of them
    __syncthreads();
    unsigned base = n_gran;
#pragma unroll
    for (int q = 0; q < kTkMaxPerThread; q++) {
      const unsigned m = __ballot_sync(0xffffffffu, km[q] == T);
      if (lane == 0) cnt[0][warp] = __popc(m);
      __syncthreads();
      unsigned before = lane < warp ? cnt[0][lane] : 0u, all = cnt[0][lane];
      before = __reduce_add_sync(0xffffffffu, before);
      all = __reduce_add_sync(0xffffffffu, all);
      const unsigned at = base + before + __popc(m & ((1u << lane) - 1u));
      if (km[q] == T && at < kTkGranules) gran[at] = tid + q * kSampT;
      base += all;
      __syncthreads();
    }
    if (tid == 0) n_gran = min(base, (unsigned)kTkGranules);
  }
  __syncthreads();
  const int ng = (int)min(n_gran, (unsigned)kTkGranules);
  uint32_t key[16], idx[16];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int gi = warp + 32 * q, at = gi < ng ? gran[gi] * kTkGranule + lane : p.V;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = at + 32 * j;
      idx[4 * q + j] = (uint32_t)i;
      key[4 * q + j] = i < p.V ? tk_key(l[i]) : 0u;
    }
  }
  // elements that reach T: usually little more than k.  Otherwise the exact k-th key, and at ties the index limit.
  uint32_t Tk = T, Ti = 0xffffffffu;
  unsigned c = 0;
#pragma unroll
  for (int q = 0; q < 16; q++) c += key[q] >= Tk;
  c = block_count(c, cnt[0], tid);
  __syncthreads();
  if (c > kTkList) {
    unsigned have;
    Tk = max(1u, kth_value<16>(key, (unsigned)p.k, kTkList, cnt, tid, have));
    if (have > kTkList) {                            // ties at the exact k-th key: the lowest indices among them
      unsigned above = 0;
#pragma unroll
      for (int q = 0; q < 16; q++) above += key[q] > Tk;
      above = block_count(above, cnt[0], tid);
      __syncthreads();
      uint32_t inv[16];                              // ~index of the tied ones: the k - above largest
#pragma unroll
      for (int q = 0; q < 16; q++) inv[q] = key[q] == Tk ? ~idx[q] : 0u;
      Ti = ~kth_value<16>(inv, (unsigned)p.k - above, kTkList / 2, cnt, tid, have);
    }
  }
#pragma unroll
  for (int q = 0; q < 16; q++)
    if (key[q] > Tk || (key[q] == Tk && idx[q] <= Ti)) {
      const unsigned at = atomicAdd(&n_list, 1u);
      if (at < kTkList) { list_k[at] = key[q]; list_i[at] = idx[q]; }
    }
  __syncthreads();
  const int nl = (int)min(n_list, (unsigned)kTkList);
  if (tid < nl) {
    const uint32_t k0 = list_k[tid], i0 = list_i[tid];
    int rank = 0;
    for (int j = 0; j < nl; j++) rank += list_k[j] > k0 || (list_k[j] == k0 && list_i[j] < i0);
    if (rank < p.k) {
      p.out_val[(size_t)row * kSampK + rank] = l[i0];
      p.out_idx[(size_t)row * kSampK + rank] = (int)i0;
    }
  }
  if (tid >= nl && tid < p.k) {                      // fewer than k numbers in the row
    p.out_val[(size_t)row * kSampK + tid] = -INFINITY;
    p.out_idx[(size_t)row * kSampK + tid] = -1;
  }
}

// ---- the same by one cluster of 8 blocks per row (topk_by_cluster): every logit stays in a register (R per thread), so nothing is
// read again and no ticket is taken.  A granule is what a warp holds in four registers per lane; all granule maxima go to every
// block, each finds the same threshold T among them (16 candidates at a time, one per warp), and the logits that reach T -- at
// least k, usually a few more than the 2 k granules that T lets through -- are stored into the first block's list and ranked
// there.  More than kTkList of them (ties, rows of few numbers): the exact k-th key, then the index limit among its ties, by a
// radix selection over the cluster.
// Bound by its chain (read, two cluster barriers, T, ranking) and from 16 values per thread on by the exponentials: 64 of 129280
// take 9.7 us in a row of launches (15.7 by the groups), of 65536 7.9; blocks of 512 threads because 1024 of 64 registers cannot hold the
// values.
constexpr int kTkBlocks = 8, kTkThreads = 512, kTkWarps = kTkThreads / 32, kTkMaxRegs = 40, kTkMaxGran = kTkBlocks * kTkWarps * (kTkMaxRegs / 4);
struct TkCluster {
  alignas(16) uint32_t gmax[kTkMaxGran];         // granule maxima of the whole row
  float2 ms[kTkBlocks * kTkWarps];               // first block: the warps' (max, sum)
  uint2 cand[kTkBlocks][kTkList];               // first block: (value, index) per block
  unsigned n[kTkBlocks];                        // the blocks' numbers of candidates
  unsigned cnt[32], n_own, hist[256], digit, above;
  uint32_t list_k[kTkList], list_i[kTkList], list_v[kTkList];
};
// The digit of the `want`-th largest element (elements counted in s.hist by every block), and how many elements have a larger one.
__device__ __noinline__ void tkc_digit(TkCluster& s, unsigned want, int tid) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  cl.sync();
  unsigned v = 0;
  if (tid < 256)
    for (int b = 0; b < kTkBlocks; b++) v += cl.map_shared_rank(s.hist, b)[255 - tid];
  const int lane = tid & 31, warp = tid >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s.cnt[warp] = x;
  __syncthreads();
  for (int w = 0; w < warp && w < 8; w++) x += s.cnt[w];
  if (tid < 256 && x - v < want && x >= want) { s.digit = 255 - tid; s.above = x - v; }
  cl.sync();                                     // every block has read the histograms
  if (tid < 256) s.hist[tid] = 0;
  __syncthreads();
}
template <int R>
__global__ void __cluster_dims__(kTkBlocks, 1, 1) __launch_bounds__(kTkThreads, 1) topk_lse_cluster_kernel(const SampleParams p) {
  static_assert(R % 4 == 0 && R <= kTkMaxRegs, "granules");
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  pdl_launch_dependents();
  pdl_wait();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // "this block runs": waited for before the first remote store
  __shared__ TkCluster s;
  constexpr int NG = R / 4, G = kTkBlocks * kTkWarps * NG;       // granules of a warp, of the row
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x % kTkBlocks, row = blockIdx.x / kTkBlocks;
  const float* l = p.logits + (size_t)row * p.V;
  const int per = (p.V + kTkBlocks - 1) / kTkBlocks, b0 = min(p.V, rank * per) + tid, b1 = min(p.V, (rank + 1) * per);
  float v[R];
#pragma unroll
  for (int q = 0; q < R; q++)      // (volatile: all requested before the first is used; short of registers, the compiler took one after the other)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\tmov.f32 %0, 0fFF800000;\n\t@p ld.global.f32 %0, [%1];\n\t}"
                 : "=f"(v[q]) : "l"(l + b0 + q * kTkThreads), "r"(b0 + q * kTkThreads), "r"(b1));
  // the key of register q, made anew each time: kept beside the values they would spill
  auto key_of = [&](int q) {
    asm volatile("" : "+f"(v[q]));
    return b0 + q * kTkThreads < b1 ? tk_key(v[q]) : 0u;
  };
  // (beyond the row: -inf.  A granule without a number then counts as one -inf, which lets nothing more through: T is at its lowest
  // there, and every number reaches it.)
  uint32_t top[NG];
  float best = -INFINITY, sum = 0.f;
#pragma unroll
  for (int g = 0; g < NG; g++) {
    const float t = fmaxf(fmaxf(v[4 * g], v[4 * g + 1]), fmaxf(v[4 * g + 2], v[4 * g + 3]));
    best = fmaxf(best, t);
    top[g] = __reduce_max_sync(0xffffffffu, tk_key(t));
  }
  float m = fmaxf(-3.0e38f, best * p.inv_temp);             // rounding keeps the order
#pragma unroll
  for (int q = 0; q < R; q++) sum += b0 + q * kTkThreads < b1 ? expf(v[q] * p.inv_temp - m) : 0.f;
  if (tid == 0) s.n_own = 0;
  if (tid < 256) s.hist[tid] = 0;
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (lane < kTkBlocks) {
    uint32_t* dst = cl.map_shared_rank(s.gmax, lane) + (rank * kTkWarps + warp) * NG;
#pragma unroll
    for (int g = 0; g < NG; g++) dst[g] = top[g];
  }
  warp_lse(m, sum);
  if (lane == 0) *cl.map_shared_rank(&s.ms[rank * kTkWarps + warp], 0) = make_float2(m, sum);
  cl.sync();
  // ---- T: the k-th largest maximum or a bound below it that at most topk_enough(k) reach; every warp counts one candidate
  const unsigned k = (unsigned)p.k, enough = topk_enough(k);
  uint32_t lo = 0, hi;                           // at least k maxima reach lo (or lo is 0), fewer reach hi
  {
    const uint4* gm = reinterpret_cast<const uint4*>(s.gmax) + lane;
    uint32_t mx = 0, mn = 0xffffffffu;
    unsigned nz = 0;
#pragma unroll
    for (int i = 0; i < G / 128; i++) {
      const uint4 t = gm[32 * i];
      mx = max(max(mx, max(t.x, t.y)), max(t.z, t.w));
      mn = min(min(mn, min(t.x - 1u, t.y - 1u)), min(t.z - 1u, t.w - 1u));           // of those that are not 0
      nz += (t.x != 0) + (t.y != 0) + (t.z != 0) + (t.w != 0);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    mn = __reduce_min_sync(0xffffffffu, mn) + 1u;
    lo = __reduce_add_sync(0xffffffffu, nz) >= k ? mn : 0u;
    hi = mx + 1u;                                // (no key is 0xffffffff: that would be a NaN's)
    while (hi - lo > 1u) {
      const uint32_t step = max(1u, (hi - lo) / (kTkWarps + 1u)), mine = lo + step * (uint32_t)(warp + 1);
      unsigned c = 0;
#pragma unroll
      for (int i = 0; i < G / 128; i++) {
        const uint4 t = gm[32 * i];
        c += (t.x >= mine) + (t.y >= mine) + (t.z >= mine) + (t.w >= mine);
      }
      c = mine < hi ? __reduce_add_sync(0xffffffffu, c) : 0u;
      if (lane == 0) s.cnt[warp] = c;
      __syncthreads();
      const unsigned all = lane < kTkWarps ? s.cnt[lane] : 0u, ok = __ballot_sync(0xffffffffu, all >= k);      // candidates in ascending order
      const int at = 31 - __clz(ok);             // -1: none
      const unsigned have = __shfl_sync(0xffffffffu, all, max(at, 0));
      __syncthreads();                           // the counts are free again
      if (at < kTkWarps - 1) hi = min(hi, lo + step * (uint32_t)(at + 2));
      lo += step * (uint32_t)(at + 1);
      if (at >= 0 && have <= enough) break;
    }
  }
  uint32_t T = max(1u, lo), Ti = 0xffffffffu;    // taken: keys above T, and those equal to T up to index Ti
  unsigned total = 0;
  for (int pass = 0; ; pass++) {
#pragma unroll
    for (int g = 0; g < NG; g++) {
      if (top[g] < T) continue;                  // few granules of the warp reach T
#pragma unroll
      for (int q = 4 * g; q < 4 * g + 4; q++) {
        const uint32_t key = key_of(q), i = (uint32_t)(b0 + q * kTkThreads);
        if (key > T || (key == T && i <= Ti)) {
          const unsigned at = atomicAdd(&s.n_own, 1u);
          if (at < kTkList) *cl.map_shared_rank(&s.cand[rank][at], 0) = make_uint2(__float_as_uint(v[q]), i);
        }
      }
    }
    __syncthreads();
    if (tid < kTkBlocks) *cl.map_shared_rank(&s.n[rank], tid) = s.n_own;
    cl.sync();
    total = 0;
#pragma unroll
    for (int b = 0; b < kTkBlocks; b++) total += s.n[b];
    if (total <= kTkList || pass == 1) break;
    // the exact k-th key, 8 bits at a time, then the index limit among the keys equal to it
    unsigned want = k;
    uint32_t pre = 0;
    for (int sh = 24; sh >= 0; sh -= 8) {
#pragma unroll
      for (int q = 0; q < R; q++) {
        const uint32_t key = key_of(q);
        if (key && (sh == 24 || (key >> (sh + 8)) == pre)) atomicAdd(&s.hist[(key >> sh) & 255u], 1u);
      }
      tkc_digit(s, want, tid);
      pre = (pre << 8) | s.digit;
      want -= s.above;
      __syncthreads();
    }
    T = pre;
    pre = 0;
    for (int sh = 24; sh >= 0; sh -= 8) {        // ~index descending: the `want` lowest indices
#pragma unroll
      for (int q = 0; q < R; q++) {
        const uint32_t inv = ~(uint32_t)(b0 + q * kTkThreads);
        if (key_of(q) == T && (sh == 24 || (inv >> (sh + 8)) == pre)) atomicAdd(&s.hist[(inv >> sh) & 255u], 1u);
      }
      tkc_digit(s, want, tid);
      pre = (pre << 8) | s.digit;
      want -= s.above;
      __syncthreads();
    }
    Ti = ~pre;
    if (tid == 0) s.n_own = 0;
    cl.sync();
  }
  if (rank) return;                              // (nobody reads the other blocks' memory any more)
  if (warp == kTkWarps - 1) {
    float2 w[kTkBlocks * kTkWarps / 32];
    float m2 = -3.0e38f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < kTkBlocks * kTkWarps / 32; i++) { w[i] = s.ms[32 * i + lane]; m2 = fmaxf(m2, w[i].x); }
#pragma unroll
    for (int i = 0; i < kTkBlocks * kTkWarps / 32; i++) s2 += w[i].y * expf(w[i].x - m2);
    warp_lse(m2, s2);
    if (lane == 0) p.out_lse[row] = m2 + logf(s2);
  }
  {
    const int b = warp / (kTkWarps / kTkBlocks);
    unsigned before = 0;
#pragma unroll
    for (int c = 0; c < kTkBlocks; c++) before += c < b ? s.n[c] : 0u;
    for (unsigned i = tid % (kTkThreads / kTkBlocks); i < s.n[b]; i += kTkThreads / kTkBlocks) {
      const uint2 c = s.cand[b][i];
      s.list_v[before + i] = c.x; s.list_i[before + i] = c.y; s.list_k[before + i] = tk_key(__uint_as_float(c.x));
    }
  }
  __syncthreads();
  const int nl = (int)total, at = tid >> 1;      // two threads per candidate
  unsigned rk = 0;
  if (at < nl) {
    const uint32_t k0 = s.list_k[at], i0 = s.list_i[at];
    for (int j = tid & 1; j < nl; j += 2) { const uint32_t kj = s.list_k[j]; rk += kj > k0 || (kj == k0 && s.list_i[j] < i0); }
  }
  rk += __shfl_xor_sync(0xffffffffu, rk, 1);
  if ((tid & 1) == 0 && at < nl && rk < k) {
    p.out_val[(size_t)row * kSampK + rk] = __uint_as_float(s.list_v[at]);
    p.out_idx[(size_t)row * kSampK + rk] = (int)s.list_i[at];
  }
  if (tid >= nl && tid < p.k) {                  // fewer than k numbers in the row
    p.out_val[(size_t)row * kSampK + tid] = -INFINITY;
    p.out_idx[(size_t)row * kSampK + tid] = -1;
  }
}

// out[r][i] = in[r][i] - logsumexp(in[r]); out may alias in.  Two forms (log_softmax_by_cluster chooses):
// one block per row, which reads it twice ...
__global__ void __launch_bounds__(kSampT) log_softmax_row_kernel(const float* in, float* out, int V) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ BlockRed r;
  const int tid = threadIdx.x, row = blockIdx.x;
  const float* x = in + (size_t)row * V;
  float* y = out + (size_t)row * V;
  float m = -3.0e38f, s = 0.f;
  for (int i = tid; i < V; i += kSampT) {
    const float v = x[i];
    if (v > m) { s = s * expf(m - v) + 1.f; m = v; }
    else s += expf(v - m);
  }
  block_lse(m, s, r, tid);
  const float lse = m + logf(s);
  for (int i = tid; i < V; i += kSampT) y[i] = x[i] - lse;
}
// ... or a cluster of 8 blocks, each of which holds its eighth of the row in registers (20 values per thread cover 163840; what is
// beyond is read again); the eight (max, sum) pairs meet through distributed shared memory, so the row is read once.  The 126
// dependent trips of one block took 37 us for 129280 logits; eight blocks take 5.
constexpr int kLsBlocks = 8, kLsRegs = 20;
__global__ void __cluster_dims__(kLsBlocks, 1, 1) __launch_bounds__(kSampT) log_softmax_kernel(const float* in, float* out, int V) {
  pdl_launch_dependents();
  pdl_wait();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // "this block runs": waited for before the first remote store
  __shared__ BlockRed r;
  __shared__ float2 pair[kLsBlocks];
  const int tid = threadIdx.x, part = blockIdx.x % kLsBlocks, row = blockIdx.x / kLsBlocks;
  const float* x = in + (size_t)row * V;
  float* y = out + (size_t)row * V;
  const int per = (V + kLsBlocks - 1) / kLsBlocks, b = min(V, part * per), e = min(V, b + per);
  float v[kLsRegs], m = -3.0e38f, s = 0.f;
#pragma unroll
  for (int q = 0; q < kLsRegs; q++) {
    const int i = b + tid + q * kSampT;
    v[q] = i < e ? x[i] : -INFINITY;
    m = fmaxf(m, v[q]);
  }
#pragma unroll
  for (int q = 0; q < kLsRegs; q++) s += expf(v[q] - m);
  for (int i = b + tid + kLsRegs * kSampT; i < e; i += kSampT) {
    const float w = x[i];
    if (w > m) { s = s * expf(m - w) + 1.f; m = w; }
    else s += expf(w - m);
  }
  block_lse(m, s, r, tid);
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (tid < kLsBlocks) cl.map_shared_rank(pair, tid)[part] = make_float2(m, s);
  cl.sync();                                         // every block's pair has arrived, and nobody writes here any more
  m = -3.0e38f; s = 0.f;
#pragma unroll
  for (int q = 0; q < kLsBlocks; q++) m = fmaxf(m, pair[q].x);
#pragma unroll
  for (int q = 0; q < kLsBlocks; q++) s += pair[q].y * expf(pair[q].x - m);
  const float lse = m + logf(s);
#pragma unroll
  for (int q = 0; q < kLsRegs; q++) {
    const int i = b + tid + q * kSampT;
    if (i < e) y[i] = v[q] - lse;
  }
  for (int i = b + tid + kLsRegs * kSampT; i < e; i += kSampT) y[i] = x[i] - lse;
}

int groups_for(int V) { return std::max(1, std::min(kSampMaxGroups, (V + 4 * kSampT - 1) / (4 * kSampT))); }
}  // namespace

// scratch: tickets [rows] | part_ms [rows][G] | part_v [rows][G][64] | part_i [rows][G][64]; must start at zero (the
// kernels leave the tickets at zero again)
size_t sample_scratch_bytes(int rows) {
  if (rows <= 0) return 0;
  const size_t R = (size_t)rows, G = kSampMaxGroups;
  return 256 + ((R * 4 + 255) & ~(size_t)255) + R * G * 8 + 2 * R * G * kSampK * 4;
}

static int fill_scratch(SampleParams& p, int rows, void* scratch, size_t scratch_bytes) {
  if (!scratch || scratch_bytes < sample_scratch_bytes(rows)) return fail(kErrScratch, "sampling: scratch too small");
  if (reinterpret_cast<uintptr_t>(scratch) & 15) return fail(kErrArg, "sampling: scratch must be 16-byte aligned");
  uint8_t* c = static_cast<uint8_t*>(scratch);
  const size_t R = (size_t)rows, G = kSampMaxGroups;
  p.ticket = reinterpret_cast<unsigned*>(c); c += (R * 4 + 255) & ~(size_t)255;
  p.part_ms = reinterpret_cast<float2*>(c); c += R * G * 8;
  p.part_v = reinterpret_cast<float*>(c); c += R * G * kSampK * 4;
  p.part_i = reinterpret_cast<uint32_t*>(c);
  return kOk;
}

int argmax_rows(const float* logits, int rows, int V, int* out_idx, float* out_val, float temperature, uint64_t seed,
                void* scratch, size_t scratch_bytes, cudaStream_t st) {
  if (rows <= 0 || V <= 0 || !logits || !out_idx) return fail(kErrArg, "argmax_rows: bad arguments");
  SampleParams p{};
  int rc = fill_scratch(p, rows, scratch, scratch_bytes);
  if (rc) return rc;
  p.logits = logits; p.rows = rows; p.V = V;
  p.groups = std::max(1, std::min(kSampMaxGroups, (V + 2047) / 2048));
  p.chunk = (V + p.groups - 1) / p.groups;
  p.inv_temp = temperature > 0.f ? 1.f / temperature : 1.f;
  p.seed_lo = (uint32_t)seed; p.seed_hi = (uint32_t)(seed >> 32);
  p.use_gumbel = temperature > 0.f ? 1 : 0;
  p.out_idx = out_idx; p.out_val = out_val;
  MSB_CUDA(launch_pdl(argmax_rows_kernel, dim3(p.groups, rows), dim3(kSampT), 0, st, p));
  MSB_LAUNCH_CHECK("argmax_rows_kernel");
  return kOk;
}

int sample_topk(const float* logits, int rows, int V, int k, float temperature, float* out_v, int* out_i, float* out_lse,
                void* scratch, size_t scratch_bytes, cudaStream_t st) {
  if (rows <= 0 || V <= 0 || !logits || !out_v || !out_i || !out_lse) return fail(kErrArg, "sample_topk: bad arguments");
  if (k < 1 || k > kSampK) return fail(kErrArg, "sample_topk: k %d outside 1..%d", k, kSampK);
  if ((size_t)V > (size_t)kSampMaxGroups * 4 * kSampT) return fail(kErrLimit, "sample_topk: V %d beyond %d", V, kSampMaxGroups * 4 * kSampT);
  SampleParams p{};
  int rc = fill_scratch(p, rows, scratch, scratch_bytes);
  if (rc) return rc;
  p.logits = logits; p.rows = rows; p.V = V; p.k = k;
  p.groups = groups_for(V);
  p.inv_temp = temperature > 0.f ? 1.f / temperature : 1.f;
  p.out_idx = out_i; p.out_val = out_v; p.out_lse = out_lse;
  static_assert(kTopkClusterMaxV <= kTkBlocks * kTkThreads * kTkMaxRegs, "registers");
  if (topk_by_cluster(rows, V, k)) {
    const int regs = (V + kTkBlocks * kTkThreads - 1) / (kTkBlocks * kTkThreads);
    const auto kern = regs <= 16 ? topk_lse_cluster_kernel<16> : regs <= 32 ? topk_lse_cluster_kernel<32> : topk_lse_cluster_kernel<kTkMaxRegs>;
    MSB_CUDA(launch_pdl(kern, dim3(rows * kTkBlocks), dim3(kTkThreads), 0, st, p));
    MSB_LAUNCH_CHECK("topk_lse_cluster_kernel");
    return kOk;
  }
  MSB_CUDA(launch_pdl(topk_lse_kernel, dim3(p.groups, rows), dim3(kSampT), 0, st, p));
  MSB_LAUNCH_CHECK("topk_lse_kernel");
  return kOk;
}

int log_softmax(const float* in, float* out, int rows, int V, cudaStream_t st) {
  if (rows <= 0 || V <= 0 || !in || !out) return fail(kErrArg, "log_softmax: bad arguments");
  int dev = 0, sms = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  MSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (!log_softmax_by_cluster(rows, V, sms)) {
    MSB_CUDA(launch_pdl(log_softmax_row_kernel, dim3(rows), dim3(kSampT), 0, st, in, out, V));
    MSB_LAUNCH_CHECK("log_softmax_row_kernel");
    return kOk;
  }
  MSB_CUDA(launch_pdl(log_softmax_kernel, dim3(rows * kLsBlocks), dim3(kSampT), 0, st, in, out, V));
  MSB_LAUNCH_CHECK("log_softmax_kernel");
  return kOk;
}

// CPU: temperature + top-p sampling from sample_topk's output.  p_i = exp(v_i / T - lse); the smallest prefix whose
// cumulative mass reaches top_p is kept and renormalised; u in [0, 1) picks inside it (arch.mm:322-342).
int sample_top_p(const float* vals, const int* ids, int k, float lse, float temperature, float top_p, double u) {
  if (temperature <= 0.0f || k <= 1) return ids[0];
  if (k > kSampK) k = kSampK;
  const double inv_t = 1.0 / temperature;
  double probs[kSampK];
  double cum = 0.0;
  int keep = k;
  for (int i = 0; i < k; i++) {
    probs[i] = std::exp((double)vals[i] * inv_t - (double)lse);
    cum += probs[i];
    if (cum >= top_p) { keep = i + 1; break; }
  }
  double tot = 0.0;
  for (int i = 0; i < keep; i++) tot += probs[i];
  const double target = u * tot;
  double acc = 0.0;
  for (int i = 0; i < keep; i++) {
    acc += probs[i];
    if (target < acc) return ids[i];
  }
  return ids[keep - 1];
}

}  // namespace msb
