// MoE router: logits = W[E x dim] . x (fp32), score = sqrt(softplus) or sigmoid, top-k of score + bias (ties -> lowest
// expert id), weights = score / (sum + 1e-20) * route_scale; plus the per-expert routing lists for the prefill grouped
// GEMM.  Replaces the reference's arch_router_fused / arch_router_topk / arch_route_count / arch_route_scatter Metal
// kernels (src/kernels/arch_router.metal:16-160) behind ms::arch::encode_router_fused / encode_router_topk /
// encode_route_lists (src/kernels/arch.hpp:79-97, arch.mm:173-239).
#include <algorithm>
#include <cooperative_groups.h>
#include "msb_common.cuh"
#include "router_route.h"

namespace msb {

constexpr int kRouterMaxE = 512;   // experts per token handled by the one-warp selection (16 per lane)
constexpr int kRouterMaxK = 16;
constexpr int kRouterKSplit = 4;   // K slices per expert row in the fused kernel

struct RouterParams {
  const float* x;
  const float* norm_w;   // not null: x is RMS-normalised with this gain before use (fused RMSNorm)
  float* x_out;          // with norm_w: the normalised x is also written here (may be null)
  float norm_eps;
  const float* W;
  const float* bias;     // may be null
  float* logits;         // [E] (written by the fused kernel; diagnostic, as the reference's Scratch::router_logits)
  float* partial;        // [E][kRouterKSplit]
  int* ids;
  float* wts;
  unsigned* ticket;      // zero between launches
  int E, dim, k, score_fn;
  float route_scale;
};

__device__ __forceinline__ float router_score(float x, int score_fn) {
  if (score_fn == 1) return 1.f / (1.f + expf(-x));
  const float sp = x > 20.f ? x : log1pf(expf(x));   // softplus, threshold 20 (arch_router.metal:20-24)
  return sqrtf(sp);
}

// One warp selects the top-k experts of one token (descending key; ties -> lowest id) and writes ids / weights; a lane holds experts
// lane + 32 i.
constexpr int kRouterEPL = kRouterMaxE / 32;
// order-preserving map of a float onto an unsigned (NaN -> 0, below everything)
__device__ __forceinline__ unsigned router_ord(float f) {
  const unsigned u = __float_as_uint(f);
  return f == f ? (u ^ ((unsigned)((int)u >> 31) | 0x80000000u)) : 0u;
}
// The selection itself: sc / key of experts lane + 32 i (key -inf beyond E)
__device__ __forceinline__ void router_select_warp(const float (&sc)[kRouterEPL], const float (&key)[kRouterEPL], int E, int k,
                                                   float route_scale, int lane, int* ids, float* wts) {
  constexpr int EPL = kRouterEPL;
  float sum = 0.f, my_w = 0.f;
  int my_e = 0;
  unsigned taken = 0;
  bool rescan = true;
  float bk = -INFINITY, bs = 0.f;
  int be = 0x7fffffff;
  for (int j = 0; j < k; j++) {
    // this lane's best remaining candidate: ascending expert id with a strict compare keeps the lowest id on ties;
    // only the lane that lost its candidate in the previous round looks again
    if (rescan) {
      bk = -INFINITY; bs = 0.f; be = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < EPL; i++) {
        const int e = lane + 32 * i;
        if (e < E && !((taken >> i) & 1u) && (be == 0x7fffffff || key[i] > bk)) { bk = key[i]; bs = sc[i]; be = e; }
      }
      rescan = false;
    }
    // warp-wide: the largest key, then the lowest expert id that holds it (one reduction instruction each)
    const unsigned uk = be == 0x7fffffff ? 0u : router_ord(bk);
    const unsigned m = __reduce_max_sync(0xffffffffu, uk);
    const int win = (int)__reduce_min_sync(0xffffffffu, (uk == m) ? (unsigned)be : 0x7fffffffu);
    const float wscore = __shfl_sync(0xffffffffu, bs, win & 31);   // the owner's best candidate is the winner
    if (lane == (win & 31)) { taken |= 1u << (win >> 5); rescan = true; }
    sum += wscore;
    if (lane == j) { my_e = win; my_w = wscore; }
  }
  const float inv = route_scale / (sum + 1e-20f);
  if (lane < k) { ids[lane] = my_e; wts[lane] = my_w * inv; }
}
// Fused decode router: every warp computes one (expert, K-slice) partial dot; the block that finishes last sums the
// slices in a fixed order, writes the logits and selects.
__global__ void __launch_bounds__(256) router_fused_kernel(const RouterParams p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = blockIdx.x * 8 + warp;
  const int slice = p.dim / kRouterKSplit;   // floats per slice, a multiple of 4
  const bool live = unit < p.E * kRouterKSplit;
  const int e = unit / kRouterKSplit, ks = unit % kRouterKSplit;
  const float4* w = reinterpret_cast<const float4*>(p.W + (size_t)(live ? e : 0) * p.dim + (size_t)ks * slice);
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  // the router matrix is constant: its first 8 x 16 bytes per lane are requested before the grid dependency resolves
  float4 a[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int c = lane + 32 * k;
    a[k] = (live && c < slice / 4) ? __ldg(w + c) : zero4;
  }
  pdl_wait();
  // Dependents are released only now: a dependent that starts may rely on everything before this launch being complete
  // (the MoE gate/up launch reads the un-normalised vector before its own dependency resolves).
  pdl_launch_dependents();
  // this unit's slice of x (and of the norm gain) is requested before the norm's reduction, not after it
  const float4* xv = reinterpret_cast<const float4*>(p.x + (size_t)ks * slice);
  const float4* gv = reinterpret_cast<const float4*>(p.norm_w ? p.norm_w + (size_t)ks * slice : p.x);
  float4 b[8], g8[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int c = lane + 32 * k;
    b[k] = (live && c < slice / 4) ? xv[c] : zero4;
    g8[k] = (live && p.norm_w && c < slice / 4) ? __ldg(gv + c) : zero4;
  }
  float mul = 1.f;
  if (p.norm_w) {   // every block needs 1/rms of the whole vector: dim floats from L2, summed in a fixed order
    __shared__ float red[8];
    float ss = 0.f;
    for (int i = threadIdx.x; i < p.dim / 4; i += 256) {
      const float4 v = reinterpret_cast<const float4*>(p.x)[i];
      ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) tot += red[i];
    mul = rsqrtf(tot / (float)p.dim + p.norm_eps);
  }
  if (live) {
    float acc = 0.f;
    for (int c0 = lane; c0 < slice / 4; c0 += 32 * 8) {   // 8 independent 16-byte loads in flight per lane
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int c = c0 + 32 * k;
        if (c0 != lane) {
          a[k] = c < slice / 4 ? __ldg(w + c) : zero4;
          b[k] = c < slice / 4 ? xv[c] : zero4;
          g8[k] = (p.norm_w && c < slice / 4) ? __ldg(gv + c) : zero4;
        }
        if (p.norm_w && c < slice / 4) {
          b[k].x = b[k].x * mul * g8[k].x; b[k].y = b[k].y * mul * g8[k].y;
          b[k].z = b[k].z * mul * g8[k].z; b[k].w = b[k].w * mul * g8[k].w;
          if (e == 0 && p.x_out) reinterpret_cast<float4*>(p.x_out + (size_t)ks * slice)[c] = b[k];
        }
      }
#pragma unroll
      for (int k = 0; k < 8; k++) {
        acc = fmaf(a[k].x, b[k].x, acc); acc = fmaf(a[k].y, b[k].y, acc);
        acc = fmaf(a[k].z, b[k].z, acc); acc = fmaf(a[k].w, b[k].w, acc);
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) p.partial[unit] = acc;
  }
  __shared__ int is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned t = atomicAdd(p.ticket, 1u);
    is_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // the finishing block: the serial tail of the launch.  Bias (constant) and partial sums are requested together; the scores, a
  // logarithm and an exponential each, are computed by all threads, one or two experts a thread, and reach the selecting warp through
  // shared memory (by that warp alone, 16 a lane, they held the launch up for 7 us: router and MoE of the reference layer 66.4 ->
  // 59.0; the logits in global memory are a diagnostic).
  __shared__ float s_score[kRouterMaxE], s_key[kRouterMaxE];
  for (int e = threadIdx.x; e < p.E; e += blockDim.x) {
    const float4 q = __ldcg(reinterpret_cast<const float4*>(p.partial) + e);
    const float bias = p.bias ? __ldg(p.bias + e) : 0.f;
    const float s = ((q.x + q.y) + q.z) + q.w;
    p.logits[e] = s;
    const float sc = router_score(s, p.score_fn);
    s_score[e] = sc;
    s_key[e] = sc + bias;
  }
  __syncthreads();
  if (warp == 0) {
    float sc[kRouterEPL], key[kRouterEPL];
#pragma unroll
    for (int i = 0; i < kRouterEPL; i++) {
      const int e = lane + 32 * i;
      sc[i] = e < p.E ? s_score[e] : 0.f;
      key[i] = e < p.E ? s_key[e] : -INFINITY;
    }
    router_select_warp(sc, key, p.E, p.k, p.route_scale, lane, p.ids, p.wts);
  }
  if (threadIdx.x == 0) *p.ticket = 0;
}

// logits [n][E] -> ids [n][k], weights [n][k].  A block per token: all threads score, the first warp selects; for calls whose
// blocks are resident at once, where a token's latency is the call's time (router_block_per_token).
__global__ void __launch_bounds__(128) router_topk_block_kernel(const float* logits, const float* bias, int* ids, float* wts, int E,
                                                                int k, int score_fn, float route_scale) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float s_score[kRouterMaxE], s_key[kRouterMaxE];
  const int t = blockIdx.x, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < E; e += 128) {
    const float b = bias ? __ldg(bias + e) : 0.f, s = router_score(logits[(size_t)t * E + e], score_fn);
    s_score[e] = s;
    s_key[e] = s + b;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  float sc[kRouterEPL], key[kRouterEPL];
#pragma unroll
  for (int i = 0; i < kRouterEPL; i++) {
    const int e = lane + 32 * i;
    sc[i] = e < E ? s_score[e] : 0.f;
    key[i] = e < E ? s_key[e] : -INFINITY;
  }
  router_select_warp(sc, key, E, k, route_scale, lane, ids + (size_t)t * k, wts + (size_t)t * k);
}
// The same with a warp per token, which scores lane + 32 i itself: no idle warps while one selects, for calls of many tokens.
__global__ void __launch_bounds__(128) router_topk_warp_kernel(const float* logits, const float* bias, int* ids, float* wts, int n,
                                                               int E, int k, int score_fn, float route_scale) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= n) return;
  const float* l = logits + (size_t)t * E;
  float bz[kRouterEPL], sc[kRouterEPL], key[kRouterEPL];
#pragma unroll
  for (int i = 0; i < kRouterEPL; i++) {
    const int e = lane + 32 * i;
    bz[i] = (bias && e < E) ? __ldg(bias + e) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < kRouterEPL; i++) {
    const int e = lane + 32 * i;
    if (e < E) {
      sc[i] = router_score(l[e], score_fn);
      key[i] = sc[i] + bz[i];
    } else {
      sc[i] = 0.f;
      key[i] = -INFINITY;
    }
  }
  router_select_warp(sc, key, E, k, route_scale, lane, ids + (size_t)t * k, wts + (size_t)t * k);
}

// ---- routing lists: entries i = t*k + j sorted by (expert, i), a counting sort in one launch.  One cluster of 8 blocks:
// block b owns the b-th eighth of the entries.  (1) It counts them per expert in shared memory; (2) through distributed
// shared memory every block reads all eight counts, so that each knows where its entries of every expert begin; (3) it
// places its entries 1024 at a time, in order: a warp ranks its 32 entries with a match, the warps' counts per expert are
// added up in warp order.  Positions depend on the entries alone (the one unordered step is the counting), so the lists are
// identical from run to run.  Bound by the latency of these steps; a warp per expert scanning all entries, as before, read
// them E times from L2: 349 us for 4096 tokens x 6 experts, 12 us now.
constexpr int kRlBlocks = 8, kRlThreads = 1024;
constexpr size_t kRlSmem = 2048 * (8 + 2 * 32);  // counts and bases of a pass over the experts, then u16 counts [warps with entries][experts]
__global__ void __cluster_dims__(kRlBlocks, 1, 1) __launch_bounds__(kRlThreads) route_lists_kernel(
    const int* __restrict__ ids, const float* __restrict__ w, unsigned* counts, unsigned* offsets, unsigned* entry, unsigned* tok,
    float* lw, unsigned* slot_of, int N, int E, int k, int pass) {      // pass: experts per pass, even
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) unsigned rl_smem[];
  __shared__ unsigned wsum[32];
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x;
  const int ep = pass;
  unsigned* hist = rl_smem;                       // [ep]
  unsigned* base = hist + ep;                     // [ep] next position of an entry of this block
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(base + ep);       // [warps][ep]
  const int per = (N + kRlBlocks - 1) / kRlBlocks, b0 = min(N, rank * per), b1 = min(N, b0 + per);
  unsigned carry = 0;
  for (int e0 = 0; e0 < E; e0 += pass) {
    const int ne = min(pass, E - e0);
    for (int e = tid; e < ne; e += kRlThreads) hist[e] = 0;
    __syncthreads();
    for (int i = b0 + tid; i < b1; i += kRlThreads) {
      const int e = ids[i] - e0;
      if (e >= 0 && e < ne) atomicAdd(&hist[e], 1u);
    }
    cl.sync();
    // per expert: entries of the blocks before this one, and of all; then a scan over the experts, 1024 at a time
    for (int c0 = 0; c0 < ne; c0 += kRlThreads) {
      const int e = c0 + tid;
      unsigned before = 0, all = 0;
      if (e < ne) {
#pragma unroll
        for (int r = 0; r < kRlBlocks; r++) {
          const unsigned v = *cl.map_shared_rank(hist + e, r);
          if (r < rank) before += v;
          all += v;
        }
      }
      unsigned x = all;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) wsum[warp] = x;
      __syncthreads();
      const unsigned ws = wsum[lane];
      const unsigned prev = __reduce_add_sync(0xffffffffu, lane < warp ? ws : 0u), total = __reduce_add_sync(0xffffffffu, ws);
      if (e < ne) {
        const unsigned off = carry + prev + x - all;
        base[e] = off + before;
        if (rank == 0) { counts[e0 + e] = all; offsets[e0 + e] = off; }
      }
      carry += total;
      __syncthreads();
    }
    cl.sync();                                    // the other blocks are done with this block's counts
    for (int i0 = b0; i0 < b1; i0 += kRlThreads) {
      const int nw = (min(b1 - i0, kRlThreads) + 31) >> 5;         // warps that have entries
      for (int j = tid; j < nw * ep / 2; j += kRlThreads) reinterpret_cast<unsigned*>(wcnt)[j] = 0;
      __syncthreads();
      const int i = i0 + tid;
      const int id = i < b1 ? ids[i] - e0 : -1;
      const bool hit = id >= 0 && id < ne;
      const unsigned m = __match_any_sync(0xffffffffu, hit ? id : -1);
      const unsigned in_warp = __popc(m & ((1u << lane) - 1u));
      if (hit && in_warp == 0) wcnt[warp * ep + id] = (uint16_t)__popc(m);
      __syncthreads();
      for (int e = tid; e < ne; e += kRlThreads) {
        unsigned run = 0;
#pragma unroll 8
        for (int q = 0; q < nw; q++) { const unsigned v = wcnt[q * ep + e]; wcnt[q * ep + e] = (uint16_t)run; run += v; }
        hist[e] = base[e];                        // where this round's entries begin
        base[e] += run;
      }
      __syncthreads();
      if (hit) {
        const unsigned q = hist[id] + wcnt[warp * ep + id] + in_warp;
        entry[q] = (unsigned)i; tok[q] = (unsigned)(i / k); lw[q] = w[i]; slot_of[i] = q;
      }
      __syncthreads();
    }
  }
  if (rank == 0 && tid == 0) offsets[E] = carry;
}

// ---------------------------------------------------------------- host side
// logits [E], padded to a multiple of 4 floats so that the partials [E][4] behind them are 16-byte aligned
size_t router_scratch_bytes(int E) { return sizeof(float) * ((size_t)((E + 3) & ~3) + (size_t)E * kRouterKSplit); }

int router_fused(const float* x, const float* norm_w, float norm_eps, float* x_out, const float* W, const float* bias,
                 int* ids, float* wts, void* scratch, size_t scratch_bytes, int E, int dim, int k, int score_fn,
                 float route_scale, cudaStream_t st) {
  if (E <= 0 || E > kRouterMaxE || k <= 0 || k > kRouterMaxK || k > E || dim <= 0 || dim % (4 * kRouterKSplit))
    return fail(kErrArg, "router: bad shape (E %d dim %d k %d)", E, dim, k);
  if (!x || !W || !ids || !wts || !scratch) return fail(kErrArg, "router: null pointer");
  if (scratch_bytes < router_scratch_bytes(E)) return fail(kErrScratch, "router: scratch too small");
  if (reinterpret_cast<uintptr_t>(scratch) & 15) return fail(kErrArg, "router: scratch must be 16-byte aligned");
  static_assert(kRouterKSplit == 4, "the finishing block reads one float4 of partials per expert");
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(W) & 15))
    return fail(kErrArg, "router: x and W must be 16-byte aligned");
  Tables tb;
  int rc = get_tables(&tb);
  if (rc) return rc;
  RouterParams p;
  if ((norm_w && (reinterpret_cast<uintptr_t>(norm_w) & 15)) || (x_out && (reinterpret_cast<uintptr_t>(x_out) & 15)))
    return fail(kErrArg, "router: norm_w and x_out must be 16-byte aligned");
  p.x = x; p.norm_w = norm_w; p.norm_eps = norm_eps; p.x_out = norm_w ? x_out : nullptr;
  p.W = W; p.bias = bias; p.ids = ids; p.wts = wts;
  p.logits = reinterpret_cast<float*>(scratch);
  p.partial = p.logits + ((E + 3) & ~3);
  p.ticket = reinterpret_cast<unsigned*>(tb.status) + 16;
  p.E = E; p.dim = dim; p.k = k; p.score_fn = score_fn; p.route_scale = route_scale;
  const int units = E * kRouterKSplit;
  MSB_CUDA(launch_pdl(router_fused_kernel, dim3((units + 7) / 8), dim3(256), 0, st, p));
  MSB_LAUNCH_CHECK("router_fused_kernel");
  return kOk;
}

int router_topk(const float* logits, const float* bias, int* ids, float* wts, int n, int E, int k, int score_fn,
                float route_scale, cudaStream_t st) {
  if (E <= 0 || E > kRouterMaxE || k <= 0 || k > kRouterMaxK || k > E || n < 0)
    return fail(kErrArg, "router_topk: bad shape (n %d E %d k %d)", n, E, k);
  if (n == 0) return kOk;
  if (!logits || !ids || !wts) return fail(kErrArg, "router_topk: null pointer");
  if (router_block_per_token(n, E))
    MSB_CUDA(launch_pdl(router_topk_block_kernel, dim3(n), dim3(128), 0, st, logits, bias, ids, wts, E, k, score_fn, route_scale));
  else
    MSB_CUDA(launch_pdl(router_topk_warp_kernel, dim3((n + 3) / 4), dim3(128), 0, st, logits, bias, ids, wts, n, E, k, score_fn,
                        route_scale));
  MSB_LAUNCH_CHECK("router_topk_kernel");
  return kOk;
}

int route_lists(const int* ids, const float* w, int n, int k, int E, unsigned* counts, unsigned* offsets,
                unsigned* entry, unsigned* tok, float* lw, unsigned* slot_of, cudaStream_t st) {
  if (n < 0 || k <= 0 || E <= 0) return fail(kErrArg, "route_lists: bad shape");
  if (!ids || !w || !counts || !offsets || !entry || !tok || !lw || !slot_of) return fail(kErrArg, "route_lists: null pointer");
  const int N = n * k;
  // experts per pass: as many as there is room for (2048 with 1024 and more entries per block, 14746 with up to 32)
  const int warps = (std::min((N + kRlBlocks - 1) / kRlBlocks, kRlThreads) + 31) / 32;
  const int pass = std::min((E + 1) & ~1, (int)(kRlSmem / (8 + 2 * (size_t)warps)) & ~1);
  const size_t smem = (size_t)pass * (8 + 2 * (size_t)warps);
  int dev = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    MSB_CUDA(cudaFuncSetAttribute(route_lists_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRlSmem));
    configured[dev & 63] = true;
  }
  MSB_CUDA(launch_pdl(route_lists_kernel, dim3(kRlBlocks), dim3(kRlThreads), smem, st, ids, w, counts, offsets, entry, tok, lw, slot_of,
                      N, E, k, pass));
  MSB_LAUNCH_CHECK("route_lists");
  return kOk;
}

}  // namespace msb
