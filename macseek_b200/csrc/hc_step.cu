// Hyper-connection step of one sublayer boundary -- ms::arch::encode_hc_step (src/kernels/arch.hpp:44-77, kernels
// src/kernels/arch_hc.metal:49-323); math as tests/ref/arch_ref.cpp:22-95:
//   h_new[i]  = x_sub ? post[i] * x_sub + sum_j comb[j][i] * h_in[j] : h_in          (4 residual streams of width D)
//   mix_out   = fn ? split + Sinkhorn( fn . h_new * rsqrt(mean(h_new^2) + 1e-20), scale, base ) : -
//   x_out     = rmsnorm( sum_j pre[j] * h_new[j] ) * norm_w                          (pre / post / comb from mix_prev)
// hc_cluster_kernel (below) takes the usual widths; hc_step_kernel every other.
// hc_step_kernel: one launch per call, all tokens: grid (blocks over D, tokens).  A block owns 32 consecutive columns d of the four
// streams; its 8 warps share the 24 rows of fn (3 rows each), so that the 96 fn values a column needs are fetched by 8
// threads at once instead of one after the other, and D / 32 blocks (128 at D = 4096) spread the 1.6 MB of fn over the
// machine.  Every thread reads its column of h_in (and x_sub) BEFORE the block's barrier and only warp 0 writes h_out
// afterwards, so h_out may alias h_in.  Each warp's shuffle sum is the block's partial of its rows; the block that
// finishes last (a ticket per token) adds the partials in block order, runs the 4 x 4 Sinkhorn on 16 lanes and scales
// x_out.  Bound by the latency of one pass over fn (24 x 4 D floats, read exactly once), not by its bytes.
#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>
#include "hc_route.h"
#include "msb_common.cuh"

namespace msb {

constexpr int kHcThreads = 256;
constexpr int kHcCols = 32;       // columns per block (one per lane); warp w takes fn rows [3 w, 3 w + 3)
constexpr int kHcMaxBlocks = 512; // D <= 16384
constexpr int kHcPart = 26;       // 24 fn rows, sum h_new^2, sum x^2

struct HcParams {
  const float* h_in;      // [n][4][D]
  float* h_out;           // [n][4][D] (written only with x_sub; may alias h_in)
  const float* x_sub;     // [n][D] or null
  const float* mix_prev;  // [n][24]
  const float* fn;        // [24][4 D] or null
  const float* scale;     // [3]
  const float* base;      // [24]
  float* mix_out;         // [n][24]
  const float* norm_w;    // [D]
  float* x_out;           // [n][D] or null
  float* part;            // [n][blocks][26] partial sums
  unsigned* ticket;       // [n], zero between launches
  int D, n, iters;
  float hc_eps;
};

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }

__global__ void __launch_bounds__(kHcThreads) hc_step_kernel(const HcParams p) {
  pdl_launch_dependents();
  __shared__ float tot[kHcPart];
  __shared__ int is_last;
  const int tok = blockIdx.y, D = p.D, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* hin = p.h_in + (size_t)tok * 4 * D;
  float* hout = p.h_out + (size_t)tok * 4 * D;
  float* xo = p.x_out ? p.x_out + (size_t)tok * D : nullptr;
  const int d = blockIdx.x * kHcCols + lane;
  const bool live = d < D;
  float h[4] = {0.f, 0.f, 0.f, 0.f}, hn[4], xs = 0.f, f[3][4];
  // fn is a weight: requested before the dependency wait, it arrives while the previous kernel finishes
  if (live && p.fn) {
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
      for (int i = 0; i < 4; i++) f[r][i] = __ldg(p.fn + ((size_t)(3 * warp + r) * 4 + i) * D + d);
  }
  pdl_wait();
  float mp[24];
#pragma unroll
  for (int i = 0; i < 24; i++) mp[i] = p.mix_prev[(size_t)tok * 24 + i];
  if (live) {
#pragma unroll
    for (int j = 0; j < 4; j++) h[j] = hin[(size_t)j * D + d];
    if (p.x_sub) xs = p.x_sub[(size_t)tok * D + d];
  }
  if (p.x_sub) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      float a = mp[4 + i] * xs;
#pragma unroll
      for (int j = 0; j < 4; j++) a = fmaf(mp[8 + 4 * j + i], h[j], a);
      hn[i] = a;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) hn[i] = h[i];
  }
  float* part = p.part + ((size_t)tok * gridDim.x + blockIdx.x) * kHcPart;
  if (p.fn) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
      float a = 0.f;
      if (live) {
#pragma unroll
        for (int i = 0; i < 4; i++) a = fmaf(f[r][i], hn[i], a);
      }
      a = warp_sum(a);
      if (lane == 0) part[3 * warp + r] = a;
    }
  }
  __syncthreads();                      // every warp has read its column of h_in: warp 0 may now overwrite it
  if (warp == 0) {
    float sq = 0.f, xq = 0.f;
    if (live) {
      if (p.x_sub) {
#pragma unroll
        for (int i = 0; i < 4; i++) hout[(size_t)i * D + d] = hn[i];
      }
      sq = hn[0] * hn[0] + hn[1] * hn[1] + hn[2] * hn[2] + hn[3] * hn[3];
      if (xo) {
        const float x = mp[0] * hn[0] + mp[1] * hn[1] + mp[2] * hn[2] + mp[3] * hn[3];
        xo[d] = x;                      // scaled by the finishing block
        xq = x * x;
      }
    }
    sq = warp_sum(sq); xq = warp_sum(xq);
    if (lane == 0) { part[24] = sq; part[25] = xq; }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) is_last = atomicAdd(&p.ticket[tok], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // entry e = warp, warp + 8, ...: its lanes take the blocks' partials 32 at a time (loads in flight together), the
  // shuffle tree then adds them in a fixed order
  for (int e = warp; e < kHcPart; e += kHcThreads / 32) {
    double v = 0.0;
    for (unsigned b = lane; b < gridDim.x; b += 32) v += (double)__ldcg(p.part + ((size_t)tok * gridDim.x + b) * kHcPart + e);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) tot[e] = (float)v;
  }
  if (tid == 0) p.ticket[tok] = 0;
  __syncthreads();
  if (p.fn && warp == 0) {
    const float rstd = rsqrtf(tot[24] / (float)(4 * D) + 1e-20f);
    float* mo = p.mix_out + (size_t)tok * 24;
    if (lane < 4) mo[lane] = sigmoidf_(tot[lane] * rstd * p.scale[0] + p.base[lane]) + p.hc_eps;
    else if (lane < 8) mo[lane] = 2.f * sigmoidf_(tot[lane] * rstd * p.scale[1] + p.base[lane]);
    // comb: lane = 4 j + k of the 4 x 4 matrix; row sums over k (xor 1, 2), column sums over j (xor 4, 8)
    const int e = lane & 15;
    float c = tot[8 + e] * rstd * p.scale[2] + p.base[8 + e];
    float mx = fmaxf(c, __shfl_xor_sync(0xffffffffu, c, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    c = expf(c - mx);
    float s = c + __shfl_xor_sync(0xffffffffu, c, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    c = c / s + p.hc_eps;
    for (int it = 0; it < p.iters; it++) {
      if (it > 0) {
        float rs = c + __shfl_xor_sync(0xffffffffu, c, 1);
        rs += __shfl_xor_sync(0xffffffffu, rs, 2);
        c = c / (rs + p.hc_eps);
      }
      float cs = c + __shfl_xor_sync(0xffffffffu, c, 4);
      cs += __shfl_xor_sync(0xffffffffu, cs, 8);
      c = c / (cs + p.hc_eps);
    }
    if (lane < 16) mo[8 + lane] = c;
  }
  if (xo) {
    const float r = rsqrtf(tot[25] / (float)D + 1e-20f);
    for (int d = tid; d < D; d += kHcThreads) xo[d] = __ldcg(xo + d) * r * p.norm_w[d];
  }
}

// ---- D a multiple of 1024 up to 5120: one cluster of 16 blocks per token (or per 4 tokens).
// Block r owns columns [r D / 16, (r + 1) D / 16): a thread holds the fn values of one column pair and 4 of the 24 rows (32
// registers, requested before the dependency wait, used for every token), so the whole step is: read the pair's four streams,
// mix them, 4 dot products, one barrier, the blocks' 26 sums to all 16 blocks through distributed shared memory, one cluster
// barrier.  x_out is then scaled out of registers and the Sinkhorn iterations run on one lane's registers (row and column
// sums without shuffles, one reciprocal per line).  Bound by that chain of latencies: the 2 MB of fn are on their way before
// it starts.  Against one ticket over D / 32 blocks with a serial finish (two passes through L2, 40 shuffles with
// divisions): two steps of D = 5120, one token, and a compressor 39 -> 24 us; a step of one token alone 6.7 to 6.9 us at D = 4096.
// More tokens: 4 at a time share the barriers and fn stays in registers, where a grid of (D / 32) x n blocks read fn once per
// token.  A step of D = 5120 takes 29.5 us for 32 tokens and 141 for 256.

// The iterations on one lane's registers, but for the last columns' division (sinkhorn_last).  A whole row or column is multiplied by
// __fdividef's reciprocal of its sum (arguments between 1e-6 and a few; an IEEE division's branches do not overlap): what is wrong
// with the factor is wrong for all four alike, and the next pass takes it out.
__device__ __forceinline__ void sinkhorn4(float (&c)[16], int iters, float eps) {   // rows 4 j.., first a softmax of each row
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float mx = fmaxf(fmaxf(c[4 * j], c[4 * j + 1]), fmaxf(c[4 * j + 2], c[4 * j + 3]));
#pragma unroll
    for (int k = 0; k < 4; k++) c[4 * j + k] = expf(c[4 * j + k] - mx);
    const float r = __fdividef(1.f, (c[4 * j] + c[4 * j + 1]) + (c[4 * j + 2] + c[4 * j + 3]));
#pragma unroll
    for (int k = 0; k < 4; k++) c[4 * j + k] = c[4 * j + k] * r + eps;
  }
  for (int it = 0; it < iters; it++) {
    if (it > 0) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float r = __fdividef(1.f, ((c[4 * j] + c[4 * j + 1]) + (c[4 * j + 2] + c[4 * j + 3])) + eps);
#pragma unroll
        for (int k = 0; k < 4; k++) c[4 * j + k] *= r;
      }
    }
    if (it + 1 == iters) break;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float r = __fdividef(1.f, ((c[k] + c[4 + k]) + (c[8 + k] + c[12 + k])) + eps);
#pragma unroll
      for (int j = 0; j < 4; j++) c[4 * j + k] *= r;
    }
  }
}

// element `lane` (0..15) after the last columns' division, which is exact: nothing comes after it
__device__ __forceinline__ float sinkhorn_last(const float (&c)[16], int lane, float eps) {
  float v = 0.f, sum = 1.f;
#pragma unroll
  for (int e = 0; e < 16; e++) v = lane == e ? c[e] : v;
#pragma unroll
  for (int k = 0; k < 4; k++) sum = (lane & 3) == k ? ((c[k] + c[4 + k]) + (c[8 + k] + c[12 + k])) + eps : sum;
  return v / sum;
}
// Sums as precise as hc_step_kernel's: chains of at most 8 products and 8 lanes in float, everything beyond in double (with the
// warps' and blocks' sums added in float the mixing weights of 1000 tokens of 4096 were 9.0e-8 from float64; they are 7.3e-8 there).
constexpr int kHcQuarters = 4 * 5;
__device__ __forceinline__ float hc_sum8(float v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float hc_total(const double (&t)[kHcRanks][kHcPart], int e) {
  double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int r = 0; r < kHcRanks; r++) s[r & 3] += t[r][e];
  return (float)((s[0] + s[1]) + (s[2] + s[3]));
}

template <int T>      // tokens per round
__global__ void __launch_bounds__(kHcThreadsMax, 1) hc_cluster_kernel(const HcParams p) {
  pdl_launch_dependents();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // "this block runs", before the first remote store
  __shared__ float part[T][kHcPart][kHcQuarters];    // per 8 lanes of a row group's warps (at most 5)
  __shared__ double tots[2][T][kHcRanks][kHcPart];   // every block's sums, by round parity
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, D = p.D;
  const int rank = blockIdx.x % kHcRanks, cluster = blockIdx.x / kHcRanks, nclusters = gridDim.x / kHcRanks;
  const int pairs = D / (2 * kHcRanks), wpg = pairs / 32;        // column pairs of the block, warps per row group
  const int rg = warp / wpg, wi = warp % wpg;                    // row group 0..5: fn rows 4 rg .. 4 rg + 3
  const int d = rank * (D / kHcRanks) + 2 * (wi * 32 + lane);
  float2 f[4][4];
  if (p.fn) {
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int i = 0; i < 4; i++) f[r][i] = __ldg(reinterpret_cast<const float2*>(p.fn + ((size_t)(4 * rg + r) * 4 + i) * D + d));
  }
  pdl_wait();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  unsigned round = 0;
  for (int t0 = cluster * T; t0 < p.n; t0 += nclusters * T, round++) {
    float2 x[T], hn[T];                              // row group 0: the mixed x; row groups 0..3: stream rg of h_new
#pragma unroll
    for (int t = 0; t < T; t++) {
      const int tk = t0 + t;
      x[t] = make_float2(0.f, 0.f);
      hn[t] = make_float2(0.f, 0.f);
      if (tk >= p.n) continue;
      const float* mp = p.mix_prev + (size_t)tk * 24;
      const float* hin = p.h_in + (size_t)tk * 4 * D + d;
      float2 h[4], xs = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 4; j++) h[j] = *reinterpret_cast<const float2*>(hin + (size_t)j * D);
      if (p.x_sub) xs = *reinterpret_cast<const float2*>(p.x_sub + (size_t)tk * D + d);
      float a[4] = {0.f, 0.f, 0.f, 0.f}, sq = 0.f;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float2 v = h[i];
        if (p.x_sub) {
          const float po = mp[4 + i];
          v = make_float2(po * xs.x, po * xs.y);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const float cj = mp[8 + 4 * j + i];
            v.x = fmaf(cj, h[j].x, v.x); v.y = fmaf(cj, h[j].y, v.y);
          }
        }
        if (p.fn) {
#pragma unroll
          for (int r = 0; r < 4; r++) { a[r] = fmaf(f[r][i].x, v.x, a[r]); a[r] = fmaf(f[r][i].y, v.y, a[r]); }
        }
        if (rg == 0) {
          const float pr = mp[i];
          x[t].x = fmaf(pr, v.x, x[t].x); x[t].y = fmaf(pr, v.y, x[t].y);
          sq = fmaf(v.x, v.x, sq); sq = fmaf(v.y, v.y, sq);
        }
        if (rg == i) hn[t] = v;
      }
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float s = hc_sum8(a[r]);
        if ((lane & 7) == 0) part[t][4 * rg + r][4 * wi + (lane >> 3)] = s;
      }
      if (rg == 0) {
        sq = hc_sum8(sq);
        const float xq = hc_sum8(x[t].x * x[t].x + x[t].y * x[t].y);
        if ((lane & 7) == 0) { part[t][24][4 * wi + (lane >> 3)] = sq; part[t][25][4 * wi + (lane >> 3)] = xq; }
      }
    }
    __syncthreads();                                 // the block's columns of h_in are read: h_out may be written
    if (p.x_sub && rg < 4) {
#pragma unroll
      for (int t = 0; t < T; t++)
        if (t0 + t < p.n) *reinterpret_cast<float2*>(p.h_out + ((size_t)(t0 + t) * 4 + rg) * D + d) = hn[t];
    }
    for (int q = tid; q < T * kHcRanks * kHcPart; q += blockDim.x) {
      const int t = q / (kHcRanks * kHcPart), dst = q / kHcPart % kHcRanks, e = q % kHcPart;
      double s[4];
#pragma unroll
      for (int k = 0; k < 4; k++) s[k] = (double)part[t][e][k];
      for (int w = 1; w < wpg; w++)
#pragma unroll
        for (int k = 0; k < 4; k++) s[k] += (double)part[t][e][4 * w + k];
      *cl.map_shared_rank(&tots[round & 1][t][rank][e], dst) = (s[0] + s[1]) + (s[2] + s[3]);
    }
    cl.sync();
    // One barrier per round is enough: a round writes the other parity, and no block can be two rounds ahead.
    if (p.x_out && rg == 0) {
#pragma unroll
      for (int t = 0; t < T; t++) {
        if (t0 + t >= p.n) continue;
        const float mul = rsqrtf(hc_total(tots[round & 1][t], 25) / (float)D + 1e-20f);
        const float2 g = *reinterpret_cast<const float2*>(p.norm_w + d);
        *reinterpret_cast<float2*>(p.x_out + (size_t)(t0 + t) * D + d) = make_float2(x[t].x * mul * g.x, x[t].y * mul * g.y);
      }
    }
    if (p.fn && warp == 5 * wpg && rank < T && t0 + rank < p.n) {       // block t of the cluster: token t's mixing weights
      const int t = rank;
      const float s = lane < 25 ? hc_total(tots[round & 1][t], lane) : 0.f;
      const float rstd = rsqrtf(__shfl_sync(0xffffffffu, s, 24) / (float)(4 * D) + 1e-20f);
      const int which = lane < 4 ? 0 : lane < 8 ? 1 : 2;
      const float y = lane < 24 ? s * rstd * p.scale[which] + p.base[lane] : 0.f;
      float* mo = p.mix_out + (size_t)(t0 + t) * 24;
      if (lane < 8) mo[lane] = lane < 4 ? sigmoidf_(y) + p.hc_eps : 2.f * sigmoidf_(y);
      float c[16];
#pragma unroll
      for (int e = 0; e < 16; e++) c[e] = __shfl_sync(0xffffffffu, y, 8 + e);
      sinkhorn4(c, p.iters, p.hc_eps);
      const float last = sinkhorn_last(c, lane, p.hc_eps);
      if (lane < 16) mo[8 + lane] = last;
    }
    __syncthreads();                                 // part[] is free again
  }
}

// clusters of hc_cluster_kernel<T> for width D that run at once (asked once per device and width), 0: none, or no width of its
template <int T>
static int hc_fit(int D, int dev) {
  static std::atomic<int> known[64][kHcThreadsMax / 192 + 1] = {};       // 1 + the number; widths are multiples of 1024
  const int threads = D / (2 * kHcRanks) * 6;
  if (D % (64 * kHcRanks) || threads > kHcThreadsMax) return 0;
  std::atomic<int>& at = known[dev & 63][threads / 192];
  int v = at.load(std::memory_order_relaxed);
  if (v == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kHcRanks); cfg.blockDim = dim3(threads);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kHcRanks; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(hc_cluster_kernel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, hc_cluster_kernel<T>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();                    // not a failure of this call: the other kernel takes it
      n = 0;
    }
    v = n + 1;
    at.store(v, std::memory_order_relaxed);
  }
  return v - 1;
}

size_t hc_scratch_bytes(int n) { return ((size_t)n * kHcMaxBlocks * kHcPart + (size_t)n) * 4 + 64; }

int hc_step(const float* h_in, float* h_out, const float* x_sub, const float* mix_prev, const float* fn, const float* scale,
            const float* base, float* mix_out, const float* norm_w, float* x_out, int D, int n, void* scratch,
            size_t scratch_bytes, cudaStream_t st) {
  if (D <= 0 || n <= 0 || !h_in || !mix_prev) return fail(kErrArg, "hc_step: bad arguments");
  if (x_sub && !h_out) return fail(kErrArg, "hc_step: h_out missing");
  if (fn && (!scale || !base || !mix_out)) return fail(kErrArg, "hc_step: fn needs scale, base and mix_out");
  if (x_out && !norm_w) return fail(kErrArg, "hc_step: x_out needs norm_w");
  if (mix_out == mix_prev) return fail(kErrArg, "hc_step: mix_out must not alias mix_prev");
  if (!scratch || scratch_bytes < hc_scratch_bytes(n)) return fail(kErrScratch, "hc_step: scratch too small");
  HcParams p;
  p.h_in = h_in; p.h_out = h_out ? h_out : const_cast<float*>(h_in); p.x_sub = x_sub; p.mix_prev = mix_prev; p.fn = fn;
  p.scale = scale; p.base = base; p.mix_out = mix_out; p.norm_w = norm_w; p.x_out = x_out;
  p.ticket = reinterpret_cast<unsigned*>(scratch);            // first n words: zero-filled by the caller once
  p.part = reinterpret_cast<float*>(scratch) + ((n + 15) & ~15);
  p.D = D; p.n = n; p.iters = 20; p.hc_eps = 1e-6f;
  if (D > kHcMaxBlocks * kHcCols) return fail(kErrLimit, "hc_step: D %d beyond %d", D, kHcMaxBlocks * kHcCols);
  const uintptr_t al = reinterpret_cast<uintptr_t>(h_in) | reinterpret_cast<uintptr_t>(p.h_out) | reinterpret_cast<uintptr_t>(x_sub) |
                       reinterpret_cast<uintptr_t>(fn) | reinterpret_cast<uintptr_t>(norm_w) | reinterpret_cast<uintptr_t>(x_out);
  int dev = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  const HcRoute route = hc_route(D, n, (al & 7) == 0, hc_fit<1>(D, dev), hc_fit<4>(D, dev));
  if (route.tokens) {
    const dim3 block(D / (2 * kHcRanks) * 6);
    MSB_CUDA(launch_clusters(route.tokens == 1 ? hc_cluster_kernel<1> : hc_cluster_kernel<4>, dim3(route.clusters * kHcRanks), block, kHcRanks, 0,
                             st, p));
    MSB_LAUNCH_CHECK("hc_cluster_kernel");
    return kOk;
  }
  const int blocks = (D + kHcCols - 1) / kHcCols;
  MSB_CUDA(launch_pdl(hc_step_kernel, dim3(blocks, n), dim3(kHcThreads), 0, st, p));
  MSB_LAUNCH_CHECK("hc_step_kernel");
  return kOk;
}

}  // namespace msb
