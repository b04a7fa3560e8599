// MoE prefill: grouped expert GEMMs on the 5th-generation tensor cores.
// Replaces the reference's prefill MoE kernels (src/kernels/quant_moe_prefill.metal:22-344) behind
// ms::q::encode_moe_prefill (src/kernels/quant.hpp:87-118, quant.mm:427-612).  Same arithmetic as the reference's
// tensor path: activations, expert weights and the intermediate H as half operands, fp32 accumulation;
//   H[e][r] = half( silu(min(g,10)) * clamp(u,-10,10) * wt[e] ),  Z[e] = H[e] . down^T,
//   Y[t] += Z[shared row of t] + sum_k Z[slot_of[t][k]]   in that fixed order.
//
// Routing arrives expert-sorted (entries [offs[j], offs[j+1]) of tok[] / wt[] belong to routed expert j).  Launches:
//   gather      Xg[entry] = half(X[tok[entry]]); the shared expert's rows (every token, weight 1) follow the routed ones
//   gate/up     grouped GEMMs with the SwiGLU in the epilogue, H stored as half
//   down        the same grouped GEMMs on the down matrices, Z stored as fp32
//   combine     the fixed-order sum into Y
// Two grouped GEMM kernels, one persistent CTA per SM each, tiles from a table the host builds from offs[]:
//   moep_ts_kernel    decodes the experts' raw blocks inside the kernel (most experts: every weight is used by few tokens)
//   moep_gemm_kernel  reads half copies by TMA (experts with so many entries that the copy pays)
// Every mbarrier wait is bounded.
#include <cuda.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <type_traits>
#include <vector>
#include "pair_gemm.cuh"

namespace msb {

// The experts of one launch, in entry order; a tile is found from its number (mp_tile), so that the host sends one small
// table instead of every tile.  An expert's entries are cut into `chunks` runs of `per` (the last may be short); chunk0 counts
// the chunks of the experts before it.
struct MpGroup { int slot, row0, m, chunk0, chunks, per; };
struct MpTile { int slot, row0, m, n0; };   // expert slot, first entry row, entries, first weight row
__device__ __forceinline__ MpTile mp_tile_in(const MpGroup& q, int steps, int step, int t) {
  const int in = t - q.chunk0 * steps, ns = q.chunks == 1 ? in : in / q.chunks, c = in - ns * q.chunks;
  return MpTile{q.slot, q.row0 + c * q.per, min(q.per, q.m - c * q.per), ns * step};
}
// Tile t of a launch over `n` groups with `steps` weight-row tiles of `step` rows each: per expert, weight-row tiles outer and
// entry chunks inner (CTAs that run together share weight rows).  Called by whole warps: 32 groups are looked at at once, two
// rounds for 1024 experts (ten dependent reads one by one, and a division, took 2800 cycles; only the loaders, ahead of the others
// anyway, still search like that).
__device__ __forceinline__ MpTile mp_tile(const MpGroup* g, int n, int steps, int step, int t) {
  const int lane = (int)threadIdx.x & 31;
  int lo = 0;
  for (int len = n; len > 1;) {
    const int w = (len + 31) >> 5, i = w * lane;
    const unsigned m = __ballot_sync(0xffffffffu, i < len && g[lo + min(i, len - 1)].chunk0 * steps <= t);      // lane 0's is
    const int at = w * (31 - __clz(m));
    lo += at;
    len = min(w, len - at);
  }
  return mp_tile_in(g[lo], steps, step, t);
}
// the same for one thread
__device__ __forceinline__ MpTile mp_tile_of_thread(const MpGroup* g, int n, int steps, int step, int t) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (g[mid].chunk0 * steps <= t) lo = mid; else hi = mid - 1;
  }
  return mp_tile_in(g[lo], steps, step, t);
}

// silu(g) = g / (1 + exp(-g)): the quotient from an approximate reciprocal and one Newton-Raphson correction by its residual, which
// leaves it within an ulp (the result is rounded to half).  The general division's range checks and branch were a fifth of the
// epilogue's time, and four warps do it for a whole tile: reference layer, division / this, 4096 tokens 3939 / 3696 us, 2137 tokens
// 2911 / 2782, 27 tokens the same.  The bound keeps an infinite exponential from making the residual 0 * inf; silu is 0 in half long
// before.
__device__ __forceinline__ float mp_silu(float g) {
  const float d = fminf(1.f + expf(-g), 8e37f);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = g * r;
  return fmaf(fmaf(-q, d, g), r, q);
}

// ---------------------------------------------------------------------------------------------------- half copies
// MODE 0: gate/up + SwiGLU -> H (half);  MODE 1: down -> Z (fp32).  The experts with many entries: their weights are dequantised to
// half once and the weight tiles come by TMA, like the activations; 256 entries x 256 weight rows per pair of blocks (pair_gemm.cuh).
// A pair's first block fetches the gate rows, the second the same up rows; every block has 128 entries and all 256 columns.
// Alone 264 us (gate/up) and 133 (down) for the 6900 dense entries of 4096 tokens of the reference layer; in a row of launches,
// which counts waiting for the decoding launch's last blocks, 389 -> 363 and 213 -> 181 against single blocks of 128 entries.
struct MpGemmParams {
  CUtensorMap a_map;        // activations [rows_total][K] half, box 64 x 128
  CUtensorMap b_map;        // half weights of the dense experts stacked by rows, box 64 x 128
  const MpGroup* groups;
  const float* wt;          // [rows_total] routing weight per entry row (mode 0)
  __half* h;                // mode 0 output [rows_total][n_out]
  float* z;                 // mode 1 output [rows_total][n_out]
  int* status;
  int ngroups, ntiles, K, n_out;     // K = contraction length (dim / inter), n_out = output row width (inter / dim)
                            // tile.slot = index of the expert in the stacked half matrix, whose rows are
                            // [slot * 2 n_out, +n_out) gate, [.. + n_out, +n_out) up (mode 0) or [slot * n_out, +n_out) down
  int late;                 // see moep_gemm_kernel
  float limit;
};
template <int MODE>
struct MoeGemm {
  const MpGemmParams& p;
  int bn, ntiles, kb;
  static constexpr int kStep = MODE == 0 ? kGmBN / 2 : kGmBN;
  struct Tile { int a_row, b_row, n0, m; };          // m: entries of this block
  __device__ explicit MoeGemm(const MpGemmParams& q) : p(q), bn(kGmBN), ntiles(q.ntiles), kb(q.K / kGmBK) {}
  __device__ int* status() const { return p.status; }
  __device__ const CUtensorMap* a_map() const { return &p.a_map; }
  __device__ const CUtensorMap* b_map() const { return &p.b_map; }
  __device__ void wait_before() const { if (!p.late) pdl_wait(); }
  __device__ void wait_after() const { if (p.late) pdl_wait(); }
  __device__ Tile tile(int t, int rank) const { return of(mp_tile(p.groups, p.ngroups, p.n_out / kStep, kStep, t), rank); }
  __device__ Tile tile_of_thread(int t, int rank) const { return of(mp_tile_of_thread(p.groups, p.ngroups, p.n_out / kStep, kStep, t), rank); }
  __device__ Tile of(const MpTile& m, int rank) const {
    const int b = MODE == 0 ? (2 * m.slot + rank) * p.n_out + m.n0 : m.slot * p.n_out + m.n0 + rank * (kGmBN / 2);
    return Tile{m.row0 + rank * kGmBM, b, m.n0, m.m - rank * kGmBM};
  }
  __device__ void epilogue(const Tile& tl, uint32_t taddr, int warp, int lane) const {
    const int lrow = 32 * warp + lane;
    const bool live = lrow < tl.m;
    const size_t grow = (size_t)tl.a_row + lrow;
    if (MODE == 0) {
      const float wt = live ? p.wt[grow] : 0.f;
#pragma unroll 1
      for (int c0 = 0; c0 < kGmBN / 2; c0 += 32) {   // gate columns [0, 128), the same rows' up columns behind them
        uint32_t g[32], u[32];
        __syncwarp();                                // lanes without an entry come here early; the loads are the whole warp's
        gm_ld32(taddr + c0, g);
        gm_ld32(taddr + kGmBN / 2 + c0, u);
        ts_wait_ld();
        if (!live) continue;
        __half2 hh[16];
#pragma unroll
        for (int q = 0; q < 16; q++) {
          float hv[2];
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const float gg = fminf(__uint_as_float(g[2 * q + e]), p.limit);
            const float uu = fminf(fmaxf(__uint_as_float(u[2 * q + e]), -p.limit), p.limit);
            hv[e] = mp_silu(gg) * uu * wt;
          }
          hh[q] = __floats2half2_rn(hv[0], hv[1]);
        }
        __half* dst = p.h + grow * p.n_out + tl.n0 + c0;              // n_out is a multiple of 256
#pragma unroll
        for (int q = 0; q < 4; q++) reinterpret_cast<uint4*>(dst)[q] = reinterpret_cast<uint4*>(hh)[q];
      }
    } else {
#pragma unroll 1
      for (int c0 = 0; c0 < kGmBN; c0 += 32) {
        uint32_t r[32];
        __syncwarp();
        gm_ld32(taddr + c0, r);
        ts_wait_ld();
        if (!live) continue;
        float* dst = p.z + grow * p.n_out + tl.n0 + c0;
#pragma unroll
        for (int q = 0; q < 8; q++)
          reinterpret_cast<float4*>(dst)[q] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                          __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
      }
    }
  }
};
// late: the launch before is the decoding one of the same stage, which shares nothing with this one and releases it only when
// everything before has completed.  Its blocks then give way to this launch's one by one, instead of the last to end holding all
// SMs up; what comes after waits for both, since every block waits for that launch before it ends.
template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGmThreads, 1) moep_gemm_kernel(const __grid_constant__ MpGemmParams p) {
  gemm_body<2>(MoeGemm<MODE>(p));
}

// ---------------------------------------------------------------------------------------------------- decoded weights as operand A
// Grouped GEMM of the experts that are not worth a half copy (ts_gemm.cuh): gate and up rows are the two halves of a tile, or
// 256 down rows; up to 128 of an expert's tokens; the whole K.
struct TsParams {
  CUtensorMap a[4];         // activations [rows_total][K] half, boxes of 16, 32, 64, 128 rows x 64
  const MpGroup* groups;
  const uint64_t* wptr;     // [slots][3] device addresses {gate, up, down}
  const float* wt;          // [rows_total] routing weight per entry row (mode 0)
  __half* h;                // mode 0 output [rows_total][n_out]
  float* z;                 // mode 1 output [rows_total][n_out]
  int ngroups, ntiles, chunk_base, K, n_out, t_r, t_s, shared_slot;      // weight types of the routed experts and of slot shared_slot
  float limit;
  Tables tb;
};
constexpr int kTsGroups = kTsExtraBytes / (int)sizeof(MpGroup);          // a larger group table stays in global memory

template <int MODE>
struct MoeTs {
  const TsParams& p;
  const MpGroup* g;         // the groups in shared memory (every role of the block looks every tile up)
  int ntiles;
  // Every tile is found anew, and nothing is fetched ahead of a tile's own pieces: the next tile's rows brought into L2 by the producers
  // and its place kept in shared memory cost more than they gave (us with / without, reference layer: 27 tokens 756 / 697, 300 of 64
  // experts 601 / 564, 4096 3810 / 3700; with Q6_K experts, 27 tokens 1935 / 1645; benchmark layer, 27 tokens 745 / 689).
  static constexpr bool kLateTrigger = true, kSingle = false, kNextInSmem = false;
  static constexpr int kStep = MODE == 0 ? 128 : 256;
  template <int T> static constexpr bool kHas = T == IQ1_S || T == IQ2_XXS || T == Q8_0 || T == Q6_K;
  __device__ bool has_type(int t) const { return p.t_r == t || p.t_s == t; }
  __device__ const CUtensorMap* a_map(int i) const { return &p.a[i]; }
  __device__ void setup(uint8_t* extra, int tid) {
    g = p.groups;
    if (p.ngroups > kTsGroups) return;
    MpGroup* dst = reinterpret_cast<MpGroup*>(extra);
    for (int i = tid; i < p.ngroups; i += kTsThreads) dst[i] = p.groups[i];
    g = dst;
  }
  __device__ TsTile tile(int t) const {
    const int steps = p.n_out / kStep;
    return of(mp_tile(g, p.ngroups, steps, kStep, p.chunk_base * steps + t));
  }
  __device__ TsTile tile_of_thread(int t) const {
    const int steps = p.n_out / kStep;
    return of(mp_tile_of_thread(g, p.ngroups, steps, kStep, p.chunk_base * steps + t));
  }
  __device__ TsTile of(const MpTile& m) const { return TsTile{m.slot, m.row0, m.m, m.n0, 0, p.K / kTsBK, m.slot == p.shared_slot ? p.t_s : p.t_r}; }
  __device__ uint32_t row_size(int type) const { return (uint32_t)row_bytes(type, p.K); }
  __device__ const uint8_t* rows(const TsTile& tl, int half, int quarter, int& live) const {
    const uint32_t rb = row_size(tl.type);
    live = 32;
    const uint64_t* wp = p.wptr + (size_t)tl.slot * 3;
    const uint8_t* base = reinterpret_cast<const uint8_t*>(MODE == 0 ? (half ? wp[1] : wp[0]) : wp[2]);
    return base + (size_t)(tl.n0 + (MODE == 0 ? 0 : 128 * half) + 32 * quarter) * rb;
  }
  __device__ void epilogue(const TsTile& tl, uint32_t d0, uint32_t d1, int quarter, int lane) const {
    const int col = tl.n0 + 32 * quarter + lane;
    for (int c0 = 0; c0 < tl.m; c0 += 16) {
      if (MODE == 0) {
        uint32_t g16[16], u16[16];
        ts_ld16(d0 + c0, g16);
        ts_ld16(d1 + c0, u16);
        const float wl = c0 + (lane & 15) < tl.m ? p.wt[tl.row0 + c0 + (lane & 15)] : 0.f;
        ts_wait_ld();
        __half* dst = p.h + (size_t)(tl.row0 + c0) * p.n_out + col;
        const int rest = tl.m - c0;
#pragma unroll
        for (int q = 0; q < 16; q++) {
          const float gg = fminf(__uint_as_float(g16[q]), p.limit);
          const float uu = fminf(fmaxf(__uint_as_float(u16[q]), -p.limit), p.limit);
          const float hv = mp_silu(gg) * uu * __shfl_sync(0xffffffffu, wl, q);
          if (q < rest) *dst = __float2half_rn(hv);
          dst += p.n_out;
        }
      } else {
        uint32_t r[2][16];
        ts_ld16(d0 + c0, r[0]);
        ts_ld16(d1 + c0, r[1]);
        ts_wait_ld();
        float* dst = p.z + (size_t)(tl.row0 + c0) * p.n_out + col;
#pragma unroll
        for (int q = 0; q < 16; q++)
          if (c0 + q < tl.m) {
            dst[(size_t)q * p.n_out] = __uint_as_float(r[0][q]);
            dst[(size_t)q * p.n_out + 128] = __uint_as_float(r[1][q]);
          }
      }
    }
  }
};
template <int MODE>
__global__ void __launch_bounds__(kTsThreads, 1) moep_ts_kernel(const __grid_constant__ TsParams p) {
  MoeTs<MODE> pr{p, nullptr, p.ntiles};
  ts_gemm_body(pr, p.tb);
}

// Xg[row] = half(X[src token]); rows [0, total) follow tok[], rows [total, total + n_tokens) are the tokens in order
// (the shared expert's entries); their routing weight 1 is written to wt_all.
__global__ void __launch_bounds__(256) moep_gather_kernel(const float* __restrict__ X, const int* __restrict__ tok,
                                                          const float* __restrict__ wt, __half* __restrict__ xg,
                                                          float* __restrict__ wt_all, int total, int n_tokens, int dim) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x;
  const int t = row < total ? tok[row] : row - total;
  if (threadIdx.x == 0) wt_all[row] = row < total ? wt[row] : 1.0f;
  const float4* src = reinterpret_cast<const float4*>(X + (size_t)t * dim);
  uint2* dst = reinterpret_cast<uint2*>(xg + (size_t)row * dim);
  for (int i = threadIdx.x; i < dim / 4; i += 256) {
    const float4 v = src[i];
    __half2 h[2] = {__floats2half2_rn(v.x, v.y), __floats2half2_rn(v.z, v.w)};
    dst[i] = *reinterpret_cast<uint2*>(h);
  }
}

// Y[t] += Z[total + t] (shared, if any) + sum over k of Z[slot_of[t * kpt + k]] (slots < 0 skipped), in that order.  Eight rows of Z
// are requested at once (one after the other, each behind its slot number, before): 4096 tokens x 7 rows of 5120, 755 MB, take 107
// us, 999 x 9 rows of 4096 28; in a row of launches 293 -> 263 and 76 -> 56, which count waiting for the launch before.
constexpr int kMpAhead = 8;
__global__ void __launch_bounds__(256) moep_combine_kernel(const float* __restrict__ z, const int* __restrict__ slot_of,
                                                           float* __restrict__ Y, int total, int n_tokens, int kpt, int dim,
                                                           int has_shared) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int* slots = slot_of + (size_t)t * kpt;
  int e[kMpAhead];
#pragma unroll
  for (int k = 0; k < kMpAhead; k++) e[k] = k < kpt ? slots[k] : -1;
  for (int i = threadIdx.x; i < dim / 4; i += 256) {
    auto row = [&](int r) { return __ldcs(reinterpret_cast<const float4*>(z + (size_t)r * dim) + i); };
    float4 v[kMpAhead], acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (has_shared) acc = row(total + t);
#pragma unroll
    for (int k = 0; k < kMpAhead; k++)
      if (e[k] >= 0) v[k] = row(e[k]);
    float4 y = reinterpret_cast<float4*>(Y + (size_t)t * dim)[i];
#pragma unroll
    for (int k = 0; k < kMpAhead; k++)
      if (e[k] >= 0) { acc.x += v[k].x; acc.y += v[k].y; acc.z += v[k].z; acc.w += v[k].w; }
    for (int k = kMpAhead; k < kpt; k++) {
      const int s = slots[k];
      if (s < 0) continue;
      const float4 w = row(s);
      acc.x += w.x; acc.y += w.y; acc.z += w.z; acc.w += w.w;
    }
    y.x += acc.x; y.y += acc.y; y.z += acc.z; y.w += acc.w;
    reinterpret_cast<float4*>(Y + (size_t)t * dim)[i] = y;
  }
}

// ---------------------------------------------------------------- host side
namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn mp_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}
int mp_make_map(CUtensorMap* map, const void* base, int64_t rows, int cols, int box_rows = kGmBM) {
  EncodeTiledFn encode = mp_encode_fn();
  if (!encode) return fail(kErrCuda, "moe_prefill: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t gstride[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kGmBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult cr = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), gdim, gstride, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) return fail(kErrCuda, "moe_prefill: tensor map encode failed (%d)", (int)cr);
  return kOk;
}

template <int MODE>
int mp_launch(MpGemmParams& p, int sms, int dev, cudaStream_t st) {
  if (p.ntiles <= 0) return kOk;
  const size_t smem = 1024 + 1024 + (size_t)gm_stages(2) * (kGmShareA + gm_share_b(2));
  auto kern = moep_gemm_kernel<MODE>;
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    MSB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[dev & 63] = true;
  }
  MSB_CUDA(launch_pdl(kern, dim3(2 * std::max(1, std::min(sms / 2, p.ntiles))), dim3(kGmThreads), smem, st, p));
  MSB_LAUNCH_CHECK("moep_gemm_kernel");
  return kOk;
}
bool ts_type_ok(int t) { return t == IQ1_S || t == IQ2_XXS || t == Q6_K || t == Q8_0; }
template <int MODE>
int ts_launch(TsParams& p, int sms, int dev, cudaStream_t st) {
  if (p.ntiles <= 0) return kOk;
  constexpr size_t smem = kTsSmem;
  auto kern = moep_ts_kernel<MODE>;
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    MSB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[dev & 63] = true;
  }
  MSB_CUDA(launch_pdl(kern, dim3(std::max(1, std::min(sms, p.ntiles))), dim3(kTsThreads), smem, st, p));
  MSB_LAUNCH_CHECK("moep_ts_kernel");
  return kOk;
}
size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }
// Routed experts with at least kMpDenseMin entries (at most kMpDenseMax, the largest first), and the shared expert from
// kMpDenseMinShared tokens on, are dequantised to half once and read by TMA; the others are decoded in the kernel.  The line for IQ
// experts is flat: against 1024, 18 calls of 2000 to 4096 tokens ran at 0.95 of its speed with 256, 0.997 with 512, 1.004 with 2048 and
// 0.975 without copies (IQ1_S, 24 experts, 4096 tokens 1838, 1754, 1762 and 1967 us for 1782).  Q8_0 and Q6_K experts, whose copy costs
// less beside their decoding, would take 256 (16 experts, 2000 tokens, Q8_0: 1276 -> 988).  The shared expert's: 24 calls of
// 150 to 2000 tokens 0.999 with 128, 1.001 with 256, 0.993 with 1024 and 0.978 without a copy.
constexpr int kMpDenseMin = 1024, kMpDenseMinShared = 512, kMpDenseMax = 24;
// one upload: groups of the decoding launches [n_exp + 1], of the TMA-fed ones [kMpDenseMax + 1], matrix addresses
// [n_exp + 1][3] and those of the dense routed experts [kMpDenseMax][3]
size_t mp_table_bytes(int n_exp) {
  return (size_t)(n_exp + 1 + kMpDenseMax + 1) * sizeof(MpGroup) + (size_t)(n_exp + 1 + kMpDenseMax) * 3 * sizeof(uint64_t);
}
}  // namespace

struct MoePrefillArgs {
  int dim, inter, t_gate_up, t_down, t_shared, n_tokens, n_exp;
  const uint64_t* slot_ptrs;   // host [n_exp][3] device addresses {gate, up, down}
  const int* offs;             // host [n_exp + 1]
  const int* tok;              // device [total]
  const float* wt;             // device [total]
  const int* slot_of;          // device [n_tokens * k_per_token]
  int k_per_token, has_shared;
  uint64_t shared_ptrs[3];
  const float* X;
  float* Y;
  void* scratch;
  size_t scratch_bytes;
  float limit;
};

size_t moe_prefill_scratch_bytes(int total, int n_tokens, int n_exp, int dim, int inter) {
  const size_t rows = (size_t)total + n_tokens;
  size_t b = 256;
  b += al256(mp_table_bytes(n_exp)) + al256(rows * sizeof(float));
  b += al256(rows * dim * 2) + al256(rows * inter * 2) + al256(rows * dim * 4);
  b += 2 * al256((size_t)(kMpDenseMax + 1) * 2 * inter * dim * 2) ;   // half copies of the dense experts: gate|up, down (+ slack)
  return b;
}

int weights_to_f16(int t, const void* W, int64_t count, __half* out, int part, cudaStream_t st);   // prefill_gemm.cu
int weights_to_f16_group(int t, const uint64_t* d_srcs, int n_mat, int64_t count, __half* out, cudaStream_t st);

int moe_prefill(const MoePrefillArgs& a, cudaStream_t st) {
  if (a.dim <= 0 || a.inter <= 0 || a.dim % 256 || a.inter % 256) return fail(kErrArg, "moe_prefill: dim/inter must be multiples of 256");
  if (a.n_tokens < 0 || a.n_exp < 0 || a.k_per_token <= 0) return fail(kErrArg, "moe_prefill: bad counts");
  if (a.n_tokens == 0) return kOk;
  if (a.n_exp > 0 && (!a.slot_ptrs || !a.offs || !a.tok || !a.wt)) return fail(kErrArg, "moe_prefill: null routing arrays");
  if (!a.slot_of || !a.X || !a.Y || !a.scratch) return fail(kErrArg, "moe_prefill: null pointer");
  const int total = a.n_exp > 0 ? a.offs[a.n_exp] : 0;
  if (a.n_exp > 0 && a.offs[0] != 0) return fail(kErrArg, "moe_prefill: offs[0] must be 0");
  for (int j = 0; j < a.n_exp; j++)
    if (a.offs[j + 1] < a.offs[j]) return fail(kErrArg, "moe_prefill: offs must not decrease");
  if (a.scratch_bytes < moe_prefill_scratch_bytes(total, a.n_tokens, a.n_exp, a.dim, a.inter))
    return fail(kErrScratch, "moe_prefill: scratch too small");
  // whichever kernels the routing will take: a type is supported or it is not
  if ((total > 0 || a.has_shared) && !(ts_type_ok(a.t_gate_up) && ts_type_ok(a.t_down) && ts_type_ok(a.t_shared)))
    return fail(kErrType, "moe_prefill: unsupported expert weight types (%s, %s, %s)", type_name(a.t_gate_up), type_name(a.t_down),
                type_name(a.t_shared));
  Tables tb;
  int rc = get_tables(&tb);
  if (rc) return rc;
  int dev = 0, sms = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  MSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int n_sh = a.has_shared ? a.n_tokens : 0;
  const size_t rows = (size_t)total + n_sh;
  // scratch carve-up
  uint8_t* cur = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(a.scratch) + 255) & ~(uintptr_t)255);
  uint8_t* d_table = cur; cur += al256(mp_table_bytes(a.n_exp));
  float* d_wt = reinterpret_cast<float*>(cur); cur += al256(rows * sizeof(float));
  __half* d_xg = reinterpret_cast<__half*>(cur); cur += al256(rows * a.dim * 2);
  __half* d_h = reinterpret_cast<__half*>(cur); cur += al256(rows * a.inter * 2);
  float* d_z = reinterpret_cast<float*>(cur); cur += al256(rows * a.dim * 4);
  __half* d_wgu = reinterpret_cast<__half*>(cur); cur += al256((size_t)(kMpDenseMax + 1) * 2 * a.inter * a.dim * 2);
  __half* d_wd = reinterpret_cast<__half*>(cur);
  // first, while the host makes the table
  if (rows > 0)
    MSB_CUDA(launch_pdl(moep_gather_kernel, dim3((unsigned)rows), dim3(256), 0, st, a.X, a.tok, a.wt, d_xg, d_wt, total, n_sh, a.dim));
  // dense experts: the largest routed experts with many entries, and the shared expert when there are many tokens
  std::vector<int> dense_slots;
  for (int j = 0; j < a.n_exp; j++)
    if (a.offs[j + 1] - a.offs[j] >= kMpDenseMin) dense_slots.push_back(j);
  std::sort(dense_slots.begin(), dense_slots.end(), [&](int x, int y) {
    const int mx = a.offs[x + 1] - a.offs[x], my = a.offs[y + 1] - a.offs[y];
    return mx != my ? mx > my : x < y;
  });
  if ((int)dense_slots.size() > kMpDenseMax) dense_slots.resize(kMpDenseMax);
  const size_t nd_r = dense_slots.size();
  if (n_sh >= kMpDenseMinShared) dense_slots.push_back(a.n_exp);
  static_assert(sizeof(MpGroup) % 8 == 0, "addresses follow the groups");
  const size_t table_bytes = mp_table_bytes(a.n_exp);
  std::vector<uint64_t> table(table_bytes / 8, 0);
  MpGroup* g_ts = reinterpret_cast<MpGroup*>(table.data());
  MpGroup* g_d = g_ts + a.n_exp + 1;
  uint64_t* wptr = reinterpret_cast<uint64_t*>(g_d + kMpDenseMax + 1);
  uint64_t* dsrc = wptr + (size_t)(a.n_exp + 1) * 3;
  std::vector<uint8_t> is_dense_slot(a.n_exp + 1, 0);
  for (int j : dense_slots) is_dense_slot[j] = 1;
  int n_ts = 0, chunks_ts = 0, n_d = 0, chunks_d = 0;
  bool routed_ts = false, shared_ts = false;
  auto entries = [&](int j) { return j == a.n_exp ? n_sh : a.offs[j + 1] - a.offs[j]; };
  auto row_of = [&](int j) { return j == a.n_exp ? total : a.offs[j]; };
  for (int jj = 0; jj <= a.n_exp; jj++) {                 // the shared expert first: its tiles take longest, so they are no tail
    const int j = jj == 0 ? a.n_exp : jj - 1, m = entries(j);
    if (m <= 0 || is_dense_slot[j]) continue;
    const int chunks = (m + kTsMaxN - 1) / kTsMaxN, per = ((m + chunks - 1) / chunks + 15) & ~15;
    g_ts[n_ts++] = MpGroup{j, row_of(j), m, chunks_ts, (m + per - 1) / per, per};
    chunks_ts += g_ts[n_ts - 1].chunks;
    (j == a.n_exp ? shared_ts : routed_ts) = true;
  }
  for (size_t q = 0; q < dense_slots.size(); q++) {       // slot = index of the half copy
    const int m = entries(dense_slots[q]), chunks = (m + 2 * kGmBM - 1) / (2 * kGmBM);
    g_d[n_d++] = MpGroup{(int)q, row_of(dense_slots[q]), m, chunks_d, chunks, 2 * kGmBM};
    chunks_d += chunks;
  }
  for (int j = 0; j < a.n_exp; j++)
    for (int q = 0; q < 3; q++) {
      wptr[(size_t)j * 3 + q] = a.slot_ptrs[(size_t)j * 3 + q];
      if (!wptr[(size_t)j * 3 + q] && a.offs[j + 1] > a.offs[j]) return fail(kErrArg, "moe_prefill: null matrix of expert slot %d", j);
    }
  for (int q = 0; q < 3; q++) wptr[(size_t)a.n_exp * 3 + q] = a.shared_ptrs[q];
  if (n_sh && (!a.shared_ptrs[0] || !a.shared_ptrs[1] || !a.shared_ptrs[2])) return fail(kErrArg, "moe_prefill: null shared expert matrix");
  for (size_t q = 0; q < nd_r; q++) {                     // gate and up of every dense routed expert, then the down matrices
    dsrc[2 * q] = wptr[(size_t)dense_slots[q] * 3];
    dsrc[2 * q + 1] = wptr[(size_t)dense_slots[q] * 3 + 1];
    dsrc[2 * nd_r + q] = wptr[(size_t)dense_slots[q] * 3 + 2];
  }
  const MpGroup* d_gts = reinterpret_cast<const MpGroup*>(d_table);
  const MpGroup* d_gd = d_gts + a.n_exp + 1;
  const uint64_t* d_wptr = reinterpret_cast<const uint64_t*>(d_gd + kMpDenseMax + 1);
  const uint64_t* d_dsrc = d_wptr + (size_t)(a.n_exp + 1) * 3;
  // (pageable source: the runtime stages it before returning)
  MSB_CUDA(cudaMemcpyAsync(d_table, table.data(), table_bytes, cudaMemcpyHostToDevice, st));
  if (rows == 0) return kOk;
  // half copies of the dense experts (gate rows then up rows per expert; down rows per expert).  The routed ones come
  // first in dense_slots and share their types: one grouped launch for all their gate / up matrices, one for the down
  // matrices; the shared expert, when it is dense, has its own type and three launches.
  {
    const size_t gu = (size_t)a.inter * a.dim;
    if (nd_r > 0 && !is_dense(a.t_gate_up) && !is_dense(a.t_down)) {
      rc = weights_to_f16_group(a.t_gate_up, d_dsrc, (int)(2 * nd_r), (int64_t)gu, d_wgu, st);
      if (rc) return rc;
      rc = weights_to_f16_group(a.t_down, d_dsrc + 2 * nd_r, (int)nd_r, (int64_t)gu, d_wd, st);
      if (rc) return rc;
    }
    for (size_t q = 0; q < dense_slots.size(); q++) {
      const int j = dense_slots[q];
      if (j != a.n_exp && !is_dense(a.t_gate_up) && !is_dense(a.t_down)) continue;    // done above
      const int t_gu = j == a.n_exp ? a.t_shared : a.t_gate_up, t_d = j == a.n_exp ? a.t_shared : a.t_down;
      rc = weights_to_f16(t_gu, reinterpret_cast<const void*>(wptr[(size_t)j * 3]), (int64_t)gu, d_wgu + (2 * q) * gu, 0, st);
      if (rc) return rc;
      rc = weights_to_f16(t_gu, reinterpret_cast<const void*>(wptr[(size_t)j * 3 + 1]), (int64_t)gu, d_wgu + (2 * q + 1) * gu, 0, st);
      if (rc) return rc;
      rc = weights_to_f16(t_d, reinterpret_cast<const void*>(wptr[(size_t)j * 3 + 2]), (int64_t)gu, d_wd + q * gu, 0, st);
      if (rc) return rc;
    }
  }
  MpGemmParams p;
  p.late = n_ts > 0;
  p.wt = d_wt; p.h = d_h; p.z = d_z; p.status = tb.status; p.limit = a.limit > 0.f ? a.limit : 10.f;
  TsParams q;
  q.wptr = d_wptr; q.wt = d_wt; q.h = d_h; q.z = d_z; q.limit = p.limit; q.tb = tb; q.shared_slot = a.n_exp;
  // Tiles of the routed experts and of the shared expert in one launch, unless both would need a (different) codebook table.
  auto ts_run = [&](auto mode, int t_r, int steps) -> int {
    constexpr int kMode = decltype(mode)::value;
    const bool split = routed_ts && shared_ts && t_r != a.t_shared && lut_bytes_for(t_r) && lut_bytes_for(a.t_shared);
    const int ch_s = shared_ts ? g_ts[0].chunks : 0;
    auto part = [&](int first, int count, int chunk0, int chunks, int tr, int ts) {
      q.groups = d_gts + first; q.ngroups = count; q.chunk_base = chunk0; q.ntiles = chunks * steps; q.t_r = tr; q.t_s = ts;
      return ts_launch<kMode>(q, sms, dev, st);
    };
    if (!split) return part(0, n_ts, 0, chunks_ts, routed_ts ? t_r : a.t_shared, shared_ts ? a.t_shared : t_r);
    int r = part(0, 1, 0, ch_s, a.t_shared, a.t_shared);
    return r ? r : part(1, n_ts - 1, ch_s, chunks_ts - ch_s, t_r, t_r);
  };
  // gate/up + SwiGLU
  rc = mp_make_map(&p.a_map, d_xg, (int64_t)rows, a.dim);
  if (rc) return rc;
  for (int i = 0; i < 4; i++) {
    rc = mp_make_map(&q.a[i], d_xg, (int64_t)rows, a.dim, 16 << i);
    if (rc) return rc;
  }
  p.K = q.K = a.dim; p.n_out = q.n_out = a.inter;
  rc = ts_run(std::integral_constant<int, 0>(), a.t_gate_up, a.inter / 128);
  if (rc) return rc;
  p.groups = d_gd; p.ngroups = n_d;
  if (n_d) {
    rc = mp_make_map(&p.b_map, d_wgu, (int64_t)dense_slots.size() * 2 * a.inter, a.dim, kGmBN / 2);
    if (rc) return rc;
    p.ntiles = chunks_d * (a.inter / (kGmBN / 2));
    rc = mp_launch<0>(p, sms, dev, st);
    if (rc) return rc;
  }
  // down
  rc = mp_make_map(&p.a_map, d_h, (int64_t)rows, a.inter);
  if (rc) return rc;
  for (int i = 0; i < 4; i++) {
    rc = mp_make_map(&q.a[i], d_h, (int64_t)rows, a.inter, 16 << i);
    if (rc) return rc;
  }
  p.K = q.K = a.inter; p.n_out = q.n_out = a.dim;
  rc = ts_run(std::integral_constant<int, 1>(), a.t_down, a.dim / 256);
  if (rc) return rc;
  if (n_d) {
    rc = mp_make_map(&p.b_map, d_wd, (int64_t)dense_slots.size() * a.dim, a.inter, kGmBN / 2);
    if (rc) return rc;
    p.ntiles = chunks_d * (a.dim / kGmBN);
    rc = mp_launch<1>(p, sms, dev, st);
    if (rc) return rc;
  }
  MSB_CUDA(launch_pdl(moep_combine_kernel, dim3((unsigned)a.n_tokens), dim3(256), 0, st, (const float*)d_z, a.slot_of, a.Y, total,
                      a.n_tokens, a.k_per_token, a.dim, a.has_shared ? 1 : 0));
  MSB_LAUNCH_CHECK("moe_prefill");
  return kOk;
}

}  // namespace msb
