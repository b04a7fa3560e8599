// Lightning indexer, decode side: query preparation, key scoring on the tensor cores, exact top-k.
//   score[t] = sum_h relu(q_h . k_t) * w_h   for t < len          (tests/ref/attn_ref.cpp:172-184 is the math spec)
//   top-k among finite scores, ties -> lower index, output sorted ascending by index, -1 padded (:186-194)
// Replaces the reference's attn_idx_prep_thread / attn_idx_score_dec2 / attn_topk_compact / attn_topk_final Metal
// kernels (src/kernels/attn_index.metal:129-145,616-677,703-797) behind ms::attn::encode_index_decode
// (src/kernels/attn.hpp:121-122, attn.mm:222-290).
//
// Scoring is a [len x 128] x [128 x heads] contraction: FP8 (e4m3) keys go straight into mma.sync m16n8k32 with the
// query held in registers as e4m3 B fragments; F16 keys use m16n8k16 with the fp32 query split into two f16 terms
// (hi + lo) so that no query precision is lost.  fp32 accumulation throughout; heads are summed in a fixed order.
// Selection: a 4096-bin histogram of the order-preserving key's top 12 bits (built by the scoring kernel) gives the
// threshold bin; a grid-wide compaction collects everything above it plus the threshold bin's members; one block
// finishes exactly (radix select on the remaining key bits, then on the index for ties) and sorts by index.
#include <cuda_fp8.h>
#include <cooperative_groups.h>
#include <algorithm>
#include <cmath>
#include "msb_common.cuh"

namespace msb {
namespace cg = cooperative_groups;

constexpr int kIdxDim = 128;
constexpr int kKeyF16 = 1, kKeyFp8 = 101;
constexpr int kHistBins = 4096;

// tcgen05 scoring kernel for FP8 keys (index_tc.cu)
int index_scores_tc(const void* keys, int len, const float* q, const float* w, int heads, float* scores, unsigned* hist,
                    int prep, const float* cs, int actq, float* q_out, float* w_out, const int* cand, int n_cand,
                    cudaStream_t st);

__device__ __forceinline__ uint32_t order_key(float f) {   // larger float <=> larger key
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ bool selectable(float f) { return f > -INFINITY; }   // finite or +inf; NaN never

__device__ __forceinline__ void mma_e4m3(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct IdxParams {
  const uint8_t* keys;
  const float* q;      // [H][128] prepared query
  const float* w;      // [H] prepared head weights
  float* scores;       // [len]
  unsigned* hist;      // [4096] or null
  int len;
};

__device__ __forceinline__ void hist_flush(unsigned* sh, unsigned* gh, int tid, int nthreads) {
  __syncthreads();
  for (int b = tid; b < kHistBins; b += nthreads) {
    const unsigned v = sh[b];
    if (v) atomicAdd(&gh[b], v);
  }
}

// ---------------------------------------------------------------- FP8 keys: direct e4m3 MMA, query in registers
// K permutation: lane (g, t) holds bytes 32t .. 32t+31 of key rows g and g+8; k-step s pairs words (2s, 2s+1) of the
// row with the same bytes of the query, so the contraction covers every dimension once.
template <int H>
__global__ void __launch_bounds__(384, 1) idx_score_fp8_kernel(const IdxParams p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int NT = H / 8;
  __shared__ unsigned sh_hist[kHistBins];
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int ntiles = (p.len + 15) / 16;
  // software pipeline: the next tile's 64 bytes per lane are requested before the current tile is multiplied
  auto fetch = [&](int tile, uint4 (&r)[4]) {
    const int k0 = tile * 16 + g, k1 = k0 + 8;
    r[0] = r[1] = r[2] = r[3] = make_uint4(0, 0, 0, 0);
    if (tile < ntiles && k0 < p.len) {
      const uint4* src = reinterpret_cast<const uint4*>(p.keys + (size_t)k0 * kIdxDim + 32 * t);
      r[0] = __ldg(src); r[1] = __ldg(src + 1);
    }
    if (tile < ntiles && k1 < p.len) {
      const uint4* src = reinterpret_cast<const uint4*>(p.keys + (size_t)k1 * kIdxDim + 32 * t);
      r[2] = __ldg(src); r[3] = __ldg(src + 1);
    }
  };
  // three tiles of keys per warp in flight (48 registers): requested before the query is staged, so that the first
  // round trips to HBM overlap the prologue
  uint4 cur[4], nx1[4], nx2[4];
  int tile = blockIdx.x * (blockDim.x >> 5) + (tid >> 5);
  fetch(tile, cur);
  fetch(tile + warps, nx1);
  fetch(tile + 2 * warps, nx2);
  if (p.hist)
    for (int b = tid; b < kHistBins; b += blockDim.x) sh_hist[b] = 0;
  // the query goes through shared memory as e4m3 bytes: a coalesced, latency-parallel load instead of 256 dependent
  // global loads per thread
  __shared__ __align__(16) uint8_t q8[H * kIdxDim];
  __shared__ __align__(16) float wsh[H];
  {
    constexpr int kQ4 = (H * kIdxDim / 4 + 383) / 384;   // 16-byte pieces per thread (block of 384)
    float4 v[kQ4];
#pragma unroll
    for (int j = 0; j < kQ4; j++) {                      // all loads in flight before the first conversion
      const int i = tid + 384 * j;
      v[j] = i < H * kIdxDim / 4 ? reinterpret_cast<const float4*>(p.q)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < kQ4; j++) {
      const int i = tid + 384 * j;
      const uint32_t b = (uint32_t)__nv_cvt_float_to_fp8(v[j].x, __NV_SATFINITE, __NV_E4M3) |
                         ((uint32_t)__nv_cvt_float_to_fp8(v[j].y, __NV_SATFINITE, __NV_E4M3) << 8) |
                         ((uint32_t)__nv_cvt_float_to_fp8(v[j].z, __NV_SATFINITE, __NV_E4M3) << 16) |
                         ((uint32_t)__nv_cvt_float_to_fp8(v[j].w, __NV_SATFINITE, __NV_E4M3) << 24);
      if (i < H * kIdxDim / 4) reinterpret_cast<uint32_t*>(q8)[i] = b;
    }
  }
  for (int i = tid; i < H; i += blockDim.x) wsh[i] = p.w[i];
  __syncthreads();
  uint32_t B[NT][4][2];
  float wr[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; nt++) {
    const uint32_t* qr = reinterpret_cast<const uint32_t*>(q8 + (size_t)(nt * 8 + g) * kIdxDim + 32 * t);
#pragma unroll
    for (int s = 0; s < 4; s++) { B[nt][s][0] = qr[2 * s]; B[nt][s][1] = qr[2 * s + 1]; }
    wr[nt][0] = wsh[nt * 8 + 2 * t];
    wr[nt][1] = wsh[nt * 8 + 2 * t + 1];
  }
  if (p.hist) __syncthreads();
  for (; tile < ntiles; tile += warps) {
    uint4 nx3[4];
    fetch(tile + 3 * warps, nx3);
    const int k0 = tile * 16 + g, k1 = k0 + 8;
    const uint32_t A0[8] = {cur[0].x, cur[0].y, cur[0].z, cur[0].w, cur[1].x, cur[1].y, cur[1].z, cur[1].w};
    const uint32_t A1[8] = {cur[2].x, cur[2].y, cur[2].z, cur[2].w, cur[3].x, cur[3].y, cur[3].z, cur[3].w};
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 4; s++) mma_e4m3(c, A0[2 * s], A1[2 * s], A0[2 * s + 1], A1[2 * s + 1], B[nt][s][0], B[nt][s][1]);
      s0 += fmaxf(c[0], 0.f) * wr[nt][0] + fmaxf(c[1], 0.f) * wr[nt][1];
      s1 += fmaxf(c[2], 0.f) * wr[nt][0] + fmaxf(c[3], 0.f) * wr[nt][1];
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1); s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1); s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    if (t == 0) {   // lanes 0, 4, ..., 28 hold the 16 scores of the tile
      if (k0 < p.len) p.scores[k0] = s0;
      if (k1 < p.len) p.scores[k1] = s1;
      if (p.hist) {   // neighbouring scores mostly share a bin: one shared-memory atomic per distinct bin per warp
        const uint32_t b0 = (k0 < p.len && selectable(s0)) ? order_key(s0) >> 20 : 0xFFFFFFFFu;
        const uint32_t b1 = (k1 < p.len && selectable(s1)) ? order_key(s1) >> 20 : 0xFFFFFFFFu;
        const unsigned m0 = __match_any_sync(0x11111111u, b0), m1 = __match_any_sync(0x11111111u, b1);
        if (b0 != 0xFFFFFFFFu && lane == __ffs(m0) - 1) atomicAdd(&sh_hist[b0], (unsigned)__popc(m0));
        if (b1 != 0xFFFFFFFFu && lane == __ffs(m1) - 1) atomicAdd(&sh_hist[b1], (unsigned)__popc(m1));
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) { cur[i] = nx1[i]; nx1[i] = nx2[i]; nx2[i] = nx3[i]; }
  }
  if (p.hist) hist_flush(sh_hist, p.hist, tid, blockDim.x);
}

// ---------------------------------------------------------------- query preparation (attn_ref.cpp:163-170)
// rope on the last 64 dims of each head (interleaved pairs), optional fp4 (e2m1, power-of-two block-32 scale)
// quant-dequant simulation, head weights scaled by dim^-0.5 * heads^-0.5.  One warp per head; v[i] = dim 32 i + lane.
__device__ __forceinline__ float pow2i(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }
__device__ __forceinline__ float round_e2m1(float x) {
  const float a = fabsf(x);
  int e = (int)((__float_as_uint(a) >> 23) & 0xFF) - 127;
  e = max(e, 0);
  return copysignf(nearbyintf(a * pow2i(1 - e)) * pow2i(e - 1), x);
}
__device__ __forceinline__ void idx_prep_head(float (&v)[4], const float* cs, int actq, int lane) {
  // dims 64..127 are roped: pair (64 + 2j, 64 + 2j + 1) with (cos, sin) j.  Lane holds dims 64+lane and 96+lane.
  {
    const float o2 = __shfl_xor_sync(0xffffffffu, v[2], 1), o3 = __shfl_xor_sync(0xffffffffu, v[3], 1);
    const int j2 = lane >> 1, j3 = 16 + (lane >> 1);
    const float c2 = cs[2 * j2], s2 = cs[2 * j2 + 1], c3 = cs[2 * j3], s3 = cs[2 * j3 + 1];
    // even element: a*c - b*s ; odd element: a*s + b*c  with (a, b) = (even, odd)
    v[2] = (lane & 1) ? __fadd_rn(__fmul_rn(o2, s2), __fmul_rn(v[2], c2)) : __fsub_rn(__fmul_rn(v[2], c2), __fmul_rn(o2, s2));
    v[3] = (lane & 1) ? __fadd_rn(__fmul_rn(o3, s3), __fmul_rn(v[3], c3)) : __fsub_rn(__fmul_rn(v[3], c3), __fmul_rn(o3, s3));
  }
  if (actq) {
#pragma unroll
    for (int i = 0; i < 4; i++) {   // block i = dims 32i .. 32i+31 = one value per lane
      float amax = fabsf(v[i]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      amax = fmaxf(amax, 6.0f * 1.17549435e-38f);
      const float r = __fmul_rn(amax, 1.0f / 6.0f);
      const uint32_t rb = __float_as_uint(r);
      const int e = (int)((rb >> 23) & 0xFF) - 127 + ((rb & 0x7FFFFF) ? 1 : 0);
      const float s = pow2i(e), inv = pow2i(-e);
      v[i] = __fmul_rn(round_e2m1(fminf(fmaxf(__fmul_rn(v[i], inv), -6.0f), 6.0f)), s);
    }
  }
}
static float idx_weight_scale(int heads) { return (float)(pow((double)kIdxDim, -0.5) * pow((double)heads, -0.5)); }
__global__ void idx_prep_kernel(const float* q_raw, const float* w_raw, const float* cs, int actq, int heads, float wscale, float* q,
                                float* w) {
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= heads) return;
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = q_raw[(size_t)h * kIdxDim + 32 * i + lane];
  idx_prep_head(v, cs, actq, lane);
#pragma unroll
  for (int i = 0; i < 4; i++) q[(size_t)h * kIdxDim + 32 * i + lane] = v[i];
  if (lane == 0) w[h] = w_raw[h] * wscale;
}

// ---------------------------------------------------------------- F16 keys (or FP8 widened to F16): m16n8k16
// The fp32 query as TERMS halfs per value, each the rounded rest of the ones before: two for the plain pass, three for the
// candidate pass, which then multiplies the whole fp32 query (scaled per head by a power of two so that no term is subnormal
// before it is negligible).  B fragments in shared memory: Bs[term][n-tile][k-step][lane] = {b0, b1}.
// K permutation: lane (g, t) holds elements 32t .. 32t+31 of its rows; k-step s uses elements 32t+4s .. 32t+4s+3.
// A warp scores 16 keys at a time and has the next 16 in flight; the first ones are requested before the query is prepared.
// LIST: position 8 i + j stands for key cand[i] * 8 + j, -inf when there is none.
// Bound by the latency of one or two rounds of loads per warp: as three launches (query, scores with 32 keys per warp and no
// prefetch, histogram) the 50003 keys of the reference shape took 25 us, and 16384 candidate keys, one warp per key on fp32
// FMAs, 33; this took 14 and 13 (as launches alone; 50 -> 35 us for the whole attention of the 50003).  With the heads' values
// requested together, the weights' scale from the host (two double powers per head before) and four chains of MMAs side by side the
// attention of the 50003 takes 31.0 in a graph of such calls (34.8 before).
constexpr int kF16Warps = 12;
struct IdxF16Params {
  const uint8_t* keys;
  const float* q;        // raw (prep) or prepared query and weights
  const float* w;
  const float* cs;       // not null: prepare the query (rope, actq), store it in q_out / w_out
  float* q_out;
  float* w_out;
  const int* cand;       // LIST
  float* scores;
  unsigned* hist;        // may be null
  int len, n, actq;      // keys, positions to score
  float wscale;          // of the raw weights
};
template <int H, bool FP8IN, int TERMS, bool LIST>
__global__ void __launch_bounds__(kF16Warps * 32, 1) idx_score_f16_kernel(const IdxF16Params p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int NTH = H / 8;
  extern __shared__ __align__(16) uint8_t f16_smem[];
  uint2* Bs = reinterpret_cast<uint2*>(f16_smem);                          // [TERMS][NTH][8][32]
  __half* Bh = reinterpret_cast<__half*>(f16_smem);
  unsigned* sh_hist = reinterpret_cast<unsigned*>(f16_smem + TERMS * NTH * 8 * 32 * sizeof(uint2));
  __shared__ __align__(16) float wsh[H], scl[H];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int warps = gridDim.x * kF16Warps, ntiles = (p.n + 15) / 16;
  auto key_of = [&](int pos) {                                             // -1: none
    if (pos >= p.n) return -1;
    if (!LIST) return pos;
    const int b = __ldg(p.cand + (pos >> 3));
    const long k = (long)b * 8 + (pos & 7);
    return b >= 0 && k < p.len ? (int)k : -1;
  };
  struct Rows { uint32_t a[2][16]; int key[2]; };
  auto fetch = [&](int tile, Rows& r) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      r.key[i] = tile < ntiles ? key_of(tile * 16 + g + 8 * i) : -1;
#pragma unroll
      for (int j = 0; j < (FP8IN ? 2 : 4); j++) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r.key[i] >= 0) v = __ldg(reinterpret_cast<const uint4*>(p.keys + ((size_t)r.key[i] * kIdxDim + 32 * t) * (FP8IN ? 1 : 2)) + j);
        r.a[i][4 * j] = v.x; r.a[i][4 * j + 1] = v.y; r.a[i][4 * j + 2] = v.z; r.a[i][4 * j + 3] = v.w;
      }
    }
  };
  int tile = blockIdx.x * kF16Warps + warp;
  Rows cur, nxt;
  fetch(tile, cur);
  fetch(tile + warps, nxt);
  if (p.hist)
    for (int b = tid; b < kHistBins; b += kF16Warps * 32) sh_hist[b] = 0;
  auto prepare = [&](int h, float (&v)[4], float w) {
    if (p.cs) {
      idx_prep_head(v, p.cs, p.actq, lane);
      w *= p.wscale;
      if (blockIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) p.q_out[(size_t)h * kIdxDim + 32 * i + lane] = v[i];
        if (lane == 0) p.w_out[h] = w;
      }
    }
    float scale = 1.f, back = 1.f;
    if (TERMS > 2) {
      float amax = 0.f;
#pragma unroll
      for (int i = 0; i < 4; i++) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      const int e = (int)((__float_as_uint(amax) >> 23) & 0xFF) - 127;     // largest value to [2^14, 2^15)
      if (e > -100 && e < 100) { scale = pow2i(14 - e); back = pow2i(e - 14); }
    }
    if (lane == 0) { wsh[h] = w; scl[h] = back; }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      // dim 32 i + lane: thread t = i of column h % 8, k-step lane / 4, half lane % 4 of the pair of words
      float rest = v[i] * scale;
#pragma unroll
      for (int c = 0; c < TERMS; c++) {
        const __half x = __float2half_rn(rest);
        rest -= __half2float(x);
        Bh[(((c * NTH + (h >> 3)) * 8 + (lane >> 2)) * 32 + (h & 7) * 4 + i) * 4 + (lane & 3)] = x;
      }
    }
  };
  // the warp's heads, three at a time so that one round trip serves them
  constexpr int kAtOnce = 3;
  for (int h0 = warp; h0 < H; h0 += kAtOnce * kF16Warps) {
    float qv[kAtOnce][4], wv[kAtOnce];
#pragma unroll
    for (int c = 0; c < kAtOnce; c++) {
      const int h = min(h0 + c * kF16Warps, H - 1);
#pragma unroll
      for (int i = 0; i < 4; i++) qv[c][i] = p.q[(size_t)h * kIdxDim + 32 * i + lane];
      wv[c] = p.w[h];
    }
#pragma unroll
    for (int c = 0; c < kAtOnce; c++) {
      const int h = h0 + c * kF16Warps;
      if (h >= H) break;
      prepare(h, qv[c], wv[c]);
    }
  }
  __syncthreads();
  for (; tile < ntiles; tile += warps) {
    Rows far;
    fetch(tile + 2 * warps, far);
    uint32_t A[2][16];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 8; j++) {
        if (FP8IN) {
          const uint32_t wd = cur.a[i][j];
          const __half2_raw lo2 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(wd & 0xFFFFu), __NV_E4M3);
          const __half2_raw hi2 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(wd >> 16), __NV_E4M3);
          A[i][2 * j] = (uint32_t)lo2.x | ((uint32_t)lo2.y << 16);
          A[i][2 * j + 1] = (uint32_t)hi2.x | ((uint32_t)hi2.y << 16);
        } else {
          A[i][2 * j] = cur.a[i][2 * j]; A[i][2 * j + 1] = cur.a[i][2 * j + 1];
        }
      }
    float s0 = 0.f, s1 = 0.f;
    // A loop: unrolled, its code comes cold from memory, which only calls of many keys make up for (a block takes 28416 keys at a time; us,
    // loop / unrolled: 1500 keys 21.9 / 22.0, 20000 24.9 / 25.2, 50003 31.1 / 31.0, 100000 36.0 / 35.2, 200000 45.1 / 43.7).
#pragma unroll 1
    for (int n2 = 0; n2 < NTH; n2 += 2) {
      // Every MMA truncates its sum: the smallest terms go first, so that only the last term's do so at the sum's full size, and
      // the two halves of K are summed apart.  (Terms inside the K steps, one chain: 4.0e-7 from float64 instead of the 2.2e-7 of
      // 128 rounded fp32 additions.)  Two tiles of heads at a time: four chains of dependent MMAs side by side.
      float c[2][2][4] = {};
#pragma unroll
      for (int term = TERMS - 1; term >= 0; term--)
#pragma unroll
        for (int s = 0; s < 4; s++) {
          uint2 b[2][2];
#pragma unroll
          for (int q = 0; q < 2; q++)
#pragma unroll
            for (int hf = 0; hf < 2; hf++) b[q][hf] = Bs[((term * NTH + n2 + q) * 8 + s + 4 * hf) * 32 + lane];
#pragma unroll
          for (int hf = 0; hf < 2; hf++)
#pragma unroll
            for (int q = 0; q < 2; q++)
              mma_f16(c[q][hf], A[0][2 * s + 8 * hf], A[1][2 * s + 8 * hf], A[0][2 * s + 8 * hf + 1], A[1][2 * s + 8 * hf + 1], b[q][hf].x, b[q][hf].y);
        }
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int nt = n2 + q;
        float r[4];
#pragma unroll
        for (int i = 0; i < 4; i++) r[i] = c[q][0][i] + c[q][1][i];
        const float2 w = *reinterpret_cast<const float2*>(&wsh[nt * 8 + 2 * t]);
        if (TERMS > 2) {
          const float2 f = *reinterpret_cast<const float2*>(&scl[nt * 8 + 2 * t]);
          r[0] *= f.x; r[1] *= f.y; r[2] *= f.x; r[3] *= f.y;
        }
        s0 += fmaxf(r[0], 0.f) * w.x + fmaxf(r[1], 0.f) * w.y;
        s1 += fmaxf(r[2], 0.f) * w.x + fmaxf(r[3], 0.f) * w.y;
      }
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1); s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1); s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    if (t == 0) {                                    // lanes 0, 4, ..., 28 hold the 16 scores of the tile
      const int k0 = tile * 16 + g, k1 = k0 + 8;
      if (LIST && cur.key[0] < 0) s0 = -INFINITY;
      if (LIST && cur.key[1] < 0) s1 = -INFINITY;
      if (k0 < p.n) p.scores[k0] = s0;
      if (k1 < p.n) p.scores[k1] = s1;
      if (p.hist) {   // neighbouring scores mostly share a bin: one shared-memory atomic per distinct bin per warp
        const uint32_t b0 = (k0 < p.n && selectable(s0)) ? order_key(s0) >> 20 : 0xFFFFFFFFu;
        const uint32_t b1 = (k1 < p.n && selectable(s1)) ? order_key(s1) >> 20 : 0xFFFFFFFFu;
        const unsigned m0 = __match_any_sync(0x11111111u, b0), m1 = __match_any_sync(0x11111111u, b1);
        if (b0 != 0xFFFFFFFFu && lane == __ffs(m0) - 1) atomicAdd(&sh_hist[b0], (unsigned)__popc(m0));
        if (b1 != 0xFFFFFFFFu && lane == __ffs(m1) - 1) atomicAdd(&sh_hist[b1], (unsigned)__popc(m1));
      }
    }
    cur = nxt; nxt = far;
  }
  if (p.hist) hist_flush(sh_hist, p.hist, tid, kF16Warps * 32);
}

// ---------------------------------------------------------------- exact top-k
struct TopkCtl { unsigned n_sel, n_cand, ticket, pad1; };

__global__ void topk_hist_kernel(const float* sc, int n, unsigned* hist) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ unsigned sh[kHistBins];
  for (int b = threadIdx.x; b < kHistBins; b += blockDim.x) sh[b] = 0;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float f = sc[i];
    if (selectable(f)) atomicAdd(&sh[order_key(f) >> 20], 1u);
  }
  hist_flush(sh, hist, threadIdx.x, blockDim.x);
}

// threshold bin: the highest bin b with (count of bins > b) < k <= (count of bins >= b); -1 when fewer than k finite
// scores exist (everything is selected).  Computed by every block of the compaction and by the final block.
// Inclusive scan of one value per thread over the block (a multiple of 32 threads, at most 1024): warp shuffles, then
// the warp totals.  `wsum` is 32 words of shared memory; the caller synchronises before reusing it.
__device__ __forceinline__ unsigned block_scan_incl(unsigned v, unsigned* wsum, unsigned* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    unsigned s = lane < nw ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    wsum[lane] = s;
  }
  __syncthreads();
  *total = wsum[nw - 1];
  return x + (warp ? wsum[warp - 1] : 0u);
}

// The thread's run of bins, from the top (blocks of kTopkThreads): issued early, consumed by threshold_from().
constexpr int kTopkThreads = 1024;                 // block size of the selection kernels
constexpr int kBinsPerThread = kHistBins / kTopkThreads;
struct BinRun { unsigned c[kBinsPerThread]; };
__device__ __forceinline__ void threshold_load(const unsigned* hist, BinRun& r) {
#pragma unroll
  for (int j = 0; j < kBinsPerThread; j++) r.c[j] = __ldcg(hist + (kHistBins - 1 - (threadIdx.x * kBinsPerThread + j)));
}
// count_out (may be null): the population of the threshold bin itself
__device__ __forceinline__ int threshold_from(const BinRun& r, int k, unsigned* sh /* [1024] */, unsigned* above_out, unsigned* count_out) {
  const int tid = threadIdx.x;
  constexpr int per = kBinsPerThread;
  unsigned mine = 0;
#pragma unroll
  for (int j = 0; j < kBinsPerThread; j++) mine += r.c[j];
  unsigned total;
  const unsigned incl = block_scan_incl(mine, sh, &total), excl = incl - mine;
  __shared__ int res_bin;
  __shared__ unsigned res_above, res_count;
  if (tid == 0) { res_bin = -1; res_above = total; res_count = 0; }
  __syncthreads();
  if (excl < (unsigned)k && incl >= (unsigned)k) {   // the threshold lies in this thread's run
    unsigned run = excl;
#pragma unroll
    for (int j = 0; j < kBinsPerThread; j++) {
      if (run + r.c[j] >= (unsigned)k) { res_bin = kHistBins - 1 - (tid * per + j); res_above = run; res_count = r.c[j]; break; }
      run += r.c[j];
    }
  }
  __syncthreads();
  *above_out = res_above;
  if (count_out) *count_out = res_count;
  return res_bin;
}
__device__ int threshold_bin(const unsigned* hist, int k, unsigned* sh /* [1024] */, unsigned* above_out) {
  BinRun r;
  threshold_load(hist, r);
  return threshold_from(r, k, sh, above_out, nullptr);
}

// forward declaration: the last step, run by the compaction block that finishes last
__device__ void topk_final_block(const float* sc, int n, int k, unsigned* hist, unsigned* fine, TopkCtl* ctl,
                                 const int* sel, const uint2* cand, int* out, int bm_words, const int* pos_map,
                                 bool have_bin, int bin_known, unsigned above_known);

// Compaction over the whole grid (blocks of 1024 threads), then the exact finish in the block that takes the last
// ticket: one launch for the whole selection after the histogram.
__global__ void __launch_bounds__(kTopkThreads, 2) topk_select_kernel(const float* sc, int n, int k, unsigned* hist, unsigned* fine,
                                                           TopkCtl* ctl, int* sel, uint2* cand, int* out, int bm_words,
                                                           int fused, const int* pos_map) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ unsigned sh[1024];
  __shared__ unsigned sh_fine[kHistBins];
  __shared__ int is_last;
  const int lane = threadIdx.x & 31;
  const int per_block = (n + gridDim.x - 1) / gridDim.x;
  const int i0 = blockIdx.x * per_block, i1 = min(n, i0 + per_block);
  // the first trip's scores (usually the only trip) are requested together with the histogram, ahead of the scan
  float f0[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int i = i0 + j * (int)blockDim.x + (int)threadIdx.x;
    f0[j] = i < i1 ? sc[i] : -INFINITY;
  }
  unsigned above;
  const int bstar = threshold_bin(hist, k, sh, &above);
  for (int b = threadIdx.x; b < kHistBins; b += blockDim.x) sh_fine[b] = 0;
  __syncthreads();
  // The block's picks are collected in shared memory first (dynamic region: per_block ints for the outright selections,
  // per_block (index, key) pairs for the threshold bin's members) and appended to the global lists with ONE atomic per
  // kind and block: thousands of same-address atomics from individual warps were the bulk of this kernel's time.
  extern __shared__ unsigned dyn_smem[];
  int* sel_buf = reinterpret_cast<int*>(dyn_smem);
  uint2* cand_buf = reinterpret_cast<uint2*>(dyn_smem + ((per_block + 1) & ~1));
  __shared__ unsigned s_n1, s_n2, s_g1, s_g2;
  if (threadIdx.x == 0) { s_n1 = 0; s_n2 = 0; }
  __syncthreads();
  // 4 independent loads per thread per trip
  for (int base = i0; base < i1; base += blockDim.x * 4) {
    float f[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = base + j * (int)blockDim.x + (int)threadIdx.x;
      f[j] = base == i0 ? f0[j] : (i < i1 ? sc[i] : -INFINITY);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int i = base + j * (int)blockDim.x + (int)threadIdx.x;
      int kind = 0;   // 1 = selected outright, 2 = threshold-bin candidate
      uint32_t key = 0;
      if (i < i1 && selectable(f[j])) {
        key = order_key(f[j]);
        const int b = (int)(key >> 20);
        kind = b > bstar ? 1 : (b == bstar ? 2 : 0);
        if (kind == 2) atomicAdd(&sh_fine[(key >> 8) & 0xFFFu], 1u);   // next 12 key bits of the threshold bin's members
      }
      const unsigned m1 = __ballot_sync(0xffffffffu, kind == 1), m2 = __ballot_sync(0xffffffffu, kind == 2);
      unsigned b1 = 0, b2 = 0;
      if (lane == 0) {
        if (m1) b1 = atomicAdd(&s_n1, (unsigned)__popc(m1));
        if (m2) b2 = atomicAdd(&s_n2, (unsigned)__popc(m2));
      }
      b1 = __shfl_sync(0xffffffffu, b1, 0);
      b2 = __shfl_sync(0xffffffffu, b2, 0);
      const unsigned lt = (1u << lane) - 1u;
      if (kind == 1) sel_buf[b1 + __popc(m1 & lt)] = i;
      if (kind == 2) cand_buf[b2 + __popc(m2 & lt)] = make_uint2((unsigned)i, key);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    s_g1 = s_n1 ? atomicAdd(&ctl->n_sel, s_n1) : 0u;
    s_g2 = s_n2 ? atomicAdd(&ctl->n_cand, s_n2) : 0u;
  }
  __syncthreads();
  for (unsigned i = threadIdx.x; i < s_n1; i += blockDim.x) { const unsigned pos = s_g1 + i; if (pos < 2048u) sel[pos] = sel_buf[i]; }
  for (unsigned i = threadIdx.x; i < s_n2; i += blockDim.x) cand[s_g2 + i] = cand_buf[i];
  hist_flush(sh_fine, fine, threadIdx.x, blockDim.x);
  if (!fused) return;
  // the block that takes the last ticket sees every other block's lists and finishes the selection
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  topk_final_block(sc, n, k, hist, fine, ctl, sel, cand, out, bm_words, pos_map, true, bstar, above);
}

// the last step as its own launch (one block)
__global__ void __launch_bounds__(kTopkThreads) topk_final_kernel(const float* sc, int n, int k, unsigned* hist, unsigned* fine,
                                                          TopkCtl* ctl, const int* sel, const uint2* cand, int* out, int bm_words,
                                                          const int* pos_map) {
  pdl_launch_dependents();
  pdl_wait();
  topk_final_block(sc, n, k, hist, fine, ctl, sel, cand, out, bm_words, pos_map, false, 0, 0u);
}

// The selection's last step, run by ONE block of 1024 threads (the compaction block that finishes last).
// out[k] ascending, -1 padded.  Resets the histograms and ctl for the next call.
// pos_map != null: the scores are indexed by virtual position 8 * i + j standing for key pos_map[i] * 8 + j (candidate
// list, ascending); the output lists key indices (still ascending, as the list is).
// have_bin: the caller already holds the coarse threshold bin and the count above it (the compaction computed them).
__device__ void topk_final_block(const float* sc, int n, int k, unsigned* hist, unsigned* fine, TopkCtl* ctl,
                                 const int* sel, const uint2* cand, int* out, int bm_words, const int* pos_map,
                                 bool have_bin, int bin_known, unsigned above_known) {
  __shared__ unsigned sh[1024];
  __shared__ int buf[2048];
  __shared__ unsigned long long c2[1024];
  __shared__ unsigned s_cnt, s_c2, s_need, s_digit;
  extern __shared__ unsigned bitmap[];          // bm_words words when the bitmap path is used (n <= 32 * bm_words)
  const int tid = threadIdx.x, NT = blockDim.x;   // kTopkThreads
  // chosen indices go into a bitmap of the n positions (read back in ascending order: no sort), or, for very long
  // inputs that do not fit shared memory, into buf[] which is then sorted
  auto emit = [&](unsigned idx) {
    if (bm_words) atomicOr(&bitmap[idx >> 5], 1u << (idx & 31));
    else { const unsigned pos = atomicAdd(&s_cnt, 1u); if (pos < 2048u) buf[pos] = (int)idx; }
  };
  // Every global read of the finish that does not depend on another one is requested here, together: the counters,
  // the fine histogram, the first 2 NT outright selections and the first NT threshold-bin candidates.  One memory
  // latency instead of four in a row on what is the serial tail of the selection.
  const unsigned n_sel = *reinterpret_cast<volatile unsigned*>(&ctl->n_sel);
  const unsigned n_cand = *reinterpret_cast<volatile unsigned*>(&ctl->n_cand);
  BinRun fr;
  threshold_load(fine, fr);
  const int sel0 = __ldcg(sel + min(tid, 2047)), sel1 = __ldcg(sel + min(tid + NT, 2047));
  const uint2 cand0 = __ldcg(cand + min(tid, max(n, 1) - 1));
  for (int i = tid; i < bm_words; i += NT) bitmap[i] = 0;
  unsigned above = above_known;
  const int bstar = have_bin ? bin_known : threshold_bin(hist, k, sh, &above);
  for (int i = tid; i < 2048; i += NT) buf[i] = 0x7fffffff;
  if (tid == 0) { s_cnt = 0; s_c2 = 0; }
  __syncthreads();
  for (unsigned i = tid, j = 0; i < n_sel && i < 2048u; i += NT, j++)
    emit((unsigned)(j == 0 ? sel0 : j == 1 ? sel1 : __ldcg(sel + i)));
  if (bstar >= 0 && n_cand > 0) {
    const unsigned need = (unsigned)k - above;   // how many of the threshold bin's members are taken
    unsigned above2, m2;
    const int fstar = threshold_from(fr, (int)need, sh, &above2, &m2);
    if (fstar >= 0 && m2 <= 1024u) {
      const unsigned need2 = need - above2;
#pragma unroll 4
      for (unsigned i = tid; i < n_cand; i += NT) {
        const uint2 cd = i == (unsigned)tid ? cand0 : __ldcg(cand + i);
        const unsigned idx = cd.x;
        const uint32_t key = cd.y;
        const int fb = (int)((key >> 8) & 0xFFFu);
        if (fb > fstar) {
          emit(idx);
        } else if (fb == fstar) {
          const unsigned pos = atomicAdd(&s_c2, 1u);
          if (pos < 1024u) c2[pos] = ((unsigned long long)(0xFFu - (key & 0xFFu)) << 32) | idx;   // ascending = better
        }
      }
      __syncthreads();
      const unsigned m = min(s_c2, 1024u);
      for (unsigned e2 = tid; e2 < m; e2 += NT) {
        const unsigned long long mine = c2[e2];
        unsigned rank = 0;
        for (unsigned j = 0; j < m; j++) rank += c2[j] < mine;
        if (rank < need2) emit((unsigned)(mine & 0xFFFFFFFFu));
      }
      __syncthreads();
    } else {
      // radix select (descending) on the low 20 bits of the key: find T = the need-th largest key among candidates
      unsigned prefix = 0, mask = 0, remaining = need;
      for (int shift = 12; shift >= -4; shift -= 8) {
        const int sft = shift < 0 ? 0 : shift;
        const unsigned dmask = shift < 0 ? 0xFu : 0xFFu;
        for (int b = tid; b < 256; b += NT) sh[b] = 0;
        __syncthreads();
        for (unsigned i = tid; i < n_cand; i += NT) {
          const unsigned key = __ldcg(cand + i).y & 0xFFFFFu;
          if ((key & mask) == prefix) atomicAdd(&sh[(key >> sft) & dmask], 1u);
        }
        __syncthreads();
        if (tid == 0) {
          unsigned run = 0;
          int d = (int)dmask;
          for (; d > 0; d--) {
            if (run + sh[d] >= remaining) break;
            run += sh[d];
          }
          s_digit = (unsigned)d; s_need = remaining - run;
        }
        __syncthreads();
        prefix |= s_digit << sft;
        mask |= dmask << sft;
        remaining = s_need;
        __syncthreads();
      }
      const unsigned T = prefix;         // exact threshold key (low 20 bits); `remaining` members equal to T are taken
      // ties at T: take the `remaining` lowest indices.  Radix select (ascending) on the index, 3 x 8 bits (n <= 2^24).
      unsigned ip = 0, im = 0, irem = remaining;
      for (int shift = 16; shift >= 0; shift -= 8) {
        for (int b = tid; b < 256; b += NT) sh[b] = 0;
        __syncthreads();
        for (unsigned i = tid; i < n_cand; i += NT) {
          const uint2 cd = __ldcg(cand + i);
          if ((cd.y & 0xFFFFFu) == T && (cd.x & im) == ip) atomicAdd(&sh[(cd.x >> shift) & 0xFFu], 1u);
        }
        __syncthreads();
        if (tid == 0) {
          unsigned run = 0;
          int d = 0;
          for (; d < 255; d++) {
            if (run + sh[d] >= irem) break;
            run += sh[d];
          }
          s_digit = (unsigned)d; s_need = irem - run;
        }
        __syncthreads();
        ip |= s_digit << shift;
        im |= 0xFFu << shift;
        irem = s_need;
        __syncthreads();
      }
      const unsigned idxT = ip;          // members equal to T with index <= idxT are taken
      for (unsigned i = tid; i < n_cand; i += NT) {
        const uint2 cd = __ldcg(cand + i);
        const unsigned idx = cd.x;
        const unsigned key = cd.y & 0xFFFFFu;
        if (key > T || (key == T && idx <= idxT)) emit(idx);
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if (bm_words) {
    // ascending read-out: every thread owns a contiguous run of bitmap words; an exclusive scan of the run
    // populations gives each run its offset in the output
    const int per = (bm_words + NT - 1) / NT;
    const int w0 = min(bm_words, tid * per), w1 = min(bm_words, w0 + per);
    unsigned cnt = 0;
    for (int w = w0; w < w1; w++) cnt += __popc(bitmap[w]);
    unsigned total;
    unsigned pos = block_scan_incl(cnt, sh, &total) - cnt;
    for (int w = w0; w < w1; w++) {
      unsigned m = bitmap[w];
      while (m) {
        const int bit = __ffs(m) - 1;
        m &= m - 1;
        if (pos < (unsigned)k) { const int v = w * 32 + bit; out[pos] = pos_map ? pos_map[v >> 3] * 8 + (v & 7) : v; }
        pos++;
      }
    }
    for (int i = tid + (int)min(total, (unsigned)k); i < k; i += NT) out[i] = -1;
  } else {
    const unsigned filled = min(s_cnt, 2048u);
    // bitonic sort of the used power-of-two prefix, ascending (unused slots hold INT_MAX)
    int P = 32;
    while (P < (int)filled) P <<= 1;
    for (int size = 2; size <= P; size <<= 1)
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int i = tid; i < P / 2; i += NT) {
          const int lo = 2 * i - (i & (stride - 1));
          const int hi = lo + stride;
          const bool up = ((lo & size) == 0);
          const int a = buf[lo], b2 = buf[hi];
          if ((a > b2) == up) { buf[lo] = b2; buf[hi] = a; }
        }
        __syncthreads();
      }
    for (int i = tid; i < k; i += NT) {
      const bool ok = i < (int)filled && buf[i] != 0x7fffffff;
      out[i] = !ok ? -1 : (pos_map ? pos_map[buf[i] >> 3] * 8 + (buf[i] & 7) : buf[i]);
    }
  }
  for (int b = tid; b < kHistBins; b += NT) { hist[b] = 0; fine[b] = 0; }
  if (tid == 0) { ctl->n_sel = 0; ctl->n_cand = 0; ctl->ticket = 0; }
  (void)n;
}

// ---- the same selection by ONE cluster of blocks, for inputs whose keys fit their registers (R per thread): no global lists, no
// tickets, no bitmap.  Every block holds a contiguous range of the positions, every warp a contiguous run of it, so the picks
// leave in ascending order at positions counted across the cluster.  The threshold is found from the coarse histogram (the
// scoring kernel's, or built here), then from a histogram of the next 12 key bits of the threshold bin's members, and only when
// that still cuts a bin from one of the last 8; each is summed over the blocks through distributed shared memory.
// Bound by the chain of cluster barriers and reads of the other blocks' shared memory.  2048 of 16384: 5 + 12 us as histogram,
// compaction and last block's finish, 10 so.
constexpr int kTcThreads = 1024, kTcBlocks = 8;
struct TcShared {
  unsigned h[kHistBins];                 // this block's histogram
  unsigned tot[kHistBins / kTcBlocks];           // its slice of the cluster's
  unsigned wsum[32], h8[256];
  unsigned slice, gt, eq;
  int bin, at;
  unsigned above, count, run, before_gt, before_eq, total;
};
// Bin (and count above it, and its own) in which the running count from the top reaches `need`, over `n` bins with thread i
// holding bin n - 1 - i; -1 when the total is below.  n <= 1024.
__device__ __forceinline__ void tc_scan(TcShared& s, unsigned v, int n, unsigned need, unsigned base) {
  const int tid = threadIdx.x;
  if (tid == 0) { s.bin = -1; s.above = 0; s.count = 0; }
  unsigned total;
  const unsigned incl = base + block_scan_incl(v, s.wsum, &total), excl = incl - v;
  if (tid < n && excl < need && incl >= need) { s.bin = n - 1 - tid; s.above = excl; s.count = v; }
  __syncthreads();
}
// The same over the cluster's sum of the blocks' 4096-bin histograms s.h (complete before the call).
__device__ __forceinline__ void tc_level(TcShared& s, cg::cluster_group& cl, int rank, unsigned need) {
  constexpr int C = kTcBlocks, per = kHistBins / C;
  const int tid = threadIdx.x, lane = tid & 31;
  cl.sync();
  unsigned v = 0;
  if (tid < per) {
#pragma unroll
    for (int c = 0; c < C; c++) v += cl.map_shared_rank(s.h, c)[rank * per + tid];
  }
  if (tid < per) s.tot[tid] = v;
  unsigned total;
  block_scan_incl(v, s.wsum, &total);
  if (tid == 0) s.slice = total;
  cl.sync();
  // which slice, from the top: lane l of one warp holds block C - 1 - l's
  if (tid < 32) {
    const unsigned x = lane < C ? *cl.map_shared_rank(&s.slice, C - 1 - lane) : 0u;
    unsigned incl = x;
#pragma unroll
    for (int o = 1; o < C; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, incl - x < need && incl >= need && lane < C);
    const unsigned run = __shfl_sync(0xffffffffu, incl - x, hit ? __ffs(hit) - 1 : 0);
    if (lane == 0) { s.at = hit ? C - __ffs(hit) : -1; s.run = run; }       // (without a hit nobody reads run)
  }
  __syncthreads();
  const int at = s.at;
  const unsigned run = s.run;
  v = at >= 0 && tid < per ? cl.map_shared_rank(s.tot, at)[per - 1 - tid] : 0u;
  tc_scan(s, v, per, need, run);
  if (tid == 0 && s.bin >= 0) s.bin += at * per;         // (no bin: nobody reads above)
  __syncthreads();
}
__global__ void __launch_bounds__(kTcThreads, 1) topk_cluster_kernel(const float* sc, int n, int k, unsigned* hist, int have_hist, int run_len,
                                                                     int* out, const int* pos_map) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ TcShared s;
  constexpr int R = 4, C = kTcBlocks;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int i0 = (rank * 32 + warp) * run_len;         // this warp's run of positions (a multiple of 32 long)
  BinRun hr;
  if (have_hist) threshold_load(hist, hr);
  uint32_t key[R];                                     // 0: not selectable (no finite score has key 0)
#pragma unroll
  for (int j = 0; j < R; j++) {
    const int i = i0 + 32 * j + lane;
    float f = -INFINITY;
    if (32 * j < run_len && i < n) f = sc[i];
    key[j] = selectable(f) ? order_key(f) : 0u;
  }
  for (int b = tid; b < kHistBins; b += kTcThreads) s.h[b] = 0;
  if (tid < 256) s.h8[tid] = 0;
  __syncthreads();
  // ---- the coarse threshold bin
  if (have_hist) {
    unsigned above, count;
    const int b = threshold_from(hr, k, s.wsum, &above, &count);
    if (tid == 0) { s.bin = b; s.above = above; s.count = count; }
    __syncthreads();
  } else {
#pragma unroll
    for (int j = 0; j < R; j++) {                      // (neighbouring scores mostly share a bin)
      if (32 * j >= run_len) break;
      const unsigned m = __match_any_sync(0xffffffffu, key[j] >> 20);
      if (key[j] && lane == __ffs(m) - 1) atomicAdd(&s.h[key[j] >> 20], (unsigned)__popc(m));
    }
    __syncthreads();
    tc_level(s, cl, rank, (unsigned)k);
    cl.sync();                                         // every block has read the others' histograms
    for (int b = tid; b < kHistBins; b += kTcThreads) s.h[b] = 0;
  }
  const int bstar = s.bin;
  uint32_t T = 0;                                      // keys above T are taken, and the `ties` lowest positions with key T
  unsigned ties = 0;
  if (bstar >= 0) {
    unsigned need = (unsigned)k - s.above;
    if (s.count == need) {
      T = ((uint32_t)bstar << 20) - 1u;                // the whole bin
      __syncthreads();
    } else {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < R; j++)
        if (key[j] && (int)(key[j] >> 20) == bstar) atomicAdd(&s.h[(key[j] >> 8) & 0xFFFu], 1u);
      __syncthreads();
      tc_level(s, cl, rank, need);
      const uint32_t pre = ((uint32_t)bstar << 12) | (uint32_t)s.bin;
      const bool whole = s.count == need - s.above;
      need -= s.above;
      __syncthreads();
      if (whole) {
        T = (pre << 8) - 1u;
      } else {
#pragma unroll
        for (int j = 0; j < R; j++)
          if (key[j] && (key[j] >> 8) == pre) atomicAdd(&s.h8[key[j] & 0xFFu], 1u);
        cl.sync();
        unsigned v = 0;
        if (tid < 256) {
#pragma unroll
          for (int c = 0; c < C; c++) v += cl.map_shared_rank(s.h8, c)[255 - tid];
        }
        tc_scan(s, v, 256, need, 0u);
        T = (pre << 8) | (uint32_t)s.bin;
        ties = need - s.above;
        if (s.count == ties) { T -= 1u; ties = 0; }
        __syncthreads();
      }
    }
  }
  // ---- counts of the warps' runs, then of the blocks before this one
  unsigned ng = 0, ne = 0;
#pragma unroll
  for (int j = 0; j < R; j++) {
    ng += __popc(__ballot_sync(0xffffffffu, key[j] > T));
    if (ties) ne += __popc(__ballot_sync(0xffffffffu, key[j] == T));
  }
  unsigned tg, te = 0;
  const unsigned bg = block_scan_incl(lane == 0 ? ng : 0u, s.wsum, &tg) - (lane == 0 ? ng : 0u);
  unsigned wg = __shfl_sync(0xffffffffu, bg, 0), we = 0;
  if (ties) {
    __syncthreads();
    const unsigned be = block_scan_incl(lane == 0 ? ne : 0u, s.wsum, &te) - (lane == 0 ? ne : 0u);
    we = __shfl_sync(0xffffffffu, be, 0);
  }
  if (tid == 0) { s.gt = tg; s.eq = te; }
  cl.sync();
  if (have_hist)
    for (int b = rank * kTcThreads + tid; b < kHistBins; b += C * kTcThreads) hist[b] = 0;      // every block has read it
  if (warp == 0) {
    const unsigned xg = lane < C ? *cl.map_shared_rank(&s.gt, lane) : 0u, xe = lane < C ? *cl.map_shared_rank(&s.eq, lane) : 0u;
    const unsigned pg = __reduce_add_sync(0xffffffffu, lane < rank ? xg : 0u), pe = __reduce_add_sync(0xffffffffu, lane < rank ? xe : 0u);
    const unsigned ag = __reduce_add_sync(0xffffffffu, xg), ae = __reduce_add_sync(0xffffffffu, xe);
    if (lane == 0) { s.before_gt = pg; s.before_eq = pe; s.total = ag + min(ae, ties); }
  }
  __syncthreads();
  wg += s.before_gt;
  we += s.before_eq;
#pragma unroll
  for (int j = 0; j < R; j++) {
    if (32 * j >= run_len) break;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned mg = __ballot_sync(0xffffffffu, key[j] > T), me = ties ? __ballot_sync(0xffffffffu, key[j] == T) : 0u;
    const unsigned e = we + __popc(me & lt), pos = wg + __popc(mg & lt) + min(e, ties);
    if (((mg >> lane) & 1u) || (((me >> lane) & 1u) && e < ties)) {
      const int v = i0 + 32 * j + lane;
      if (pos < (unsigned)k) out[pos] = pos_map ? pos_map[v >> 3] * 8 + (v & 7) : v;
    }
    wg += __popc(mg); we += __popc(me);
  }
  const unsigned filled = s.total;
  if (rank == 0)
    for (int i = tid + (int)min(filled, (unsigned)k); i < k; i += kTcThreads) out[i] = -1;
  cl.sync();                                           // nobody leaves while its shared memory is being read
}

// block maxima over `bs` consecutive scores; the newest (possibly partial) block is pinned to +inf
// (attn_ref.cpp:196-202)
__global__ void block_max_kernel(const float* sc, int len, int bs, float* out, int nb) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  float m = -INFINITY;
  for (int i = b * bs; i < min(len, (b + 1) * bs); i++) m = fmaxf(m, sc[i]);
  if (b == (len - 1) / bs) m = INFINITY;
  out[b] = m;
}

// ---------------------------------------------------------------- host side
size_t topk_scratch_bytes(int n_max) {
  return 2 * sizeof(unsigned) * kHistBins + 64 + sizeof(int) * 2048 + sizeof(uint2) * (size_t)std::max(n_max, 1);
}

// scratch layout: hist[4096] | fine[4096] | ctl (64 B) | sel[2048] | cand[n_max] as (index, key) pairs.  The histograms and ctl must be zero
// on entry; the final kernel leaves them zero again.
// What topk() refuses.  A caller whose scoring kernel adds into the scratch's histogram asks before that launch: a call that is
// refused leaves the scratch as it was, zeroed.
int topk_check(const float* sc, int n, int k, const int* out, const void* scratch, size_t scratch_bytes) {
  if (n < 0 || k <= 0 || k > 2048) return fail(kErrArg, "topk: n %d k %d (k must be 1..2048)", n, k);
  if (!out || !scratch || (n > 0 && !sc)) return fail(kErrArg, "topk: null pointer");
  if (scratch_bytes < topk_scratch_bytes(n)) return fail(kErrScratch, "topk: scratch too small");
  return kOk;
}

int topk(const float* sc, int n, int k, int* out, void* scratch, size_t scratch_bytes, bool hist_ready, const int* pos_map,
         cudaStream_t st) {
  const int bad = topk_check(sc, n, k, out, scratch, scratch_bytes);
  if (bad) return bad;
  unsigned* hist = reinterpret_cast<unsigned*>(scratch);
  unsigned* fine = hist + kHistBins;
  TopkCtl* ctl = reinterpret_cast<TopkCtl*>(fine + kHistBins);
  int* sel = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(ctl) + 64);
  uint2* cand = reinterpret_cast<uint2*>(sel + 2048);
  int dev = 0, sms = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  MSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // A cluster of 8 blocks up to 4 keys per thread, up to 2 where it has to make the histogram as well (2048 of 16384 11.8 us against
  // 12.7, of 24576 12.9 / 12.5, of 32768 14.3 / 12.8).  Beyond, the compaction over the whole GPU: larger clusters and more keys
  // per thread lose there (16 blocks: 50003 keys 16 against 12 us, 200000 24 against 16).
  if (n > 0 && n <= kTcBlocks * kTcThreads * (hist_ready ? 4 : 2)) {
    const int run = ((n + kTcBlocks * 32 - 1) / (kTcBlocks * 32) + 31) & ~31;
    MSB_CUDA(launch_clusters(topk_cluster_kernel, dim3(kTcBlocks), dim3(kTcThreads), kTcBlocks, 0, st, sc, n, k, hist, hist_ready ? 1 : 0,
                             run, out, pos_map));
    MSB_LAUNCH_CHECK("topk_cluster_kernel");
    return kOk;
  }
  // positions bitmap in shared memory for n up to 1M (128 KB); longer inputs use the sorting read-out
  const int bm_words = n <= (1 << 20) ? std::max(1, (n + 31) / 32) : 0;
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    MSB_CUDA(cudaFuncSetAttribute(topk_select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024));
    MSB_CUDA(cudaFuncSetAttribute(topk_final_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024));
    configured[dev & 63] = true;
  }
  // MSB_TOPK_FUSED=0: selection and read-out as two launches (topk_select_kernel + topk_final_kernel) instead of one
  static const int fused = getenv("MSB_TOPK_FUSED") ? atoi(getenv("MSB_TOPK_FUSED")) : 1;
  const int nthreads = kTopkThreads;
  // one element per thread and up to two blocks per SM: the per-block fixed work (threshold, fine histogram) is small
  // next to the latency of a longer per-thread loop
  int blocks = std::max(1, std::min(2 * sms * (1024 / nthreads), (n + nthreads - 1) / nthreads));
  // staging of a block's picks: per_block ints + per_block (index, key) pairs; blocks are added until that fits
  auto stage_of = [&](int nb) { const size_t pb = ((size_t)n + nb - 1) / nb; return ((pb + 1) & ~(size_t)1) * 4 + pb * 8 + 16; };
  while (stage_of(blocks) > 100 * 1024) blocks *= 2;
  const size_t stage_bytes = stage_of(blocks);
  if (n > 0 && !hist_ready) MSB_CUDA(launch_pdl(topk_hist_kernel, dim3(std::max(1, std::min(sms * 2, (n + 1023) / 1024))), dim3(256), 0, st, sc, n, hist));
  if (fused) {
    MSB_CUDA(launch_pdl(topk_select_kernel, dim3(blocks), dim3(nthreads), std::max((size_t)bm_words * 4, stage_bytes), st, sc, n, k, hist,
                        fine, ctl, sel, cand, out, bm_words, 1, pos_map));
  } else {
    if (n > 0) MSB_CUDA(launch_pdl(topk_select_kernel, dim3(blocks), dim3(nthreads), stage_bytes, st, sc, n, k, hist, fine, ctl, sel, cand, out, bm_words, 0, pos_map));
    MSB_CUDA(launch_pdl(topk_final_kernel, dim3(1), dim3(kTopkThreads), (size_t)bm_words * 4, st, sc, n, k, hist, fine, ctl,
                        (const int*)sel, (const uint2*)cand, out, bm_words, pos_map));
  }
  MSB_LAUNCH_CHECK("topk");
  return kOk;
}

int index_prep(const float* q_raw, const float* w_raw, const float* cs, int actq, int heads, float* q, float* w,
               cudaStream_t st) {
  if (heads <= 0 || !q_raw || !w_raw || !cs || !q || !w) return fail(kErrArg, "index_prep: bad arguments");
  MSB_CUDA(launch_pdl(idx_prep_kernel, dim3((heads + 3) / 4), dim3(128), 0, st, q_raw, w_raw, cs, actq, heads, idx_weight_scale(heads), q, w));
  MSB_LAUNCH_CHECK("idx_prep_kernel");
  return kOk;
}

template <bool FP8IN, int TERMS, bool LIST, int H>
static int launch_f16_heads(const IdxF16Params& p, int sms, int dev, cudaStream_t st) {
  auto kern = idx_score_f16_kernel<H, FP8IN, TERMS, LIST>;
  const size_t smem = (size_t)TERMS * (H / 8) * 8 * 32 * sizeof(uint2) + (p.hist ? kHistBins * sizeof(unsigned) : 0);
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    MSB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
    configured[dev & 63] = true;
  }
  const int grid = std::max(1, std::min(sms, (p.n + 16 * kF16Warps - 1) / (16 * kF16Warps)));
  MSB_CUDA(launch_pdl(kern, dim3(grid), dim3(kF16Warps * 32), smem, st, p));
  return kOk;
}
template <bool FP8IN, int TERMS, bool LIST>
static int launch_f16(const IdxF16Params& p, int heads, int sms, int dev, cudaStream_t st) {
  return heads == 64 ? launch_f16_heads<FP8IN, TERMS, LIST, 64>(p, sms, dev, st) : launch_f16_heads<FP8IN, TERMS, LIST, 32>(p, sms, dev, st);
}
// F16 keys, the query preparation inside (q_out / w_out are written); cand null: keys [0, len), else the candidate blocks' keys;
// hist may be null.  Arguments checked by the caller.
int index_scores_f16(const void* keys, int len, const float* q_raw, const float* w_raw, const float* cs, int actq, int heads, float* q_out,
                     float* w_out, const int* cand, int n_cand, float* scores, unsigned* hist, cudaStream_t st) {
  int dev = 0, sms = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  MSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const IdxF16Params p{(const uint8_t*)keys, q_raw, w_raw, cs, q_out, w_out, cand, scores, hist, len, cand ? 8 * n_cand : len, actq, idx_weight_scale(heads)};
  const int rc = cand ? launch_f16<false, 3, true>(p, heads, sms, dev, st) : launch_f16<false, 2, false>(p, heads, sms, dev, st);
  if (rc) return rc;
  MSB_LAUNCH_CHECK("idx_score_f16_kernel");
  return kOk;
}

int index_scores(int key_type, const void* keys, int len, const float* q, const float* w, int heads, float* scores,
                 unsigned* hist, int exact_query, cudaStream_t st) {
  if (len < 0 || (heads != 32 && heads != 64)) return fail(kErrArg, "index_scores: heads must be 32 or 64 (got %d)", heads);
  if (key_type != kKeyF16 && key_type != kKeyFp8) return fail(kErrType, "index_scores: key type %d", key_type);
  if (len == 0) return kOk;
  if (!keys || !q || !w || !scores || (reinterpret_cast<uintptr_t>(keys) & 15))
    return fail(kErrArg, "index_scores: null or misaligned pointer");
  int dev = 0, sms = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  MSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  IdxParams p{(const uint8_t*)keys, q, w, scores, hist, len};
  // MSB_IDX_LEGACY=1: FP8 scoring on mma.sync (idx_score_fp8_kernel) instead of the tcgen05 kernel
  static const bool legacy = getenv("MSB_IDX_LEGACY") && atoi(getenv("MSB_IDX_LEGACY")) != 0;
  if (key_type == kKeyFp8 && !exact_query && !legacy) return index_scores_tc(keys, len, q, w, heads, scores, hist, 0, nullptr, 0, nullptr, nullptr, nullptr, 0, st);
  if (key_type == kKeyFp8 && !exact_query) {
    const int grid = std::max(1, std::min(sms, (len + 16 * 12 - 1) / (16 * 12)));
    if (heads == 64) MSB_CUDA(launch_pdl(idx_score_fp8_kernel<64>, dim3(grid), dim3(384), 0, st, p));
    else MSB_CUDA(launch_pdl(idx_score_fp8_kernel<32>, dim3(grid), dim3(384), 0, st, p));
  } else {
    IdxF16Params f{(const uint8_t*)keys, q, w, nullptr, nullptr, nullptr, nullptr, scores, nullptr, len, len, 0, 1.f};
    const int rc = key_type == kKeyFp8 ? launch_f16<true, 2, false>(f, heads, sms, dev, st) : launch_f16<false, 2, false>(f, heads, sms, dev, st);
    if (rc) return rc;
  }
  MSB_LAUNCH_CHECK("idx_score_kernel");
  return kOk;
}

int block_max(const float* sc, int len, int bs, float* out, cudaStream_t st) {
  if (len <= 0 || bs <= 0 || !sc || !out) return fail(kErrArg, "block_max: bad arguments");
  const int nb = (len + bs - 1) / bs;
  MSB_CUDA(launch_pdl(block_max_kernel, dim3((nb + 255) / 256), dim3(256), 0, st, sc, len, bs, out, nb));
  MSB_LAUNCH_CHECK("block_max_kernel");
  return kOk;
}

}  // namespace msb
