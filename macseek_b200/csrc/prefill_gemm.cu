// Prefill projection GEMM on the 5th-generation tensor cores:  Y[n x rows] (+)= X16[n x cols] . W^T
// Replaces the reference's q_mm / q_mm_dense / q_deq_f16 Metal kernels (src/kernels/quant_mm.metal:87-154) behind
// ms::q::encode_matmul / encode_matmul_h / encode_f32_to_f16 (src/kernels/quant.hpp:37-46, quant.mm:189-248).
// Same arithmetic as the reference: activations and weights as half operands, fp32 accumulation.
//
// Two forms; mm_dense_us / mm_splits estimate which ends first:
//   mm_ts_kernel    short prompts: the raw blocks are decoded inside the kernel (ts_gemm.cuh), one launch
//   gemm_tc_kernel  the weight matrix is dequantised to half first (exactly the reference's values, rounded to half once) into
//                   caller-provided scratch, as the reference does for n >= 512 (quant.mm:225-240); the contraction is then one
//                   persistent kernel of block PAIRS: a 256 token x (up to 256) weight row tile, each block fetching half of
//                   either operand by TMA (128-byte swizzle) -> tcgen05.mma.cta_group::2 kind::f16 -> 128 fp32 accumulator rows
//                   per block in TMEM (two sets, so the epilogue of one tile overlaps the main loop of the next) -> tcgen05.ld
//                   -> Y.  Fetching the operands from L2 bounds it, hence the pairs: 32 KB per block and 128 x 256 x 64
//                   products instead of 48 (4096 x 4096 x 5120: 178 -> 150 us, 1.14 PFLOP/s).  Warp roles: 0..3 epilogue, 4 MMA
//                   issue (first block of the pair), 5 TMA.  The same kernel with single blocks, 128 tokens per tile, where 256
//                   leave more of the machine or of the last tile idle than the pairs save (gemm_shape).
// Every mbarrier wait is bounded.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cooperative_groups.h>
#include <algorithm>
#include <atomic>
#include "pair_gemm.cuh"

namespace msb {
namespace cg = cooperative_groups;

struct GemmParams {
  CUtensorMap a_map;   // X16 [n][cols] half, box 64 x 128
  CUtensorMap b_map;   // W16 [rows][cols] half, box 64 x bn / (blocks of a tile)
  float* y;            // [n][rows]
  int* status;
  int n, rows, cols, accumulate, bn;
};

// The projection's tiles: token tiles fastest, so that neighbouring pairs share a weight tile.
template <int G>
struct GemmProj {
  const GemmParams& p;
  int bn, mt, ntiles, kb;
  bool vec_ok;
  struct Tile { int a_row, b_row, col; };
  __device__ explicit GemmProj(const GemmParams& q) : p(q), bn(q.bn) {
    mt = (q.n + G * kGmBM - 1) / (G * kGmBM);
    ntiles = mt * ((q.rows + bn - 1) / bn);
    kb = (q.cols + kGmBK - 1) / kGmBK;
    vec_ok = q.rows % 4 == 0 && (reinterpret_cast<uintptr_t>(q.y) & 15) == 0;
  }
  __device__ int* status() const { return p.status; }
  __device__ void wait_before() const { pdl_wait(); }   // X16 (and W16) come from kernels that ran before
  __device__ void wait_after() const {}
  __device__ const CUtensorMap* a_map() const { return &p.a_map; }
  __device__ const CUtensorMap* b_map() const { return &p.b_map; }
  __device__ Tile tile(int t, int rank) const {
    const int m = t % mt, nn = t / mt;
    return Tile{(G * m + rank) * kGmBM, nn * bn + rank * (bn / G), nn * bn};
  }
  __device__ Tile tile_of_thread(int t, int rank) const { return tile(t, rank); }
  __device__ void epilogue(const Tile& tl, uint32_t taddr, int warp, int lane) const {
    const int token = tl.a_row + 32 * warp + lane;
#pragma unroll 1
    for (int c0 = 0; c0 < bn; c0 += 32) {
      uint32_t r[32];
      __syncwarp();                                    // lanes without a token come here early; the load is the whole warp's
      gm_ld32(taddr + c0, r);
      ts_wait_ld();
      const int col0 = tl.col + c0;
      if (token < p.n && col0 < p.rows) {
        float* dst = p.y + (size_t)token * p.rows + col0;
        if (vec_ok && col0 + 32 <= p.rows) {
#pragma unroll
          for (int q = 0; q < 8; q++) {
            float4 v = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]),
                                   __uint_as_float(r[4 * q + 3]));
            if (p.accumulate) {
              const float4 o = reinterpret_cast<const float4*>(dst)[q];
              v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
            }
            reinterpret_cast<float4*>(dst)[q] = v;
          }
        } else {
#pragma unroll
          for (int q = 0; q < 32; q++)
            if (col0 + q < p.rows) dst[q] = p.accumulate ? dst[q] + __uint_as_float(r[q]) : __uint_as_float(r[q]);
        }
      }
    }
  }
};
template <int G>
__global__ void __cluster_dims__(G, 1, 1) __launch_bounds__(kGmThreads, 1) gemm_tc_kernel(const __grid_constant__ GemmParams p) {
  gemm_body<G>(GemmProj<G>(p));
}

// ---------------------------------------------------------------- decoded weights as operand A
// The same product for short prompts, straight from the raw blocks (ts_gemm.cuh): no half copy of W.  Few activation rows make
// few tiles of 256 weight rows, so a tile's K is split over the blocks of a cluster; each leaves its fp32 sums in its own
// shared memory and the cluster adds them up in block order, every block a share of the activation rows (no second launch, no
// atomics, the same result every time).
struct MmTsParams {
  CUtensorMap a[4];           // X16 [n][cols] half, boxes of 16, 32, 64, 128 rows x 64
  const uint8_t* w;
  float* y;                   // [n][rows]
  int n, rows, cols, accumulate;
  int chunks, per;            // activation rows: chunks of `per` (the last may be short)
  int row_tiles, splits;
  Tables tb;
};
template <int T>
struct MmTs {
  const MmTsParams& p;
  int ntiles;
  float* part;                // this block's sums [m][256] in shared memory (splits > 1)
  static constexpr bool kLateTrigger = false, kSingle = TsPiece<T>::kK == kTsBK;
  // A tile is a few divisions here; finding it anew is sooner, except where the decoders leave no registers for it (speed against the
  // kernel before, shared memory / anew: IQ4_NL 0.993 / 1.006, IQ1_S 1.026 / 1.037, BF16 0.995 / 1.006, F16 1.000 / 1.006, IQ2_XXS 1.029 /
  // 1.030; Q8_0 1.017 / 1.003, Q6_K 1.013 / 1.001, Q5_K 1.006 / 1.000; 28 shapes each of 17 to 128 tokens).
  static constexpr bool kNextInSmem = T == Q8_0 || T == Q6_K || T == Q5_K;
  template <int U> static constexpr bool kHas = U == T;
  __device__ bool has_type(int t) const { return t == T; }
  __device__ const CUtensorMap* a_map(int i) const { return &p.a[i]; }
  __device__ void setup(uint8_t*, int) {}
  __device__ TsTile tile_of_thread(int t) const { return tile(t); }
  // splits innermost (a cluster), then the activation chunks (they share weight rows)
  __device__ TsTile tile(int t) const {
    constexpr int PB2 = 2 * TsPiece<T>::kK / kTsBK;      // K blocks of a pair of pieces
    const int s = t % p.splits, q = t / p.splits, c = q % p.chunks, r = q / p.chunks;
    const int kb = p.cols / kTsBK, pairs = (kb + PB2 - 1) / PB2;
    const int k0 = (int)((int64_t)pairs * s / p.splits) * PB2, k1 = min(kb, (int)((int64_t)pairs * (s + 1) / p.splits) * PB2);
    return TsTile{0, c * p.per, min(p.per, p.n - c * p.per), 256 * r, k0, k1 - k0, T};
  }
  __device__ uint32_t row_size(int) const { return (uint32_t)row_bytes(T, p.cols); }
  __device__ const uint8_t* rows(const TsTile& tl, int half, int quarter, int& live) const {
    const uint32_t rb = row_size(T);
    const int r0 = min(tl.n0 + 128 * half + 32 * quarter, p.rows - 1);
    live = min(32, p.rows - r0);
    return p.w + (size_t)r0 * rb;
  }
  __device__ void epilogue(const TsTile& tl, uint32_t d0, uint32_t d1, int quarter, int lane) const {
    const int in = 32 * quarter + lane;
    for (int c0 = 0; c0 < tl.m; c0 += 16) {
#pragma unroll
      for (int hf = 0; hf < 2; hf++) {
        uint32_t r[16];
        __syncwarp();                                  // (lanes beyond the last row)
        ts_ld16((hf ? d1 : d0) + c0, r);
        ts_wait_ld();
        if (p.splits > 1) {
#pragma unroll
          for (int q = 0; q < 16; q++)
            if (c0 + q < tl.m) part[(c0 + q) * 256 + 128 * hf + in] = __uint_as_float(r[q]);
        } else {
          const int col = tl.n0 + 128 * hf + in;
          float* dst = p.y + (size_t)(tl.row0 + c0) * p.rows + col;
          if (col < p.rows) {
#pragma unroll
            for (int q = 0; q < 16; q++)
              if (c0 + q < tl.m) {
                float v = __uint_as_float(r[q]);
                if (p.accumulate) v += dst[(size_t)q * p.rows];
                dst[(size_t)q * p.rows] = v;
              }
          }
        }
      }
    }
  }
};
template <int T>
// Bound by a block's producers and its start and end: 100 activation rows of a 5120 x 4096 Q6_K matrix take 23 us (conversion
// and GEMM 49 before, 39 with the block-pair GEMM), of IQ1_S 18, of BF16 19 (116 before).
__global__ void __launch_bounds__(kTsThreads, 1) mm_ts_kernel(const __grid_constant__ MmTsParams p) {
  // the sums take the place of the activation ring, the tables and the staged pieces: all of them have been read when the last
  // MMA has finished, which is when the epilogue starts (one tile per block when splits > 1)
  const uint32_t base = ((smem_u32(ts_smem_raw) + 1023u) & ~1023u) + 1024u;
  static_assert(kTsRing * kTsSlotBytes + kTsLutBytes + kTsRawBytes >= kTsMaxN * 256 * 4, "the sums fit");
  MmTs<T> pr{p, p.row_tiles * p.chunks * p.splits, reinterpret_cast<float*>(ts_smem_raw + (base - smem_u32(ts_smem_raw)))};
  ts_gemm_body(pr, p.tb);
  if (p.splits == 1) return;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  const TsTile tl = pr.tile((int)blockIdx.x);
  const int rank = (int)cl.block_rank();
  const bool vec = p.rows % 4 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
  for (int i = threadIdx.x; ; i += kTsThreads) {
    const int j = (i >> 6) * p.splits + rank, c = 4 * (i & 63);
    if (j >= tl.m) break;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < p.splits; s++) {
      const float4 v = *reinterpret_cast<const float4*>(cl.map_shared_rank(pr.part, s) + j * 256 + c);
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
    const int col = tl.n0 + c;
    float* dst = p.y + (size_t)(tl.row0 + j) * p.rows + col;
    if (vec) {
      if (col >= p.rows) continue;
      if (p.accumulate) {
        const float4 o = *reinterpret_cast<const float4*>(dst);
        a.x += o.x; a.y += o.y; a.z += o.z; a.w += o.w;
      }
      *reinterpret_cast<float4*>(dst) = a;
    } else {
      const float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (col + q < p.rows) dst[q] = p.accumulate ? dst[q] + v[q] : v[q];
    }
  }
  cl.sync();                                              // nobody leaves while its sums are being read
}

// ---------------------------------------------------------------- operand preparation
// weights -> half, the reference's dequantised value rounded to half once (q_deq_f16, quant_mm.metal:131-154)
template <int T>
__global__ void dequant_f16_kernel(const uint8_t* __restrict__ src, __half* __restrict__ out, int64_t n8, Tables tb) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  constexpr int per_block = block_elems(T) / 8;
  const uint8_t* blk = src + (i / per_block) * block_bytes(T);
  float y[8];
  dequant8<T>(blk, (int)(i % per_block), tb, y);
  __half2 h[4];
#pragma unroll
  for (int k = 0; k < 4; k++) h[k] = __floats2half2_rn(y[2 * k], y[2 * k + 1]);
  *reinterpret_cast<uint4*>(out + 8 * i) = *reinterpret_cast<uint4*>(h);
}
// the same for a group of equally sized matrices in one launch (blockIdx.y = matrix; srcs[g] = its device address, its
// half copy at out + g * count): a few-microsecond launch per 8 M-weight matrix never reaches the memory system's pace
template <int T>
__global__ void dequant_f16_group_kernel(const uint64_t* __restrict__ srcs, __half* __restrict__ out, int64_t n8, Tables tb) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  const uint8_t* src = reinterpret_cast<const uint8_t*>(srcs[blockIdx.y]);
  constexpr int per_block = block_elems(T) / 8;
  const uint8_t* blk = src + (i / per_block) * block_bytes(T);
  float y[8];
  dequant8<T>(blk, (int)(i % per_block), tb, y);
  __half2 h[4];
#pragma unroll
  for (int k = 0; k < 4; k++) h[k] = __floats2half2_rn(y[2 * k], y[2 * k + 1]);
  *reinterpret_cast<uint4*>(out + ((int64_t)blockIdx.y * n8 + i) * 8) = *reinterpret_cast<uint4*>(h);
}
// dense sources: part 0 = half(w); part 1 (F32 only) = half(w - half(w)), the second term of a two-pass product.  Eight values
// per thread (one 8-byte value per thread took 83 us for 21 M BF16 weights, this 14); src at any alignment of its type.
template <int T>
__global__ void __launch_bounds__(256) dense_f16_kernel(const uint8_t* __restrict__ src, __half* __restrict__ out, int64_t n8, int part) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  constexpr int B = block_bytes(T);
  uint32_t raw[2 * B];
  const uint8_t* s = src + i * 8 * B;
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
    for (int k = 0; k < B / 2; k++) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(s) + k);
      raw[4 * k] = v.x; raw[4 * k + 1] = v.y; raw[4 * k + 2] = v.z; raw[4 * k + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 2 * B; k++)
      raw[k] = T == F32 ? __ldg(reinterpret_cast<const uint32_t*>(s) + k)
                        : __ldg(reinterpret_cast<const uint16_t*>(s) + 2 * k) | ((uint32_t)__ldg(reinterpret_cast<const uint16_t*>(s) + 2 * k + 1) << 16);
  }
  __half h[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const float w = T == F32 ? __uint_as_float(raw[k % (2 * B)]) : __uint_as_float(k & 1 ? raw[k >> 1] & 0xFFFF0000u : raw[k >> 1] << 16);
    h[k] = __float2half_rn(w);
    if (T == F32 && part) h[k] = __float2half_rn(w - __half2float(h[k]));
  }
  reinterpret_cast<uint4*>(out)[i] = *reinterpret_cast<uint4*>(h);
}
// activations -> half (encode_f32_to_f16); count % 4 == 0
__global__ void __launch_bounds__(256) f32_to_f16_kernel(const float* __restrict__ x, __half* __restrict__ out, size_t n4) {
  pdl_launch_dependents();
  pdl_wait();
  // four values 256 apart per thread: four loads in flight
  const size_t i0 = (size_t)blockIdx.x * 1024 + threadIdx.x;
  float4 v[4];
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (i0 + 256 * k < n4) v[k] = __ldcs(reinterpret_cast<const float4*>(x) + i0 + 256 * k);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    __half2 h[2] = {__floats2half2_rn(v[k].x, v[k].y), __floats2half2_rn(v[k].z, v[k].w)};
    if (i0 + 256 * k < n4) reinterpret_cast<uint2*>(out)[i0 + 256 * k] = *reinterpret_cast<uint2*>(h);
  }
}

// ---------------------------------------------------------------- host side
namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn gm_encode_fn() {
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
// Which of the forms is faster, estimated in us.  The figures are fitted to the times of every form at 1810 combinations of type, 512
// to 8192 rows, 1024 to 8192 columns and 17 to 4096 activation rows (rms error 6 to 13 %); the form chosen is 0.7 % slower than the
// fastest on average, more than 8 % at 3 % of them (again on the present kernels: 0.5 % and 3 % of 134 drawn shapes).
//   decoded operand  the start and the epilogue, the producers' time per 256 of a block's K (by type), and what each further
//                    wave starts anew
//   half copy        the conversion (by type, per 2^20 weights) and the GEMM (gemm_us)
// Odd rows, no multiples of 4: output rows are no multiples of 16 bytes and either form's epilogue stores word by word, the half GEMM's
// lanes each into a row of their own (18.6 us for a tile of 128 tokens x 256; 1.7 times that where all blocks store beside their main
// loops).  Fitted to both forms at 1500 odd shapes of the same ranges: the form chosen is 0.3 % slower than the faster one on average, more
// than 8 % at 1 %.  (Estimates of waves x share of K instead: 12 % and 31 %; 546 x 5632 of F16, 24 tokens, 22.2 us for 11.4.)
constexpr int kMmMaxSplits = 8;
struct MmCost {
  double conv0, conv;                              // conversion: fixed, per 2^20 weights
  double split256;                                 // per 256 of K, for the choice of the split
  double start, k256, k256_m, epi_m, wave, cluster;   // start + epi_m m / 128, (k256 + k256_m m / 128) per 256 of K, per further wave, per wave of clusters
};
constexpr MmCost mm_cost(int t) {
  switch (t) {
    case Q6_K: return {0.46, 0.65, 3.9, 9.98, 4.19, -0.94, 6.91, 12.02, -3.18};
    case Q5_K: return {0.79, 0.61, 4.5, 10.42, 4.39, -0.52, 6.50, 10.13, -3.44};
    case Q8_0: return {0.27, 0.67, 3.7, 8.61, 4.09, -1.12, 7.85, 14.38, -3.00};
    case IQ4_NL: return {0.87, 0.63, 3.5, 8.90, 3.58, -0.67, 6.65, 11.88, -3.02};
    case IQ1_S: return {2.00, 0.55, 2.7, 10.51, 1.43, 0.60, 4.51, 10.83, -3.62};
    case IQ2_XXS: return {1.30, 0.61, 2.9, 9.70, 2.31, -0.20, 6.55, 11.91, -3.71};
    case BF16: return {0.73, 0.65, 3.2, 8.89, 2.02, 0.16, 6.21, 11.59, -2.85};
    default: return {0.0, 0.0, 3.2, 9.37, 2.15, 0.0, 5.42, 12.99, -2.67};
  }
}
// The half GEMM alone: `tiles` of bn weight rows by 128 g tokens, kb K blocks.  Whole waves, and a last one whose steps are the
// shorter the fewer blocks load.
double gemm_us(int g, int bn, int tiles, int kb, int n, bool odd, int sms) {
  const int at_once = sms / g, full = tiles / at_once, rest = tiles % at_once;
  const double w = (128.0 * g + bn) / (128.0 * g + 256.0), fill = (double)rest / at_once;
  const double step = g == 2 ? 0.746 * w - 0.318 : 0.598 * w - 0.105;
  const double last = g == 2 ? 0.607 * w - 0.318 + 0.139 * w * fill : 0.426 * w - 0.105 + 0.172 * w * fill;
  if (odd) {
    const double epi = bn / 256.0 * (4.6 + 14.0 * std::min(n, kGmBM) / kGmBM), first = kb * (full ? step : last);
    return 3.6 + first + std::max(full - 1, 0) * std::max(kb * step, 1.74 * epi) + (full && rest ? std::max(kb * last, 1.74 * epi) : 0.0) + epi;
  }
  return (g == 2 ? 6.9 : 6.1) + kb * (full * step + (rest ? last : 0.0));
}

// half matrix [rows][cols] with row stride `stride` halfs, tiles of box_rows x 64 halfs, 128-byte swizzle
int make_map(CUtensorMap* map, const void* base, int rows, int cols, int64_t stride, int box_rows) {
  EncodeTiledFn encode = gm_encode_fn();
  if (!encode) return fail(kErrCuda, "matmul: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t gstride[1] = {(cuuint64_t)stride * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kGmBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult cr = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), gdim, gstride, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) return fail(kErrCuda, "matmul: tensor map encode failed (%d)", (int)cr);
  return kOk;
}

// Blocks of a tile and its weight rows: 256, or less where that fills the last wave better.  A step costs about what its operands
// cost to fetch from L2 (the tensor core needs less): proportional to the tile's tokens + bn.
struct GemmShape { int g, bn; };
GemmShape gemm_shape(int n, int rows, int cols, int sms, double* us) {
  GemmShape best{2, kGmBN};
  *us = 1e30;
  const bool odd = rows % 4 != 0;
  for (int g : {2, 1}) {
    if (odd && g == 1) break;
    const int mt = (n + g * kGmBM - 1) / (g * kGmBM), at_once = sms / g;
    int bn = kGmBN, tiles = 0;
    int64_t cost = INT64_MAX;
    for (int b = kGmBN; b >= 128; b -= 32) {
      const int t = mt * ((rows + b - 1) / b);
      const int64_t c = (int64_t)((t + at_once - 1) / at_once) * (128 * g + b);
      if (c < cost) { cost = c; bn = b; tiles = t; }
    }
    const double t = gemm_us(g, bn, tiles, (cols + kGmBK - 1) / kGmBK, n, odd, sms);
    if (t < *us / (g == 1 ? 1.03 : 1.0)) best = GemmShape{g, bn};           // pairs, unless single blocks are clearly faster
    *us = std::min(*us, t);
  }
  return best;
}

template <int G>
int gemm_launch(GemmParams& p, const void* x16, int64_t x_stride, const void* w16, int sms, int dev, cudaStream_t st) {
  int rc = make_map(&p.a_map, x16, p.n, p.cols, x_stride, kGmBM);
  if (rc) return rc;
  rc = make_map(&p.b_map, w16, p.rows, p.cols, p.cols, p.bn / G);
  if (rc) return rc;
  const int tiles = ((p.n + G * kGmBM - 1) / (G * kGmBM)) * ((p.rows + p.bn - 1) / p.bn);
  const size_t smem = 1024 + 1024 + (size_t)gm_stages(G) * (kGmShareA + gm_share_b(G));
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    MSB_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[dev & 63] = true;
  }
  MSB_CUDA(launch_pdl(gemm_tc_kernel<G>, dim3(G * std::max(1, std::min(sms / G, tiles))), dim3(kGmThreads), smem, st, p));
  MSB_LAUNCH_CHECK("gemm_tc_kernel");
  return kOk;
}

// Y (+)= X16 . W16^T, both operands half in global memory
int gemm_f16(const void* x16, int64_t x_stride, const void* w16, float* y, int n, int rows, int cols, bool accumulate,
             cudaStream_t st) {
  Tables tb;
  int rc = get_tables(&tb);
  if (rc) return rc;
  int dev = 0, sms = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  MSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  GemmParams p;
  double us;
  const GemmShape shape = gemm_shape(n, rows, cols, sms, &us);
  p.bn = shape.bn;
  p.y = y; p.status = tb.status; p.n = n; p.rows = rows; p.cols = cols; p.accumulate = accumulate ? 1 : 0;
  return shape.g == 2 ? gemm_launch<2>(p, x16, x_stride, w16, sms, dev, st) : gemm_launch<1>(p, x16, x_stride, w16, sms, dev, st);
}

double mm_dense_us(int t, int n, int rows, int cols, int sms) {
  double us;
  gemm_shape(n, rows, cols, sms, &us);
  const MmCost c = mm_cost(t);
  return c.conv0 + c.conv * rows * cols / 1048576.0 + us;
}
// Blocks of a cluster that share a tile's K: the split that ends first; a cluster needs its blocks on one GPC, so how many run
// at once comes from the driver (asked once per device and size).
template <int T>
int mm_splits(int tiles, int chunks, int cols, int m, bool odd, int sms, int dev, double& us) {
  static std::atomic<int> active[64][kMmMaxSplits + 1] = {};
  constexpr int kPair = 2 * TsPiece<T>::kK;
  const int pairs = (cols + kPair - 1) / kPair;
  constexpr MmCost c = mm_cost(T);
  int best = 1;
  double best_t = 1e30;
  for (int s = 1; s <= std::min(kMmMaxSplits, pairs); s++) {
    int act = active[dev & 63][s].load(std::memory_order_relaxed);
    if (act == 0) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(s); cfg.blockDim = dim3(kTsThreads); cfg.dynamicSmemBytes = kTsSmem;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = s; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
      cfg.attrs = &attr; cfg.numAttrs = 1;
      int n = 0;
      act = s == 1 ? sms : cudaOccupancyMaxActiveClusters(&n, mm_ts_kernel<T>, &cfg) == cudaSuccess && n > 0 ? n : -1;
      if (act < 0) (void)cudaGetLastError();              // a size that cannot run is not a failure of this call
      active[dev & 63][s].store(act, std::memory_order_relaxed);
    }
    if (act < 0) continue;
    const int waves = (tiles + act - 1) / act;            // of one persistent block per SM, or of clusters that start anew
    const double k = (pairs + s - 1) / s * kPair / 256.0, t = s == 1 ? 9.0 + waves * k * c.split256 : waves * (9.0 + k * c.split256);
    if (t < best_t) {
      best_t = t; best = s;
      const double start = c.start + c.epi_m * m / 128.0, work = k * (c.k256 + c.k256_m * m / 128.0);
      us = s == 1 ? start + waves * work + (waves - 1) * c.wave : waves * (start + work + c.cluster);
    }
  }
  // (BF16 and F16 rows are fetched once per chunk of activation rows, which the fit to whole rows does not see)
  if (odd) us *= 0.95 * (is_dense(T) ? 1.0 + 0.07 * std::max(0, chunks - 2) : 1.0);
  return best;
}
// taken = false: the half copy is faster
template <int T>
int mm_ts(const void* W, const void* x16, int64_t x_stride, float* y, int n, int rows, int cols, bool accumulate, cudaStream_t st,
          bool& taken) {
  MmTsParams p;
  taken = true;
  int rc = get_tables(&p.tb);
  if (rc) return rc;
  int dev = 0, sms = 0;
  MSB_CUDA(cudaGetDevice(&dev));
  MSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    MSB_CUDA(cudaFuncSetAttribute(mm_ts_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTsSmem));
    configured[dev & 63] = true;
  }
  const int ch = (n + kTsMaxN - 1) / kTsMaxN;
  p.per = ((n + ch - 1) / ch + 15) & ~15;
  p.chunks = (n + p.per - 1) / p.per;
  p.row_tiles = (rows + 255) / 256;
  const int tiles = p.row_tiles * p.chunks;
  double us;
  p.splits = mm_splits<T>(tiles, p.chunks, cols, std::min(n, p.per), rows % 4 != 0, sms, dev, us);
  if (us >= mm_dense_us(T, n, rows, cols, sms)) { taken = false; return kOk; }
  for (int i = 0; i < 4; i++) {
    rc = make_map(&p.a[i], x16, n, cols, x_stride, 16 << i);
    if (rc) return rc;
  }
  p.w = (const uint8_t*)W; p.y = y; p.n = n; p.rows = rows; p.cols = cols; p.accumulate = accumulate ? 1 : 0;
  if (p.splits == 1) {
    MSB_CUDA(launch_pdl(mm_ts_kernel<T>, dim3(std::min(sms, tiles)), dim3(kTsThreads), kTsSmem, st, p));
  } else {
    MSB_CUDA(launch_clusters(mm_ts_kernel<T>, dim3(tiles * p.splits), dim3(kTsThreads), p.splits, kTsSmem, st, p));
  }
  MSB_LAUNCH_CHECK("mm_ts_kernel");
  return kOk;
}
// Y (+)= X16 . W^T from the raw blocks; taken = false: not for this type or shape (a row is no whole number of pieces)
int mm_ts_run(int t, const void* W, const void* x16, int64_t x_stride, float* y, int n, int rows, int cols, bool accumulate,
              cudaStream_t st, bool& taken) {
  taken = false;
  if (cols % ts_piece_k(t) || (is_dense(t) && (reinterpret_cast<uintptr_t>(W) & 15))) return kOk;
  switch (t) {
#define MM_TS(T) case T: return mm_ts<T>(W, x16, x_stride, y, n, rows, cols, accumulate, st, taken);
    MM_TS(Q8_0) MM_TS(Q5_K) MM_TS(Q6_K) MM_TS(IQ2_XXS) MM_TS(IQ1_S) MM_TS(IQ4_NL) MM_TS(BF16) MM_TS(F16)
#undef MM_TS
  }
  return kOk;
}

}  // namespace

// W (type t) -> half [rows x cols]; part 1 = the F32 remainder term (also used by the MoE prefill for its dense experts)
int weights_to_f16(int t, const void* W, int64_t count, __half* out, int part, cudaStream_t st) {
  Tables tb;
  int rc = get_tables(&tb);
  if (rc) return rc;
  const int threads = 256;
  const int64_t n8 = count / 8;                       // rows are multiples of 8
  const dim3 grid((unsigned)((n8 + threads - 1) / threads));
  const uint8_t* s = (const uint8_t*)W;
  if (t == F16) {
    MSB_CUDA(cudaMemcpyAsync(out, W, (size_t)count * 2, cudaMemcpyDeviceToDevice, st));
  } else if (t == F32) {
    MSB_CUDA(launch_pdl(dense_f16_kernel<F32>, grid, dim3(threads), 0, st, s, out, n8, part));
  } else if (t == BF16) {
    MSB_CUDA(launch_pdl(dense_f16_kernel<BF16>, grid, dim3(threads), 0, st, s, out, n8, part));
  } else {
    switch (t) {
      case Q8_0: MSB_CUDA(launch_pdl(dequant_f16_kernel<Q8_0>, grid, dim3(threads), 0, st, s, out, n8, tb)); break;
      case Q5_K: MSB_CUDA(launch_pdl(dequant_f16_kernel<Q5_K>, grid, dim3(threads), 0, st, s, out, n8, tb)); break;
      case Q6_K: MSB_CUDA(launch_pdl(dequant_f16_kernel<Q6_K>, grid, dim3(threads), 0, st, s, out, n8, tb)); break;
      case IQ2_XXS: MSB_CUDA(launch_pdl(dequant_f16_kernel<IQ2_XXS>, grid, dim3(threads), 0, st, s, out, n8, tb)); break;
      case IQ1_S: MSB_CUDA(launch_pdl(dequant_f16_kernel<IQ1_S>, grid, dim3(threads), 0, st, s, out, n8, tb)); break;
      case IQ4_NL: MSB_CUDA(launch_pdl(dequant_f16_kernel<IQ4_NL>, grid, dim3(threads), 0, st, s, out, n8, tb)); break;
      default: return fail(kErrType, "matmul: unsupported weight type %d", t);
    }
  }
  MSB_LAUNCH_CHECK("weights_to_f16");
  return kOk;
}

// n_mat block-quantised matrices of `count` weights each, addresses in the device array d_srcs, to half copies laid
// back to back at out
int weights_to_f16_group(int t, const uint64_t* d_srcs, int n_mat, int64_t count, __half* out, cudaStream_t st) {
  if (n_mat <= 0) return kOk;
  if (is_dense(t) || n_mat > 65535) return fail(kErrType, "matmul: grouped conversion needs a block-quantised type");
  Tables tb;
  int rc = get_tables(&tb);
  if (rc) return rc;
  const int threads = 256;
  const int64_t n8 = count / 8;
  const dim3 grid((unsigned)((n8 + threads - 1) / threads), (unsigned)n_mat);
  switch (t) {
    case Q8_0: MSB_CUDA(launch_pdl(dequant_f16_group_kernel<Q8_0>, grid, dim3(threads), 0, st, d_srcs, out, n8, tb)); break;
    case Q5_K: MSB_CUDA(launch_pdl(dequant_f16_group_kernel<Q5_K>, grid, dim3(threads), 0, st, d_srcs, out, n8, tb)); break;
    case Q6_K: MSB_CUDA(launch_pdl(dequant_f16_group_kernel<Q6_K>, grid, dim3(threads), 0, st, d_srcs, out, n8, tb)); break;
    case IQ2_XXS: MSB_CUDA(launch_pdl(dequant_f16_group_kernel<IQ2_XXS>, grid, dim3(threads), 0, st, d_srcs, out, n8, tb)); break;
    case IQ1_S: MSB_CUDA(launch_pdl(dequant_f16_group_kernel<IQ1_S>, grid, dim3(threads), 0, st, d_srcs, out, n8, tb)); break;
    case IQ4_NL: MSB_CUDA(launch_pdl(dequant_f16_group_kernel<IQ4_NL>, grid, dim3(threads), 0, st, d_srcs, out, n8, tb)); break;
    default: return fail(kErrType, "matmul: unsupported weight type %d", t);
  }
  MSB_LAUNCH_CHECK("weights_to_f16_group");
  return kOk;
}

int f32_to_f16(const float* x, void* x16, size_t count, cudaStream_t st) {
  if (count % 4) return fail(kErrArg, "f32_to_f16: count %zu is not a multiple of 4", count);
  if (count == 0) return kOk;
  if (!x || !x16 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(x16) & 7))
    return fail(kErrArg, "f32_to_f16: null or misaligned pointer");
  const size_t n4 = count / 4;
  MSB_CUDA(launch_pdl(f32_to_f16_kernel, dim3((unsigned)((n4 + 1023) / 1024)), dim3(256), 0, st, x, (__half*)x16, n4));
  MSB_LAUNCH_CHECK("f32_to_f16_kernel");
  return kOk;
}

// scratch of matmul_h: the half copy of W (nothing for F16 weights); matmul adds the half copy of X
size_t matmul_scratch_bytes(int t, int rows, int cols, int n, bool with_x) {
  size_t b = t == F16 ? 0 : (size_t)rows * cols * 2;
  b = (b + 255) & ~(size_t)255;
  if (with_x) b += ((size_t)n * cols * 2 + 255) & ~(size_t)255;
  return b ? b + 256 : 0;   // + room to align the base
}

int matmul_h(int t, const void* W, int rows, int cols, const void* X16, int x_stride, float* Y, int n, bool accumulate,
             void* scratch, size_t scratch_bytes, cudaStream_t st) {
  if (!type_known(t)) return fail(kErrType, "matmul: unsupported weight type %d", t);
  if (rows <= 0 || cols <= 0 || n < 0 || cols % block_elems(t) || cols % 8)
    return fail(kErrArg, "matmul: bad shape (rows %d cols %d n %d, type %s)", rows, cols, n, type_name(t));
  if (n == 0) return kOk;
  if (x_stride == 0) x_stride = cols;
  if (x_stride < cols || x_stride % 8) return fail(kErrArg, "matmul: x_stride %d must be >= cols and a multiple of 8", x_stride);
  if (!W || !X16 || !Y || (reinterpret_cast<uintptr_t>(X16) & 15)) return fail(kErrArg, "matmul: null or misaligned pointer");
  if (scratch_bytes < matmul_scratch_bytes(t, rows, cols, n, false) || (t != F16 && !scratch))
    return fail(kErrScratch, "matmul: scratch too small");
  bool taken;
  int rc = mm_ts_run(t, W, X16, x_stride, Y, n, rows, cols, accumulate, st, taken);
  if (rc || taken) return rc;
  const void* w16 = W;
  if (t == F16) {
    if (reinterpret_cast<uintptr_t>(W) & 15) return fail(kErrArg, "matmul: F16 weights must be 16-byte aligned");
  } else {
    __half* wbuf = reinterpret_cast<__half*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~(uintptr_t)255);
    rc = weights_to_f16(t, W, (int64_t)rows * cols, wbuf, 0, st);
    if (rc) return rc;
    w16 = wbuf;
  }
  rc = gemm_f16(X16, x_stride, w16, Y, n, rows, cols, accumulate, st);
  if (rc || t != F32) return rc;
  // F32 weights keep their precision: second pass with the remainder term w - half(w)
  __half* wbuf = reinterpret_cast<__half*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~(uintptr_t)255);
  rc = weights_to_f16(t, W, (int64_t)rows * cols, wbuf, 1, st);
  if (rc) return rc;
  return gemm_f16(X16, x_stride, wbuf, Y, n, rows, cols, true, st);
}

int matmul(int t, const void* W, int rows, int cols, const float* X, float* Y, int n, bool accumulate, void* scratch,
           size_t scratch_bytes, cudaStream_t st) {
  if (rows <= 0 || cols <= 0 || n < 0) return fail(kErrArg, "matmul: bad shape");
  if (n == 0) return kOk;
  if (!scratch || scratch_bytes < matmul_scratch_bytes(t, rows, cols, n, true)) return fail(kErrScratch, "matmul: scratch too small");
  const size_t wpart = matmul_scratch_bytes(t, rows, cols, n, false);
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~(uintptr_t)255);
  void* x16 = base + ((wpart + 255) & ~(size_t)255);
  int rc = f32_to_f16(X, x16, (size_t)n * cols, st);
  if (rc) return rc;
  return matmul_h(t, W, rows, cols, x16, cols, Y, n, accumulate, scratch, wpart, st);
}

}  // namespace msb
