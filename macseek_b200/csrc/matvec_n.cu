// Projections of 2 to 16 tokens with block-quantised weights: Y[n][rows] (+)= X[n][cols] . W^T on the integer tensor cores.
// The arithmetic of the one-token kernel (quant_blocks.cuh): integer codes times a 16-bit fixed-point copy of the activations
// (two int8 limbs), exact in int32 inside a 32-element unit (Q6_K: inside its 16-element halves), scaled and added in fp32.
//
// mma.sync m16n8k32: A = 16 weight rows x one unit of codes, B = 4 tokens x 2 limbs as the 8 columns, so that a decoded code
// serves 4 tokens per instruction where dp4a needs two instructions per token and 4 codes, and the two limb sums of a (row,
// token) pair land in one thread.  The sums start at the bit pattern of 1.5 * 2^23, so that reading them as floats and
// subtracting that converts them (they stay below 2^20).  Bound by instruction issue (decode, conversion of the sums): Q6_K
// 9000 x 5120 takes 14.2 us with 2 tokens, 15.6 with 4, 26.2 with 8, 52.5 with 16; 16384 x 4096 with 4 went from 31.5 to 19.0.
//
// A block is 16 consumer warps + 1 producer warp (stream_pipe.cuh).  A piece is 16 * RT consecutive rows, whole (one bulk copy)
// or, when that does not fit, a run of their units; KW = 16 / RT warps share the 16 rows of one MMA, each taking every KW-th
// group of 4 units, and their sums are added in warp order through shared memory.
#include <algorithm>
#include "stream_pipe.cuh"

namespace msb {

constexpr int kMnNW = 16;
constexpr float kMnMagic = 12582912.f;              // 1.5 * 2^23, bits 0x4B400000

struct MnParams {
  const uint8_t* W;
  const float* x;
  float* y;
  int64_t x_stride, y_stride;
  int rows, units, n;                               // n <= 4 * NG tokens
  uint32_t row_bytes, pitch, stage_bytes;
  int accumulate, rt, chunk_units, stages, tiles, one_copy;
  Tables tb;
};
struct MnHead {
  uint64_t full[kMaxStages], empty[kMaxStages], lutbar;
  int abort_flag;
};

__host__ __device__ constexpr bool mn_by_lookup(int t) { return t == IQ1_S || t == IQ2_XXS; }

__device__ __forceinline__ void mn_mma32(int (&d)[4], const uint32_t (&a)[4], uint2 b) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "r"(0x4B400000));
}
__device__ __forceinline__ void mn_mma16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a0), "r"(a1), "r"(b), "r"(0x4B400000));
}
// 256 * hi + lo of the two sums
__device__ __forceinline__ float mn_sum(int hi, int lo) {
  return fmaf(__int_as_float(hi) - kMnMagic, 256.f, __int_as_float(lo) - kMnMagic);
}

// Activations in shared memory as B fragments: unit u, token group q: 32 lanes x 8 bytes, lane 4 g + t holding column g = token
// (g >> 1), limb (g & 1; 0 = high) of thread t's 8 elements, and 4 pairs {scale, scale * sum}.
// Thread t's elements: 4 t .. and 16 + 4 t .. (4 each), for the look-up types 8 t .. 8 t + 7.
// x ~= scale * (256 hi + lo) with both limbs signed: that covers -32768 .. 32639, so the unit's larger extreme is made the
// negative one (the scale carries the sign) and only a smaller extreme within 0.4 % of it costs range.
template <int T, int NG>
__device__ __forceinline__ void mn_quantize(const MnParams& p, uint8_t* frag, float2* meta, int tid) {
  // Four threads per unit, 8 elements each; the loads of up to four tokens are in flight together.  Columns of tokens past n
  // stay as they are: nothing of them reaches another column.
  const int l4 = tid & 3, total = p.units * 4;
  for (int base = 0; base < total; base += kMnNW * 32) {
    const bool live = base + tid < total;           // whole quads are live or not
    const int u = live ? (base + tid) >> 2 : 0;
    const float* src = p.x + 32 * u + 8 * l4;
#pragma unroll 1
    for (int q = 0; q < NG; q++) {
      const int nc = min(4, p.n - 4 * q);
      float v[4][8];
#pragma unroll
      for (int c = 0; c < 4; c++)
        if (c < nc) {
          const float4* s4 = reinterpret_cast<const float4*>(src + (size_t)(4 * q + c) * p.x_stride);
          const float4 a = s4[0], b = s4[1];
          v[c][0] = a.x; v[c][1] = a.y; v[c][2] = a.z; v[c][3] = a.w; v[c][4] = b.x; v[c][5] = b.y; v[c][6] = b.z; v[c][7] = b.w;
        }
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (c >= nc) break;
        float P = 0.f, N = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) { P = fmaxf(P, v[c][i]); N = fmaxf(N, -v[c][i]); }
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
          P = fmaxf(P, __shfl_xor_sync(0xffffffffu, P, o));
          N = fmaxf(N, __shfl_xor_sync(0xffffffffu, N, o));
        }
        const float big = fmaxf(P, N), small = fminf(P, N);
        const bool edge = small * 32767.f > big * 32639.f;
        const float top = edge ? small : big, lim = edge ? 32639.f : 32767.f, sign = P > N ? -1.f : 1.f;
        const float inv = top > 0.f ? sign * (lim / top) : 0.f, sc = sign * (top * (edge ? 1.f / 32639.f : 1.f / 32767.f));
        uint32_t f[8];
#pragma unroll
        for (int i = 0; i < 8; i++) f[i] = __float_as_uint(fmaf(v[c][i], inv, kMnMagic));
        uint32_t hw[2], lw[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
          lw[j] = __byte_perm(__byte_perm(f[4 * j], f[4 * j + 1], 0x0040), __byte_perm(f[4 * j + 2], f[4 * j + 3], 0x0040), 0x5410);
          hw[j] = __byte_perm(__byte_perm(f[4 * j] + 128u, f[4 * j + 1] + 128u, 0x0051),
                              __byte_perm(f[4 * j + 2] + 128u, f[4 * j + 3] + 128u, 0x0051), 0x5410);
        }
        const int slot = u * NG + q, g = 2 * c;
        if constexpr (T == Q5_K) {
          int sum = 256 * dp4a_ss(hw[1], 0x01010101u, dp4a_ss(hw[0], 0x01010101u, 0)) + dp4a_ss(lw[1], 0x01010101u, dp4a_ss(lw[0], 0x01010101u, 0));
          sum += __shfl_xor_sync(0xffffffffu, sum, 1);
          sum += __shfl_xor_sync(0xffffffffu, sum, 2);
          if (live && l4 == 0) meta[slot * 4 + c] = make_float2(sc, sc * (float)sum);
        } else if (live && l4 == 0) {
          meta[slot * 4 + c] = make_float2(sc, 0.f);
        }
        if (live) {
          uint32_t* d = reinterpret_cast<uint32_t*>(frag) + (size_t)slot * 64;
          // word index of (column, thread t, half b): 2 * (4 column + t) + b
          const int w0 = mn_by_lookup(T) ? 2 * l4 : 2 * ((2 * l4) & 3) + (l4 >> 1), w1 = mn_by_lookup(T) ? w0 + 1 : w0 + 2;
          d[8 * g + w0] = hw[0]; d[8 * g + w1] = hw[1];
          d[8 * (g + 1) + w0] = lw[0]; d[8 * (g + 1) + w1] = lw[1];
        }
      }
    }
  }
}

// 32-bit word at a 2-byte aligned shared address
__device__ __forceinline__ uint32_t mn_word(saddr_t p) {
  const saddr_t a = p & ~3u;
  return __funnelshift_r(lds_u32(a), lds_u32(a + 4u), (p & 2u) * 8u);
}
// bytes b + k of a word, k a byte constant: no carry between bytes as long as the sums fit
__device__ __forceinline__ uint32_t mn_signed(uint32_t codes, uint32_t minus) {   // codes (below 128) - minus, per byte, two's complement
  return ((codes | 0x80808080u) - minus) ^ 0x80808080u;
}
// Codes of 4 consecutive units (128 elements; `nu` of them exist) of the thread's two rows, as A fragments, and their scales;
// `each(k, a, s0, s1, m0, m1)` is called per unit: a = {row 0 words t, row 1 words t, row 0 words t + 4, row 1 words t + 4}.
template <int T, class F>
__device__ __forceinline__ void mn_item(const saddr_t (&row)[2], int item, int nu, int t, const LaneLuts& L, F&& each) {
  if constexpr (T == Q8_0) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (k >= nu) break;
      uint32_t a[4];
      float s[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const saddr_t b = row[i] + (uint32_t)(4 * item + k) * 34u;
        a[i] = mn_word(b + 2u + 4u * t); a[2 + i] = mn_word(b + 18u + 4u * t);
        s[i] = lds_half(b);
      }
      each(k, a, s[0], s[1], 0.f, 0.f);
    }
  } else if constexpr (T == IQ4_NL) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (k >= nu) break;
      uint32_t a[4];
      float s[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const saddr_t b = row[i] + (uint32_t)(4 * item + k) * 18u;
        const uint32_t w = mn_word(b + 2u + 4u * t);
        a[i] = iq4_levels(w); a[2 + i] = iq4_levels(w >> 4);
        s[i] = lds_half(b);
      }
      each(k, a, s[0], s[1], 0.f, 0.f);
    }
  } else if constexpr (T == Q5_K) {
    uint32_t qh[2][2], sc[2][3];
    float d[2], dm[2];
    saddr_t q[2];
    const int half = item & 1;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const saddr_t b = row[i] + (uint32_t)(item >> 1) * 176u;
      d[i] = lds_half(b); dm[i] = lds_half(b + 2u);
#pragma unroll
      for (int j = 0; j < 3; j++) sc[i][j] = mn_word(b + 4u + 4u * j);
      qh[i][0] = mn_word(b + 16u + 4u * t) >> (4 * half); qh[i][1] = mn_word(b + 32u + 4u * t) >> (4 * half);
      q[i] = b + 48u + 64u * half + 4u * t;
    }
#pragma unroll
    for (int P = 0; P < 2; P++) {
      uint32_t w[2][2];
#pragma unroll
      for (int i = 0; i < 2; i++) { w[i][0] = mn_word(q[i] + 32u * P); w[i][1] = mn_word(q[i] + 32u * P + 16u); }
#pragma unroll
      for (int o = 0; o < 2; o++) {
        const int k = 2 * P + o;
        uint32_t a[4];
        float s[2], m[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
#pragma unroll
          for (int j = 0; j < 2; j++) a[2 * j + i] = ((w[i][j] >> (4 * o)) & 0x0F0F0F0Fu) | (((qh[i][j] >> k) & 0x01010101u) << 4);
          uint32_t sv, mv;
          if (half == 0) { sv = (sc[i][0] >> (8 * k)) & 63u; mv = (sc[i][1] >> (8 * k)) & 63u; }
          else {
            const uint32_t hi = sc[i][2] >> (8 * k);
            sv = (hi & 15u) | (((sc[i][0] >> (8 * k + 6)) & 3u) << 4);
            mv = ((hi >> 4) & 15u) | (((sc[i][1] >> (8 * k + 6)) & 3u) << 4);
          }
          s[i] = d[i] * (float)sv; m[i] = dm[i] * (float)mv;
        }
        each(k, a, s[0], s[1], m[0], m[1]);
      }
    }
  } else if constexpr (T == Q6_K) {
    uint32_t qh[2][2], sc[2][2];
    float d[2];
    saddr_t q[2];
    const int half = item & 1;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const saddr_t b = row[i] + (uint32_t)(item >> 1) * 210u;
      qh[i][0] = mn_word(b + 128u + 32u * half + 4u * t); qh[i][1] = mn_word(b + 144u + 32u * half + 4u * t);
      sc[i][0] = mn_word(b + 192u + 8u * half); sc[i][1] = mn_word(b + 196u + 8u * half);
      d[i] = lds_half(b + 208u);
      q[i] = b + 64u * half + 4u * t;
    }
    uint32_t w[2][4];                                // [row][2 * (32-byte run) + 16-byte half]
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) w[i][j] = mn_word(q[i] + 16u * j);
#pragma unroll
    for (int k = 0; k < 4; k++) {                    // sub-block k: run k & 1, low nibbles for k < 2
      uint32_t a[4];
      float s[2], s2[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const uint32_t lo = w[i][2 * (k & 1) + j] >> (4 * (k >> 1)), hi = qh[i][j] >> (2 * k);
          a[2 * j + i] = mn_signed((lo & 0x0F0F0F0Fu) | ((hi & 0x03030303u) << 4), 0x20202020u);
        }
        const uint32_t v = sc[i][k >> 1] >> (16 * (k & 1));
        s[i] = d[i] * (float)(int8_t)(v & 0xFFu); s2[i] = d[i] * (float)(int8_t)((v >> 8) & 0xFFu);
      }
      each(k, a, s[0], s[1], s2[0], s2[1]);
    }
  } else if constexpr (T == IQ1_S) {
    saddr_t b[2];
    float d[2];
    const int u0 = 4 * (item & 1);
#pragma unroll
    for (int i = 0; i < 2; i++) { b[i] = row[i] + (uint32_t)(item >> 1) * 50u; d[i] = lds_half(b[i]) * 0.125f; }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      uint32_t a[4];
      float s[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const uint32_t qs = lds_u8(b[i] + 2u + 4u * (u0 + k) + t), h = lds_u16(b[i] + 34u + 2u * (u0 + k));
        const uint32_t w = lds_u32(L.iq1s + (qs | (((h >> (3 * t)) & 7u) << 8)) * (4u * kIq1sCopies));
        const uint32_t off = h & 0x8000u ? 0x09090909u : 0x07070707u;          // 8 code - 7 or - 9
        a[i] = mn_signed((w & 0x0F0F0F0Fu) * 8u, off); a[2 + i] = mn_signed(((w >> 4) & 0x0F0F0F0Fu) * 8u, off);
        s[i] = d[i] * (float)(((h >> 11) & 14u) | 1u);
      }
      each(k, a, s[0], s[1], 0.f, 0.f);
    }
  } else {
    constexpr uint32_t kPoolA = 0xF82B1908u, kPoolB = 0x0000D5E7u;             // bytes 8, 25, 43, -8 | -25, -43
    saddr_t b[2];
    float d[2];
    const int u0 = 4 * (item & 1);
#pragma unroll
    for (int i = 0; i < 2; i++) { b[i] = row[i] + (uint32_t)(item >> 1) * 66u; d[i] = lds_half(b[i]) * 0.25f; }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      uint32_t a[4];
      float s[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const saddr_t q = b[i] + 2u + 8u * (u0 + k);
        const uint32_t a1 = lds_u32_a2(q + 4u);
        const uint32_t sel = lds_u32(L.iq2g + lds_u8(q + t) * (4u * kIq2Copies)) + lds_u32(L.iq2s + ((a1 >> (7 * t)) & 127u) * (4u * kIq2Copies));
        a[i] = __byte_perm(kPoolA, kPoolB, sel); a[2 + i] = __byte_perm(kPoolA, kPoolB, sel >> 16);
        s[i] = d[i] * (0.5f + (float)(a1 >> 28));
      }
      each(k, a, s[0], s[1], 0.f, 0.f);
    }
  }
}

template <int T, int NG>
__global__ void __launch_bounds__((kMnNW + 1) * 32, 1) matvec_mma_kernel(const MnParams p) {
  pdl_launch_dependents();
  extern __shared__ __align__(128) uint8_t smem[];
  MnHead* hd = reinterpret_cast<MnHead*>(smem);
  uint8_t* cur = smem + 128;
  uint8_t* lut = cur;
  constexpr size_t kLut = mn_by_lookup(T) ? lut_bytes_for(T) : 0;
  cur += kLut;
  const int U = p.units;
  uint8_t* frag = cur; cur += (size_t)U * NG * 256;
  float2* meta = reinterpret_cast<float2*>(cur); cur += (size_t)U * NG * 32;
  constexpr int kTok = 4 * NG;
  float* part = reinterpret_cast<float*>(cur);      // [2][16 warps][kTok][16 rows]
  cur += (size_t)2 * kMnNW * 16 * kTok * 4;
  Ring ring;
  ring.full = hd->full; ring.empty = hd->empty;
  ring.abort_flag = &hd->abort_flag; ring.status = p.tb.status; ring.stages = p.stages;
  ring.slot0 = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(cur) + 127) & ~(uintptr_t)127);
  ring.slot_bytes = p.stage_bytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  ring_init(ring, tid, kMnNW);
  if (tid == 0) { mbar_init(&hd->lutbar, 1); mbar_fence_init(); }
  __syncthreads();
  const int RT = p.rt, KW = kMnNW / RT, R = 16 * RT;
  const bool whole = p.chunk_units >= U;
  const int nchunks = whole ? 1 : (U + p.chunk_units - 1) / p.chunk_units;
  uint32_t n = 0;
  if (warp == kMnNW) {
    const uint8_t* srcv[1];
    Piece pc;
    pc.src = srcv; pc.nsrc = 1; pc.row_stride = p.row_bytes;
    for (int tl = blockIdx.x; tl < p.tiles; tl += gridDim.x) {
      const int r0 = tl * R, nrows = min(R, p.rows - r0);
      for (int c = 0; c < nchunks; c++, n++) {
        const int u0 = c * p.chunk_units, nu = min(p.chunk_units, U - u0);
        srcv[0] = p.W + (size_t)r0 * p.row_bytes + units_bytes(T, u0);
        if (p.one_copy) { pc.rows_per_src = 1; pc.nrows = 1; pc.bytes = (uint32_t)nrows * p.row_bytes; }
        else { pc.rows_per_src = R; pc.nrows = nrows; pc.bytes = units_bytes(T, nu); }
        if (!produce_piece(ring, n, pc, p.pitch, lane)) return;
      }
    }
    return;
  }
  LaneLuts L;
  const bool luts_ok = load_luts(lut, T == IQ1_S, T == IQ2_XXS, p.tb, tid, &hd->lutbar, &hd->abort_flag, L, lane);
  pdl_wait();                                       // the weights are constants; x (and y, when accumulating) are not
  mn_quantize<T, NG>(p, frag, meta, tid);
  bar_sync_named(1, kMnNW * 32);
  bool ok = luts_ok;                                 // after an abandoned wait a warp still takes part in the block's barriers
  const int rt = warp / KW, kw = warp % KW, g = lane >> 2, t = lane & 3;
  const saddr_t frag_s = smem_u32(frag) + 8u * lane, meta_s = smem_u32(meta) + 8u * t;
  uint32_t count = 0;
  for (int tl = blockIdx.x; tl < p.tiles; tl += gridDim.x, count++) {
    const int r0 = tl * R;
    float acc[2][NG];
#pragma unroll
    for (int q = 0; q < NG; q++) acc[0][q] = acc[1][q] = 0.f;
    for (int c = 0; c < nchunks; c++, n++) {
      const int u0 = c * p.chunk_units, nu = min(p.chunk_units, U - u0);
      const uintptr_t a0 = reinterpret_cast<uintptr_t>(p.W) + (size_t)r0 * p.row_bytes + units_bytes(T, u0);
      saddr_t row[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const uint32_t lr = 16u * rt + g + 8u * i;
        row[i] = smem_u32(ring.slot(n)) + lr * p.pitch + (uint32_t)((p.one_copy ? a0 : a0 + (uintptr_t)lr * p.row_bytes) & 15u);
      }
      ok = ok && consumer_wait(ring, n);
      for (int item = kw; ok && 4 * item < nu; item += KW) {
        mn_item<T>(row, item, nu - 4 * item, t, L, [&](int k, const uint32_t (&a)[4], float s0, float s1, float m0, float m1) {
#pragma unroll
          for (int q = 0; q < NG; q++) {
            const uint32_t at = (uint32_t)((u0 + 4 * item + k) * NG + q);
            const uint2 b = lds_u64(frag_s + 256u * at), me = lds_u64(meta_s + 32u * at);
            const float xs = __uint_as_float(me.x);
            int d[4];
            if constexpr (T == Q6_K) {
              int e[4];
              mn_mma16(d, a[0], a[1], b.x);
              mn_mma16(e, a[2], a[3], b.y);
              acc[0][q] = fmaf(xs, fmaf(m0, mn_sum(e[0], e[1]), s0 * mn_sum(d[0], d[1])), acc[0][q]);
              acc[1][q] = fmaf(xs, fmaf(m1, mn_sum(e[2], e[3]), s1 * mn_sum(d[2], d[3])), acc[1][q]);
            } else {
              mn_mma32(d, a, b);
              acc[0][q] = fmaf(s0 * xs, mn_sum(d[0], d[1]), acc[0][q]);
              acc[1][q] = fmaf(s1 * xs, mn_sum(d[2], d[3]), acc[1][q]);
              if constexpr (T == Q5_K) {
                const float sx = __uint_as_float(me.y);
                acc[0][q] = fmaf(-m0, sx, acc[0][q]);
                acc[1][q] = fmaf(-m1, sx, acc[1][q]);
              }
            }
          }
        });
      }
      consumer_release(ring, n, lane);
    }
    float* pw = part + (size_t)(count & 1u) * (kMnNW * 16 * kTok);
#pragma unroll
    for (int q = 0; q < NG; q++)
#pragma unroll
      for (int i = 0; i < 2; i++) pw[(warp * kTok + 4 * q + t) * 16 + g + 8 * i] = acc[i][q];
    bar_sync_named(1, kMnNW * 32);
    for (int o = tid; o < R * p.n; o += kMnNW * 32) {
      const int tok = o / R, r = o - tok * R;
      if (r0 + r >= p.rows) continue;
      float v = 0.f;
      for (int k = 0; k < KW; k++) v += pw[(((r >> 4) * KW + k) * kTok + tok) * 16 + (r & 15)];
      float* yp = p.y + (size_t)tok * p.y_stride + r0 + r;
      *yp = p.accumulate ? *yp + v : v;
    }
  }
}

namespace {
size_t mn_x_bytes(int units, int ng) { return (size_t)units * ng * 288 + (size_t)2 * kMnNW * 16 * 16 * ng; }
// What the ring must at least hold: two pieces of 16 whole rows, or three runs of 64 units (128 for the look-up types, whose
// units are a third as long)
size_t mn_ring_bytes(int t, int cols) {
  return std::min<size_t>(48 * ((size_t)units_bytes(t, mn_by_lookup(t) ? 128 : 64) + 62) + 1024, 2 * (16 * (row_bytes(t, cols) + 62) + 192));
}

template <int T, int NG>
int mn_launch(MnParams& p, cudaStream_t st, int dev, int sms) {
  const size_t fixed = 128 + (mn_by_lookup(T) ? lut_bytes_for(T) : 0) + mn_x_bytes(p.units, NG) + 128;
  const size_t avail = kSmemLimit - fixed;
  const int items = (p.units + 3) / 4;
  p.chunk_units = p.units; p.rt = 1;
  // Rows of 1.5 KB and more come one copy each, an odd multiple of 16 bytes apart, so that the 8 rows a load touches lie in
  // different banks (at a distance of 5440 bytes they met four in a bank: 27 us instead of 17); shorter rows as one copy of
  // the piece, the copy engine's time per copy being what matters then -- but where all 8 would meet in a bank (multiples of 128
  // bytes: 16384 x 2048 Q5_K, 4 tokens, 25 us in one copy, 13 apart), or four of them and the rows are not the shortest
  // (16384 x 1024 Q8_0 9.7 / 8.1; x 1024 IQ4_NL 7.7 / 9.4).
  p.one_copy = p.row_bytes < 1536 && p.row_bytes % 128 != 0 && (p.row_bytes % 64 != 0 || p.row_bytes < 1024);
  p.pitch = p.one_copy ? p.row_bytes : piece_pitch(p.row_bytes);
  size_t slot = 0;
  auto whole_slot = [&](int rt) { return ((size_t)16 * rt * p.pitch + 64 + 127) & ~(size_t)127; };
  if (2 * whole_slot(1) <= avail) {
    // more rows per piece as long as a warp would have fewer than 4 items, every SM still has a piece, and two pieces fit
    while (p.rt < 8 && items * p.rt < 4 * kMnNW && (long)p.rows >= 32L * p.rt * sms && 2 * whole_slot(2 * p.rt) <= avail) p.rt *= 2;
    slot = whole_slot(p.rt);
    p.stages = (int)std::min<size_t>(kMaxStages, avail / slot);
  } else {
    // runs of units, whole rounds of the 16 warps where that fits (64 units), whole super-blocks always
    const size_t third = (avail / 3) & ~(size_t)127;
    int cu = (int)((third / 16 - 64) / (size_t)units_bytes(T, 8)) * 8;
    if (cu >= 64) cu = cu / 64 * 64;
    if (cu < 8) return fail(kErrLimit, "matvec: no staging shape fits (type %s units %d)", type_name(T), p.units);
    p.chunk_units = std::min(cu, p.units);
    p.one_copy = 0;
    p.pitch = piece_pitch(units_bytes(T, p.chunk_units));
    slot = ((size_t)16 * p.pitch + 64 + 127) & ~(size_t)127;
    p.stages = (int)std::min<size_t>(kMaxStages, avail / slot);
  }
  p.stage_bytes = (uint32_t)slot;
  p.tiles = (p.rows + 16 * p.rt - 1) / (16 * p.rt);
  auto kern = matvec_mma_kernel<T, NG>;
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    MSB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    configured[dev & 63] = true;
  }
  MSB_CUDA(launch_pdl(kern, dim3(std::min(p.tiles, sms)), dim3((kMnNW + 1) * 32), fixed + p.stages * slot, st, p));
  MSB_LAUNCH_CHECK("matvec_mma_kernel");
  return kOk;
}
template <int NG>
int mn_type(int t, MnParams& p, cudaStream_t st, int dev, int sms) {
  switch (t) {
    case Q8_0: return mn_launch<Q8_0, NG>(p, st, dev, sms);
    case Q5_K: return mn_launch<Q5_K, NG>(p, st, dev, sms);
    case Q6_K: return mn_launch<Q6_K, NG>(p, st, dev, sms);
    case IQ2_XXS: return mn_launch<IQ2_XXS, NG>(p, st, dev, sms);
    case IQ1_S: return mn_launch<IQ1_S, NG>(p, st, dev, sms);
    default: return mn_launch<IQ4_NL, NG>(p, st, dev, sms);
  }
}
}  // namespace

// Tokens one pass of matvec_mma can take: as many groups of four as leave the ring its room; 0: not even one group
int matvec_mma_tokens(int t, int cols) {
  const size_t lut = mn_by_lookup(t) ? lut_bytes_for(t) : 0;
  for (int ng : {4, 3, 2, 1})
    if (256 + lut + mn_x_bytes(cols / 32, ng) + mn_ring_bytes(t, cols) <= (size_t)kSmemLimit) return 4 * ng;
  return 0;
}
// n <= matvec_mma_tokens(t, cols) tokens; arguments checked by the caller (matvec_n)
int matvec_mma(int t, const void* W, int rows, int cols, const float* X, int64_t x_stride, float* Y, int64_t y_stride, int n,
               int accumulate, cudaStream_t st, int dev, int sms, const Tables& tb) {
  MnParams p{};
  p.tb = tb;
  p.W = (const uint8_t*)W; p.x = X; p.y = Y; p.x_stride = x_stride; p.y_stride = y_stride;
  p.rows = rows; p.units = cols / 32; p.n = n; p.row_bytes = (uint32_t)row_bytes(t, cols); p.accumulate = accumulate;
  switch ((n + 3) / 4) {
    case 1: return mn_type<1>(t, p, st, dev, sms);
    case 2: return mn_type<2>(t, p, st, dev, sms);
    case 3: return mn_type<3>(t, p, st, dev, sms);
    default: return mn_type<4>(t, p, st, dev, sms);
  }
}

}  // namespace msb
