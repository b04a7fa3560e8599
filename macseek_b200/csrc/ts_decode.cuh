// Weight decoding for contractions whose weights are the tensor core's A operand in TMEM: raw GGUF rows -> half pairs in
// registers, written with tcgen05.st (lane = weight row, one 32-bit column = two consecutive K elements).
//
// A producer warp owns 32 consecutive weight rows of a tile, one per lane.  The rows' bytes come a PIECE at a time (a run of
// K elements whose blocks lie together): the warp copies the 32 rows' pieces into shared memory with cp.async, four to eight
// lanes per row, so that a copy instruction touches four or eight rows' lines instead of 32, and lane l then reads row l.
//   IQ1_S, IQ2_XXS  the piece is one 256-element block; it is copied as the 16-byte chunks it touches (4 or 5 however it is
//                   aligned), read back with 16-byte loads and shifted into place in registers once (5 or 6 instructions per
//                   32 weights; 4-byte copies and loads took 15 and, per piece, 16 copy instructions instead of 4 or 5)
//   Q8_0, Q6_K, Q5_K, IQ4_NL   128 elements, 4-byte copies (an odd number of words per row: no bank conflicts)
//   F16, BF16       64 elements of 16-byte aligned rows
// Against an operand tile in shared memory this takes two trips out of the
// shared-memory pipe per weight (the producers' stores and the tensor core's reads), which is what bounded that form.
#pragma once
#include "quant_blocks.cuh"

namespace msb {

// K elements of a piece, and 32-bit words staged per row of it (4-byte copies: the piece plus up to 2 bytes)
template <int T> struct TsPiece;
template <> struct TsPiece<IQ1_S> { static constexpr int kK = 256, kWords = 16; };      // 4 chunks of 16 bytes, chunk c of row r at c ^ (r / 2 % 4)
template <> struct TsPiece<IQ2_XXS> { static constexpr int kK = 256, kWords = 20; };    // 5 chunks
template <> struct TsPiece<Q8_0> { static constexpr int kK = 128, kWords = 35; };       // four 34-byte blocks
template <> struct TsPiece<Q6_K> { static constexpr int kK = 128, kWords = 31; };       // half a block: ql 17, qh 9, scales + d 5
template <> struct TsPiece<Q5_K> { static constexpr int kK = 128, kWords = 31; };       // half a block: d, dmin, scales, qh 13; qs 17 (+ 1 to be odd)
template <> struct TsPiece<IQ4_NL> { static constexpr int kK = 128, kWords = 19; };     // four 18-byte blocks
template <> struct TsPiece<F16> { static constexpr int kK = 64, kWords = 36; };         // 8 chunks (16-byte aligned rows), 9 apart
template <> struct TsPiece<BF16> { static constexpr int kK = 64, kWords = 36; };
__host__ __device__ constexpr int ts_piece_k(int t) { return t == IQ1_S || t == IQ2_XXS ? 256 : t == F16 || t == BF16 ? 64 : 128; }

#ifdef __CUDACC__
// byte offset of staged word w of a piece (half h of its block), from the piece's (Q6_K, Q5_K: the block's) first byte
template <int T>
__device__ __forceinline__ uint32_t ts_seg(uint32_t w, uint32_t h) {
  if (T == Q6_K) return w < 17u ? 64u * h + 4u * w : w < 26u ? 128u + 32u * h + 4u * (w - 17u) : 192u + 4u * (w - 26u);
  if (T == Q5_K) return w < 13u ? 4u * w : 48u + 64u * h + 4u * (w - 13u);
  return 4u * w;
}
// first byte of a row's piece; the staged words start there rounded down to 4
template <int T>
__device__ __forceinline__ uint32_t ts_piece_off(uint32_t p) {
  return T == Q6_K || T == Q5_K ? (p >> 1) * (uint32_t)block_bytes(T) : T == Q8_0 || T == IQ4_NL ? p * 4u * (uint32_t)block_bytes(T) : p * (uint32_t)block_bytes(T);
}
__device__ __forceinline__ void ts_cp4(uint32_t dst, const uint8_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ts_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void ts_cp16(uint32_t dst, const uint8_t* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <int N>
__device__ __forceinline__ void ts_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// rows [0, 32) at `rows` (stride rb; those from `live` on do not exist: the last one stands in): copy piece p of each to
// dst[row * kWords].
// IQ types: a chunk's 16 bytes hold at least one byte of the block, so no copy leaves the matrix's last 16-byte line.
template <int T>
__device__ __forceinline__ void ts_stage(uint32_t dst, const uint8_t* rows, uint32_t rb, int live, uint32_t p, int lane) {
  if constexpr (T == IQ1_S || T == IQ2_XXS) {
    constexpr uint32_t C = TsPiece<T>::kWords / 4;
    static_assert((block_bytes(T) - 1) / 16 + 1 == C && (14 + block_bytes(T) - 1) / 16 + 1 == C, "the same number of chunks at every offset");
    const uintptr_t base = reinterpret_cast<uintptr_t>(rows) + p * (uint32_t)block_bytes(T);
    auto copy = [&](uint32_t to, uintptr_t from) { ts_cp16(to, reinterpret_cast<const uint8_t*>(from & ~(uintptr_t)15)); };
    if (T == IQ1_S && live == 32) {                      // four chunks: a lane's are of rows 8 apart, at the same place in each
      const uint32_t r = (uint32_t)lane >> 2, c = (uint32_t)lane & 3u;
      const uintptr_t from = base + r * rb + 16u * c;
      const uint32_t to = dst + 16u * (4u * r + (c ^ ((r >> 1) & 3u)));
#pragma unroll
      for (uint32_t i = 0; i < C; i++) copy(to + 512u * i, from + (uintptr_t)(8u * rb) * i);
      return;
    }
#pragma unroll
    for (uint32_t i = 0; i < C; i++) {
      const uint32_t f = (uint32_t)lane + 32u * i, r = f / C, c = f - r * C, pos = T == IQ1_S ? c ^ ((r >> 1) & 3u) : c;
      copy(dst + 16u * (r * C + pos), base + (uintptr_t)(min((int)r, live - 1) * rb) + 16u * c);
    }
    return;
  }
  if constexpr (T == F16 || T == BF16) {               // rows are 16-byte aligned: eight whole chunks, nine per row in shared memory
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) {
      const uint32_t r = (uint32_t)(lane >> 3) + 4u * i, c = (uint32_t)lane & 7u;
      ts_cp16(dst + 144u * r + 16u * c, rows + (size_t)min((int)r, live - 1) * rb + p * 128u + 16u * c);
    }
    return;
  }
  // Eight lanes per row, four rows per pass.
  constexpr uint32_t W = TsPiece<T>::kWords, J = (W + 7) / 8;
  const uint32_t w0 = (uint32_t)lane & 7u, r0 = (uint32_t)lane >> 3;
  const uint8_t* base = rows + ts_piece_off<T>(p);
  const uint32_t d = dst + 4u * (r0 * W + w0);
  uint32_t off[J];                                   // from the piece's first byte, a multiple of 4
#pragma unroll
  for (uint32_t j = 0; j < J; j++) off[j] = ts_seg<T>(w0 + 8u * j, p & 1u);
#pragma unroll
  for (uint32_t k = 0; k < 8; k++) {
    const uint8_t* q = base + (size_t)min((int)(r0 + 4u * k), live - 1) * rb;
    const uint8_t* a = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(q) & ~(uintptr_t)3);
#pragma unroll
    for (uint32_t j = 0; j < J; j++) {
      if (8u * j + 8u > W && w0 + 8u * j >= W) continue;
      // the last word of an aligned row lies past its piece (and past the matrix at its end), Q5_K's padding always; nobody reads it
      constexpr uint32_t kEnd = T == Q5_K ? W - 2 : W - 1;
      if (T == Q5_K && w0 + 8u * j > kEnd) continue;
      if (T != Q6_K && 8u * j + 8u > W && w0 + 8u * j == kEnd && (reinterpret_cast<uintptr_t>(q) & 2) == 0) continue;
      ts_cp4(d + 16u * k * W + 32u * j, a + off[j]);
    }
  }
}

__device__ __forceinline__ uint32_t ts_prmt(uint32_t a, uint32_t b, uint32_t sel) {   // byte permute; every selector nibble here is below 8
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ uint32_t ts_sign_bytes(uint32_t x) {   // 0xFF for the bytes of x with the top bit set, else 0
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, 0xBA98;" : "=r"(r) : "r"(x));
  return r;
}
__device__ __forceinline__ uint32_t ts_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

// ---- decoding.  TsRow: the lane's row of the staged piece; unit u = 32 elements, o[k] = halfs of elements 2k, 2k + 1.
// IQ types: f[k] = the 32-bit word at byte 2 + 4 k of the block (qs, then for IQ1_S qh), d2 = the block scale twice.
// Q types: the whole piece in registers too, so that its one buffer can be filled again while it is decoded.
template <int T> struct TsRow;
template <> struct TsRow<Q8_0> { uint32_t w[4][8], d[4]; };
template <> struct TsRow<Q6_K> { uint32_t ql[2][8], qh[8], sc[2]; float d; };
template <> struct TsRow<Q5_K> { uint32_t qs[2][8], qh[8], sc[3], half; float d, dmin; };
template <> struct TsRow<IQ4_NL> { uint32_t w[4][4], d[4]; };
template <> struct TsRow<F16> { uint32_t w[32]; };
template <> struct TsRow<BF16> { uint32_t w[32]; };
template <> struct TsRow<IQ1_S> { uint32_t f[12], d2; };
template <> struct TsRow<IQ2_XXS> { uint32_t f[16], d2; };
template <int T>
__device__ __forceinline__ void ts_open(TsRow<T>& r, saddr_t staged, uintptr_t row_addr, uint32_t piece, int lane) {
  if constexpr (T == IQ1_S || T == IQ2_XXS) {
    constexpr int C = TsPiece<T>::kWords / 4, N = sizeof(r.f) / 4;
    const uint32_t o = (uint32_t)(row_addr + piece * (uint32_t)block_bytes(T)) & 15u;     // the block's first byte in chunk 0
    const uint32_t x = T == IQ1_S ? ((uint32_t)lane >> 1) & 3u : 0u;
    uint32_t w[4 * C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      const uint4 v = lds_u128(staged + 16u * ((uint32_t)c ^ x));
      w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
    }
    r.d2 = ts_prmt(lds_u16(staged + 16u * x + o), 0, 0x1010);
    const bool two = (o & 8u) != 0, one = (o & 4u) != 0;
#pragma unroll
    for (int i = 0; i < N + 2; i++) w[i] = two ? w[i + 2] : w[i];
#pragma unroll
    for (int i = 0; i < N + 1; i++) w[i] = one ? w[i + 1] : w[i];
    const uint32_t sh = 16u + 8u * (o & 2u);           // 16 or 32
#pragma unroll
    for (int i = 0; i < N; i++) r.f[i] = __funnelshift_rc(w[i], w[i + 1], sh);
  } else if constexpr (T == F16 || T == BF16) {
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const uint4 v = lds_u128(staged + 16u * c);
      r.w[4 * c] = v.x; r.w[4 * c + 1] = v.y; r.w[4 * c + 2] = v.z; r.w[4 * c + 3] = v.w;
    }
  } else {
    const saddr_t b = staged + ((uint32_t)(row_addr + ts_piece_off<T>(piece)) & 2u);
    if constexpr (T == Q8_0) {
#pragma unroll
      for (int u = 0; u < 4; u++) { load_words<8>(b + 34u * u + 2u, r.w[u]); r.d[u] = lds_u16(b + 34u * u); }
    } else if constexpr (T == IQ4_NL) {
#pragma unroll
      for (int u = 0; u < 4; u++) { load_words<4>(b + 18u * u + 2u, r.w[u]); r.d[u] = lds_u16(b + 18u * u); }
    } else if constexpr (T == Q5_K) {
      r.half = piece & 1u;
      r.d = lds_half(b); r.dmin = lds_half(b + 2u);
      load_words<3>(b + 4u, r.sc);
      load_words<8>(b + 16u, r.qh);
      load_words<8>(b + 52u, r.qs[0]);
      load_words<8>(b + 84u, r.qs[1]);
    } else {
      load_words<8>(b, r.ql[0]);
      load_words<8>(b + 32u, r.ql[1]);
      load_words<8>(b + 68u, r.qh);
      load_words<2>(b + 104u + 8u * (piece & 1u), r.sc);
      r.d = lds_half(b + 104u + 16u);
    }
  }
}
// The byte permutes fill the ALU (half the issue rate), so what else can goes to the multiply-add pipe: address arithmetic
// and shifts as multiplications with multipliers the compiler cannot see through (powers of two would come back as shifts).
struct TsMul { uint32_t byte, hi[4], top; };         // byte -> table bytes; IQ1_S: the four qh fields -> table bytes; 2^16
template <int T>
__device__ __forceinline__ void ts_mul_init(TsMul& m) {
  constexpr uint32_t kByte = T == IQ1_S ? 8 * kIq1selCopies : 4 * kIq2Copies;
  asm volatile("mov.u32 %0, %1;" : "=r"(m.byte) : "n"(kByte));
  asm volatile("mov.u32 %0, 65536;" : "=r"(m.top));
#pragma unroll
  for (int l = 0; l < 4; l++) { const uint32_t v = (2048u * kIq1selCopies) >> (3 * l); asm volatile("mov.u32 %0, %1;" : "=r"(m.hi[l]) : "r"(v)); }
}
__device__ __forceinline__ uint32_t ts_top16(uint32_t x, const TsMul& m) {     // x >> 16
  uint32_t r;
  asm("mul.hi.u32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(m.top));
  return r;
}
__device__ __forceinline__ uint32_t ts_hmul2(uint32_t a, uint32_t b) {
  return ts_u32(__hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b)));
}
// The distinct values of a unit are d times a factor that is exact in half (IQ1_S: (2 s + 1) (g + delta), at most 8 bits;
// IQ2_XXS: (2 s + 1) / 8 times 8, 25 or 43, at most 11 bits), and d is a half: one half multiplication rounds the exact
// product once, as the float product rounded to half does.  The 16 factor triples are a table: entry s | (delta < 0) << 3 for
// IQ1_S, entry s for IQ2_XXS; 8 bytes {f0, f1, f2, 0}, 128 bytes in all, no bank conflicts.
template <int T>
__device__ __forceinline__ uint2 ts_factors(int e) {
  float f[3];
  if (T == IQ1_S) {
    const float m = (float)(2 * (e & 7) + 1), delta = e & 8 ? -0.125f : 0.125f;
    f[0] = m * (delta - 1.f); f[1] = m * delta; f[2] = m * (delta + 1.f);
  } else {
    const float m = (float)(2 * e + 1) * 0.125f;
    f[0] = m * 8.f; f[1] = m * 25.f; f[2] = m * 43.f;
  }
  return make_uint2(ts_u32(__floats2half2_rn(f[0], f[1])), ts_u32(__floats2half2_rn(f[2], 0.f)));
}
// IQ1_S: a table entry holds the byte-permute selectors of its four pairs of values
__device__ __forceinline__ void ts_unit_iq1s(uint32_t qs, uint32_t h, uint32_t d2, saddr_t lut, saddr_t fac, const TsMul& mul, uint32_t (&o)[16]) {
  const uint2 f = lds_u64(fac + ((h >> 9) & 0x78u));
  const uint32_t h01 = ts_hmul2(f.x, d2), h2 = ts_hmul2(f.y, d2);
#pragma unroll
  for (int l = 0; l < 4; l++) {
    const uint32_t at = ts_prmt(qs, 0, 0x4440 | l) * mul.byte + ((h & (7u << (3 * l))) * mul.hi[l] + lut);
    const uint2 w = lds_u64(at);
    o[4 * l] = ts_prmt(h01, h2, w.x); o[4 * l + 1] = ts_prmt(h01, h2, ts_top16(w.x, mul));
    o[4 * l + 2] = ts_prmt(h01, h2, w.y); o[4 * l + 3] = ts_prmt(h01, h2, ts_top16(w.y, mul));
  }
}
// IQ2_XXS: three magnitudes and their negatives; grid nibble (0..2) + 3 for a negative element, in element order, picks low
// and high bytes with one permute each per four elements, two more put the halfs together
__device__ __forceinline__ void ts_unit_iq2(uint32_t q, uint32_t a1, uint32_t d2, saddr_t lutg, saddr_t luts, saddr_t fac, const TsMul& mul,
                                            uint32_t (&o)[16]) {
  const uint2 f = lds_u64(fac + ((a1 >> 25) & 0x78u));
  const uint32_t m01 = ts_hmul2(f.x, d2), m2 = ts_hmul2(f.y, d2);
  const uint32_t n01 = m01 ^ 0x80008000u, n2 = m2 ^ 0x80008000u;
  // low bytes (the same for both signs) and high bytes of {m0, m1, m2, -m0 | -m1, -m2}
  const uint32_t l4 = ts_prmt(m01, m2, 0x0420), l2 = ts_prmt(m01, m2, 0x0042);
  const uint32_t h3 = ts_prmt(m01, m2, 0x0531);
  const uint32_t h4 = ts_prmt(h3, n01, 0x5210), h2 = ts_prmt(n01, n2, 0x0053);
#pragma unroll
  for (int l = 0; l < 4; l++) {
    const uint32_t g = lds_u32(ts_prmt(q, 0, 0x4440 | l) * mul.byte + lutg);
    const uint32_t m = lds_u32(((a1 >> (7 * l)) & 127u) * mul.byte + luts);
    const uint32_t w = g + m, t = ts_top16(w, mul);
    const uint32_t a = ts_prmt(l4, l2, w), b = ts_prmt(h4, h2, w);                // elements 0..3
    const uint32_t c = ts_prmt(l4, l2, t), e = ts_prmt(h4, h2, t);                // elements 4..7
    o[4 * l] = ts_prmt(a, b, 0x5140); o[4 * l + 1] = ts_prmt(a, b, 0x7362);
    o[4 * l + 2] = ts_prmt(c, e, 0x5140); o[4 * l + 3] = ts_prmt(c, e, 0x7362);
  }
}
// Q8_0: code and scale are halfs, their product rounds once (as the float product rounded to half does)
__device__ __forceinline__ void ts_unit_q8(const uint32_t (&w)[8], uint32_t dbits, uint32_t (&o)[16]) {
  const uint32_t d2 = dbits | (dbits << 16);
  const __half2 dd = *reinterpret_cast<const __half2*>(&d2);
  const __half2 off = __floats2half2_rn(1152.f, 1152.f);
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint32_t b = w[i] ^ 0x80808080u;                                     // code + 128
    const uint32_t v0 = ts_prmt(b, 0x64646464u, 0x4140), v1 = ts_prmt(b, 0x64646464u, 0x4342);   // 1024 + code + 128
    o[2 * i] = ts_u32(__hmul2(__hsub2(*reinterpret_cast<const __half2*>(&v0), off), dd));
    o[2 * i + 1] = ts_u32(__hmul2(__hsub2(*reinterpret_cast<const __half2*>(&v1), off), dd));
  }
}
// Q6_K: (d * scale) * (code - 32) in float, rounded to half; two scales of 16 elements
__device__ __forceinline__ void ts_unit_q6(const uint32_t (&ql)[8], const uint32_t (&qh)[8], int nsh, int hsh, float s0, float s1,
                                           uint32_t (&o)[16]) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint32_t c = ((ql[i] >> nsh) & 0x0F0F0F0Fu) | (((qh[i] >> hsh) & 0x03030303u) << 4);
    const float sc = i < 4 ? s0 : s1;
    float f[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      f[k] = __fmul_rn(sc, __uint_as_float(ts_prmt(c, 0x4B000000u, 0x7540 | k)) - 8388640.f);   // 2^23 + code - (2^23 + 32)
    o[2 * i] = ts_u32(__floats2half2_rn(f[0], f[1]));
    o[2 * i + 1] = ts_u32(__floats2half2_rn(f[2], f[3]));
  }
}
// Q5_K: d1 * code - m1 in float (each operation rounded, as the reference), rounded to half; u = sub-block 4 half + u of 8
__device__ __forceinline__ void ts_unit_q5(const uint32_t (&qs)[8], const uint32_t (&qh)[8], int nsh, int hsh, float d1, float m1, uint32_t (&o)[16]) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint32_t c = ((qs[i] >> nsh) & 0x0F0F0F0Fu) | (((qh[i] >> hsh) & 0x01010101u) << 4);
    float f[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      f[k] = __fsub_rn(__fmul_rn(d1, __uint_as_float(ts_prmt(c, 0x4B000000u, 0x7540 | k)) - 8388608.f), m1);
    o[2 * i] = ts_u32(__floats2half2_rn(f[0], f[1]));
    o[2 * i + 1] = ts_u32(__floats2half2_rn(f[2], f[3]));
  }
}
// IQ4_NL: levels + 128 from four 4-byte tables (the low three bits of a code select in each pair, its top bit between the
// pairs), then as Q8_0; low nibbles are elements 0..15, high nibbles 16..31
__device__ __forceinline__ void ts_unit_iq4(const uint32_t (&w)[4], uint32_t dbits, uint32_t (&o)[16]) {
  // levels -127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113, each + 128
  constexpr uint32_t a0 = 0x3F2D1801u, a1 = 0x766A5D4Fu, b0 = 0xA6998D81u, b1 = 0xF1D9C5B5u;
  const uint32_t d2 = dbits | (dbits << 16);
  const __half2 dd = *reinterpret_cast<const __half2*>(&d2);
  const __half2 off = __floats2half2_rn(1152.f, 1152.f);
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t n = h ? w[i] >> 4 : w[i];                                   // codes in the low nibble of each byte
      const uint32_t lo3 = n & 0x07070707u;
      const uint32_t sel = ts_prmt(lo3 | (lo3 >> 4), 0, 0x0020);                 // nibbles c0, c1, c2, c3 in the low 16 bits
      const uint32_t top = ts_sign_bytes(n << 4);                                // 0xFF in the bytes whose code is 8 or more
      const uint32_t b = (ts_prmt(a0, a1, sel) & ~top) | (ts_prmt(b0, b1, sel) & top);
      const uint32_t v0 = ts_prmt(b, 0x64646464u, 0x4140), v1 = ts_prmt(b, 0x64646464u, 0x4342);
      o[8 * h + 2 * i] = ts_u32(__hmul2(__hsub2(*reinterpret_cast<const __half2*>(&v0), off), dd));
      o[8 * h + 2 * i + 1] = ts_u32(__hmul2(__hsub2(*reinterpret_cast<const __half2*>(&v1), off), dd));
    }
}
// unit u of the piece (0 .. kK / 32 - 1)
template <int T>
__device__ __forceinline__ void ts_unit(const TsRow<T>& r, int u, const LaneLuts& L, saddr_t fac, const TsMul& mul, uint32_t (&o)[16]) {
  if constexpr (T == IQ1_S) {
    ts_unit_iq1s(r.f[u], r.f[8 + (u >> 1)] >> (16 * (u & 1)), r.d2, L.iq1s, fac, mul, o);       // bits above the unit's 16 are masked off
  } else if constexpr (T == IQ2_XXS) {
    ts_unit_iq2(r.f[2 * u], r.f[2 * u + 1], r.d2, L.iq2g, L.iq2s, fac, mul, o);
  } else if constexpr (T == Q8_0) {
    ts_unit_q8(r.w[u], r.d[u], o);
  } else if constexpr (T == IQ4_NL) {
    ts_unit_iq4(r.w[u], r.d[u], o);
  } else if constexpr (T == F16) {
#pragma unroll
    for (int i = 0; i < 16; i++) o[i] = r.w[16 * u + i];
  } else if constexpr (T == BF16) {
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t v = r.w[16 * u + i];
      o[i] = ts_u32(__floats2half2_rn(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u)));
    }
  } else if constexpr (T == Q5_K) {
    // scales: sub-blocks 0..3 the low 6 bits of bytes j and j + 4; 4..7 nibbles of byte j + 4 with the top bits of bytes j - 4 and j
    const int sh = 8 * u;
    uint32_t scale, mn;
    if (r.half == 0) { scale = (r.sc[0] >> sh) & 63u; mn = (r.sc[1] >> sh) & 63u; }
    else {
      const uint32_t hi = r.sc[2] >> sh;
      scale = (hi & 15u) | (((r.sc[0] >> (sh + 6)) & 3u) << 4);
      mn = ((hi >> 4) & 15u) | (((r.sc[1] >> (sh + 6)) & 3u) << 4);
    }
    ts_unit_q5(r.qs[u >> 1], r.qh, 4 * (u & 1), 4 * (int)r.half + u, __fmul_rn(r.d, (float)scale), __fmul_rn(r.dmin, (float)mn), o);
  } else if constexpr (T == Q6_K) {
    const uint32_t sc = r.sc[u >> 1] >> (16 * (u & 1));                        // two int8 scales
    ts_unit_q6(r.ql[u & 1], r.qh, 4 * (u >> 1), 2 * u, __fmul_rn(r.d, (float)(int8_t)(sc & 0xFFu)), __fmul_rn(r.d, (float)(int8_t)((sc >> 8) & 0xFFu)), o);
  }
}
// TMEM: 16 columns (32 halfs) of the warp's 32 lanes
__device__ __forceinline__ void ts_st16(uint32_t taddr, const uint32_t (&o)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]),
      "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(o[15])
      : "memory");
}
__device__ __forceinline__ void ts_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[128 lanes x N] (+)= A[TMEM: 128 lanes x 16 halfs] . B[shared: N rows x 16 halfs]^T
__device__ __forceinline__ void ts_mma_f16(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void ts_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
#endif  // __CUDACC__

}  // namespace msb
