// Contraction of raw GGUF weight rows with half activations on tcgen05, the weights decoded inside the kernel into TMEM as
// the A operand (ts_decode.cuh: lane = weight row), the activations the B operand (shared memory, TMA).  One decode serves up
// to 128 activation rows, and a tile's M is always full however few rows there are.  Used by the MoE prefill (experts with
// few entries) and by the prefill projections of short prompts.
//   tile      256 weight rows (two M = 128 halves) x up to 128 activation rows x a range of K blocks of 64
//   warps     0..3 epilogue (one per TMEM lane quarter), 4..19 producers (four groups of four: half of the tile x parity of
//             the K piece; every group owns two of the eight 32-column operand slots), 20 and 21 MMA issuers (a half each),
//             22 activation loader (TMA)
//   TMEM      columns [0, 256): accumulators -- two tiles of up to 64 activation rows in turn, or one wider tile;
//             [256, 512): operand slots.  (Sixteen slots of half the size were slower, 2.50 -> 3.07 ms for 300 tokens of the
//             reference MoE layer: the hand-over costs more than the elasticity gives.)
// Every mbarrier wait is bounded.
#pragma once
#include <cuda.h>
#include "ts_decode.cuh"

namespace msb {

constexpr int kTsBK = 64;
constexpr int kTsMaxN = 128, kTsSmallN = 64;
constexpr int kTsEpiWarps = 4, kTsProdWarps = 16;
constexpr int kTsMmaWarp = kTsEpiWarps + kTsProdWarps;                        // two MMA warps, then the activation loader
constexpr int kTsThreads = (kTsMmaWarp + 3) * 32;
constexpr int kTsSlots = 8;                       // operand slots of 32 columns, two per producer group
constexpr int kTsRing = 4, kTsSlotBytes = kTsMaxN * kTsBK * 2;
constexpr int kTsRawWarp = 5120, kTsRawBytes = kTsProdWarps * kTsRawWarp;      // staged raw pieces of one producer warp
constexpr int kTsLutBytes = kIq1selLutBytes;
constexpr uint32_t kTsSlotCol = 2 * kTsMaxN;
constexpr int kTsExtraBytes = 16 * 1024;          // shared memory for the caller's own tables
constexpr size_t kTsSmem = 1024 + 1024 + (size_t)kTsRing * kTsSlotBytes + kTsLutBytes + kTsRawBytes + kTsExtraBytes;
static_assert(kTsSmem <= 227 * 1024, "shared memory");

// slot: the caller's; activation rows [row0, row0 + m), m <= kTsMaxN; weight rows from n0; K blocks [k0, k0 + kb), k0 on a piece
struct TsTile { int slot, row0, m, n0, k0, kb, type; };

struct TsHead {
  uint64_t full[kTsRing], empty[kTsRing], wfull[kTsSlots], wempty[kTsSlots], accfull[2], accempty[2], lutbar;
  uint32_t tmem_base;
  int abort_flag;
  uint2 fac[16];        // factor triples of the IQ type in use (ts_factors)
};

#ifdef __CUDACC__
extern __shared__ __align__(1024) uint8_t ts_smem_raw[];
__device__ __forceinline__ uint64_t ts_desc(uint32_t saddr) {   // K-major, 128-byte swizzle, 8-row groups 1024 B apart
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void ts_tma_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void ts_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void ts_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ts_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ts_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K block of step `st`: the two producer parities take pieces of 1 << sh K blocks in turn (piece 2 i by parity 0, 2 i + 1 by
// parity 1) and the MMA alternates between them; a last odd piece is parity 0's alone.
__device__ __forceinline__ int ts_kblock(int st, int kb, int sh, int& par) {
  const int pair = st >> (sh + 1), in = st & ((2 << sh) - 1);
  if (((pair + 1) << (sh + 1)) <= kb) { par = in & 1; return ((2 * pair + par) << sh) + (in >> 1); }
  par = 0;
  return st;
}
__device__ __forceinline__ int ts_piece_shift(int t) { const int k = ts_piece_k(t); return k == 256 ? 2 : k == 128 ? 1 : 0; }

// A producer warp's share of one tile: its 32 rows (the first `live`, at least one, exist), pieces p0 + (those of its parity
// below np).  `use` counts the group's operand slot uses.
template <int T>
__device__ __forceinline__ bool ts_produce(const uint8_t* rows, uint32_t rb, int live, int p0, int np, int par, uint32_t raw, uint32_t tslot,
                                           uint32_t& use, uint64_t* wfull, uint64_t* wempty, const LaneLuts& L, saddr_t fac, int lane,
                                           volatile int* abort_flag, int* status) {
  constexpr int PK = TsPiece<T>::kK, PB = PK / kTsBK, W = TsPiece<T>::kWords;
  constexpr bool kTwo = 2 * 32 * 4 * W <= kTsRawWarp;     // (room for two of the larger pieces too changed nothing)
  static_assert(32 * 4 * W <= kTsRawWarp, "a piece of 32 rows fits");
  const int last = np & 1 ? np - 1 : np;                 // pieces [last, np): parity 0
  TsMul mul;
  ts_mul_init<T>(mul);
  const uintptr_t my_row = reinterpret_cast<uintptr_t>(rows) + (uintptr_t)min(lane, live - 1) * rb;
  if (par < np) ts_stage<T>(raw, rows, rb, live, (uint32_t)(p0 + par), lane);
  ts_cp_commit();
  uint32_t buf = 0;
  for (int p = par; p < np && (p < last || par == 0); p += 2, buf ^= kTwo ? 1u : 0u) {
    // two buffers: the next piece is requested before this one is read; one: as soon as this one is in registers
    if (kTwo && p + 2 < np) ts_stage<T>(raw + (buf ^ 1u) * (32u * 4u * W), rows, rb, live, (uint32_t)(p0 + p + 2), lane);
    if (kTwo) ts_cp_commit();
    ts_cp_wait<kTwo ? 1 : 0>();
    __syncwarp();
    TsRow<T> r;
    ts_open<T>(r, raw + buf * (32u * 4u * W) + (uint32_t)lane * (4u * W), my_row, (uint32_t)(p0 + p), lane);
    if (!kTwo) {
      __syncwarp();
      if (p + 2 < np) ts_stage<T>(raw, rows, rb, live, (uint32_t)(p0 + p + 2), lane);
      ts_cp_commit();
    }
#pragma unroll
    for (int i = 0; i < PB; i++, use++) {
      const uint32_t sl = use & 1u;                      // the group's two slots in turn
      uint32_t o[16];
      ts_unit<T>(r, 2 * i, L, fac, mul, o);
      if (!__all_sync(0xffffffffu, mbar_wait(wempty + sl, ((use >> 1) & 1u) ^ 1u, abort_flag, status, kDevWaitEmpty))) return false;
      ts_fence_after();
      ts_st16(tslot + 32u * sl, o);
      ts_unit<T>(r, 2 * i + 1, L, fac, mul, o);
      ts_st16(tslot + 32u * sl + 16u, o);
      ts_wait_st();
      ts_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(wfull + sl);
    }
    __syncwarp();                                        // every lane has read its row before the buffer is filled again
  }
  return true;
}

// The kernel body.  Prob describes the work (see its uses): types() the weight types that may occur (at most one IQ type with
// a codebook among them), setup() copies its tables to `extra` after the dependency wait, tile(i) the i-th tile of this block,
// rows() a producer warp's 32 rows, a_small / a_large the activation maps with boxes of 16 / 64 rows x 64, epilogue() stores.
template <class Prob>
__device__ __forceinline__ void ts_gemm_body(Prob& pr, const Tables& tb) {
  pdl_launch_dependents();
  extern __shared__ __align__(1024) uint8_t ts_smem_raw[];
  uint8_t* smem = ts_smem_raw + ((1024u - (smem_u32(ts_smem_raw) & 1023u)) & 1023u);
  TsHead* hd = reinterpret_cast<TsHead*>(smem);
  uint8_t* ring = smem + 1024;
  uint8_t* lut = ring + kTsRing * kTsSlotBytes;
  uint8_t* raw = lut + kTsLutBytes;
  int* status = tb.status;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool iq1 = pr.has_type(IQ1_S), iq2 = pr.has_type(IQ2_XXS);    // not both
  if (tid == 0) {
    for (int s = 0; s < kTsRing; s++) { mbar_init(&hd->full[s], 1); mbar_init(&hd->empty[s], 2); }
    for (int s = 0; s < kTsSlots; s++) { mbar_init(&hd->wfull[s], 4); mbar_init(&hd->wempty[s], 1); }
    for (int b = 0; b < 2; b++) { mbar_init(&hd->accfull[b], 2); mbar_init(&hd->accempty[b], kTsEpiWarps); }
    mbar_init(&hd->lutbar, 1);
    hd->abort_flag = 0;
    mbar_fence_init();
  }
  if (tid >= 32 && tid < 48) hd->fac[tid - 32] = iq1 ? ts_factors<IQ1_S>(tid - 32) : ts_factors<IQ2_XXS>(tid - 32);
  if (warp == kTsMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&hd->tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  if (tid == 0 && (iq1 || iq2)) {                      // constant tables: before the dependency wait
    mbar_arrive_expect_tx(&hd->lutbar, iq1 ? (uint32_t)kIq1selLutBytes : (uint32_t)(kIq2GridLutBytes + kIq2SignLutBytes));
    if (iq1) {
      for (uint32_t o = 0; o < kIq1selLutBytes; o += 16384) tma_load_1d(lut + o, tb.img_iq1sel + o, 16384, &hd->lutbar);
    } else {
      for (uint32_t o = 0; o < kIq2GridLutBytes; o += 16384) tma_load_1d(lut + o, tb.img_iq2g + o, 16384, &hd->lutbar);
      tma_load_1d(lut + kIq2GridLutBytes, tb.img_iq2s, (uint32_t)kIq2SignLutBytes, &hd->lutbar);
    }
  }
  pdl_wait();
  pr.setup(raw + kTsRawBytes, tid);
  ts_fence_before();
  __syncthreads();
  ts_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, hd->tmem_base, 0);      // warp-uniform, and known to be
  volatile int* abort_flag = &hd->abort_flag;
  const int my_tiles = pr.ntiles > (int)blockIdx.x ? (pr.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  auto tile = [&](int i) { return pr.tile((int)blockIdx.x + i * (int)gridDim.x); };

  if (warp == kTsMmaWarp + 2) {
    // ------------------------------------------------------------------ activation loader (one thread)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int i = 0; ok && i < my_tiles; i++) {
        const TsTile tl = tile(i);
        const int sh = ts_piece_shift(tl.type);
        const bool small = tl.m <= 32;
        const int step = small ? 16 : 64, boxes = (tl.m + step - 1) / step;
        for (int st = 0; st < tl.kb; st++, it++) {
          int par;
          const int k = tl.k0 + ts_kblock(st, tl.kb, sh, par), s = it % kTsRing;
          if (!mbar_wait(&hd->empty[s], ((it / kTsRing) & 1u) ^ 1u, abort_flag, status, kDevWaitEmpty)) { ok = false; break; }
          uint8_t* slot = ring + (size_t)s * kTsSlotBytes;
          mbar_arrive_expect_tx(&hd->full[s], (uint32_t)(boxes * step * kTsBK * 2));
          for (int b = 0; b < boxes; b++)
            ts_tma_2d(slot + b * step * kTsBK * 2, small ? pr.a_small() : pr.a_large(), k * kTsBK, tl.row0 + b * step, &hd->full[s]);
        }
      }
    }
  } else if (warp >= kTsMmaWarp) {
    // ------------------------------------------------------------------ MMA issuers: one warp per half of the tile
    const int half = warp - kTsMmaWarp;
    const bool leader = elect_one();
    uint32_t it = 0, acc = 0, use0 = 0, use1 = 0;        // slot uses of the groups of parity 0 / 1
    bool ok = true;
    auto wait_acc = [&](uint32_t b) {
      return __all_sync(0xffffffffu, mbar_wait_sleep(&hd->accempty[b], ((acc >> 1) & 1u) ^ 1u, abort_flag, status, kDevWaitEmpty, 100)) != 0;
    };
    for (int i = 0; ok && i < my_tiles; i++) {
      const TsTile tl = tile(i);
      const int sh = ts_piece_shift(tl.type);
      const bool wide = tl.m > kTsSmallN;
      const uint32_t idesc = (1u << 4) | ((uint32_t)((tl.m + 15) >> 4) << 18) | (8u << 24);   // f16 x f16 -> f32, N / 8 at bit 17, M 128
      if (wide && (acc & 1u)) {                          // a wide tile takes both accumulators, from the first one on
        if (!wait_acc(1)) break;
        if (leader) mbar_arrive(&hd->accfull[1]);
        acc++;
      }
      const uint32_t b0 = acc & 1u;
      if (!wait_acc(b0)) break;
      if (wide && !wait_acc(1)) break;
      ts_fence_after();
      const uint32_t d = tmem + b0 * (uint32_t)kTsMaxN + (uint32_t)(half ? (wide ? kTsMaxN : kTsSmallN) : 0);
      for (int st = 0; st < tl.kb; st++, it++) {
        int par;
        ts_kblock(st, tl.kb, sh, par);
        const int s = it % kTsRing;
        const uint32_t n = par ? use1 : use0;
        const uint32_t slot = 2u * (uint32_t)(2 * par + half) + (n & 1u), b_s = smem_u32(ring) + (uint32_t)s * (uint32_t)kTsSlotBytes;
        ok = __all_sync(0xffffffffu, mbar_wait(&hd->full[s], (it / kTsRing) & 1u, abort_flag, status, kDevWaitFull) &&
                                         mbar_wait(&hd->wfull[slot], (n >> 1) & 1u, abort_flag, status, kDevWaitFull));
        if (!ok) break;
        ts_fence_after();
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < kTsBK / 16; ks++)
            ts_mma_f16(d, tmem + kTsSlotCol + 32u * slot + 8u * ks, ts_desc(b_s + ks * 32), idesc, (st > 0 || ks > 0) ? 1u : 0u);
          ts_commit(&hd->wempty[slot]);
          ts_commit(&hd->empty[s]);
        }
        __syncwarp();
        if (par) use1++; else use0++;
      }
      if (!ok) break;
      if (leader) {
        ts_commit(&hd->accfull[b0]);
        if (wide) ts_commit(&hd->accfull[1]);
      }
      __syncwarp();
      acc += wide ? 2 : 1;
    }
  } else if (warp >= kTsEpiWarps) {
    // ------------------------------------------------------------------ producers
    const int pw = warp - kTsEpiWarps, group = pw >> 2, quarter = warp & 3, half = group & 1, par = group >> 1;
    LaneLuts L;
    L.iq1s = smem_u32(lut) + 8u * (lane % kIq1selCopies);
    L.iq2g = smem_u32(lut) + 4u * lane;
    L.iq2s = L.iq2g + (uint32_t)kIq2GridLutBytes;
    const saddr_t fac = smem_u32(hd->fac);
    bool ok = !(iq1 || iq2) || __all_sync(0xffffffffu, mbar_wait(&hd->lutbar, 0, abort_flag, status, kDevWaitFull));
    const uint32_t my_raw = smem_u32(raw) + (uint32_t)pw * kTsRawWarp;
    const uint32_t tslot = tmem + ((uint32_t)(32 * quarter) << 16) + kTsSlotCol + 64u * group;
    uint32_t use = 0;
    TsTile nx = my_tiles > 0 ? tile(0) : TsTile{};
    for (int i = 0; ok && i < my_tiles; i++) {
      const TsTile tl = nx;
      int live;
      uint32_t rb;
      if (i + 1 < my_tiles) nx = tile(i + 1);
      if (Prob::kWholeK && i + 1 < my_tiles) {
        // the next tile's rows into L2 (this parity's half of the lines): its pieces then come at L2 latency
        const uint8_t* q = pr.rows(nx, half, quarter, rb, live);
        const uint32_t bytes = (uint32_t)live * rb;
        for (uint32_t o = 128u * (lane * 2 + par); o < bytes; o += 128u * 64u) asm volatile("prefetch.global.L2 [%0];" ::"l"(q + o));
      }
      const uint8_t* rows = pr.rows(tl, half, quarter, rb, live);
#define TS_PRODUCE(T)                                                                                                                     \
  case T:                                                                                                                                 \
    if constexpr (Prob::template kHas<T>)                                                                                                 \
      ok = ts_produce<T>(rows, rb, live, tl.k0 / (TsPiece<T>::kK / kTsBK), tl.kb / (TsPiece<T>::kK / kTsBK), par, my_raw, tslot, use,      \
                         &hd->wfull[2 * group], &hd->wempty[2 * group], L, fac, lane, abort_flag, status);                                \
    break;
      switch (tl.type) {
        TS_PRODUCE(IQ1_S)
        TS_PRODUCE(IQ2_XXS)
        TS_PRODUCE(Q8_0)
        TS_PRODUCE(Q6_K)
        TS_PRODUCE(Q5_K)
        TS_PRODUCE(IQ4_NL)
        TS_PRODUCE(BF16)
        TS_PRODUCE(F16)
      }
#undef TS_PRODUCE
    }
    ts_cp_wait<0>();
  } else {
    // ------------------------------------------------------------------ epilogue: TMEM lane = weight row, column = activation row
    const int quarter = warp & 3;
    uint32_t acc = 0;
    for (int i = 0; i < my_tiles; i++) {
      const TsTile tl = tile(i);
      const bool wide = tl.m > kTsSmallN;
      if (wide && (acc & 1u)) {
        if (!__all_sync(0xffffffffu, mbar_wait_sleep(&hd->accfull[1], (acc >> 1) & 1u, abort_flag, status, kDevWaitFull, 100))) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(&hd->accempty[1]);
        acc++;
      }
      const uint32_t b0 = acc & 1u, ph = (acc >> 1) & 1u;
      if (!__all_sync(0xffffffffu, mbar_wait_sleep(&hd->accfull[b0], ph, abort_flag, status, kDevWaitFull, 100))) break;
      if (wide && !__all_sync(0xffffffffu, mbar_wait_sleep(&hd->accfull[1], ph, abort_flag, status, kDevWaitFull, 100))) break;
      ts_fence_after();
      const uint32_t d0 = tmem + ((uint32_t)(32 * quarter) << 16) + b0 * (uint32_t)kTsMaxN;
      pr.epilogue(tl, d0, d0 + (uint32_t)(wide ? kTsMaxN : kTsSmallN), quarter, lane);
      ts_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&hd->accempty[b0]);
        if (wide) mbar_arrive(&hd->accempty[1]);
      }
      acc += wide ? 2 : 1;
    }
  }
  ts_fence_before();
  __syncthreads();
  if (warp == kTsMmaWarp) {
    ts_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}
#endif  // __CUDACC__

}  // namespace msb
