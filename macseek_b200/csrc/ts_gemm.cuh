// Contraction of raw GGUF weight rows with half activations on tcgen05, the weights decoded inside the kernel into TMEM as
// the A operand (ts_decode.cuh: lane = weight row), the activations the B operand (shared memory, TMA).  One decode serves up
// to 128 activation rows, and a tile's M is always full however few rows there are.  Used by the MoE prefill (experts with
// few entries) and by the prefill projections of short prompts.
//   tile      256 weight rows (two M = 128 halves) x up to 128 activation rows x a range of K blocks of 64
//   warps     0..3 epilogue (one per TMEM lane quarter), 4..19 producers (four groups of four: half of the tile x parity of
//             the K piece; every group owns two of the eight 32-column operand slots), 20 and 21 MMA issuers (a half each),
//             22 activation loader (TMA)
//             What bounds a tile: a fifth of a call's time is decoding, the rest is there without it -- fetching the raw pieces, the
//             hand-over of slots, a tile's start and end (MoE prefill of the reference layer, us, as it is / decoded values replaced by
//             constants / nothing fetched either: 27 tokens 697 / 539 / 432, 300 tokens 1982 / 1505 / 1300, 4096 tokens 3490 / 2854 / 2801)
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

// A producer warp's part of a tile: its 32 rows (the first `live` exist), K blocks as above.
struct TsWork { const uint8_t* rows; int live, k0, kb, type; };

struct TsHead {
  uint64_t full[kTsRing], empty[kTsRing], wfull[kTsSlots], wempty[kTsSlots], accfull[2], accempty[2], lutbar;
  uint32_t tmem_base;
  int abort_flag;
  uint2 fac[16];        // factor triples of the IQ type in use (ts_factors)
  TsWork next[kTsProdWarps];   // every producer warp's next tile (kNextInSmem)
};
static_assert(sizeof(TsHead) <= 1024, "the ring follows");

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

// The pieces of 1 << sh K blocks go to the two producer parities in turn (even pieces to the tile's first parity, odd ones to its
// second) and the MMA alternates between them: couple c is K block ts_kblock(c, sh) of the first and the one 1 << sh behind it of the
// second; what is left after the couples (a last odd piece) is the first's alone, in order.  After a tile with such a piece the
// parities change places, so that neither has the extra work every time (9 pieces a row: 5 and 4).
__device__ __forceinline__ int ts_couples(int kb, int sh) { return (kb >> (sh + 1)) << sh; }
__device__ __forceinline__ bool ts_odd(int kb, int sh) { return (kb >> sh) & 1; }
__device__ __forceinline__ int ts_kblock(int c, int sh) { return ((c >> sh) << (sh + 1)) + (c & ((1 << sh) - 1)); }
__device__ __forceinline__ int ts_piece_shift(int t) { const int k = ts_piece_k(t); return k == 256 ? 2 : k == 128 ? 1 : 0; }

__device__ __forceinline__ TsTile uniform_tile(const TsTile& t) {
  return TsTile{uniform(t.slot), uniform(t.row0), uniform(t.m), uniform(t.n0), uniform(t.k0), uniform(t.kb), uniform(t.type)};
}

// A producer warp's share of one tile: pieces p0 + (those of its parity below np) of its 32 rows.  `use` counts the group's operand
// slot uses.  meanwhile() is called once, when the first piece has been requested.
template <int T, class Meanwhile>
__device__ __forceinline__ bool ts_produce(const uint8_t* rows, uint32_t rb, int live, int p0, int np, int par, uint32_t raw, uint32_t tslot,
                                           uint32_t& use, uint64_t* wfull, uint64_t* wempty, const LaneLuts& L, saddr_t fac, int lane,
                                           volatile int* abort_flag, int* status, Meanwhile meanwhile) {
  constexpr int PK = TsPiece<T>::kK, PB = PK / kTsBK, W = TsPiece<T>::kWords;
  constexpr bool kTwo = 2 * 32 * 4 * W <= kTsRawWarp;     // (room for two of the larger pieces too changed nothing)
  static_assert(32 * 4 * W <= kTsRawWarp, "a piece of 32 rows fits");
  const int last = np & 1 ? np - 1 : np;                 // pieces [last, np): parity 0
  TsMul mul;
  ts_mul_init<T>(mul);
  const uintptr_t my_row = reinterpret_cast<uintptr_t>(rows) + (uintptr_t)min(lane, live - 1) * rb;
  if (par < np) ts_stage<T>(raw, rows, rb, live, (uint32_t)(p0 + par), lane);
  ts_cp_commit();
  meanwhile();
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
// a codebook among them), setup() copies its tables to `extra` after the dependency wait, tile(t) the t-th tile
// (called by whole warps; tile_of_thread by one thread), kSingle whether every type's pieces are one K block,
// kNextInSmem whether producers find their next tile while a piece is under way and keep it in shared memory,
// rows() a producer warp's 32 rows of row_size() bytes, a_map(i) the activation map with boxes of 16 << i rows x 64, epilogue() stores.
template <class Prob>
__device__ __forceinline__ void ts_gemm_body(Prob& pr, const Tables& tb) {
  if (!Prob::kLateTrigger) pdl_launch_dependents();
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
  if (Prob::kLateTrigger) pdl_launch_dependents();     // what is launched next may rely on everything before this launch
  pr.setup(raw + kTsRawBytes, tid);
  ts_fence_before();
  __syncthreads();
  ts_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, hd->tmem_base, 0);      // warp-uniform, and known to be
  volatile int* abort_flag = &hd->abort_flag;
  const int my_tiles = pr.ntiles > (int)blockIdx.x ? (pr.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  auto tile = [&](int i) { return pr.tile((int)blockIdx.x + i * (int)gridDim.x); };

  if (warp == kTsMmaWarp + 2) {
    // ------------------------------------------------------------------ activation loader (one thread; the others of its warp idle)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int i = 0; ok && i < my_tiles; i++) {
        const TsTile tl = pr.tile_of_thread((int)blockIdx.x + i * (int)gridDim.x);
        const int sh = ts_piece_shift(tl.type), couples = ts_couples(tl.kb, sh), steps = tl.kb - couples;
        const int box = tl.m <= 16 ? 0 : tl.m <= 32 ? 1 : tl.m <= 64 ? 2 : 3;
        const uint32_t bytes = (16u << box) * kTsBK * 2u;
        const CUtensorMap* map = pr.a_map(box);
        auto load = [&](int k) {
          const uint32_t s = it % kTsRing;
          ok = mbar_wait(&hd->empty[s], ((it / kTsRing) & 1u) ^ 1u, abort_flag, status, kDevWaitEmpty);
          if (!ok) return;
          mbar_arrive_expect_tx(&hd->full[s], bytes);
          ts_tma_2d(ring + s * kTsSlotBytes, map, (tl.k0 + k) * kTsBK, tl.row0, &hd->full[s]);
          it++;
        };
        for (int c = 0; ok && c < steps; c++) {
          const int k = c < couples ? ts_kblock(c, sh) : couples + c;
          load(k);
          if (ok && c < couples) load(k + (1 << sh));
        }
      }
    }
  } else if (warp >= kTsMmaWarp) {
    // ------------------------------------------------------------------ MMA issuers: one warp per half of the tile
    // A couple of K blocks at a time, its four barriers looked at by four lanes at once.  Everything between the operands' arrival and
    // the release of their slots is on the producers' way: with a K block at a time and one barrier after the other they waited a
    // third of the time for these warps, although the tensor core was idle.  Pieces of one K block (BF16, F16: kSingle) are hardly
    // decoded at all and these warps wait for data: there a K block at a time is sooner (us, couples / one at a time: BF16 4096 x 4096,
    // 17 tokens 12.01 / 11.60, 200 tokens 18.46 / 17.91; 5120 x 8192, 50 tokens 20.52 / 19.57; F16 19.46 / 18.64).
    const int half = warp - kTsMmaWarp;
    const bool leader = elect_one();
    const uint32_t role = (uint32_t)lane & 3u;           // 0, 1: the activations of the first, the second; 2, 3: their weights
    static_assert(kTsRing == 4, "phase of the ring");
    uint32_t my = role == 1 ? 1 : 0;                     // number of the next use of this lane's kind
    const uint64_t desc0 = ts_desc(smem_u32(ring));
    uint32_t it = 0, acc = 0, flip = 0, use[2] = {0, 0}; // flip: the parity that is first; uses of the slots of the first, the second
    bool ok = true;
    auto wait_acc = [&](uint32_t b) {
      return __all_sync(0xffffffffu, mbar_wait_sleep(&hd->accempty[b], ((acc >> 1) & 1u) ^ 1u, abort_flag, status, kDevWaitEmpty, 100)) != 0;
    };
    for (int i = 0; ok && i < my_tiles; i++) {
      const TsTile tl = uniform_tile(tile(i));
      const int sh = Prob::kSingle ? 0 : ts_piece_shift(tl.type);
      const int couples = Prob::kSingle ? 0 : ts_couples(tl.kb, sh), steps = Prob::kSingle ? 0 : tl.kb - couples;
      const uint32_t g0 = 2 * flip + half, g1 = 2 * (flip ^ 1u) + half;        // the groups that are first, second
      uint64_t* const my_bars = role < 2 ? hd->full : hd->wfull + 2 * (role == 2 ? g0 : g1);
      auto my_bar = [&]() { return my_bars + (my & (role < 2 ? kTsRing - 1 : 1)); };
      auto my_phase = [&]() { return (my >> (role < 2 ? 2 : 1)) & 1u; };
      auto wait_for = [&](uint32_t which) {              // 0: the first's barriers, 1: the second's
        return __all_sync(0xffffffffu, (role & 1u) != which || mbar_wait(my_bar(), my_phase(), abort_flag, status, kDevWaitFull)) != 0;
      };
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
      auto issue = [&](uint32_t g, uint32_t n, uint32_t s, uint32_t more) {      // slot n & 1 of group g, ring stage s
        const uint32_t a = tmem + kTsSlotCol + 32u * (2u * g + (n & 1u));
        const uint64_t b = desc0 + (uint64_t)(s * (kTsSlotBytes >> 4));
#pragma unroll
        for (int ks = 0; ks < kTsBK / 16; ks++) ts_mma_f16(d, a + 8u * ks, b + 2u * ks, idesc, ks > 0 ? 1u : more);
        ts_commit(&hd->wempty[2u * g + (n & 1u)]);
        ts_commit(&hd->empty[s]);
      };
      for (int st = 0; Prob::kSingle && st < tl.kb; st++, it++) {
        const bool second = st & 1;
        const uint32_t g = second ? g1 : g0, n = second ? use[1] : use[0], slot = 2u * g + (n & 1u);
        ok = __all_sync(0xffffffffu, mbar_wait(&hd->full[it & 3u], (it >> 2) & 1u, abort_flag, status, kDevWaitFull) &&
                                         mbar_wait(&hd->wfull[slot], (n >> 1) & 1u, abort_flag, status, kDevWaitFull));
        if (!ok) break;
        ts_fence_after();
        if (leader) issue(g, n, it & 3u, st > 0 ? 1u : 0u);
        __syncwarp();
        if (second) use[1]++; else use[0]++;
      }
      for (int c = 0; c < couples; c++) {
        bool mine;                                       // the first's barriers are waited for, the second's looked at
        if (role & 1u) mine = mbar_test_wait(my_bar(), my_phase());
        else mine = mbar_wait(my_bar(), my_phase(), abort_flag, status, kDevWaitFull);
        const unsigned there = __ballot_sync(0xffffffffu, mine);
        ok = (there & 5u) == 5u;
        if (!ok) break;
        __syncwarp();                                    // what the other lanes have seen is there for the issuing one
        ts_fence_after();
        if (leader) issue(g0, use[0], it & 3u, c > 0 ? 1u : 0u);
        __syncwarp();
        ok = (there & 10u) == 10u || wait_for(1);
        if (!ok) break;
        __syncwarp();
        ts_fence_after();
        if (leader) issue(g1, use[1], (it + 1) & 3u, 1u);
        __syncwarp();
        it += 2; use[0]++; use[1]++;
        my += role < 2 ? 2 : 1;
      }
      for (int c = couples; ok && c < steps; c++) {
        ok = wait_for(0);
        if (!ok) break;
        __syncwarp();
        ts_fence_after();
        if (leader) issue(g0, use[0], it & 3u, c > 0 ? 1u : 0u);
        __syncwarp();
        it++; use[0]++;
        my += role == 3 ? 0 : 1;
      }
      if (ts_odd(tl.kb, sh)) {                           // first and second change places
        flip ^= 1u;
        const uint32_t t = use[0];
        use[0] = use[1]; use[1] = t;
        const uint32_t other = __shfl_xor_sync(0xffffffffu, my, 1);
        if (role >= 2) my = other;
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
    const int pw = warp - kTsEpiWarps, group = pw >> 2, quarter = warp & 3, half = group & 1;
    int par = group >> 1;                                // first (0) or second in the tile
    LaneLuts L;
    L.iq1s = smem_u32(lut) + 8u * (lane % kIq1selCopies);
    L.iq2g = smem_u32(lut) + 4u * lane;
    L.iq2s = L.iq2g + (uint32_t)kIq2GridLutBytes;
    const saddr_t fac = smem_u32(hd->fac);
    bool ok = !(iq1 || iq2) || __all_sync(0xffffffffu, mbar_wait(&hd->lutbar, 0, abort_flag, status, kDevWaitFull));
    const uint32_t my_raw = smem_u32(raw) + (uint32_t)pw * kTsRawWarp;
    const uint32_t tslot = tmem + ((uint32_t)(32 * quarter) << 16) + kTsSlotCol + 64u * group;
    uint32_t use = 0;
    auto work = [&](int i) {
      const TsTile tl = tile(i);
      int live;
      const uint8_t* r = pr.rows(tl, half, quarter, live);
      return TsWork{r, live, tl.k0, tl.kb, tl.type};
    };
    auto put = [&](const TsWork& w) { if (lane == 0) hd->next[pw] = w; };
    if (Prob::kNextInSmem && my_tiles > 0) put(work(0));
    for (int i = 0; ok && i < my_tiles; i++) {
      TsWork tl;
      if constexpr (Prob::kNextInSmem) {
        __syncwarp();
        tl = hd->next[pw];
        __syncwarp();
      } else {
        tl = work(i);
      }
      const uint32_t rb = pr.row_size(tl.type);
      auto meanwhile = [&]() {
        if (Prob::kNextInSmem && i + 1 < my_tiles) put(work(i + 1));
      };
#define TS_PRODUCE(T)                                                                                                                     \
  case T:                                                                                                                                 \
    if constexpr (Prob::template kHas<T>)                                                                                                 \
      ok = ts_produce<T>(tl.rows, rb, tl.live, tl.k0 / (TsPiece<T>::kK / kTsBK), tl.kb / (TsPiece<T>::kK / kTsBK), par, my_raw, tslot,     \
                         use, &hd->wfull[2 * group], &hd->wempty[2 * group], L, fac, lane, abort_flag, status, meanwhile);                 \
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
      if (ts_odd(tl.kb, ts_piece_shift(tl.type))) par ^= 1;
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
