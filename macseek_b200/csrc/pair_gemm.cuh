// Persistent tcgen05 GEMM of half operands in global memory, fp32 accumulation: a tile is (128 tokens per block) x bn weight rows, shared
// by a cluster of G = 2 blocks (cta_group::2: each fetches its 128 tokens and half of the weight rows) or worked on by one block.
// Operands by TMA (128-byte swizzle); two accumulator sets in TMEM, so the epilogue of one tile overlaps the main loop of the next.
// Warp roles: 0..3 epilogue, 4 MMA issue (first block of a pair), 5 TMA.  Fetching the operands from L2 bounds it, hence the pairs: 32
// KB per block and 128 x 256 x 64 products instead of 48.  Every mbarrier wait is bounded.
#pragma once
#include <cooperative_groups.h>
#include "ts_gemm.cuh"

namespace msb {

constexpr int kGmBM = 128, kGmBN = 256, kGmBK = 64;          // a block's tokens, a tile's largest number of weight rows, contraction (halfs)
constexpr int kGmShareA = kGmBM * kGmBK * 2;                 // a block's share of a stage: its tokens ...
__host__ __device__ constexpr int gm_share_b(int G) { return kGmBN / G * kGmBK * 2; }      // ... and its share of the weight rows
__host__ __device__ constexpr int gm_stages(int G) { return G == 2 ? 6 : 4; }              // 192 KB either way
constexpr int kGmThreads = 6 * 32;

#ifdef __CUDACC__
struct GemmHead {
  uint64_t full[gm_stages(2)], empty[gm_stages(2)], accfull[2], accempty[2];
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t gm_leader(const void* p) {     // the address of the pair's first block for the same variable
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
  return r;
}
// to this block's shared memory; the bytes are counted on a barrier of the pair's first block
__device__ __forceinline__ void gm_tma_2d(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
template <int G>
__device__ __forceinline__ void gm_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  if constexpr (G == 2)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void gm_commit(uint64_t* bar) {          // arrives on the barrier of both blocks
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void gm_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void gm_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// Prob: ntiles, bn, kb (K blocks of 64), status, a_map (boxes of 128 rows), b_map (boxes of bn / G rows); tile(t, rank), called by
// whole warps, and tile_of_thread() name the block's first token row (a_row) and first weight row (b_row) of tile t; epilogue(tile, taddr,
// warp, lane): lane = token row 32 warp + lane of the block, column = weight row of the tile; wait_before() and wait_after() surround the
// work, one of them waits for the launch before.
template <int G, class Prob>      // G: blocks that share a tile, 2 or 1
__device__ __forceinline__ void gemm_body(const Prob& p) {
  namespace cg = cooperative_groups;
  constexpr int kStages = gm_stages(G), kShareB = gm_share_b(G);
  pdl_launch_dependents();
  uint8_t* smem = ts_smem_raw + ((1024u - (smem_u32(ts_smem_raw) & 1023u)) & 1023u);   // swizzled tiles: 1024-byte aligned
  GemmHead* hd = reinterpret_cast<GemmHead*>(smem);
  uint8_t* stage0 = smem + 1024;                                   // per stage: this block's share of A, then of B
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)blockIdx.x % G, pair = (int)blockIdx.x / G, npairs = (int)gridDim.x / G;
  constexpr uint32_t kCols = 2 * kGmBN;
  cg::cluster_group cl = cg::this_cluster();

  if (tid == 0) {
    for (int s = 0; s < kStages; s++) { mbar_init(&hd->full[s], 1); mbar_init(&hd->empty[s], 1); }
    for (int b = 0; b < 2; b++) { mbar_init(&hd->accfull[b], 1); mbar_init(&hd->accempty[b], 4 * G); }
    hd->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4) {
    if constexpr (G == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&hd->tmem_base)), "r"(kCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&hd->tmem_base)), "r"(kCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  ts_fence_before();
  cl.sync();                                                       // every block's barriers exist
  ts_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, hd->tmem_base, 0);      // warp-uniform, and known to be
  volatile int* abort_flag = &hd->abort_flag;
  const int bn = p.bn, kb = p.kb, ntiles = p.ntiles;
  const int my_tiles = ntiles > pair ? (ntiles - 1 - pair) / npairs + 1 : 0;
  p.wait_before();       // for the operands

  if (warp == 5) {
    // ------------------------------------------------------------------ TMA producer: one thread per block, the others of its warp have
    // nothing to do until the end (a warp that polls, or that waits for this thread after every tile, costs a product of 16 us 2)
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)(G * kGmShareA + bn * kGmBK * 2);           // of the tile's blocks
      uint32_t it = 0;
      for (int i = 0; i < my_tiles; i++) {
        const auto tl = p.tile_of_thread(pair + i * npairs, rank);
        bool ok = true;
        for (int k = 0; k < kb; k++, it++) {
          const int s = it % kStages;
          if (!mbar_wait(&hd->empty[s], ((it / kStages) & 1u) ^ 1u, abort_flag, p.status(), kDevWaitEmpty)) { ok = false; break; }
          uint8_t* slot = stage0 + (size_t)s * (kGmShareA + kShareB);
          if (rank == 0) mbar_arrive_expect_tx(&hd->full[s], bytes);
          if constexpr (G == 2) {
            const uint32_t bar = gm_leader(&hd->full[s]);
            gm_tma_2d(slot, p.a_map(), k * kGmBK, tl.a_row, bar);
            gm_tma_2d(slot + kGmShareA, p.b_map(), k * kGmBK, tl.b_row, bar);
          } else {
            ts_tma_2d(slot, p.a_map(), k * kGmBK, tl.a_row, &hd->full[s]);
            ts_tma_2d(slot + kGmShareA, p.b_map(), k * kGmBK, tl.b_row, &hd->full[s]);
          }
        }
        if (!ok) break;
      }
    }
  } else if (warp == 4) {
    // ------------------------------------------------------------------ MMA issuer (one elected lane of the first block)
    if (rank == 0) {
      // instruction descriptor: D fp32, A and B f16, both K-major, N = bn, M = 128 per block
      const uint32_t idesc = (1u << 4) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(G * kGmBM >> 4) << 24);
      const bool leader = elect_one();
      uint32_t it = 0;
      bool ok = true;
      for (int i = 0; ok && i < my_tiles; i++) {
        const int buf = i & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(&hd->accempty[buf], ((i >> 1) & 1u) ^ 1u, abort_flag, p.status(), kDevWaitEmpty))) break;
        ts_fence_after();
        for (int k = 0; k < kb; k++, it++) {
          const int s = it % kStages;
          ok = __all_sync(0xffffffffu, mbar_wait(&hd->full[s], (it / kStages) & 1u, abort_flag, p.status(), kDevWaitFull));
          if (!ok) break;
          ts_fence_after();
          const uint32_t a_s = smem_u32(stage0) + (uint32_t)s * (uint32_t)(kGmShareA + kShareB), b_s = a_s + kGmShareA;
          if (leader) {
#pragma unroll
            for (int ks = 0; ks < kGmBK / 16; ks++)     // K = 16 halfs = 32 bytes per instruction
              gm_mma_f16<G>(tmem + (uint32_t)(buf * kGmBN), ts_desc(a_s + ks * 32), ts_desc(b_s + ks * 32), idesc, (k > 0 || ks > 0) ? 1u : 0u);
            if constexpr (G == 2) {
              gm_commit(&hd->empty[s]);
              if (k == kb - 1) gm_commit(&hd->accfull[buf]);
            } else {
              ts_commit(&hd->empty[s]);
              if (k == kb - 1) ts_commit(&hd->accfull[buf]);
            }
          }
          __syncwarp();
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: TMEM lane = token of this block
    for (int i = 0; i < my_tiles; i++) {
      const int buf = i & 1;
      const auto tl = p.tile(pair + i * npairs, rank);
      if (!__all_sync(0xffffffffu, mbar_wait(&hd->accfull[buf], (i >> 1) & 1u, abort_flag, p.status(), kDevWaitFull))) break;
      ts_fence_after();
      p.epilogue(tl, tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(buf * kGmBN), warp, lane);
      ts_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (G == 2) gm_arrive(gm_leader(&hd->accempty[buf]));
        else mbar_arrive(&hd->accempty[buf]);
      }
    }
  }
  // ------------------------------------------------------------------ teardown (every thread of the tile's blocks arrives here)
  p.wait_after();
  ts_fence_before();
  cl.sync();
  if (warp == 4) {
    ts_fence_after();
    if constexpr (G == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
  }
}
#endif  // __CUDACC__

}  // namespace msb
