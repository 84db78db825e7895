// Two-SM variant of the persistent bf16 GEMM core: a cluster of two CTAs works on one 256 x 256 tile (or, see Config2Flat256, one of
// 128 rows) with
// tcgen05.mma.cta_group::2. Each CTA stages its own 128 rows of A and 128 of the tile's 256 B rows (so a k-block
// costs 32 KB of shared-memory fill per SM instead of 48 KB, and each MMA reads half of B from the peer SM), holds
// the accumulator rows of its A half in its own TMEM and runs its own epilogue. The leader CTA (cluster rank 0)
// issues every MMA; completion is signalled to both CTAs with tcgen05.commit ... multicast::cluster.
//
//   D[M,N] = A[M,K] * B[N,K]^T        A, B bf16 K-major; fp32 accumulate; N % 256 == 0; K % 64 == 0
//
// Loads never use cluster multicast: both CTAs fetch their halves with plain tiled TMA loads whose byte counts
// land on the leader's mbarrier. Same hooks as the one-SM core (AGate, Epilogue); row blocks handed to them are
// 128-row blocks (block = 2 * pairRowBlock + cluster rank). Every wait is bounded.
#pragma once

#include "gemm_sm100.cuh"

namespace mscclpp {
namespace gemm {

template <int kStages_, int kStagingBytes_, int kBarrierBytes_, int kPairM_ = 2 * kBlockM, int kBlockN_ = 256>
struct Config2Of {
  static constexpr int kBlockN = kBlockN_;
  static constexpr int kPairM = kPairM_;                           // rows per tile
  static_assert((kPairM == 256 && kBlockN == 256) || (kPairM == 128 && (kBlockN == 128 || kBlockN == 256)), "unsupported tile");
  static constexpr int kRows = kPairM / 2;                         // of this CTA's A half
  static constexpr int kStageABytes = kRows * kBlockK * 2;         // 256 rows: 16 KB
  static constexpr int kStageBBytes = (kBlockN / 2) * kBlockK * 2;  // this CTA's B half, 256 columns: 16 KB
  // k blocks per stage (see Config::kKb in gemm_sm100.cuh; 128 x 4096 in tiles of 128 x 128 160 -> 93 ns per k block, with four of them per stage 95)
  static constexpr int kKb = kPairM == 128 && kBlockN == 128 ? 2 : 1;
  static constexpr int kStageBytes = kKb * (kStageABytes + kStageBBytes);  // A blocks, then B blocks
  static constexpr int kStages = kStages_ / kKb;
  // An accumulator with 256 rows per tile: lane = row of this CTA's half, column = column of the tile. With 128 rows: lanes 0 to 63
  // are the 64 rows and the columns the first half of the tile's, lanes 64 to 127 the same rows and the second half.
  static constexpr bool kFolded = kPairM == 128;
  static constexpr int kAccCols = kFolded ? kBlockN / 2 : kBlockN;
  static constexpr int kTmemCols = 2 * kAccCols;  // two accumulator buffers
  static constexpr int kBarrierBytes = kBarrierBytes_;
  static constexpr int kStagingBytes = kStagingBytes_;  // of the epilogue
  static constexpr int kEpiWarps = kAccCols >= 128 ? kNumEpilogueWarps : 4;
  static constexpr int kColsPerWarp = kAccCols / (kEpiWarps / 4);
  static constexpr int kCoreBars = 2 * kStages + 6 > 20 ? 2 * kStages + 6 : 20;  // words; barriers of a row epilogue follow
  static constexpr int kSmemBytes = kStages * kStageBytes + kStagingBytes + kBarrierBytes + 1024;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");
};
using Config2 = Config2Of<6, kEpilogueStagingBytes, 256>;
using Config2Rows = Config2Of<5, 2 * kEpilogueStagingBytes, 512>;  // row epilogues: every block of a warp's tile is staged
// Tiles of 128 rows, for problems of too few rows or tiles for the above: 64 rows of A and half of B per CTA and k block, 24 KB for 128 x
// 256 and 16 KB for 128 x 128, where one SM takes 32 KB for half of the former and 24 KB for half of the latter. (A warp stages one
// block, row epilogue or not.)
using Config2Flat256 = Config2Of<8, kEpilogueStagingBytes, 512, 128, 256>;
using Config2Flat128 = Config2Of<12, kEpilogueStagingBytes / 2, 512, 128, 128>;

template <typename Cfg>
MSCCLPP_HOST_DEVICE_INLINE constexpr uint32_t makeInstrDescPair() {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(Cfg::kBlockN >> 3) << 17) |
         (static_cast<uint32_t>(Cfg::kPairM >> 4) << 24);
}

// Body of one CTA of a pair. All threads call it; `pairIdx` / `numPairs` index the persistent tile loop.
// shape.mOrder / mOrderParam apply to 256-row blocks here.
template <typename Cfg = Config2, typename AGate, typename Epilogue>
MSCCLPP_DEVICE_INLINE void gemmCtaPair(const CUtensorMap* tmapA, const CUtensorMap* tmapB, Shape shape, int pairIdx, int numPairs,
                                       AGate& gate, Epilogue& epi, DeviceStatus* status, uint64_t budgetNs, uint8_t* smemRaw) {
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t ctaRank = ptx::cluster_ctarank();
  const bool leader = ctaRank == 0;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
  uint8_t* tiles = smem;
  uint8_t* staging = smem + Cfg::kStages * Cfg::kStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + Cfg::kStagingBytes);
  SharedState st;
  st.full = bars;
  st.empty = bars + Cfg::kStages;
  st.tmemFull = bars + 2 * Cfg::kStages;
  st.tmemEmpty = bars + 2 * Cfg::kStages + 2;
  st.tmemBase = reinterpret_cast<uint32_t*>(bars + 2 * Cfg::kStages + 4);
  st.abortFlag = reinterpret_cast<volatile uint32_t*>(st.tmemBase + 1);
  st.epiArrivals = reinterpret_cast<volatile uint32_t*>(st.tmemBase + 2);

  const int numMBlk2 = (shape.M + Cfg::kPairM - 1) / Cfg::kPairM;
  const int numNBlk = (shape.N + Cfg::kBlockN - 1) / Cfg::kBlockN;
  const int numTiles = numMBlk2 * numNBlk;
  const int numKBlk = shape.K / kBlockK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; s++) {
      ptx::mbar_init(&st.full[s], 1);   // the leader's producer arrives once and announces both CTAs' bytes
      ptx::mbar_init(&st.empty[s], 1);  // one multicast commit per use
    }
    for (int s = 0; s < 2; s++) {
      ptx::mbar_init(&st.tmemFull[s], 1);
      ptx::mbar_init(&st.tmemEmpty[s], 2 * Cfg::kEpiWarps);  // the epilogue warps of both CTAs arrive at the leader's
    }
    *st.abortFlag = 0;
    *st.epiArrivals = 0;
    ptx::fence_mbar_init();
    ptx::tma_prefetch_desc(tmapA);
    ptx::tma_prefetch_desc(tmapB);
  }
  if constexpr (IsRowEpilogue<Epilogue>::value) {
    if (warp >= 2) epi.setup(staging + (warp - 2) * Epilogue::kBlocks * kStagingBytesPerWarp, bars + Cfg::kCoreBars + (warp - 2) * Epilogue::kBlocks, lane);
  }
  __syncthreads();
  // the peer's barriers must exist before anything of mine can signal them
  ptx::cluster_sync_all();
  if (warp == 1) {
    ptx::tmem_alloc_pair(st.tmemBase, Cfg::kTmemCols);
    ptx::tmem_relinquish_pair();
  }
  ptx::tcgen05_fence_before_sync();
  __syncthreads();
  ptx::tcgen05_fence_after_sync();
  const uint32_t tmemBase = *st.tmemBase;
  // everything up to here is this pair's own: with a programmatic dependent launch it ran under the kernel before
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  if (warp == 0) {
    // ===================================================== TMA producer (one thread per CTA)
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int issuedUses = 0;
      for (int tile = pairIdx; tile < numTiles && ok; tile += numPairs) {
        int mBlk2, nBlk;
        tileCoord(shape, tile, numMBlk2, numNBlk, mBlk2, nBlk);
        const int mBlk = 2 * mBlk2 + static_cast<int>(ctaRank);
        ok = gate.waitRowBlock(mBlk);
        int aRow;
        const CUtensorMap* tmapARows = gate.tmapA(mBlk, tmapA, aRow);
        if constexpr (Cfg::kFolded) aRow = mBlk * Cfg::kRows;  // (no gate)
        for (int kb = 0; kb < numKBlk && ok; kb += Cfg::kKb) {
          ok = mbarWaitFast(&st.empty[stage], phase ^ 1u, status, budgetNs, 100 + stage, st.abortFlag);
          if (!ok) break;
          uint8_t* sa = tiles + stage * Cfg::kStageBytes;
          uint8_t* sb = sa + Cfg::kKb * Cfg::kStageABytes;
          const uint32_t leaderFull = ptx::mapa_shared(ptx::smem_u32(&st.full[stage]), 0);
          if (shape.probe & 1) {
            if (leader) ptx::mbar_arrive(&st.full[stage]);
          } else {
            const int blocks = Cfg::kKb == 1 || numKBlk - kb > Cfg::kKb ? Cfg::kKb : numKBlk - kb;  // (the last stage may not be full)
            if (leader) ptx::mbar_expect_tx(&st.full[stage], 2 * blocks * (Cfg::kStageABytes + Cfg::kStageBBytes));
#pragma unroll
            for (int j = 0; j < Cfg::kKb; j++) {
              if (j >= blocks) break;
              ptx::tma_load_2d_pair(sa + j * Cfg::kStageABytes, tmapARows, (kb + j) * kBlockK, aRow, leaderFull);
              ptx::tma_load_2d_pair(sb + j * Cfg::kStageBBytes, tmapB, (kb + j) * kBlockK,
                                    nBlk * Cfg::kBlockN + static_cast<int>(ctaRank) * (Cfg::kBlockN / 2), leaderFull);
            }
          }
          issuedUses++;
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok) *st.abortFlag = 1;
      // Loads in flight land in this CTA's shared memory: the CTA stays resident until the cluster barrier at the
      // end, which every thread of both CTAs reaches, and the leader's consumer either uses them or has given up.
      (void)issuedUses;
    }
  } else if (warp == 1) {
    // ===================================================== MMA issuer (one thread of the leader CTA)
    if (leader && ptx::elect_one()) {
      constexpr uint32_t idesc = makeInstrDescPair<Cfg>();
      // one thread feeds the tensor cores of both SMs: descriptors are stepped by adds, waits cost one instruction when
      // the data is already there
      const uint64_t descA0 = makeSmemDesc(ptx::smem_u32(tiles));
      const uint64_t descB0 = makeSmemDesc(ptx::smem_u32(tiles) + Cfg::kKb * Cfg::kStageABytes);
      constexpr uint64_t kStageStep = Cfg::kStageBytes >> 4;
      const bool issue = (shape.probe & 2) == 0;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int it = 0;
      for (int tile = pairIdx; tile < numTiles && ok; tile += numPairs, it++) {
        const int acc = it & 1;
        const uint32_t accPhase = (it >> 1) & 1;
        ok = mbarWaitFast<true>(&st.tmemEmpty[acc], accPhase ^ 1u, status, budgetNs, 200 + acc, st.abortFlag);
        if (!ok) break;
        ptx::tcgen05_fence_after_sync();
        const uint32_t tmemD = tmemBase + acc * Cfg::kAccCols;
        for (int kb = 0; kb < numKBlk; kb += Cfg::kKb) {
          ok = mbarWaitFast(&st.full[stage], phase, status, budgetNs, 300 + stage, st.abortFlag);
          if (!ok) break;
          ptx::tcgen05_fence_after_sync();
          const uint64_t descA = descA0 + stage * kStageStep;
          const uint64_t descB = descB0 + stage * kStageStep;
          if (issue) {
            ptx::tcgen05_mma_f16_pair(tmemD, descA, descB, idesc, kb != 0 ? 1u : 0u);
#pragma unroll
            for (int k = 1; k < kBlockK / kUmmaK; k++) ptx::tcgen05_mma_f16_pair_acc(tmemD, descA + 2 * k, descB + 2 * k, idesc);
#pragma unroll
            for (int j = 1; j < Cfg::kKb; j++) {
              if (kb + j >= numKBlk) break;
#pragma unroll
              for (int k = 0; k < kBlockK / kUmmaK; k++)
                ptx::tcgen05_mma_f16_pair_acc(tmemD, descA + j * (Cfg::kStageABytes >> 4) + 2 * k, descB + j * (Cfg::kStageBBytes >> 4) + 2 * k, idesc);
            }
          }
          ptx::tcgen05_commit_pair(&st.empty[stage], 3);  // both CTAs may refill this stage once the MMAs retire
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) ptx::tcgen05_commit_pair(&st.tmemFull[acc], 3);
      }
      if (!ok) *st.abortFlag = 1;
    }
  } else if (warp < 2 + Cfg::kEpiWarps) {
    // ===================================================== epilogue (8 warps per CTA, or 4, on this CTA's accumulator rows)
    const int quarter = warp & 3;
    const int part = (warp - 2) >> 2;
    // this warp's corner of the CTA's part of a tile
    const int rowOfWarp = Cfg::kFolded ? (quarter & 1) * 32 : quarter * 32;
    const int colOfWarp = part * Cfg::kColsPerWarp + (Cfg::kFolded ? (quarter >> 1) * Cfg::kAccCols : 0);
    uint8_t* stage = staging + (warp - 2) * kStagingBytesPerWarp;
    bool ok = true;
    int it = 0;
    for (int tile = pairIdx; tile < numTiles && ok; tile += numPairs, it++) {
      int mBlk2, nBlk;
      tileCoord(shape, tile, numMBlk2, numNBlk, mBlk2, nBlk);
      const int mBlk = 2 * mBlk2 + static_cast<int>(ctaRank);
      const int acc = it & 1;
      const uint32_t accPhase = (it >> 1) & 1;
      const int row0 = mBlk * Cfg::kRows + rowOfWarp;
      const int col0 = nBlk * Cfg::kBlockN + colOfWarp;
      // lets the epilogue put loads it will need (a residual, a bias) in flight while the MMAs of this tile still run
      if constexpr (IsRowEpilogue<Epilogue>::value) {
        if (it == 0) epi.request(row0, col0, lane);
      } else {
        epi.tileBegin(row0, col0, lane);
      }
      ok = mbarWait(&st.tmemFull[acc], accPhase, status, budgetNs, 400 + acc);
      ok = __all_sync(0xffffffffu, ok) && (*st.abortFlag == 0);
      if (!ok) break;
      ptx::tcgen05_fence_after_sync();
      const uint32_t taddr = tmemBase + (static_cast<uint32_t>(quarter * 32) << 16) + acc * Cfg::kAccCols + part * Cfg::kColsPerWarp;
      // The accumulator goes back by a relaxed arrive between fences of tensor memory. A release at cluster scope instead, one B200:
      // 2305 x 8192 x 128 layer 43.1 us (now 37.5), 8192 x 8192 x 1024 layer 166.4 (162.9), GEMM of 4096 x 8192 x 256 26.0 (22.6),
      // GEMM of 8192 x 8192 x 1024 111.5 (111.4): what it costs is paid per tile, behind the stores of the tile before.
      const uint32_t leaderEmpty = ptx::mapa_shared(ptx::smem_u32(&st.tmemEmpty[acc]), 0);
      if constexpr (IsRowEpilogue<Epilogue>::value) {
        ok = epi.tile(taddr, row0, col0, it, lane, [&] { ptx::mbar_arrive_tmem_read(leaderEmpty); });
        if (!ok) break;
        if (tile + numPairs < numTiles) {  // the next tile's residual, under its MMAs
          int m, n;
          tileCoord(shape, tile + numPairs, numMBlk2, numNBlk, m, n);
          epi.request((2 * m + static_cast<int>(ctaRank)) * Cfg::kRows + rowOfWarp, n * Cfg::kBlockN + colOfWarp, lane);
        }
      } else {
        stagedEpilogueTile<Cfg::kColsPerWarp>(epi, taddr, stage, row0, col0, lane, [&] { ptx::mbar_arrive_tmem_read(leaderEmpty); }, shape.probe);
      }
      if constexpr (Epilogue::kNeedsTileBarrier) {
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          atomicAdd(const_cast<uint32_t*>(st.epiArrivals), 1u);
          const uint32_t target = static_cast<uint32_t>(it + 1) * Cfg::kEpiWarps;
          SpinGuard g(status, budgetNs);
          while (static_cast<int32_t>(*st.epiArrivals - target) < 0) {
            if (*st.abortFlag || !g.keepSpinning()) {
              *st.abortFlag = 1;
              break;
            }
          }
          __threadfence_block();
        }
        __syncwarp();
        if (*st.abortFlag) {
          ok = false;
          break;
        }
        if (warp == 2) epi.tileDone(mBlk, nBlk, lane);
      }
      // per-warp hook: this warp's part of the tile is stored (fused epilogues count it and may take on follow-up work)
      epi.warpTileDone(mBlk, lane);
    }
    if (ok) epi.warpDrain(lane);  // follow-up work that is left once the warp has no tile of its own any more
    if (!ok && lane == 0) *st.abortFlag = 1;
    if constexpr (IsRowEpilogue<Epilogue>::value) {
      if (!ok) epi.drain(it);
    }
    if constexpr (Epilogue::kBulkStore) {
      if (lane == 0) ptx::bulk_wait<0>();
    }
  } else if (warp >= 2 + kNumEpilogueWarps) {
    // warps beyond the ten of the GEMM roles (a kernel may launch more threads): follow-up work of a fused epilogue that
    // must stay off the epilogue warps' critical path
    epi.auxWarp(warp - (2 + kNumEpilogueWarps), lane);
  }

  // ---- teardown: both CTAs meet (the peer may still read my shared memory or signal my barriers until then)
  ptx::tcgen05_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync_all();
  ptx::tcgen05_fence_after_sync();
  if (warp == 1) ptx::tmem_dealloc_pair(tmemBase, Cfg::kTmemCols);
}

}  // namespace gemm
}  // namespace mscclpp
