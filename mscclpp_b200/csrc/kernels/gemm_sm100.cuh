// Warp-specialised persistent bf16 GEMM core for sm_100a: TMA (cp.async.bulk.tensor, no cluster
// multicast) stages 128B-swizzled A/B tiles in shared memory, ONE thread issues tcgen05.mma with
// the fp32 accumulator in tensor memory (TMEM), and four epilogue warps read the accumulator back
// with tcgen05.ld while the next tile's MMAs already run on the second TMEM buffer.
//
//   D[M,N] = A[M,K] * B[N,K]^T        A, B bf16 K-major (row-major [rows, K]); fp32 accumulate
//
// The reference library has no GEMM (it is a pure communication library); this core exists so that
// the tensor-parallel collectives can be fused with the matmul that produces or consumes them.
// Hooks for that fusion:
//   * AGate     - called by the TMA producer before it loads the A tiles of a row block, so an
//                 all-gather that is still in flight can be waited for block by block;
//   * Epilogue  - each epilogue warp converts a 32-row x 64-column block of the accumulator to bf16 and
//                 writes it into its own 4 KB of shared memory in the 128-byte-swizzled layout of a TMA
//                 box; Epilogue::block() then moves it out with ONE cp.async.bulk.tensor store, or re-reads
//                 it with a row-contiguous lane mapping (stagedRead) so that every global load and store
//                 of a fused epilogue (residual add, partial products for a collective) covers whole
//                 128-byte lines. tileDone() follows once all epilogue warps have stored their part; there
//                 a fused kernel signals consumers (reduce-scatter / allreduce owners);
//   * aux CTAs  - blocks with blockIdx.x >= number of GEMM CTAs run a caller-supplied role
//                 (reducer, copier) inside the same launch.
// Every wait is bounded; on expiry the kernel records a DeviceStatus, drains its own TMA copies,
// frees its TMEM and returns.
#pragma once

#include <type_traits>
#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <mscclpp/device/ptx.cuh>
#include <mscclpp/poll_device.hpp>

#include "gemm.cuh"

namespace mscclpp {
namespace gemm {

constexpr int kBlockM = 128;
constexpr int kBlockK = 64;          // 64 bf16 = 128 bytes = one swizzle row
constexpr int kUmmaK = 16;           // K of one tcgen05.mma for 16-bit inputs
constexpr int kNumEpilogueWarps = 8;  // two warps per TMEM lane quarter, each takes half of the tile's columns
constexpr int kNumEpilogueThreads = kNumEpilogueWarps * 32;
constexpr int kNumThreads = 64 + kNumEpilogueThreads;  // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2-9: epilogue
constexpr int kStagingBytesPerWarp = 32 * 128;  // 32 rows x 64 bf16 columns
constexpr int kEpilogueStagingBytes = kNumEpilogueWarps * kStagingBytesPerWarp;
constexpr int kPartBytes = 32 * 64 * 4;  // a 32-row x 64-column block of the accumulator on its way to the CTA that finishes it

// kSplit > 1: a cluster of kSplit CTAs shares one tile, each with its part of the reduction (see splitEpilogueTile).
template <int kBlockN, int kSplit = 1>
struct Config {
  // k blocks per stage. The two threads that feed the tensor core spend 135 ns on a stage even without its loads and products, however many
  // stages there are. Two k blocks instead of one: 128 x 4096 in tiles of 64 columns 186 -> 146 ns per k block. Wider tiles are left
  // with too few stages: 128 columns 184 -> 173 ns with few SMs busy, but 266 -> 281 with all of them.
  static constexpr int kKb = kBlockN == 64 ? 2 : 1;
  static_assert(kBlockN == 64 || kBlockN == 128 || kBlockN == 256, "unsupported N tile");
  static constexpr int kStageABytes = kBlockM * kBlockK * 2;
  static constexpr int kStageBBytes = kBlockN * kBlockK * 2;
  static constexpr int kStageBytes = kKb * (kStageABytes + kStageBBytes);  // A blocks, then B blocks
  // 32-row x 64-column blocks of the tile, how many of them a CTA of the cluster finishes, and what its peers send it for them
  static constexpr int kBlocks = 4 * kBlockN / 64;
  static_assert(kBlocks % kSplit == 0 && (kSplit == 1 || kBlockN == 64), "a CTA finishes whole blocks, a warp sends or finishes one");
  static constexpr int kOwnBlocks = kBlocks / kSplit;
  static constexpr int kRecvBytes = (kSplit - 1) * kOwnBlocks * kPartBytes;
  static constexpr int kStages = (kBlockN == 256 ? 4 : (kBlockN == 128 ? 6 : 8)) / kKb;
  static constexpr int kTmemCols = (kSplit > 1 ? 1 : 2) * kBlockN;  // two accumulator buffers (power of two >= 32); one tile needs one
  static constexpr int kBarrierBytes = 256;
  // epilogue warps that take part: every warp owns 32 rows (its TMEM lane quarter) x a multiple of 64 columns
  static constexpr int kEpiWarps = kBlockN >= 128 ? kNumEpilogueWarps : 4;
  static constexpr int kColsPerWarp = kBlockN / (kEpiWarps / 4);
  // (where the reduction is split, a CTA has one tile: its blocks are staged in the operand stages, which are done with by then)
  static constexpr int kStagingBytes = kSplit > 1 ? 0 : kEpilogueStagingBytes;
  static constexpr int kSmemBytes = kStages * kStageBytes + kRecvBytes + kStagingBytes + kBarrierBytes + 1024;  // +1024: manual alignment
  static_assert(kSmemBytes <= 227 * 1024 && kEpilogueStagingBytes + kNumEpilogueWarps * kPartBytes <= kStages * kStageBytes, "shared memory of one CTA");
};

MSCCLPP_DEVICE_INLINE void tileCoord(const Shape& s, int tile, int numMBlk, int numNBlk, int& mBlk, int& nBlk) {
  if (s.rowMajorTiles) {
    mBlk = tile / numNBlk;
    nBlk = tile % numNBlk;
  } else {
    mBlk = tile % numMBlk;
    nBlk = tile / numMBlk;
  }
  if (s.mOrder == 1) {
    const int per = numMBlk / s.mOrderParam;
    mBlk = (mBlk % s.mOrderParam) * per + mBlk / s.mOrderParam;
  } else if (s.mOrder == 2) {
    mBlk += s.mOrderParam;
    if (mBlk >= numMBlk) mBlk -= numMBlk;
  } else if (s.mOrder == 3) {
    // bands of mOrderParam row blocks, walked row-block-first inside a band: the tiles that run at the same time cover
    // a near-square region, so each wave re-reads a band of A and a few column panels of B from L2 instead of all of A
    const int g = s.mOrderParam;
    const int perBand = g * numNBlk;
    const int band = tile / perBand;
    const int first = band * g;
    const int rows = numMBlk - first < g ? numMBlk - first : g;  // the last band may be shorter
    const int t = tile - band * perBand;
    mBlk = first + t % rows;
    nBlk = t / rows;
  }
}

// 64-bit shared-memory matrix descriptor: K-major operand, 128-byte swizzle, tile base 1024B-aligned.
// bits [0,14) start address >> 4; [16,30) leading byte offset >> 4 (unused for swizzled K-major, 1);
// [32,46) stride byte offset >> 4 (8 rows x 128 B = 1024 B between 8-row groups); [46,48) version = 1
// on sm_100; [61,64) layout = 2 (SWIZZLE_128B).
MSCCLPP_DEVICE_INLINE uint64_t makeSmemDesc(uint32_t smemAddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smemAddr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// 32-bit instruction descriptor for kind::f16: bf16 x bf16 -> fp32, both operands K-major.
// [4,6) D format (1 = f32); [7,10) A format (1 = bf16); [10,13) B format (1 = bf16);
// bit 15 / 16 A / B major (0 = K); [17,23) N >> 3; [24,29) M >> 4.
template <int kBlockN>
MSCCLPP_HOST_DEVICE_INLINE constexpr uint32_t makeInstrDesc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kBlockN >> 3) << 17) |
         (static_cast<uint32_t>(kBlockM >> 4) << 24);
}

struct NoGate {
  MSCCLPP_DEVICE_INLINE bool waitRowBlock(int /*mBlk*/) const { return true; }
  // Tensor map and first row (in that map) of row block mBlk's A tiles.
  MSCCLPP_DEVICE_INLINE const CUtensorMap* tmapA(int mBlk, const CUtensorMap* dflt, int& row) const {
    row = mBlk * kBlockM;
    return dflt;
  }
};

// ---- epilogue staging: a warp's 32 x 64 bf16 block in shared memory, laid out like a SWIZZLE_128B TMA box
// (row r at byte r * 128, its 16-byte chunk c at position c ^ (r & 7)); the buffer is 1024-byte aligned.
MSCCLPP_DEVICE_INLINE uint32_t stagedOffset(int r, int c) { return static_cast<uint32_t>(r * 128 + ((c ^ (r & 7)) << 4)); }
// Row-contiguous view for fused epilogues: in step i (0..7) lane l holds chunk (l & 7) of row 4 * i + (l >> 3), so a
// warp-wide global access built on it touches four complete 128-byte lines.
MSCCLPP_DEVICE_INLINE int stagedRow(int i, int lane) { return 4 * i + (lane >> 3); }
MSCCLPP_DEVICE_INLINE int stagedCol(int lane) { return (lane & 7) * 8; }
MSCCLPP_DEVICE_INLINE uint4 stagedRead(const uint8_t* stage, int i, int lane) {
  return *reinterpret_cast<const uint4*>(stage + stagedOffset(stagedRow(i, lane), lane & 7));
}

struct SharedState {
  uint64_t* full;       // [stages] TMA -> MMA
  uint64_t* empty;      // [stages] MMA -> TMA
  uint64_t* tmemFull;   // [2] MMA -> epilogue
  uint64_t* tmemEmpty;  // [2] epilogue -> MMA
  uint32_t* tmemBase;
  volatile uint32_t* abortFlag;
  volatile uint32_t* epiArrivals;  // epilogue warps that finished storing, summed over the tiles so far
};

// Columns [8k, 8k+8) of a thread's 32 accumulator values as packed bf16.
template <typename Epilogue>
MSCCLPP_DEVICE_INLINE uint4 packChunk(const uint32_t (&v)[32], int k) {
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    __nv_bfloat162 h = __floats2bfloat162_rn(Epilogue::convert(__uint_as_float(v[8 * k + 2 * j])),
                                             Epilogue::convert(__uint_as_float(v[8 * k + 2 * j + 1])));
    w[j] = *reinterpret_cast<uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Epilogues that combine the two 32-column halves of every 64-column block into 32 output columns (gated activations: the
// weight rows are interleaved so that columns [0, 32) of a block are "gate" features and [32, 64) the matching "up"
// features) say so with `static constexpr bool kGatedPairs = true` and a `static float gatePair(float gate, float up)`.
// Only chunks 0-3 of a staged row then carry data.
template <typename E, typename = void>
struct IsGatedEpilogue : std::false_type {};
template <typename E>
struct IsGatedEpilogue<E, std::void_t<decltype(E::kGatedPairs)>> : std::bool_constant<E::kGatedPairs> {};

// Epilogues that do a whole tile themselves, with a row of the accumulator per lane and their own staging memory and
// barriers, say so with `static constexpr bool kRowEpilogue = true` (two-SM core only; see ResidualSumsqRows).
template <typename E, typename = void>
struct IsRowEpilogue : std::false_type {};
template <typename E>
struct IsRowEpilogue<E, std::void_t<decltype(E::kRowEpilogue)>> : std::bool_constant<E::kRowEpilogue> {};

// A warp's 32 x 64 block of the accumulator, packed, into its staging buffer.
template <typename Epilogue>
MSCCLPP_DEVICE_INLINE void stageBlock(uint32_t (&v0)[32], uint32_t (&v1)[32], uint8_t* stage, int lane) {
  // the buffer is free once the bulk store of the previous block has read it (or block() has ended)
  if constexpr (Epilogue::kBulkStore) {
    if (lane == 0) ptx::bulk_wait_read<0>();
  }
  __syncwarp();
  if constexpr (IsGatedEpilogue<Epilogue>::value) {
#pragma unroll
    for (int i = 0; i < 32; i++) v0[i] = __float_as_uint(Epilogue::gatePair(__uint_as_float(v0[i]), __uint_as_float(v1[i])));
#pragma unroll
    for (int c = 0; c < 4; c++) *reinterpret_cast<uint4*>(stage + stagedOffset(lane, c)) = packChunk<Epilogue>(v0, c);
  } else {
#pragma unroll
    for (int c = 0; c < 4; c++) {
      *reinterpret_cast<uint4*>(stage + stagedOffset(lane, c)) = packChunk<Epilogue>(v0, c);
      *reinterpret_cast<uint4*>(stage + stagedOffset(lane, c + 4)) = packChunk<Epilogue>(v1, c);
    }
  }
  if constexpr (Epilogue::kBulkStore) ptx::fence_proxy_async_smem();
  __syncwarp();
}

// One epilogue warp, one tile: `taddr` is the TMEM address of the warp's lane quarter at its first column,
// (row0, col0) the global coordinates of that corner. Calls arriveEmpty() as soon as the warp's last accumulator
// read has completed, i.e. before the last block is written out.
template <int kColsPerWarp, typename Epilogue, typename ArriveEmpty>
MSCCLPP_DEVICE_INLINE void stagedEpilogueTile(Epilogue& epi, uint32_t taddr, uint8_t* stage, int row0, int col0, int lane,
                                              ArriveEmpty&& arriveEmpty, int probe = 0) {
  static_assert(kColsPerWarp % 64 == 0, "an epilogue warp works in blocks of 64 columns");
  constexpr int kBlocks = kColsPerWarp / 64;
  const bool drop = (probe & 4) != 0;
  if (probe & 8) {  // diagnostics: hand the accumulator back unread
    ptx::tcgen05_fence_before_sync();
    __syncwarp();
    if (lane == 0) arriveEmpty();
    return;
  }
#pragma unroll
  for (int b = 0; b < kBlocks; b++) {
    uint32_t v0[32], v1[32];
    ptx::tmem_ld_32x32b_x32(taddr + b * 64, v0);
    ptx::tmem_ld_32x32b_x32(taddr + b * 64 + 32, v1);
    ptx::tmem_ld_wait();
    if (b == kBlocks - 1) {
      ptx::tcgen05_fence_before_sync();
      __syncwarp();
      if (lane == 0) arriveEmpty();
    }
    stageBlock<Epilogue>(v0, v1, stage, lane);
    if (!drop) epi.block(stage, row0, col0 + b * 64, lane, b);
  }
}

// One epilogue warp of a CTA whose cluster shares one tile: every CTA holds the products of its part of the reduction, and each
// finishes kOwnBlocks of the tile's 32 x 64 blocks. A warp has one block. It either copies it into the shared memory of the CTA that finishes
// it (fp32, a float4 of every lane next to one another: no bank conflicts on either side; a bulk copy, whose bytes count on the
// block's barrier there - plain stores to the other CTA and a release took 0.3-0.7 us longer), or it adds what comes for it to its
// accumulator, in the order of the ranks, and finishes it like any other. Returns false if a part did not come.
template <int kBlockN, int kSplit, typename Epilogue>
MSCCLPP_DEVICE_INLINE bool splitEpilogueTile(Epilogue& epi, uint32_t taddr, uint8_t* recv, uint64_t* got, uint8_t* send, uint8_t* stage, int row0,
                                             int col0, int quarter, int part, int lane, DeviceStatus* status, uint64_t budgetNs) {
  using Cfg = Config<kBlockN, kSplit>;
  const int rank = static_cast<int>(ptx::cluster_ctarank());
  const int block = part * 4 + quarter, owner = block / Cfg::kOwnBlocks, slot = block % Cfg::kOwnBlocks;
  uint32_t v0[32], v1[32];
  ptx::tmem_ld_32x32b_x32(taddr + part * 64, v0);
  ptx::tmem_ld_32x32b_x32(taddr + part * 64 + 32, v1);
  ptx::tmem_ld_wait();
  if (owner != rank) {
    uint4* out = reinterpret_cast<uint4*>(send) + lane;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      out[j * 32] = make_uint4(v0[4 * j], v0[4 * j + 1], v0[4 * j + 2], v0[4 * j + 3]);
      out[(j + 8) * 32] = make_uint4(v1[4 * j], v1[4 * j + 1], v1[4 * j + 2], v1[4 * j + 3]);
    }
    ptx::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      ptx::bulk_s2cluster(ptx::mapa_shared(ptx::smem_u32(recv) + (slot * (kSplit - 1) + (rank < owner ? rank : rank - 1)) * kPartBytes, owner), send,
                          kPartBytes, ptx::mapa_shared(ptx::smem_u32(&got[slot]), owner));
    }
    return true;
  }
  const bool ok = __all_sync(0xffffffffu, mbarWait(&got[slot], 0, status, budgetNs, 460 + slot));
  if (!ok) return false;
  const float4* in = reinterpret_cast<const float4*>(recv + slot * (kSplit - 1) * kPartBytes) + lane;
#pragma unroll
  for (int s = 0; s < kSplit - 1; s++) {
#pragma unroll
    for (int j = 0; j < 16; j++) {
      uint32_t* v = j < 8 ? &v0[4 * j] : &v1[4 * j - 32];
      const float4 p = in[s * (kPartBytes / 16) + j * 32];
      v[0] = __float_as_uint(__uint_as_float(v[0]) + p.x);
      v[1] = __float_as_uint(__uint_as_float(v[1]) + p.y);
      v[2] = __float_as_uint(__uint_as_float(v[2]) + p.z);
      v[3] = __float_as_uint(__uint_as_float(v[3]) + p.w);
    }
  }
  stageBlock<Epilogue>(v0, v1, stage, lane);
  epi.block(stage, row0, col0 + part * 64, lane, 0);
  return true;
}

// Body of a GEMM CTA. All 192 threads call it. `ctaIdx`/`numCtas` index the persistent tile loop. kSplit > 1: they index clusters of
// kSplit CTAs, as many as there are tiles.
template <int kBlockN, typename AGate, typename Epilogue, int kSplit = 1>
MSCCLPP_DEVICE_INLINE void gemmCta(const CUtensorMap* tmapA, const CUtensorMap* tmapB, Shape shape, int ctaIdx,
                                   int numCtas, AGate& gate, Epilogue& epi, DeviceStatus* status, uint64_t budgetNs,
                                   uint8_t* smemRaw) {
  using Cfg = Config<kBlockN, kSplit>;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // ---- carve shared memory (tiles need 1024-byte alignment for the 128B swizzle)
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
  uint8_t* tiles = smem;
  [[maybe_unused]] uint8_t* recv = smem + Cfg::kStages * Cfg::kStageBytes;
  uint8_t* staging = kSplit > 1 ? tiles : recv;  // 1024-byte aligned: every stage is a multiple of 1024 bytes
  uint64_t* bars = reinterpret_cast<uint64_t*>(recv + Cfg::kRecvBytes + Cfg::kStagingBytes);
  SharedState st;
  st.full = bars;
  st.empty = bars + Cfg::kStages;
  st.tmemFull = bars + 2 * Cfg::kStages;
  st.tmemEmpty = bars + 2 * Cfg::kStages + 2;
  st.tmemBase = reinterpret_cast<uint32_t*>(bars + 2 * Cfg::kStages + 4);
  st.abortFlag = reinterpret_cast<volatile uint32_t*>(st.tmemBase + 1);
  st.epiArrivals = reinterpret_cast<volatile uint32_t*>(st.tmemBase + 2);
  [[maybe_unused]] uint64_t* got = bars + 2 * Cfg::kStages + 6;  // [kOwnBlocks] the peers' parts of a block have come
  static_assert(kSplit == 1 || (2 * Cfg::kStages + 6 + Cfg::kOwnBlocks) * 8 <= Cfg::kBarrierBytes, "barriers");
  static_assert(kSplit == 1 || !Epilogue::kNeedsTileBarrier, "the split form finishes single blocks");

  const int numMBlk = (shape.M + kBlockM - 1) / kBlockM;
  const int numNBlk = (shape.N + kBlockN - 1) / kBlockN;  // (the last tile may reach beyond N: see StoreBf16)
  const int numTiles = numMBlk * numNBlk;
  const int numKBlkAll = shape.K / kBlockK;
  const int split = kSplit > 1 ? static_cast<int>(ptx::cluster_ctarank()) : 0;
  const int kBlk0 = kSplit > 1 ? numKBlkAll * split / kSplit : 0;  // this CTA's part of the reduction
  const int kBlkEnd = kSplit > 1 ? numKBlkAll * (split + 1) / kSplit : numKBlkAll;
  unsigned long long* tl = shape.stamps != nullptr ? shape.stamps + static_cast<size_t>(blockIdx.x) * kStampWords : nullptr;
  if (tl != nullptr && threadIdx.x == 0) tl[0] = ptx::globaltimer();

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; s++) {
      ptx::mbar_init(&st.full[s], 1);
      ptx::mbar_init(&st.empty[s], 1);
    }
    for (int s = 0; s < 2; s++) {
      ptx::mbar_init(&st.tmemFull[s], 1);
      ptx::mbar_init(&st.tmemEmpty[s], Cfg::kEpiWarps);  // one arrival per epilogue warp that takes part
    }
    if constexpr (kSplit > 1) {
      for (int s = 0; s < Cfg::kOwnBlocks; s++) {
        ptx::mbar_init(&got[s], 1);
        ptx::mbar_expect_tx(&got[s], (kSplit - 1) * kPartBytes);
      }
    }
    *st.abortFlag = 0;
    *st.epiArrivals = 0;
    ptx::fence_mbar_init();
    ptx::tma_prefetch_desc(tmapA);
    ptx::tma_prefetch_desc(tmapB);
  }
  if (warp == 1) {
    ptx::tmem_alloc(st.tmemBase, Cfg::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tcgen05_fence_before_sync();
  __syncthreads();
  // every CTA of the cluster runs and its barriers exist before a peer writes into its shared memory
  if constexpr (kSplit > 1) ptx::cluster_sync_all();
  ptx::tcgen05_fence_after_sync();
  const uint32_t tmemBase = *st.tmemBase;
  // everything up to here is this CTA's own: with a programmatic dependent launch it ran under the kernel before
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  if (warp == 0) {
    // ===================================================== TMA producer (one thread)
    // The single threads of this warp and the next are taken with elect.sync, not by lane number: the compiler then knows
    // that exactly one thread runs the loop and keeps descriptors and barrier addresses uniform. Measured on a B200 (128 x
    // 128 tiles, K = 4096, operands in L2): 0.41 us per 64-wide k block with `lane == 0`, 0.28 us with elect.sync; 333 x
    // 6144 x 4096 26.7 -> 18.0 us, 128 x 8192 x 1024 9.5 -> 7.2 us, and with the two-SM core 8192 x 7168 x 8192 779 -> 684 us.
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t armed = 0;        // bit s: stage s has a load in flight that nobody has waited for yet
      uint32_t armedParity = 0;  // parity those loads complete
      bool ok = true;
      for (int tile = ctaIdx; tile < numTiles && ok; tile += numCtas) {
        int mBlk, nBlk;
        tileCoord(shape, tile, numMBlk, numNBlk, mBlk, nBlk);
        ok = gate.waitRowBlock(mBlk);
        int aRow;
        const CUtensorMap* tmapARows = gate.tmapA(mBlk, tmapA, aRow);
        for (int kb = kBlk0; kb < kBlkEnd && ok; kb += Cfg::kKb) {
          if (tl != nullptr) {
            const unsigned long long t0 = ptx::globaltimer();
            ok = mbarWaitFast(&st.empty[stage], phase ^ 1u, status, budgetNs, 100 + stage, st.abortFlag);
            tl[8] += ptx::globaltimer() - t0;
          } else {
            ok = mbarWaitFast(&st.empty[stage], phase ^ 1u, status, budgetNs, 100 + stage, st.abortFlag);
          }
          if (!ok) break;
          uint8_t* sa = tiles + stage * Cfg::kStageBytes;
          uint8_t* sb = sa + Cfg::kKb * Cfg::kStageABytes;
          if (shape.probe & 1) {
            ptx::mbar_arrive(&st.full[stage]);
          } else {
            const int blocks = Cfg::kKb == 1 || kBlkEnd - kb > Cfg::kKb ? Cfg::kKb : kBlkEnd - kb;  // (the last stage may not be full)
            ptx::mbar_expect_tx(&st.full[stage], blocks * (shape.aBoxRows * kBlockK * 2 + Cfg::kStageBBytes));
#pragma unroll
            for (int j = 0; j < Cfg::kKb; j++) {
              if (j >= blocks) break;
              ptx::tma_load_2d(sa + j * Cfg::kStageABytes, tmapARows, (kb + j) * kBlockK, aRow, &st.full[stage]);
              ptx::tma_load_2d(sb + j * Cfg::kStageBBytes, tmapB, (kb + j) * kBlockK, nBlk * kBlockN, &st.full[stage]);
            }
          }
          armed |= 1u << stage;
          armedParity = (armedParity & ~(1u << stage)) | (phase << stage);
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok) {
        *st.abortFlag = 1;
        // drain: wait (bounded) until every load this thread issued has landed
        for (int s = 0; s < Cfg::kStages; s++) {
          if (armed & (1u << s)) mbarWait(&st.full[s], (armedParity >> s) & 1u, nullptr, 2000000ull, 0);
        }
      }
    }
  } else if (warp == 1) {
    // ===================================================== MMA issuer (one thread)
    if (ptx::elect_one()) {
      constexpr uint32_t idesc = makeInstrDesc<kBlockN>();
      // The issue loop is ONE thread feeding the tensor core: every instruction in it is on the critical path of the
      // whole SM. Descriptors are formed once and stepped by adds; the common case of each wait is one instruction.
      const uint64_t descA0 = makeSmemDesc(ptx::smem_u32(tiles));
      const uint64_t descB0 = makeSmemDesc(ptx::smem_u32(tiles) + Cfg::kKb * Cfg::kStageABytes);
      constexpr uint64_t kStageStep = Cfg::kStageBytes >> 4;  // a stage, in the descriptor's 16-byte address units
      const bool issue = (shape.probe & 2) == 0;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int it = 0;
      for (int tile = ctaIdx; tile < numTiles && ok; tile += numCtas, it++) {
        const int acc = it & 1;
        const uint32_t accPhase = (it >> 1) & 1;
        if (tl != nullptr) {
          const unsigned long long t0 = ptx::globaltimer();
          ok = mbarWaitFast(&st.tmemEmpty[acc], accPhase ^ 1u, status, budgetNs, 200 + acc, st.abortFlag);
          tl[2] += ptx::globaltimer() - t0;
        } else {
          ok = mbarWaitFast(&st.tmemEmpty[acc], accPhase ^ 1u, status, budgetNs, 200 + acc, st.abortFlag);
        }
        if (!ok) break;
        ptx::tcgen05_fence_after_sync();
        const uint32_t tmemD = tmemBase + acc * kBlockN;
        for (int kb = kBlk0; kb < kBlkEnd; kb += Cfg::kKb) {
          if (tl != nullptr) {
            const unsigned long long t0 = ptx::globaltimer();
            ok = mbarWaitFast(&st.full[stage], phase, status, budgetNs, 300 + stage, st.abortFlag);
            tl[3] += ptx::globaltimer() - t0;
          } else {
            ok = mbarWaitFast(&st.full[stage], phase, status, budgetNs, 300 + stage, st.abortFlag);
          }
          if (!ok) break;
          ptx::tcgen05_fence_after_sync();
          const uint64_t descA = descA0 + stage * kStageStep;
          const uint64_t descB = descB0 + stage * kStageStep;
          if (issue) {
            // advancing K by 16 elements = 32 bytes inside the 128-byte swizzle row: +2 in the (>>4) address field
            ptx::tcgen05_mma_f16(tmemD, descA, descB, idesc, kb != kBlk0 ? 1u : 0u);
#pragma unroll
            for (int k = 1; k < kBlockK / kUmmaK; k++) ptx::tcgen05_mma_f16_acc(tmemD, descA + 2 * k, descB + 2 * k, idesc);
#pragma unroll
            for (int j = 1; j < Cfg::kKb; j++) {
              if (kb + j >= kBlkEnd) break;
#pragma unroll
              for (int k = 0; k < kBlockK / kUmmaK; k++)
                ptx::tcgen05_mma_f16_acc(tmemD, descA + j * (Cfg::kStageABytes >> 4) + 2 * k, descB + j * (Cfg::kStageBBytes >> 4) + 2 * k, idesc);
            }
          }
          ptx::tcgen05_commit(&st.empty[stage]);  // frees the smem stage once these MMAs retire
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) ptx::tcgen05_commit(&st.tmemFull[acc]);
      }
      if (tl != nullptr) tl[1] = ptx::globaltimer();
      if (!ok) *st.abortFlag = 1;
    }
  } else if (warp < 2 + Cfg::kEpiWarps) {
    // ===================================================== epilogue (lane quarter x column part per warp)
    const int quarter = warp & 3;  // a warp may only touch TMEM lanes [32*(warpid%4), +32)
    const int part = (warp - 2) >> 2;
    uint8_t* stage = staging + (warp - 2) * kStagingBytesPerWarp;
    bool ok = true;
    int it = 0;
    for (int tile = ctaIdx; tile < numTiles && ok; tile += numCtas, it++) {
      int mBlk, nBlk;
      tileCoord(shape, tile, numMBlk, numNBlk, mBlk, nBlk);
      const int acc = it & 1;
      const uint32_t accPhase = (it >> 1) & 1;
      const int row0 = mBlk * kBlockM + quarter * 32;
      const int col0 = nBlk * kBlockN + part * Cfg::kColsPerWarp;
      // lets the epilogue put loads it will need (a residual, a bias) in flight while the MMAs of this tile still run
      if constexpr (kSplit > 1) {
        if ((part * 4 + quarter) / Cfg::kOwnBlocks == split) epi.tileBegin(row0, col0, lane);
      } else {
        epi.tileBegin(row0, col0, lane);
      }
      const bool stampIt = tl != nullptr && warp == 2 && lane == 0;
      unsigned long long tw0 = 0;
      if (stampIt) tw0 = ptx::globaltimer();
      ok = mbarWait(&st.tmemFull[acc], accPhase, status, budgetNs, 400 + acc);
      ok = __all_sync(0xffffffffu, ok) && (*st.abortFlag == 0);
      if (!ok) break;
      if (stampIt) {
        const unsigned long long now = ptx::globaltimer();
        tl[5] += now - tw0;
        tw0 = now;
      }
      ptx::tcgen05_fence_after_sync();
      if constexpr (kSplit > 1) {
        ok = splitEpilogueTile<kBlockN, kSplit>(epi, tmemBase + (static_cast<uint32_t>(quarter * 32) << 16), recv, got, staging + kEpilogueStagingBytes + (warp - 2) * kPartBytes, stage, row0, nBlk * kBlockN,
                                                quarter, part, lane, status, budgetNs);
        break;
      }
      const uint32_t taddr = tmemBase + (static_cast<uint32_t>(quarter * 32) << 16) + acc * kBlockN + part * Cfg::kColsPerWarp;
      // the accumulator buffer can be overwritten by the MMA warp as soon as every warp has read its part
      stagedEpilogueTile<Cfg::kColsPerWarp>(epi, taddr, stage, row0, col0, lane, [&] { ptx::mbar_arrive(&st.tmemEmpty[acc]); }, shape.probe);
      if (stampIt) {
        const unsigned long long now = ptx::globaltimer();
        tl[6] += now - tw0;
        tl[4] = now;
      }
      if constexpr (Epilogue::kNeedsTileBarrier) {
        // All epilogue warps have issued their stores -> let the fused kernel publish the tile. The
        // meeting point is a counter with a bounded wait (not bar.sync): if one warp gave up on the
        // accumulator barrier above, the others must not wait for it forever.
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
    if (tl != nullptr && warp == 2 && lane == 0) tl[7] = ptx::globaltimer();
    if (!ok && lane == 0) *st.abortFlag = 1;
    // bulk stores of this warp still read its staging buffer: the CTA must not end before they have
    if constexpr (Epilogue::kBulkStore) {
      if (lane == 0) ptx::bulk_wait<0>();
    }
  } else if (warp >= 2 + kNumEpilogueWarps) {
    // warps beyond the ten of the GEMM roles (a kernel may launch more threads): follow-up work of a fused epilogue that
    // must stay off the epilogue warps' critical path
    epi.auxWarp(warp - (2 + kNumEpilogueWarps), lane);
  }

  // ---- teardown: everybody meets, then the allocating warp frees TMEM
  ptx::tcgen05_fence_before_sync();
  __syncthreads();
  // (a peer may still write into this CTA's shared memory, or this one into a peer's)
  if constexpr (kSplit > 1) ptx::cluster_sync_all();
  ptx::tcgen05_fence_after_sync();
  if (warp == 1) ptx::tmem_dealloc(tmemBase, Cfg::kTmemCols);
}

// Plain epilogue: every staged 32 x 64 block leaves with one tiled bulk store (rows beyond M are clipped by the
// tensor map, whose box is 64 columns x 32 rows with the 128-byte swizzle of the staging layout). N is a multiple of 64, not
// necessarily of the tile: rows of B beyond N are read as zeros, blocks beyond it stay where they are.
struct StoreBf16 {
  static constexpr bool kNeedsTileBarrier = false;
  static constexpr bool kBulkStore = true;
  const CUtensorMap* tmapD;
  int M, N;
  MSCCLPP_DEVICE_INLINE static float convert(float x) { return x; }
  MSCCLPP_DEVICE_INLINE void tileBegin(int, int, int) const {}
  MSCCLPP_DEVICE_INLINE void block(const uint8_t* stage, int row0, int col0, int lane, int /*b*/) const {
    if (lane == 0 && row0 < M && col0 < N) {
      ptx::tma_store_2d(tmapD, stage, col0, row0);
      ptx::bulk_commit();
    }
  }
  MSCCLPP_DEVICE_INLINE void tileDone(int, int, int) const {}
  MSCCLPP_DEVICE_INLINE void warpTileDone(int, int) const {}
  MSCCLPP_DEVICE_INLINE void warpDrain(int) const {}
  MSCCLPP_DEVICE_INLINE void auxWarp(int, int) const {}
};

}  // namespace gemm
}  // namespace mscclpp
