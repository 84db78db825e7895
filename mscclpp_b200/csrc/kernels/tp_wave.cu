// The layer of one GPU for prompts, in ONE launch that never re-reads what it has computed:
//
//     h   = X[M,K] * W[N,K]^T + residual          (bf16, fp32 accumulation)
//     out = h * rsqrt(mean(h^2) + eps) * gamma
//
// The two-launch form stores h and reads it back for the norm: at 8192 x 8192 that is 268 MB of the 570 MB it moves, in a
// pass of its own. Here a tile of h stays on chip until the sums of squares of its rows are complete, under the matrix products of
// the tiles after it:
//   * the tiles are walked row block by row block, so the N / 256 tiles that share rows run on different pairs of SMs in the same
//     wave or in two consecutive ones;
//   * the eight epilogue warps of the GEMM core make h: accumulator + residual, stored by bulk copies; the sums of squares
//     of the rows over a warp's columns go to a table in global memory;
//   * eight more warps make `out`: each takes 16 rows of the tile out of the staging boxes into registers, which frees the boxes for
//     the next residual, adds up the rows' parts in a fixed order once they are complete, scales and stores, a row's 512 bytes per instruction;
//   * one extra warp per CTA does the exchange: it counts the CTA's finished tile on its 128-row block (one release per tile)
//     and waits until all N / 256 tiles of the block are counted.
// What bounds it (8192 x 8192 x 1024, 139 us in graph replay; two launches 160, 185 once the power limit has brought the clocks
// down): the SMs' inputs and the power. The operand tiles alone are 1.07 GB into the SMs, 64 us at full clock; with residual and
// matrix products that path, the memory's 436 MB (67 us) and the tensor cores (60 us at full clock, 90 at the power limit)
// overlap only in part. The residual and `out` carry evict-first policies, which keeps the operands in L2: DRAM reads 240 -> 176 MB.
// Tried instead: the epilogue warps making `out` too, with h of two tiles in their registers, 215 us, or fetched back by
// bulk copies, 144: two warps per scheduler cannot hide the latencies of both; separate warps that read h back from L2, 143.
// Blocks wait for one another's tiles, so the launch is cooperative. It always ends: a tile is published before its CTA
// waits for anything, and what a CTA waits for are tiles of the same row block, at most one tile further in every pair's list.
// Every wait is bounded all the same.
//
// The reference library has no counterpart (it offers the allreduce alone).
#include <mutex>
#include <map>

#include <mscclpp/gpu_data_types.hpp>

#include "bf16x8.cuh"
#include "gemm2_sm100.cuh"
#include "tp_fused.cuh"

namespace mscclpp {

namespace {

using bf16 = __nv_bfloat16;
constexpr int kScaleWarps = 8;                        // 16 rows of a tile each
constexpr int kWaveThreads = gemm::kNumThreads + 32 * (kScaleWarps + 1);
constexpr int kBoxesOfWarp = 2;                       // 32 rows x 64 columns: an epilogue warp's part of a tile
// barriers: 20 words of the core, the boxes' loads, 6 of the exchange
constexpr int kBarWords = 20 + gemm::kNumEpilogueWarps * kBoxesOfWarp + 6;
using ConfigWave = gemm::Config2Of<5, kBoxesOfWarp * gemm::kEpilogueStagingBytes, kBarWords * 8>;
static_assert(kBoxesOfWarp * 64 == ConfigWave::kColsPerWarp && kScaleWarps * 16 == gemm::kBlockM, "");

MSCCLPP_DEVICE_INLINE uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
MSCCLPP_DEVICE_INLINE void sts128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

struct LayerRows {
  static constexpr bool kNeedsTileBarrier = false;
  static constexpr bool kBulkStore = true;
  static constexpr bool kRowEpilogue = true;
  static constexpr int kBlocks = kBoxesOfWarp;
  const CUtensorMap* tmapResidual;  // boxes of 64 columns x 32 rows; null = no residual
  const CUtensorMap* tmapH;
  bf16* out;           // [M, N]
  const bf16* gamma;   // [N] or null
  float* parts;        // [128-row block][2 * N / 256][128] sums of squares of the rows over a warp's 128 columns
  uint32_t* counters;  // [128-row block] tiles published; zero at launch
  int M, N, numTiles, pairIdx, numPairs;
  float eps;
  DeviceStatus* status;
  uint64_t budgetNs;
  uint32_t boxes = 0;        // shared-memory address of this warp's boxes
  uint64_t* here = nullptr;  // ... and the barriers of their loads
  // By tile parity. The boxes are taken before the next tile may be worked on, and a tile is taken when the one before is through: no
  // barrier gets a whole turn ahead of one who waits for it.
  uint64_t* sums = nullptr;   // [2] h of a tile is in the boxes and its rows' sums of squares in the table: eight epilogue warps arrive
  uint64_t* taken = nullptr;  // [2] ... and in the registers of the scale warps, which arrive
  uint64_t* ready = nullptr;  // [2] all tiles of the row block are counted
  uint64_t once = 0;           // L2 policy of what is read or written once: it makes room before the operands do
  int loads = 0;               // of tiles requested so far
  int tiles = 0;               // whose h is computed
  bool came = true;            // (lane 0) the boxes were taken in time

  MSCCLPP_DEVICE_INLINE void setup(uint8_t* boxes_, uint64_t* here_, int lane) {
    const int idx = static_cast<int>(threadIdx.x >> 5) - 2;
    boxes = ptx::smem_u32(boxes_);
    here = here_;
    sums = here_ - idx * kBlocks + gemm::kNumEpilogueWarps * kBlocks;
    taken = sums + 2;
    ready = sums + 4;
    once = ptx::l2_evict_first();
    if (lane == 0) {
      if (idx < gemm::kNumEpilogueWarps) {
        for (int b = 0; b < kBlocks; b++) ptx::mbar_init(&here[b], 1);
      } else if (idx == gemm::kNumEpilogueWarps) {
        for (int p = 0; p < 2; p++) {
          ptx::mbar_init(&sums[p], gemm::kNumEpilogueWarps);
          ptx::mbar_init(&taken[p], kScaleWarps);
          ptx::mbar_init(&ready[p], 1);
        }
      }
      ptx::fence_mbar_init();
    }
    __syncwarp();
  }
  // The residual of the next tile, as soon as h has left the boxes both ways.
  MSCCLPP_DEVICE_INLINE void request(int row0, int col0, int lane) {
    loads++;
    if (lane != 0) return;
    if (tiles > 0) came = mbarWait(&taken[(tiles - 1) & 1], ((tiles - 1) >> 1) & 1, status, budgetNs, 460);
    if (tmapResidual == nullptr) return;
#pragma unroll
    for (int b = 0; b < kBlocks; b++) {
      if (b == 0) ptx::bulk_wait_read<kBlocks - 1>();
      else ptx::bulk_wait_read<0>();
      ptx::mbar_expect_tx(&here[b], gemm::kStagingBytesPerWarp);
      ptx::tma_load_2d_hint(boxes + b * gemm::kStagingBytesPerWarp, tmapResidual, col0 + b * 64, row0, &here[b], once);
    }
  }

  // h of one tile. Returns false if something did not come.
  template <typename ArriveEmpty>
  MSCCLPP_DEVICE_INLINE bool tile(uint32_t taddr, int row0, int col0, int it, int lane, ArriveEmpty&& arriveEmpty) {
    uint64_t ss = 0, ss1 = 0;  // two sums each
    bool ok = __all_sync(0xffffffffu, came);
    if (!ok) return false;
#pragma unroll 1
    for (int b = 0; b < kBlocks; b++) {
      const uint32_t box = boxes + b * gemm::kStagingBytesPerWarp;
      if (tmapResidual != nullptr) {
        ok = mbarWait(&here[b], it & 1, status, budgetNs, 450 + b);
        if (!__all_sync(0xffffffffu, ok)) return false;
      } else {
        if (lane == 0) ptx::bulk_wait_read<0>();  // the stores of the tile before
        __syncwarp();
      }
#pragma unroll 1
      for (int q = 0; q < 2; q++) {
        uint32_t v[32];
        ptx::tmem_ld_32x32b_x32(taddr + b * 64 + q * 32, v);
        uint4 r[4];
        uint32_t at[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          at[c] = box + gemm::stagedOffset(lane, q * 4 + c);
          r[c] = make_uint4(0, 0, 0, 0);
          if (tmapResidual != nullptr) r[c] = lds128(at[c]);
        }
        ptx::tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; c++) {
          uint4 x = gemm::packChunk<LayerRows>(v, c);
          if (tmapResidual != nullptr) x = addBf16x8(x, r[c]);
          sts128(at[c], x);
          const uint64_t p0 = pairOf(x.x), p1 = pairOf(x.y), p2 = pairOf(x.z), p3 = pairOf(x.w);
          ss = fmaPair(p0, p0, ss);
          ss1 = fmaPair(p1, p1, ss1);
          ss = fmaPair(p2, p2, ss);
          ss1 = fmaPair(p3, p3, ss1);
        }
      }
      if (b == kBlocks - 1) {
        ptx::tcgen05_fence_before_sync();
        __syncwarp();
        if (lane == 0) arriveEmpty();
      }
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (row0 < M) ptx::tma_store_2d(tmapH, box, col0 + b * 64, row0);
        ptx::bulk_commit();  // (an empty group keeps the count of groups the same in every tile)
      }
    }
    const int row = row0 + lane, perRow = 2 * (N / ConfigWave::kBlockN);
    const float2 s0 = valuesOf(ss), s1 = valuesOf(ss1);
    if (row < M) {
      parts[(static_cast<size_t>(row0 / gemm::kBlockM) * perRow + col0 / ConfigWave::kColsPerWarp) * gemm::kBlockM + (row & (gemm::kBlockM - 1))] =
          (s0.x + s0.y) + (s1.x + s1.y);
    }
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&sums[it & 1]);
    tiles = it + 1;
    return true;
  }
  MSCCLPP_DEVICE_INLINE void warpDrain(int) const {}
  // After an abort: what is still on its way into the boxes must land before the CTA may end.
  MSCCLPP_DEVICE_INLINE void drain(int done) const {
    if (tmapResidual == nullptr || loads <= done) return;
    for (int b = 0; b < kBlocks; b++) (void)mbarWait(&here[b], (loads - 1) & 1, nullptr, 2000000ull, 0);
  }

  MSCCLPP_DEVICE_INLINE void auxWarp(int idx, int lane) const {
    const int perRow = N / ConfigWave::kBlockN;  // tiles that share a row block
    const int count = numTiles > pairIdx ? (numTiles - pairIdx + numPairs - 1) / numPairs : 0;
    if (idx == kScaleWarps) {
      if (lane == 0) exchange(perRow, count);
    } else {
      scaleTiles(idx, lane, perRow, count);
    }
  }
  MSCCLPP_DEVICE_INLINE int rowBlock(int it, int perRow) const {
    return 2 * ((pairIdx + it * numPairs) / perRow) + static_cast<int>(ptx::cluster_ctarank());
  }
  // One thread. Publishing waits for nothing but this CTA's own epilogue: while the thread polls for the rows of one tile it also
  // looks whether the next tile has to be published.
  MSCCLPP_DEVICE_INLINE void exchange(int perRow, int count) const {
    int published = 0;
    for (int it = 0; it < count; it++) {
      const int mBlk = rowBlock(it, perRow);
      SpinGuard guard(status, budgetNs);
      for (;;) {
        if (published < count && published <= it + 1 && ptx::mbar_test_wait(&sums[published & 1], (published >> 1) & 1)) {
          // cumulative: the eight warps' parts, observed through the barrier, are released with the count
          ptx::red_release_gpu_add(counters + rowBlock(published, perRow), 1);
          published++;
          continue;
        }
        if (published > it && static_cast<int32_t>(ptx::ld_acquire_gpu(counters + mBlk)) >= perRow) break;
        if (!guard.keepSpinning()) {
          guard.report(kDevTimeoutFlag, 0, 470, mBlk, perRow, published);
          return;  // the scale warps' wait for this tile runs out too
        }
      }
      ptx::mbar_arrive(&ready[it & 1]);
    }
  }
  MSCCLPP_DEVICE_INLINE void scaleTiles(int idx, int lane, int perRow, int count) const {
    const size_t words = static_cast<size_t>(N / 8);
    // This lane's eight columns of a row: box (lane / 8) & 1 of the epilogue warp with that column half and this warp's row quarter.
    // (An epilogue warp's quarter is its number modulo 4, so warp 2 has quarter 2: the boxes of quarter q are the (q + 2) % 4th.)
    const uint32_t firstBox = boxes - (gemm::kNumEpilogueWarps + idx) * (kBlocks * gemm::kStagingBytesPerWarp);
    const int owner = ((idx / 2 + 2) & 3) + 4 * (lane >> 4);
    const uint32_t mine = firstBox + (owner * kBlocks + ((lane >> 3) & 1)) * gemm::kStagingBytesPerWarp;
    for (int it = 0; it < count; it++) {
      const int mBlk = rowBlock(it, perRow);
      const int row0 = mBlk * gemm::kBlockM + idx * 16;
      const size_t word = static_cast<size_t>((pairIdx + it * numPairs) % perRow) * (ConfigWave::kBlockN / 8) + lane;  // of a row
      bool ok = mbarWait(&sums[it & 1], (it >> 1) & 1, status, budgetNs, 480);
      if (!__all_sync(0xffffffffu, ok)) return;
      uint4 v[16];
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = lds128(mine + gemm::stagedOffset((idx & 1) * 16 + j, lane & 7));
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&taken[it & 1]);
      uint4 gw = make_uint4(0, 0, 0, 0);
      if (gamma != nullptr) gw = ptx::ld_weak_v4(reinterpret_cast<const uint4*>(gamma) + word);
      ok = mbarWait(&ready[it & 1], (it >> 1) & 1, status, budgetNs, 490);
      if (!__all_sync(0xffffffffu, ok)) return;
      // the parts of 16 rows, the even ones in the lower half of the warp, the odd ones in the upper
      const float* src = parts + (static_cast<size_t>(mBlk) * (2 * perRow) + (lane >> 4)) * gemm::kBlockM + idx * 16 + (lane & 15);
      float total = 0.f;
      constexpr int kDepth = 8;
#pragma unroll 1
      for (int p0 = 0; p0 < perRow; p0 += kDepth) {
        float f[kDepth];
#pragma unroll
        for (int k = 0; k < kDepth; k++) {
          f[k] = 0.f;
          if (p0 + k < perRow) f[k] = __ldcg(src + static_cast<size_t>(p0 + k) * (2 * gemm::kBlockM));
        }
#pragma unroll
        for (int k = 0; k < kDepth; k++) total += f[k];
      }
      total += __shfl_xor_sync(0xffffffffu, total, 16);
      const float rinv = rsqrtf(total / static_cast<float>(N) + eps);
      const uint64_t g[4] = {pairOf(gw.x), pairOf(gw.y), pairOf(gw.z), pairOf(gw.w)};
      uint4* to = reinterpret_cast<uint4*>(out) + static_cast<size_t>(row0) * words + word;
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const float s = __shfl_sync(0xffffffffu, rinv, j);
        const uint64_t sc = pairOf(s, s);
        uint64_t p[4] = {mulPair(pairOf(v[j].x), sc), mulPair(pairOf(v[j].y), sc), mulPair(pairOf(v[j].z), sc), mulPair(pairOf(v[j].w), sc)};
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          if (gamma != nullptr) p[i] = mulPair(p[i], g[i]);
          o[i] = packPair(p[i]);
        }
        if (row0 + j < M) ptx::st_weak_v4_hint(to, make_uint4(o[0], o[1], o[2], o[3]), once);
        to += words;
      }
    }
  }
  MSCCLPP_DEVICE_INLINE static float convert(float x) { return x; }
  MSCCLPP_DEVICE_INLINE void warpTileDone(int, int) const {}
};

struct WaveArgs {
  bf16* out;
  const bf16* gamma;
  float* parts;
  uint32_t* counters;  // [0]: CTAs that are through; then a counter per 128-row block
  int hasResidual;
  float eps;
  DeviceStatus* status;
  uint64_t budgetNs;
};

__global__ void __launch_bounds__(kWaveThreads, 1)
    tpLayerWaveKernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB,
                      const __grid_constant__ CUtensorMap tmapResidual, const __grid_constant__ CUtensorMap tmapH, gemm::Shape shape,
                      WaveArgs a) {
  extern __shared__ uint8_t smemRaw[];
  const int numBlocks = 2 * ((shape.M + ConfigWave::kPairM - 1) / ConfigWave::kPairM);
  const int numTiles = numBlocks / 2 * (shape.N / ConfigWave::kBlockN);
  const int pairIdx = blockIdx.x / 2, numPairs = gridDim.x / 2;
  gemm::NoGate gate;
  LayerRows epi{a.hasResidual ? &tmapResidual : nullptr, &tmapH, a.out, a.gamma, a.parts, a.counters + 1, shape.M, shape.N,
                numTiles, pairIdx, numPairs, a.eps, a.status, a.budgetNs};
  gemm::gemmCtaPair<ConfigWave>(&tmapA, &tmapB, shape, pairIdx, numPairs, gate, epi, a.status, a.budgetNs, smemRaw);
  // nobody of this CTA looks at the counters any more; the last CTA to come here clears them for the next launch
  if (threadIdx.x == 0 && ptx::atom_add_acqrel_gpu(a.counters, 1) == gridDim.x - 1) {
    for (int i = 0; i <= numBlocks; i++) a.counters[i] = 0;
  }
}

// Pairs of SMs that can run this kernel at the same time on the current device.
int residentPairs() {
  static std::mutex mu;
  static std::map<int, int> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find(dev);
  if (it != known.end()) return it->second;
  const void* kernel = reinterpret_cast<const void*>(tpLayerWaveKernel);
  if (gemm::ensureDynamicSmem(kernel, ConfigWave::kSmemBytes) != cudaSuccess) return 0;  // (the query fails without it)
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(kWaveThreads);
  cfg.dynamicSmemBytes = ConfigWave::kSmemBytes;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) return 0;
  known[dev] = n;
  return n;
}

}  // namespace

bool tpLayerWaveFits(int N) { return N > 0 && N % ConfigWave::kBlockN == 0 && N / ConfigWave::kBlockN <= residentPairs(); }

size_t tpLayerWaveCounterWords(int M) { return 1 + 2 * static_cast<size_t>((M + ConfigWave::kPairM - 1) / ConfigWave::kPairM); }

cudaError_t launchTpLayerWave(const void* A, const void* B, const void* residual, void* h, void* out, const void* gamma, float* parts,
                              uint32_t* counters, int M, int N, int K, float eps, DeviceStatus* status, uint64_t budgetNs, cudaStream_t stream) {
  if (M < ConfigWave::kPairM || N <= 0 || K <= 0 || K % gemm::kBlockK != 0 || N % ConfigWave::kBlockN != 0) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(parts)) & 15) return cudaErrorInvalidValue;
  // row block by row block: what shares rows runs at the same time
  gemm::Shape shape{M, N, K, gemm::kBlockM, 1, 0, 0};
  const uint64_t pitch = static_cast<uint64_t>(N) * 2;
  CUtensorMap ta, tb, tr, th;
  cudaError_t e = gemm::makeTensorMapBf16(&ta, A, M, K, static_cast<uint64_t>(K) * 2, gemm::kBlockM);
  if (e == cudaSuccess) e = gemm::makeTensorMapBf16(&tb, B, N, K, static_cast<uint64_t>(K) * 2, ConfigWave::kBlockN / 2);
  if (e == cudaSuccess) e = gemm::makeTensorMapBf16(&tr, residual != nullptr ? residual : h, M, N, pitch, 32);
  if (e == cudaSuccess) e = gemm::makeTensorMapBf16(&th, h, M, N, pitch, 32);
  const void* kernel = reinterpret_cast<const void*>(tpLayerWaveKernel);
  if (e == cudaSuccess) e = gemm::ensureDynamicSmem(kernel, ConfigWave::kSmemBytes);
  if (e != cudaSuccess) return e;
  const int tiles = ((M + ConfigWave::kPairM - 1) / ConfigWave::kPairM) * (N / ConfigWave::kBlockN);
  if (!tpLayerWaveFits(N)) return cudaErrorInvalidValue;  // a row block has to fit two consecutive waves
  int pairs = residentPairs();
  if (pairs > tiles) pairs = tiles;
  WaveArgs args{static_cast<bf16*>(out), static_cast<const bf16*>(gamma), parts, counters, residual != nullptr, eps, status, budgetNs};
  void* params[] = {&ta, &tb, &tr, &th, &shape, &args};
  return gemm::launchClusterPair(kernel, dim3(2 * pairs), dim3(kWaveThreads), ConfigWave::kSmemBytes, params, true, stream);
}

}  // namespace mscclpp
