// The layer for a handful of tokens (decode) on one GPU, ONE launch in which no thread block waits for another:
//
//     h   = X[T,K] * W[N,K]^T + residual          T <= kTpDecodeMaxTokens (bf16, fp32 accumulation)
//     out = h * rsqrt(mean(h^2) + eps) * gamma
//
// A decode step is a chain of such layers, each a stream over its weights (16 MB at 8192 x 1024, 2.6 us) behind a chain of
// round trips. tp_decode.cu, which also serves several GPUs, is launched cooperatively (its blocks exchange the rows' sums),
// so layer n + 1 starts when layer n has ended. Here
//   * the launch overlaps the kernel before it (programmatic dependent launch): as soon as a block of layer n has ended, one of layer
//     n + 1 takes its place and prefetches its weights, activations and residual into L2. Only then does it wait for
//     layer n. A prefetch moves data to the point of coherence and shows it to nobody, so it does not matter who writes them;
//   * weights and activations come as tiles of 128 reduction elements (cp.async.bulk.tensor, 128-byte swizzle, two boxes), a few dozen
//     requests per block instead of one per weight row: the copy engine takes about ten cycles per request, 1.4 us for 256 of them. The
//     block waits for the thread that requests them: with one barrier per box instead of one per tile 8 x 5120 x 2560 took 11.6 us, not 10.7;
//   * the products are warp-level tensor-core instructions with the weights as the 16-row operand and the tokens as the
//     8-column one, as in tp_decode.cu (a tcgen05 tile starts at 64 rows, and this is a stream); sixteen warps split a block's columns four ways and its tiles four ways;
//   * the rows' sums of squares need every column. Instead of exchanging them, each block counts itself, and the block (with more
//     than two tokens: the pair of blocks) that counts last reads all shares and h back and writes `out`.
//
// One B200, a chain of layers in a CUDA graph, us per layer before / now (floor: the weights from memory): 1 x 8192 x 1024 11.4 / 7.1
// (2.6), 8 x 5120 x 2560 17.4 / 10.7 (4.0), 8 x 8192 x 1024 11.6 / 9.3, 5 x 4160 x 3072 19.3 / 11.8, 3 x 1032 x 256 7.2 / 5.1. What
// bounds it, 1 x 8192 x 1024: 0.7 us from the last store of the layer before to the end of the wait, 0.7 to the first tile,
// 1.8 for the rest (9.3 TB/s, out of L2), 1.3 for the sums, 0.9 for the count, 1.3 for the last block.
// Tried instead: splitting K over clusters of four blocks (one more cluster barrier and the partial sums through
// distributed shared memory) 10.5 us; two blocks per SM, so that layer n + 1 prefetches under the products of layer n: 9.0 against
// 8.9 us with one token at that time, but 16.4 against 13.0 with eight (fewer tiles in flight).
//
// The reference library has no counterpart (it offers the allreduce alone, allreduce_packet.cu).
#include <mscclpp/gpu_data_types.hpp>

#include "bf16x8.cuh"
#include "gemm.cuh"
#include "tp_fused.cuh"

namespace mscclpp {

namespace {

using bf16 = __nv_bfloat16;
constexpr int kWorkers = 512;              // sixteen warps: four column groups x four tiles at a time
constexpr int kThreads = kWorkers + 32;    // and the one that requests the tiles
constexpr int kTileK = 128;                // reduction elements per tile: two boxes of 128 bytes
constexpr int kBoxK = kTileK / 2;
constexpr int kMaxCols = 128;              // output columns per block
constexpr int kMaxTiles = 16;              // in flight
constexpr int kXBytes = kTpDecodeMaxTokens * kTileK * 2;  // both boxes
constexpr int kMaxSmem = 216 * 1024;       // of a block: tiles in flight are worth more than a second block

struct DecodeLocalArgs {
  const bf16* residualIn;  // may be null
  bf16* residualOut;
  bf16* out;
  const bf16* gamma;       // may be null
  float* shares;           // [gridDim.x][kTpDecodeMaxTokens]
  uint32_t* counted;       // blocks that are through; zero between launches
  int T, N, K;
  float eps;
  int cols;                // output columns per block, a multiple of 8
  int stages;              // tiles in flight
  DeviceStatus* status;
  uint64_t budgetNs;
};

MSCCLPP_DEVICE_INLINE void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// kPair: clusters of two blocks, which share the work of the last one.
template <bool kPair>
__global__ void __launch_bounds__(kThreads, 1)
    tpDecodeLocalKernel(const __grid_constant__ CUtensorMap tmapW, const __grid_constant__ CUtensorMap tmapX, const __grid_constant__ DecodeLocalArgs a) {
  extern __shared__ uint8_t smemRaw[];
  __shared__ __align__(8) uint64_t full[kMaxTiles], empty[kMaxTiles];
  __shared__ uint32_t order[2];
  __shared__ float rinv[kTpDecodeMaxTokens];
  ptx::grid_launch_dependents();
  const int T = a.T, N = a.N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col0 = blockIdx.x * a.cols;
  const int tiles = a.K / kTileK;
  const uint32_t tileBytes = a.cols * (kTileK * 2) + kXBytes;
  const uint32_t tile0 = (ptx::smem_u32(smemRaw) + 1023u) & ~1023u;  // a tile of weights, then one of activations, `stages` times
  // partial products of the four warps of a column group: [4][kTpDecodeMaxTokens][partRow]
  const int partRow = (a.cols + 15) / 16 * 16;
  float* part = reinterpret_cast<float*>(smemRaw + (tile0 - ptx::smem_u32(smemRaw)) + a.stages * tileBytes);
  // a thread per eight columns of a row of the results
  const int t = threadIdx.x / (kMaxCols / 8), ju = threadIdx.x % (kMaxCols / 8);
  const int col = col0 + ju * 8;
  const bool mine = t < T && ju * 8 < a.cols && col < N;

  if (warp == kWorkers / 32) {
    if (ptx::elect_one()) {
      for (int s = 0; s < a.stages; s++) {
        ptx::mbar_init(&full[s], 1);
        ptx::mbar_init(&empty[s], 4);  // the four warps that work on a tile
      }
      ptx::fence_mbar_init();
      for (int k = 0; k < a.K; k += kBoxK) ptx::tma_prefetch_2d(&tmapW, k, col0);
      for (int k = 0; k < a.K; k += kBoxK) ptx::tma_prefetch_2d(&tmapX, k, 0);
    }
  } else if (mine) {
    if (a.residualIn != nullptr) prefetch_l2(a.residualIn + static_cast<size_t>(t) * N + col);
    if (a.gamma != nullptr && t == 0) prefetch_l2(a.gamma + col);
  }
  __syncthreads();
  // both blocks run before one writes into the other's shared memory (below); under the layer before it costs nothing
  if constexpr (kPair) ptx::cluster_sync_all();
  ptx::grid_dependency_wait();

  uint4 residual = make_uint4(0, 0, 0, 0);
  if (mine && a.residualIn != nullptr) residual = ptx::ld_weak_v4(a.residualIn + static_cast<size_t>(t) * N + col);
  if (warp == kWorkers / 32) {
    if (ptx::elect_one()) {
      int s = 0;
      uint32_t phase = 0;
      for (int k = 0; k < tiles; k++) {
        if (k >= a.stages && !mbarWait(&empty[s], phase ^ 1u, a.status, a.budgetNs, 630)) break;
        ptx::mbar_expect_tx(&full[s], static_cast<uint32_t>(a.cols + T) * (kTileK * 2));
        const uint32_t at = tile0 + s * tileBytes;
        const uint32_t boxBytes = a.cols * (kBoxK * 2), atX = at + 2 * boxBytes;
        ptx::tma_load_2d(at, &tmapW, k * kTileK, col0, &full[s]);
        ptx::tma_load_2d(atX, &tmapX, k * kTileK, 0, &full[s]);
        ptx::tma_load_2d(at + boxBytes, &tmapW, k * kTileK + kBoxK, col0, &full[s]);
        ptx::tma_load_2d(atX + kXBytes / 2, &tmapX, k * kTileK + kBoxK, 0, &full[s]);
        if (++s == a.stages) {
          s = 0;
          phase ^= 1u;
        }
      }
    }
  } else {
    // ---- products. Warp (g, sl): columns [16 g, + 16) and [16 g + 64, + 16) of the slab, tiles sl, sl + 4, ...: the
    // elements [128 sl, + 128) of every 512 of the reduction, the slices of tp_decode.cu, whose sums these are to the bit. The rows of
    // absent columns and tokens hold whatever was there: they reach only their own results, which nobody reads.
    const int g = warp & 3, sl = warp >> 2;
    const int groups = (a.cols + 15) / 16;
    const uint32_t aRow = g * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, aHigh = (lane >> 4) & 1, swz = lane & 7;
    float acc[2][4] = {};
    // The number of stages is a multiple of four or that of the tiles, so that a stage is always this warp's or never: it
    // sees every turn of the barrier. (A warp that met a barrier only every other turn could take the turn before last for the one it waits for.)
    int s = sl;
    uint32_t phase = 0;
    bool healthy = true;
    for (int k = sl; k < tiles; k += 4) {
      // After a wait that ran out the warp only sees the remaining copies land (bounded): the block must not end before they have.
      const bool ok = mbarWait(&full[s], phase, healthy ? a.status : nullptr, healthy ? a.budgetNs : 2000000ull, 620);
      healthy = __all_sync(0xffffffffu, ok) && healthy;
      const uint32_t boxBytes = a.cols * (kBoxK * 2);
#pragma unroll
      for (int box = 0; box < 2; box++) {
        const uint32_t w = tile0 + s * tileBytes + box * boxBytes, x = tile0 + s * tileBytes + 2 * boxBytes + box * (kXBytes / 2);
        uint32_t b[2][4];
#pragma unroll
        for (int half = 0; half < 2; half++) ldmatrix_x4(b[half], x + (lane & 7) * 128 + (((half * 4 + (lane >> 3)) ^ swz) << 4));
#pragma unroll
        for (int j = 0; j < 2; j++) {
          if (g + j * 4 < groups) {
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
              uint32_t af[4];
              ldmatrix_x4(af, w + (aRow + j * 64) * 128 + (((kk * 2 + aHigh) ^ swz) << 4));
              mma_m16n8k16(acc[j], af, b[kk >> 1][(kk & 1) * 2], b[kk >> 1][(kk & 1) * 2 + 1]);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&empty[s]);
      s += 4;
      if (s >= a.stages) {
        s -= a.stages;
        phase ^= 1u;
      }
    }
    // accumulator layout: rows lane / 4 and lane / 4 + 8 (columns of the slab), columns 2 (lane % 4) and + 1 (tokens)
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (g + j * 4 >= groups) break;
      float* dst = part + (sl * kTpDecodeMaxTokens + (lane & 3) * 2) * partRow + (g + j * 4) * 16 + (lane >> 2);
      dst[0] = acc[j][0];
      dst[partRow] = acc[j][1];
      dst[8] = acc[j][2];
      dst[partRow + 8] = acc[j][3];
    }
  }
  __syncthreads();

  // ---- sums, residual, squares
  if (threadIdx.x < kTpDecodeMaxTokens * (kMaxCols / 8)) {
    float ss = 0.f;
    if (mine) {
      float f[8], r[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float* src = part + t * partRow + ju * 8 + j;
        const int slice = kTpDecodeMaxTokens * partRow;
        f[j] = ((src[0] + src[slice]) + src[2 * slice]) + src[3 * slice];  // (in the order of tp_decode.cu)
      }
      // the product rounded to bf16, then the sum with the residual: the roundings of the unfused composition
      uint4 h = Vec16<bf16>::fromFloat(f);
      Vec16<bf16>::toFloat(h, f);
      Vec16<bf16>::toFloat(residual, r);
#pragma unroll
      for (int j = 0; j < 8; j++) f[j] += r[j];
      h = Vec16<bf16>::fromFloat(f);
      Vec16<bf16>::toFloat(h, f);
#pragma unroll
      for (int j = 0; j < 8; j++) ss += f[j] * f[j];
      *reinterpret_cast<uint4*>(a.residualOut + static_cast<size_t>(t) * N + col) = h;
    }
#pragma unroll
    for (int o = kMaxCols / 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (ju == 0 && t < T) a.shares[blockIdx.x * kTpDecodeMaxTokens + t] = ss;
  }
  __syncthreads();
  const int half = kPair ? static_cast<int>(ptx::cluster_ctarank()) : 0;
  if (threadIdx.x == 0) {
    const uint32_t old = ptx::atom_add_acqrel_gpu(a.counted, 1);  // releases what the block has written, cumulatively
    order[half] = old;
    if constexpr (kPair) {
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(ptx::mapa_shared(ptx::smem_u32(&order[half]), half ^ 1)), "r"(old) : "memory");
    }
  }
  __syncthreads();  // (the barrier of the cluster is for whole warps, behind the store to the other block)
  if constexpr (kPair) ptx::cluster_sync_all();
  const bool last = order[0] == gridDim.x - 1 || (kPair && order[1] == gridDim.x - 1);
  if (!last || warp == kWorkers / 32) return;

  // ---- who counted last: every share and all of h are in memory. Short code: only this block runs it, so it comes from L2.
  const int words = N / 8;
  constexpr int kRows = kPair ? kTpDecodeMaxTokens : 2, kWide = kTpDecodeMaxTokens / kRows;  // eight words per thread at a time
  constexpr int kStep = (kPair ? 2 : 1) * kWorkers;
  const int first = half * kWorkers + static_cast<int>(threadIdx.x);
  const uint4* h = reinterpret_cast<const uint4*>(a.residualOut);
  const uint4* gamma = reinterpret_cast<const uint4*>(a.gamma);
  uint4* out = reinterpret_cast<uint4*>(a.out);
  bool summed = false;
#pragma unroll 1
  for (int w0 = first; w0 < words || !summed; w0 += kWide * kStep) {
    uint4 v[kWide][kRows], g[kWide];
#pragma unroll
    for (int c = 0; c < kWide; c++) {
      const int w = w0 + c * kStep;
#pragma unroll
      for (int r = 0; r < kRows; r++) {
        if (w < words && r < T) v[c][r] = ptx::ld_cg_v4(h + r * words + w);
      }
      if (w < words && gamma != nullptr) g[c] = ptx::ld_weak_v4(gamma + w);
    }
    if (!summed) {
      summed = true;
      if (warp < T) {
        float share[kBarrierSlots / 32], sum = 0.f;
#pragma unroll
        for (int i = 0; i < kBarrierSlots / 32; i++) {  // (all requested before the first is looked at: one after the other took 1.7 us)
          share[i] = 0.f;
          if (lane + i * 32 < static_cast<int>(gridDim.x)) share[i] = __ldcg(a.shares + (lane + i * 32) * kTpDecodeMaxTokens + warp);
        }
#pragma unroll
        for (int i = 0; i < kBarrierSlots / 32; i++) sum += share[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) rinv[warp] = rsqrtf(sum / static_cast<float>(N) + a.eps);
      }
      ptx::named_barrier(1, kWorkers);
    }
#pragma unroll
    for (int c = 0; c < kWide; c++) {
      const int w = w0 + c * kStep;
      if (w >= words) break;
      const uint64_t gp[4] = {pairOf(g[c].x), pairOf(g[c].y), pairOf(g[c].z), pairOf(g[c].w)};
#pragma unroll
      for (int r = 0; r < kRows; r++) {
        if (r >= T) break;
        const uint64_t sc = pairOf(rinv[r], rinv[r]);
        const uint4 x = v[c][r];
        uint64_t p[4] = {mulPair(pairOf(x.x), sc), mulPair(pairOf(x.y), sc), mulPair(pairOf(x.z), sc), mulPair(pairOf(x.w), sc)};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) o[j] = packPair(gamma != nullptr ? mulPair(p[j], gp[j]) : p[j]);
        out[r * words + w] = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
  if (first == 0) *a.counted = 0;  // for the next launch
}

}  // namespace

size_t tpDecodeLocalWorkspaceWords() { return 4 + static_cast<size_t>(kBarrierSlots) * kTpDecodeMaxTokens; }

namespace {

int maxBlocks() {
  const int even = gemm::smCount() & ~1;
  return even < kBarrierSlots ? even : kBarrierSlots;
}
int columnsPerBlock(int N) { return ((N + maxBlocks() - 1) / maxBlocks() + 7) / 8 * 8; }

}  // namespace

bool tpDecodeLocalCovers(const TpDecodeArgs& args, const void* workspace) {
  const int T = args.T, N = args.N, K = args.K;
  if (workspace == nullptr || args.comm.world != 1 || args.nvls || args.numCtas != 0 || args.stamps != nullptr) return false;
  const uintptr_t aligned = reinterpret_cast<uintptr_t>(args.w[0]) | reinterpret_cast<uintptr_t>(args.x[0]) | reinterpret_cast<uintptr_t>(args.out) |
                            reinterpret_cast<uintptr_t>(args.residualIn) | reinterpret_cast<uintptr_t>(args.residualOut) |
                            reinterpret_cast<uintptr_t>(args.gamma) | reinterpret_cast<uintptr_t>(workspace);
  if (T < 1 || T > kTpDecodeMaxTokens || N < 8 || N % 8 != 0 || K < 256 || K % 256 != 0 || args.residualOut == nullptr || aligned % 16 != 0) return false;
  return columnsPerBlock(N) <= kMaxCols;
}

cudaError_t launchTpDecodeLocal(const TpDecodeArgs& args, void* workspace, cudaStream_t stream) {
  if (!tpDecodeLocalCovers(args, workspace)) return cudaErrorInvalidValue;
  const int T = args.T, N = args.N, K = args.K;
  DecodeLocalArgs a{args.residualIn, args.residualOut, args.out, args.gamma, static_cast<float*>(workspace) + 4, static_cast<uint32_t*>(workspace),
                    T, N, K, args.eps, 0, 0, args.comm.status, args.comm.timeoutNs};
  a.cols = columnsPerBlock(N);
  int blocks = (N + a.cols - 1) / a.cols;
  const uint32_t tileBytes = static_cast<uint32_t>(a.cols) * kTileK * 2 + kXBytes;
  const int partBytes = 4 * kTpDecodeMaxTokens * ((a.cols + 15) / 16 * 16) * 4;
  a.stages = static_cast<int>((kMaxSmem - 1024 - partBytes) / tileBytes);
  if (a.stages > kMaxTiles) a.stages = kMaxTiles;
  // Tile k and the one that comes after it in a stage belong to the same warps (see the kernel), unless none comes after any.
  a.stages = a.stages >= K / kTileK ? K / kTileK : a.stages & ~3;
  const bool pair = T > 2;
  if (pair) blocks = (blocks + 1) & ~1;  // (the odd one out has no columns: its weights are out of the map's bounds, read as zeros)
  const void* kernel = pair ? reinterpret_cast<const void*>(tpDecodeLocalKernel<true>) : reinterpret_cast<const void*>(tpDecodeLocalKernel<false>);
  CUtensorMap tw, tx;
  cudaError_t e = gemm::makeTensorMapBf16(&tw, args.w[0], N, K, static_cast<uint64_t>(K) * 2, a.cols);
  if (e == cudaSuccess) e = gemm::makeTensorMapBf16(&tx, args.x[0], T, K, static_cast<uint64_t>(K) * 2, T);
  const int smem = static_cast<int>(a.stages * tileBytes) + partBytes + 1024;
  if (e == cudaSuccess) e = gemm::ensureDynamicSmem(kernel, kMaxSmem);
  if (e != cudaSuccess) return e;
  void* params[] = {&tw, &tx, &a};
  return pair ? gemm::launchClusterPair(kernel, dim3(blocks), dim3(kThreads), smem, params, false, stream, true)
              : gemm::launchOverlapped(kernel, dim3(blocks), dim3(kThreads), smem, params, stream);
}

}  // namespace mscclpp
