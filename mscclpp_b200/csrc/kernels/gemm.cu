// Plain bf16 GEMM on tcgen05/TMEM (see gemm_sm100.cuh for the kernel body) and tensor-map helpers.
#include "gemm.cuh"

#include <atomic>
#include <cmath>
#include <map>
#include <mutex>
#include <set>
#include <tuple>
#include <utility>

#include "gemm2_sm100.cuh"
#include "gemm_sm100.cuh"

namespace mscclpp {
namespace gemm {

namespace {

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encodeFn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeFn>(p);
    }
  });
  return fn;
}

template <int kBlockN, int kSplit>
__global__ void __launch_bounds__(kNumThreads, 1)
    gemmBf16Kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB,
                   const __grid_constant__ CUtensorMap tmapD, Shape shape, DeviceStatus* status, uint64_t budgetNs) {
  extern __shared__ uint8_t smemRaw[];
  NoGate gate;
  StoreBf16 epi{&tmapD, shape.M, shape.N};
  if (threadIdx.x == 0) ptx::tma_prefetch_desc(&tmapD);
  gemmCta<kBlockN, NoGate, StoreBf16, kSplit>(&tmapA, &tmapB, shape, blockIdx.x / kSplit, gridDim.x / kSplit, gate, epi, status, budgetNs, smemRaw);
}

template <int kBlockN, int kSplit = 1>
cudaError_t launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, Shape shape, int numCtas,
                   DeviceStatus* status, cudaStream_t stream, uint64_t budgetNs) {
  using Cfg = Config<kBlockN, kSplit>;
  const void* kernel = reinterpret_cast<const void*>(gemmBf16Kernel<kBlockN, kSplit>);
  cudaError_t e = ensureDynamicSmem(kernel, Cfg::kSmemBytes);
  if (e != cudaSuccess) return e;
  const int tiles = ((shape.M + kBlockM - 1) / kBlockM) * ((shape.N + kBlockN - 1) / kBlockN);
  int grid = numCtas > 0 ? numCtas : smCount();
  if (grid > tiles) grid = tiles;
  void* params[] = {const_cast<CUtensorMap*>(&ta), const_cast<CUtensorMap*>(&tb), const_cast<CUtensorMap*>(&td), &shape, &status, &budgetNs};
  if constexpr (kSplit > 1) return launchClusters(kernel, kSplit, dim3(tiles * kSplit), dim3(kNumThreads), Cfg::kSmemBytes, params, false, stream, true);
  return launchOverlapped(kernel, dim3(grid), dim3(kNumThreads), Cfg::kSmemBytes, params, stream);
}

template <typename Cfg>
__global__ void __launch_bounds__(kNumThreads, 1)
    gemmBf16PairKernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB,
                       const __grid_constant__ CUtensorMap tmapD, Shape shape, DeviceStatus* status, uint64_t budgetNs) {
  extern __shared__ uint8_t smemRaw[];
  NoGate gate;
  StoreBf16 epi{&tmapD, shape.M, shape.N};
  if (threadIdx.x == 0) ptx::tma_prefetch_desc(&tmapD);
  gemmCtaPair<Cfg>(&tmapA, &tmapB, shape, blockIdx.x / 2, gridDim.x / 2, gate, epi, status, budgetNs, smemRaw);
}

// Tile order of a plain GEMM: bands of `band` row blocks (0 = the default for the tile shape, < 0 = plain column-major walk).
void setBandOrder(Shape& shape, int numMBlk, int band, int dflt) {
  if (band == 0) band = dflt;
  if (band > 0 && numMBlk > band) {
    shape.mOrder = 3;
    shape.mOrderParam = band;
  }
}

}  // namespace

cudaError_t ensureDynamicSmem(const void* kernel, int bytes) {
  // the attribute belongs to the (kernel, device) pair: a process that drives several GPUs sets it on each of them
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({kernel, dev})) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.insert({kernel, dev});
  return e;
}

int residentClusters(const void* kernel, int ctas, int nThreads, int smemBytes) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, int, int, int>, int> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(kernel, dev, ctas, nThreads, smemBytes);
  const auto it = known.find(key);
  if (it != known.end()) return it->second;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(nThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smemBytes);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = static_cast<unsigned>(ctas);
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  known[key] = n;
  return n;
}

cudaError_t launchClusters(const void* kernel, int ctas, dim3 grid, dim3 block, size_t smemBytes, void** params, bool cooperative,
                           cudaStream_t stream, bool overlapped) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = static_cast<unsigned>(ctas);
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 1;
  if (cooperative) {
    attrs[cfg.numAttrs].id = cudaLaunchAttributeCooperative;
    attrs[cfg.numAttrs++].val.cooperative = 1;
  } else if (overlapped) {
    attrs[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  return cudaLaunchKernelExC(&cfg, kernel, params);
}

cudaError_t launchClusterPair(const void* kernel, dim3 grid, dim3 block, size_t smemBytes, void** params, bool cooperative,
                              cudaStream_t stream, bool overlapped) {
  return launchClusters(kernel, 2, grid, block, smemBytes, params, cooperative, stream, overlapped);
}

cudaError_t launchOverlapped(const void* kernel, dim3 grid, dim3 block, size_t smemBytes, void** params, cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, kernel, params);
}

namespace {

bool validGemm(const void* D, int M, int N, int K, int ldd) {
  return M > 0 && N > 0 && K > 0 && K % kBlockK == 0 && ldd % 8 == 0 && (reinterpret_cast<uintptr_t>(D) & 15) == 0;
}

template <typename Cfg>
cudaError_t launchPair(const void* A, const void* B, void* D, int M, int N, int K, int ldd, int numCtas, DeviceStatus* status, cudaStream_t stream,
                       int probe, int band, uint64_t budgetNs) {
  Shape shape{M, N, K, Cfg::kRows, 0, 0, 0, probe};
  const int rowBlocks = (M + Cfg::kPairM - 1) / Cfg::kPairM;
  setBandOrder(shape, rowBlocks, band, 2048 / Cfg::kPairM);
  CUtensorMap ta, tb, td;
  cudaError_t e = makeTensorMapBf16(&ta, A, M, K, static_cast<uint64_t>(K) * 2, Cfg::kRows);
  if (e != cudaSuccess) return e;
  e = makeTensorMapBf16(&tb, B, N, K, static_cast<uint64_t>(K) * 2, Cfg::kBlockN / 2);
  if (e != cudaSuccess) return e;
  e = makeTensorMapBf16(&td, D, M, N, static_cast<uint64_t>(ldd) * 2, 32);
  if (e != cudaSuccess) return e;
  const void* kernel = reinterpret_cast<const void*>(gemmBf16PairKernel<Cfg>);
  e = ensureDynamicSmem(kernel, Cfg::kSmemBytes);
  if (e != cudaSuccess) return e;
  const int tiles = rowBlocks * ((N + Cfg::kBlockN - 1) / Cfg::kBlockN);
  int grid = numCtas > 0 ? numCtas : smCount();
  grid &= ~1;
  if (grid > 2 * tiles) grid = 2 * tiles;
  if (grid < 2) grid = 2;
  void* params[] = {&ta, &tb, &td, &shape, &status, &budgetNs};
  return launchClusterPair(kernel, dim3(grid), dim3(kNumThreads), Cfg::kSmemBytes, params, false, stream, true);
}

}  // namespace

cudaError_t gemmBf16TwoSm(const void* A, const void* B, void* D, int M, int N, int K, int ldd, int numCtas, DeviceStatus* status,
                          cudaStream_t stream, int probe, int band, uint64_t budgetNs) {
  if (!validGemm(D, M, N, K, ldd) || N % Config2::kBlockN != 0) return cudaErrorInvalidValue;
  return launchPair<Config2>(A, B, D, M, N, K, ldd, numCtas, status, stream, probe, band, budgetNs);
}

int smCount() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

cudaError_t makeTensorMapBf16(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint64_t rowStrideBytes,
                              uint32_t boxRows) {
  EncodeFn fn = encodeFn();
  if (fn == nullptr) return cudaErrorNotSupported;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || (rowStrideBytes & 15) != 0) return cudaErrorInvalidValue;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {rowStrideBytes};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(kBlockK), boxRows};
  cuuint32_t elemStrides[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elemStrides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

namespace {

template <int kBlockN, int kSplit = 1>
cudaError_t launchOne(const void* A, const void* B, void* D, int M, int N, int K, int ldd, int numCtas, DeviceStatus* status, cudaStream_t stream,
                      int probe, int band, uint64_t budgetNs) {
  Shape shape{M, N, K, M < kBlockM ? M : kBlockM, 0, 0, 0, probe};
  setBandOrder(shape, (M + kBlockM - 1) / kBlockM, band, 16);
  CUtensorMap ta, tb, td;
  cudaError_t e = makeTensorMapBf16(&ta, A, M, K, static_cast<uint64_t>(K) * 2, shape.aBoxRows);
  if (e == cudaSuccess) e = makeTensorMapBf16(&tb, B, N, K, static_cast<uint64_t>(K) * 2, kBlockN);
  if (e == cudaSuccess) e = makeTensorMapBf16(&td, D, M, N, static_cast<uint64_t>(ldd) * 2, 32);  // 64-column x 32-row boxes of the output
  if (e != cudaSuccess) return e;
  return launch<kBlockN, kSplit>(ta, tb, td, shape, numCtas, status, stream, budgetNs);
}

}  // namespace

cudaError_t gemmBf16(const void* A, const void* B, void* D, int M, int N, int K, int ldd, int blockN, int numCtas,
                     DeviceStatus* status, cudaStream_t stream, int probe, int band, uint64_t budgetNs) {
  if ((blockN != 64 && blockN != 128 && blockN != 256) || !validGemm(D, M, N, K, ldd) || N % blockN != 0) return cudaErrorInvalidValue;
  switch (blockN) {
    case 64:
      return launchOne<64>(A, B, D, M, N, K, ldd, numCtas, status, stream, probe, band, budgetNs);
    case 128:
      return launchOne<128>(A, B, D, M, N, K, ldd, numCtas, status, stream, probe, band, budgetNs);
    default:
      return launchOne<256>(A, B, D, M, N, K, ldd, numCtas, status, stream, probe, band, budgetNs);
  }
}

namespace {

// What a form costs: `fixed` us (launch, first loads, last stores), its k blocks one after the other, and `wave` us for every further wave
// of tiles (their epilogues and the ragged end; a cluster's start). A k block takes what its issue costs, `block` us, or its
// bytes at the rate of an SM's input, whichever is longer.
struct Cost {
  Form form;
  float fixed, block, wave;
};
struct Rates {
  float sm, all, memory;  // KB per us into one SM and into all of them, and TB/s of the memory
};

// Clusters of four of the split form that run at the same time: they leave SMs over in the groups that they may not leave (34 of 148 SMs on a
// B200, where 37 would have them).
int clustersOfFour() {
  static std::atomic<int> known[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return smCount() / 4 - 3;
  int n = known[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    const void* kernel = reinterpret_cast<const void*>(gemmBf16Kernel<64, 4>);
    constexpr int kSmemBytes = Config<64, 4>::kSmemBytes;
    if (ensureDynamicSmem(kernel, kSmemBytes) != cudaSuccess) return 0;
    n = residentClusters(kernel, 4, kNumThreads, kSmemBytes);
    known[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// 0: nothing of this form fits the device.
float timeOf(const Cost& c, const Rates& rates, int M, int N, int K, int sms, int fours) {
  const int tileM = c.form.pairM != 0 ? c.form.pairM : kBlockM, ctas = c.form.pairM != 0 ? 2 : c.form.split;
  const int64_t tiles = static_cast<int64_t>((M + tileM - 1) / tileM) * ((N + c.form.blockN - 1) / c.form.blockN);
  const int slots = ctas == 4 ? fours : sms / ctas;
  if (slots < 1) return 0.f;
  const int64_t waves = (tiles + slots - 1) / slots;
  const float active = static_cast<float>((tiles < slots ? tiles : slots) * ctas);
  const float kb = static_cast<float>((M < tileM ? M : tileM) + c.form.blockN) * (2 * kBlockK) / 1000.f / (c.form.pairM != 0 ? 2 : 1);
  const float rate = rates.all / active < rates.sm ? rates.all / active : rates.sm;
  const float block = kb / rate > c.block ? kb / rate : c.block;
  const int blocks = (K / kBlockK + c.form.split - 1) / c.form.split;
  return static_cast<float>(waves) * blocks * block + static_cast<float>(waves - 1) * c.wave;
}

}  // namespace

// The form whose time by the model above is the least: `fixed` and the fourth root of the sum of the fourth powers of the k blocks' time and
// of the operands' and the result's at the rate of the memory. The constants are a fit to all forms on 140 shapes drawn from M 9-8192, N
// 512-8192, K 256-8192 (one B200, graph replay, operands of three calls in turn). The model is within 6.3 % (rms); what it picks is
// 0.6 % slower than the best form (geometric mean; at worst 14 %), where the rule before it - 256 x 256 pairs if there are 74, else
// the widest one-SM tile of which N is a multiple and there are 120 - lost 16 % on the same kernels (at worst 2.2 times).
// gemm_bf16, us before / now: 80 x 1408 x 4992 17.4 / 8.5, 645 x 704 x 6144 21.1 / 12.0, 840 x 5696 x 1600 27.9 / 20.5, 333 x 6144 x 4096
// 23.7 / 22.0, 5510 x 1728 x 640 23.4 / 15.6, 2233 x 6592 x 4160 184 / 107; shapes of up to 8.4 us wait for the host either way.
// Split over clusters of two, tiles of 128 or 256 columns split over 2, 4 or 8: never more than 3 % ahead.
Form planForm(int M, int N, int K, int sms, int fours) {
  static constexpr Cost kCosts[] = {
      {{256, 256, 1}, 3.99f, 0.299f, 1.05f}, {{128, 256, 1}, 3.54f, 0.154f, 0.84f}, {{128, 128, 1}, 3.00f, 0.093f, 0.60f}, {{0, 64, 1}, 2.65f, 0.145f, 0.25f},
      {{0, 128, 1}, 2.94f, 0.182f, 0.62f},   {{0, 256, 1}, 3.65f, 0.274f, 1.50f},   {{0, 64, 4}, 4.34f, 0.134f, 4.70f},
  };
  static constexpr Rates kRates = {147.f, 21100.f, 5.4f};
  const float memory = 2e-6f / kRates.memory * (static_cast<float>(M) * K + static_cast<float>(N) * K + static_cast<float>(M) * N);
  const float memory2 = memory * memory;
  if (sms <= 0) sms = smCount(), fours = clustersOfFour();
  Form best{0, 64, 1};
  float least = 0.f;
  for (const Cost& c : kCosts) {
    if (K / kBlockK < c.form.split) continue;
    const float loop = timeOf(c, kRates, M, N, K, sms, fours), loop2 = loop * loop;
    if (loop == 0.f) continue;
    const float t = c.fixed + sqrtf(sqrtf(loop2 * loop2 + memory2 * memory2));
    if (least == 0.f || t < least) {
      least = t;
      best = c.form;
    }
  }
  return best;
}

// Here the pairs of SMs are always ahead, for their epilogue (ResidualSumsqRows). Same model with squares; fitted to 60 shapes drawn from M
// 9-8192, N 1024-8192, K 256-2048 (with the scale pass behind them): within 3.8 %, the pick 0.1 % slower than the best form, at worst
// 4 %. Both launches, us by the rule before (one-SM tiles below 64 pairs or 256 rows) / now: 61 x 7680 x 1536 11.3 / 10.0,
// 66 x 4352 x 1024 9.3 / 8.0, 128 x 8192 x 1024 11.5 / 10.3, 185 x 6144 x 1600 17.0 / 13.1, 596 x 2816 x 320 11.9 / 9.5.
Form planLayerForm(int M, int N, int K, int sms) {
  static constexpr Cost kCosts[] = {{{256, 256, 1}, 4.2f, 0.31f, 0.05f}, {{128, 256, 1}, 3.65f, 0.092f, 1.f}, {{128, 128, 1}, 3.2f, 0.07f, 1.f}};
  static constexpr Rates kRates = {162.f, 24000.f, 7.8f};
  const float memory = 2e-6f / kRates.memory * (static_cast<float>(M) * K + static_cast<float>(N) * K + 2.f * static_cast<float>(M) * N);
  if (sms <= 0) sms = smCount();
  Form best{0, 64, 1};  // where N is no multiple of 128
  float least = 0.f;
  for (const Cost& c : kCosts) {
    if (N % c.form.blockN != 0 || (c.form.pairM == 256 && M < 256)) continue;
    const float loop = timeOf(c, kRates, M, N, K, sms, 0);
    if (loop == 0.f) continue;
    const float t = c.fixed + sqrtf(loop * loop + memory * memory);
    if (least == 0.f || t < least) {
      least = t;
      best = c.form;
    }
  }
  return best;
}

cudaError_t gemmBf16Form(const void* A, const void* B, void* D, int M, int N, int K, int ldd, Form form, DeviceStatus* status, cudaStream_t stream,
                         uint64_t budgetNs) {
  if (!validGemm(D, M, N, K, ldd) || N % 64 != 0 || form.split > K / kBlockK) return cudaErrorInvalidValue;
  switch (form.pairM * 1000000 + form.blockN * 1000 + form.split) {
    case 64001:
      return launchOne<64>(A, B, D, M, N, K, ldd, 0, status, stream, 0, 0, budgetNs);
    case 64004:
      return launchOne<64, 4>(A, B, D, M, N, K, ldd, 0, status, stream, 0, 0, budgetNs);
    case 128001:
      return launchOne<128>(A, B, D, M, N, K, ldd, 0, status, stream, 0, 0, budgetNs);
    case 256001:
      return launchOne<256>(A, B, D, M, N, K, ldd, 0, status, stream, 0, 0, budgetNs);
    case 256256001:
      return launchPair<Config2>(A, B, D, M, N, K, ldd, 0, status, stream, 0, 0, budgetNs);
    case 128256001:
      return launchPair<Config2Flat256>(A, B, D, M, N, K, ldd, 0, status, stream, 0, 0, budgetNs);
    case 128128001:
      return launchPair<Config2Flat128>(A, B, D, M, N, K, ldd, 0, status, stream, 0, 0, budgetNs);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace gemm
}  // namespace mscclpp
