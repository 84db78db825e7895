// MoE expert-parallel dispatch and combine, one kernel each, over peer memory.
//
// dispatch: every (token, expert) pair of this rank is PUSHED into the hosting rank's receive buffer, directly
//   into its place in an expert-grouped layout (rows of local expert 0 from source ranks 0..n-1, then expert 1,
//   ...), so the grouped expert GEMM can run on the buffer as it is. The sizes are data dependent:
//     A. one pass over topkIdx assigns each pair its position inside its (source rank, expert) group and counts
//        the groups (atomics on 64..256 counters);
//     B. the counts travel to every rank as (value, epoch) pairs - 8-byte stores, no separate flag;
//     C. every block reads the full [rank][expert] count matrix and derives the first row of each of its groups
//        at the destination;
//     D. a block's tokens are cut into pieces of 128 16-byte words, a warp loads a piece once and stores it to the
//        token's top-k destinations (16-byte peer stores); with fp8 = 1 the piece is quantised in registers to e4m3
//        with one scale per 128 elements, which halves the bytes on NVLink.
// combine: the reverse direction is a PULL - the source rank reads the expert outputs of its tokens out of the
//   hosting ranks' buffers (16-byte peer loads), applies the routing weights in fp32 and writes the bf16 result.
//   No staging buffer and no second pass. With fp8 = 1 the expert outputs are e4m3 with 1 x 128 scales (quantised by
//   the expert GEMM's epilogue or by launchMoeQuantizeRows), half the bytes over NVLink.
// With one rank there is nobody to exchange counts with or to wait for: neither launch is cooperative, both overlap the kernel
// before them, and every block of the dispatch counts all pairs by itself (up to 8192 of them). Dispatch and combine together
// on one B200, with the cooperative dispatch / now: 4096 tokens x 4096 bf16, top-2 of 64 experts 51 / 37 us (201 MB, 5.4 TB/s), 777
// tokens x 7168 fp8, top-8 of 256 experts 39 / 27 us.
// With several ranks both end with a cross-rank barrier: after dispatch returns every row sent to this rank has landed; after combine
// returns the peers are done reading this rank's expert outputs.
//
// The reference library has no MoE kernels of its own; its bulk-copy device primitives
// (include/mscclpp/bulk_device.hpp) exist to let users write them.
#include "moe.cuh"

#include <mscclpp/gpu_data_types.hpp>
#include <mscclpp/poll_device.hpp>

#include "gemm.cuh"

namespace mscclpp {

namespace {

using bf16 = __nv_bfloat16;
constexpr int kThreads = 512;
constexpr int kMaxWordsPerLane = 32;  // hidden <= 32 lanes * 32 words * 8 elements = 8192
constexpr int kBatchTokens = 32;      // dispatch: tokens whose destinations are worked out together
constexpr int kPieceWords = 4;        // dispatch: 16-byte words per lane of the piece of a row that a warp moves at a time
static_assert(kBatchTokens * kMoeMaxTopk <= kThreads && kMoeMaxExperts < kThreads && kPieceWords % 2 == 0, "one thread per pair and per expert");

struct Workspace {
  uint32_t* cnt;      // [kMoeMaxExperts] pairs of this rank per expert (zero between launches)
  uint2* matrix;      // [kMaxRanks][kMoeMaxExperts] (count, epoch) written by the source ranks
};

MSCCLPP_DEVICE_INLINE Workspace workspaceOf(const DeviceComm& c, int rank, uint64_t wsOff) {
  Workspace w;
  w.cnt = reinterpret_cast<uint32_t*>(c.peerBase[rank] + wsOff);
  w.matrix = reinterpret_cast<uint2*>(c.peerBase[rank] + wsOff + kMoeMaxExperts * sizeof(uint32_t));
  return w;
}


// Quantises the 8 values of one lane to e4m3 with the scale of its 128-element group (the 16 consecutive lanes that
// hold the group): returns the packed bytes, sets `scale` (the same on all 16 lanes).
MSCCLPP_DEVICE_INLINE uint2 quantizeWordE4m3(const float (&f)[8], float& scale) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(f[i]));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  scale = amax > 0.f ? amax * (1.f / 448.f) : 1.f;
  const float inv = 1.f / scale;
  uint32_t q2[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * i] * inv, f[4 * i + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * i + 2] * inv, f[4 * i + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    q2[i] = lo | (hi << 16);
  }
  return make_uint2(q2[0], q2[1]);
}

// 16 e4m3 bytes -> 16 floats (not yet scaled).
MSCCLPP_DEVICE_INLINE void e4m3x16ToFloat(const uint4& v, float (&f)[16]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w[i] & 0xffffu), __NV_E4M3);
    const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w[i] >> 16), __NV_E4M3);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&lo));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&hi));
    f[4 * i] = a.x;
    f[4 * i + 1] = a.y;
    f[4 * i + 2] = b.x;
    f[4 * i + 3] = b.y;
  }
}

// kOne: one rank and few enough pairs that every block counts them all by itself (moeCountsAlone). No block waits for another
// then, so the launch is not cooperative and overlaps the kernel before it, and the heap's epoch plays no part.
template <bool kOne>
__global__ void __launch_bounds__(kThreads, 1) moeDispatchKernel(MoeDispatchArgs a) {
  const DeviceComm& c = a.comm;
  const int rank = deviceRank(c);
  const int world = kOne ? 1 : c.world;
  uint32_t epoch = 0;
  if constexpr (kOne) ptx::grid_launch_dependents();
  else epoch = launchEpoch(c, rank);
  const uint64_t base = c.peerBase[c.rank];
  const uint64_t local = c.peerBase[rank];
  const uint64_t wsOff = reinterpret_cast<uint64_t>(a.workspace) - base;
  const Workspace ws = workspaceOf(c, rank, wsOff);
  // local operands: addressed through the (emulated) rank's heap base
  const bf16* x = reinterpret_cast<const bf16*>(local + (reinterpret_cast<uint64_t>(a.x) - base));
  const int32_t* topkIdx = reinterpret_cast<const int32_t*>(local + (reinterpret_cast<uint64_t>(a.topkIdx) - base));
  int32_t* slotMap = reinterpret_cast<int32_t*>(local + (reinterpret_cast<uint64_t>(a.slotMap) - base));
  int32_t* recvCounts = reinterpret_cast<int32_t*>(local + (reinterpret_cast<uint64_t>(a.recvCounts) - base));
  const uint64_t recvXOff = reinterpret_cast<uint64_t>(a.recvX) - base;
  const uint64_t recvScalesOff = a.recvScales ? reinterpret_cast<uint64_t>(a.recvScales) - base : 0;
  const uint64_t recvSrcOff = reinterpret_cast<uint64_t>(a.recvSrc) - base;
  const int E = a.numExperts, El = E / world;
  SymmControl* ctl = control(c, rank);

  __shared__ uint32_t counts[kMaxRanks][kMoeMaxExperts];  // [source rank][expert]
  __shared__ uint32_t firstRow[kMoeMaxExperts];           // first destination row of my group of expert e
  __shared__ uint32_t prefix[kMoeMaxExperts + 1];         // rows of the experts before e
  __shared__ uint32_t warpTotal[kThreads / 32];
  __shared__ uint64_t rowAddr[2][kBatchTokens * kMoeMaxTopk];    // destination row of a pair, 0 = none
  __shared__ uint64_t scaleAddr[2][kBatchTokens * kMoeMaxTopk];  // its scales
  __shared__ int overflow;

  // this block's tokens; the rows of the first batch start on their way to L2 now, under the exchange of the counts
  const int words = a.hidden / 8;  // 16-byte words per bf16 row
  const int chunks = (words + 32 * kPieceWords - 1) / (32 * kPieceWords);
  const MoeTokenShare share = moeTokenShare(a.tokens, blockIdx.x, gridDim.x);
  const int tokBegin = share.begin, tokEnd = share.end;
  if (threadIdx.x < kBatchTokens && tokBegin + static_cast<int>(threadIdx.x) < tokEnd)
    ptx::bulk_prefetch_l2(x + static_cast<size_t>(tokBegin + threadIdx.x) * a.hidden, static_cast<uint32_t>(a.hidden) * 2);

  bool healthy = true;
  if constexpr (kOne) {
    // ---- A-C. every expert's pairs before this block's share, in it and behind it
    for (int i = threadIdx.x; i < 3 * kMoeMaxExperts; i += blockDim.x) counts[i / kMoeMaxExperts][i % kMoeMaxExperts] = 0;
    if (threadIdx.x == 0) overflow = 0;
    __syncthreads();
    ptx::grid_dependency_wait();
    const int lo = tokBegin * a.topk, hi = tokEnd * a.topk, pairs = a.tokens * a.topk;
    // All expert ids are requested at once, sixteen per thread, and counted one by one: additions to one word of shared memory take turns, but
    // finding the ids that a warp's lanes have in common first (__match_any_sync) took 7 us for 8192 pairs.
    auto count = [&](int i, int e) {
      if (e >= 0 && e < E) atomicAdd(&counts[static_cast<int>(i >= lo) + static_cast<int>(i >= hi)][e], 1u);
    };
    const bool vectors = (reinterpret_cast<uintptr_t>(topkIdx) & 15) == 0;
    constexpr int kDepth = 4;
    for (int v0 = threadIdx.x; 4 * (v0 - static_cast<int>(threadIdx.x)) < pairs; v0 += kDepth * kThreads) {
      int e[kDepth][4];
#pragma unroll
      for (int k = 0; k < kDepth; k++) {
        const int i = 4 * (v0 + k * kThreads);
        const uint32_t* at = reinterpret_cast<const uint32_t*>(topkIdx) + i;
        if (vectors && i + 3 < pairs) {
          const uint4 v = ptx::ld_weak_v4(at);
          e[k][0] = static_cast<int>(v.x);
          e[k][1] = static_cast<int>(v.y);
          e[k][2] = static_cast<int>(v.z);
          e[k][3] = static_cast<int>(v.w);
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) e[k][j] = i + j < pairs ? static_cast<int>(ptx::ld_weak_u32(at + j)) : -1;
        }
      }
#pragma unroll
      for (int k = 0; k < kDepth; k++) {
#pragma unroll
        for (int j = 0; j < 4; j++) count(4 * (v0 + k * kThreads) + j, e[k][j]);
      }
    }
  } else {
    // ---- A. position of every pair inside its (me, expert) group
    for (int i = tokBegin * a.topk + threadIdx.x; i < tokEnd * a.topk; i += blockDim.x) {
      const int e = topkIdx[i];
      slotMap[i] = (e >= 0 && e < E) ? static_cast<int32_t>(atomicAdd(&ws.cnt[e], 1u)) : -1;
    }
    healthy = gridBarrier(c, rank, &ctl->gridSync[0], gridDim.x);

    // ---- B. block 0 sends my counts to everybody (its own matrix row included), then re-arms the counters
    if (blockIdx.x == 0 && healthy) {
      for (int i = threadIdx.x; i < world * E; i += blockDim.x) {
        const int p = i / E, e = i % E;
        uint2* dst = workspaceOf(c, p, wsOff).matrix + rank * kMoeMaxExperts + e;
        ptx::st_volatile_v2(dst, make_uint2(ws.cnt[e], epoch));
      }
      __syncthreads();
      for (int e = threadIdx.x; e < E; e += blockDim.x) ws.cnt[e] = 0;
    }

    // ---- C. every block collects the whole matrix and derives the first row of each of its groups
    if (threadIdx.x == 0) overflow = 0;
    __syncthreads();
    if (healthy) {
      for (int i = threadIdx.x; i < world * E; i += blockDim.x) {
        const int s = i / E, e = i % E;
        const uint2* src = ws.matrix + s * kMoeMaxExperts + e;
        SpinGuard g(c.status, c.timeoutNs);
        uint2 v = ptx::ld_volatile_v2(src);
        while (v.y != epoch) {
          if (!g.keepSpinning()) {
            g.report(kDevTimeoutFlag, rank, 6000 + s, e, epoch, v.y);
            overflow = 2;
            break;
          }
          v = ptx::ld_volatile_v2(src);
        }
        counts[s][e] = v.x;
      }
    }
  }
  __syncthreads();
  {
    // prefix[e] = rows of all experts before e, over all source ranks (one expert per thread, kMoeMaxExperts <= blockDim.x):
    // a scan of shuffles, where summing up the experts before each one took 4 us with 256 experts on one rank
    const bool known = healthy && overflow == 0;
    const int e = threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t tot = 0, before = 0;
    if (known && e < E) {
      if constexpr (kOne) {
        before = counts[0][e];
        tot = before + counts[1][e] + counts[2][e];
      } else {
        for (int s = 0; s < world; s++) {
          const uint32_t n = counts[s][e];
          if (s < rank) before += n;
          tot += n;
        }
      }
    }
    uint32_t incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) warpTotal[warp] = incl;
    __syncthreads();
    if (e <= E && e <= kMoeMaxExperts) {
      uint32_t base = 0;
      for (int q = 0; q < warp; q++) base += warpTotal[q];
      prefix[e] = base + incl - tot;
    }
    __syncthreads();
    if (known && e < E) {
      const int d = e / El;
      const uint32_t first = prefix[d * El];
      firstRow[e] = prefix[e] - first + before;
      const uint32_t rankTotal = prefix[(d + 1) * El] - first;
      if (rankTotal > static_cast<uint32_t>(a.capacity)) atomicExch(&overflow, 1);
      if (blockIdx.x == 0 && d == rank) {
        recvCounts[e - d * El] = static_cast<int32_t>(tot);
        if (e == d * El) recvCounts[El] = static_cast<int32_t>(rankTotal);
      }
    }
  }
  __syncthreads();
  if (overflow == 1 && blockIdx.x == 0 && threadIdx.x == 0 && c.status != nullptr) {
    // a destination would receive more rows than its buffer holds: nothing is sent, the host sees the error
    SpinGuard g(c.status, c.timeoutNs);
    g.report(kDevErrorCapacity, rank, 6100, 0, static_cast<uint64_t>(a.capacity), 0);
  }
  const bool send = healthy && overflow == 0;

  // ---- D. rows to their destinations. Every block has a contiguous share of the tokens, and their slotMap entries to itself:
  // a block that gave up above may not take back what another one, which got through, is about to read. Destinations of a
  // batch of tokens are worked out by one thread per pair (one reader and writer per entry), then the warps take the
  // (token, piece) units of the batch in turn, with the next unit's loads in flight while the current one is stored.
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  const int scalesPerRow = a.hidden / kMoeScaleGroup;
  const bool wide = (recvXOff & 15) == 0;  // the quantised rows may be stored in 16-byte words
  auto storeWord = [](uint32_t* p, uint32_t v) {
    if constexpr (kOne) *p = v;
    else ptx::st_relaxed_sys(p, v);
  };
  if (send) {
    auto stage = [&](int t0, int n, int buf) {
      const int i = threadIdx.x;
      if (i >= n * a.topk) return;
      const int p = t0 * a.topk + i;
      const int e = topkIdx[p];
      uint64_t row = 0, scales = 0;
      int r = -1;
      if (e >= 0 && e < E) {
        if constexpr (kOne) r = moeDestinationRow(atomicAdd(&firstRow[e], 1u), 0, a.capacity);
        else r = moeDestinationRow(firstRow[e], slotMap[p], a.capacity);  // slotMap holds the position in the group
      }
      slotMap[p] = r;
      if (r >= 0) {
        const uint64_t peer = c.peerBase[e / El];
        row = peer + recvXOff + static_cast<uint64_t>(r) * a.hidden * (a.fp8 ? 1 : 2);
        scales = peer + recvScalesOff + static_cast<uint64_t>(r) * scalesPerRow * 4;
        storeWord(reinterpret_cast<uint32_t*>(peer + recvSrcOff) + r, (static_cast<uint32_t>(rank) << 24) | static_cast<uint32_t>(t0 + i / a.topk));
      }
      rowAddr[buf][i] = row;
      scaleAddr[buf][i] = scales;
    };
    if (tokBegin < tokEnd) stage(tokBegin, min(kBatchTokens, tokEnd - tokBegin), 0);
    int buf = 0;
    for (int t0 = tokBegin; t0 < tokEnd; t0 += kBatchTokens, buf ^= 1) {
      const int n = min(kBatchTokens, tokEnd - t0);
      __syncthreads();
      if (t0 + n < tokEnd) stage(t0 + n, min(kBatchTokens, tokEnd - t0 - n), buf ^ 1);
      const int units = n * chunks;
      uint4 cur[kPieceWords];
      auto load = [&](int u, uint4 (&v)[kPieceWords]) {
        const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(t0 + u / chunks) * a.hidden);
        const int w0 = (u % chunks) * (32 * kPieceWords) + lane;
#pragma unroll
        for (int j = 0; j < kPieceWords; j++) {
          v[j] = make_uint4(0, 0, 0, 0);
          if (w0 + j * 32 < words) v[j] = kOne ? ptx::ld_weak_v4(src + w0 + j * 32) : ptx::ld_input_v4(src + w0 + j * 32);
        }
      };
      if (warp < units) load(warp, cur);
      for (int u = warp; u < units; u += warps) {
        uint4 next[kPieceWords];
        if (u + warps < units) load(u + warps, next);
        const int w0 = (u % chunks) * (32 * kPieceWords);
        const uint64_t* rows = &rowAddr[buf][(u / chunks) * a.topk];
        if (!a.fp8) {
          for (int k = 0; k < a.topk; k++) {
            const uint64_t row = rows[k];
            if (row == 0) continue;
#pragma unroll
            for (int j = 0; j < kPieceWords; j++) {
              const int w = w0 + j * 32 + lane;
              if (w < words) ptx::st_weak_v4(reinterpret_cast<void*>(row + static_cast<uint64_t>(w) * 16), cur[j]);
            }
          }
        } else {
          // 32 lanes x 8 elements = 256 elements per step = two scale groups (lanes 0-15, 16-31)
          uint2 q8[kPieceWords];
          float scale = 0.f;  // lane 2 j + g: the scale of step j's group g
#pragma unroll
          for (int j = 0; j < kPieceWords; j++) {
            float f[8];
            Vec16<bf16>::toFloat(cur[j], f);
            float sc;
            q8[j] = quantizeWordE4m3(f, sc);
            sc = __shfl_sync(0xffffffffu, sc, (lane & 1) * 16);
            if ((lane >> 1) == j) scale = sc;
          }
          // neighbouring lanes swap halves: even lanes end up with 16 bytes of step j, odd lanes with 16 bytes of step j + 1
          uint4 out16[kPieceWords / 2];
#pragma unroll
          for (int j = 0; j < kPieceWords; j += 2) {
            const uint2 give = (lane & 1) ? q8[j] : q8[j + 1];
            const uint32_t gx = __shfl_xor_sync(0xffffffffu, give.x, 1), gy = __shfl_xor_sync(0xffffffffu, give.y, 1);
            out16[j / 2] = (lane & 1) ? make_uint4(gx, gy, q8[j + 1].x, q8[j + 1].y) : make_uint4(q8[j].x, q8[j].y, gx, gy);
          }
          const uint64_t* scaleRows = &scaleAddr[buf][(u / chunks) * a.topk];
          for (int k = 0; k < a.topk; k++) {
            const uint64_t row = rows[k];
            if (row == 0) continue;
            if (wide) {
#pragma unroll
              for (int j = 0; j < kPieceWords; j += 2) {
                const int w = w0 + (j + (lane & 1)) * 32 + (lane & ~1);
                if (w < words) ptx::st_weak_v4(reinterpret_cast<void*>(row + static_cast<uint64_t>(w) * 8), out16[j / 2]);
              }
            } else {
#pragma unroll
              for (int j = 0; j < kPieceWords; j++) {
                const int w = w0 + j * 32 + lane;
                if (w < words) ptx::st_volatile_v2(reinterpret_cast<void*>(row + static_cast<uint64_t>(w) * 8), q8[j]);
              }
            }
            const int sw = w0 / 16 + lane;
            if (lane < 2 * kPieceWords && sw < scalesPerRow)
              storeWord(reinterpret_cast<uint32_t*>(scaleRows[k]) + sw, __float_as_uint(scale));
          }
        }
#pragma unroll
        for (int j = 0; j < kPieceWords; j++) cur[j] = next[j];
      }
    }
  } else {
    for (int i = tokBegin * a.topk + threadIdx.x; i < tokEnd * a.topk; i += blockDim.x) slotMap[i] = -1;
  }
  if constexpr (!kOne) {
    // every row of mine is on its way: after this barrier the rows sent TO me have landed
    if (healthy) rankBarrier(c, rank, 0, blockIdx.x, epoch);
    finishLaunch(c, rank, epoch);
  }
}

// A unit of the combine is 32 x kWords 16-byte words of one token's result (kFp8: of its quantised rows). A warp takes the
// units in turn over the whole grid; the rows of kRows experts are requested together (kWords x kRows = 8 loads per lane
// in flight; launchMoeCombine picks the form), and the expert ids, rows and weights of its next unit while it waits for them (lane k holds the k-th).
// kOne: one rank. There is nobody to wait for: the launch is not cooperative and overlaps the kernel before it.
template <int kWords, int kRows, bool kFp8, bool kOne>
__global__ void __launch_bounds__(kThreads, 1) moeCombineKernel(MoeCombineArgs a) {
  const DeviceComm& c = a.comm;
  const int rank = deviceRank(c);
  const int world = kOne ? 1 : c.world;
  uint32_t epoch = 0;
  if constexpr (kOne) {
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
  } else {
    epoch = launchEpoch(c, rank);
  }
  const uint64_t base = c.peerBase[c.rank];
  const uint64_t local = c.peerBase[rank];
  const int32_t* topkIdx = reinterpret_cast<const int32_t*>(local + (reinterpret_cast<uint64_t>(a.topkIdx) - base));
  const float* weights = reinterpret_cast<const float*>(local + (reinterpret_cast<uint64_t>(a.topkWeights) - base));
  const int32_t* slotMap = reinterpret_cast<const int32_t*>(local + (reinterpret_cast<uint64_t>(a.slotMap) - base));
  bf16* y = reinterpret_cast<bf16*>(local + (reinterpret_cast<uint64_t>(a.y) - base));
  const uint64_t outOff = reinterpret_cast<uint64_t>(a.expertOut) - base;
  const uint64_t scalesOff = kFp8 ? reinterpret_cast<uint64_t>(a.outScales) - base : 0;
  const int scalesPerRow = a.hidden / kMoeScaleGroup;
  const int El = a.numExperts / world;
  constexpr int kElems = kFp8 ? 16 : 8;  // values in a 16-byte word
  const int words = a.hidden / kElems;
  const int chunks = (words + 32 * kWords - 1) / (32 * kWords);
  const int64_t units = static_cast<int64_t>(a.tokens) * chunks;

  // the peers' expert outputs are final once their kernels run
  const bool healthy = kOne || rankBarrier(c, rank, 0, blockIdx.x, epoch);
  const int lane = threadIdx.x & 31;
  const int warpsPerBlock = blockDim.x >> 5;
  const int numWarps = gridDim.x * warpsPerBlock;
  if (healthy) {
    int e = -1, row = -1;
    float wgt = 0.f;
    auto fetch = [&](int64_t u) {  // lane k: the k-th expert of unit u's token
      e = row = -1;
      if (u < units && lane < a.topk) {
        const size_t p = static_cast<size_t>(u / chunks) * a.topk + lane;
        e = topkIdx[p];
        row = slotMap[p];
        wgt = weights[p];
      }
    };
    const int warp = threadIdx.x >> 5;
    const bool roundTheBlocks = kWords == 8 ? a.roundTheBlocks != 0 : units < 3 * static_cast<int64_t>(numWarps);  // (see launchCombine)
    int64_t u = roundTheBlocks ? static_cast<int64_t>(warp) * gridDim.x + blockIdx.x : static_cast<int64_t>(blockIdx.x) * warpsPerBlock + warp;
    fetch(u);
    for (; u < units; u += numWarps) {
      const int t = static_cast<int>(u / chunks);
      const int w0 = static_cast<int>(u % chunks) * (32 * kWords) + lane;
      uint64_t rowBase = 0, scaleBase = 0;  // 0 = this lane's slot is not in use
      const float weight = wgt;
      if (e >= 0 && e < a.numExperts && row >= 0) {
        const uint64_t peer = c.peerBase[e / El];
        rowBase = peer + outOff + static_cast<uint64_t>(row) * a.hidden * (kFp8 ? 1 : 2);
        scaleBase = peer + scalesOff + static_cast<uint64_t>(row) * scalesPerRow * 4;
      }
      fetch(u + numWarps);
      float acc[kWords][kElems];
#pragma unroll
      for (int j = 0; j < kWords; j++) {
#pragma unroll
        for (int i = 0; i < kElems; i++) acc[j][i] = 0.f;
      }
#pragma unroll 1
      for (int k0 = 0; k0 < a.topk; k0 += kRows) {
        uint4 v[kRows][kWords];
        [[maybe_unused]] float sc[kRows][kWords];
        bool used[kRows];
        float wq[kRows];
#pragma unroll
        for (int q = 0; q < kRows; q++) {  // (slots at or beyond topk carry rowBase 0)
          const uint64_t rb = __shfl_sync(0xffffffffu, rowBase, k0 + q);
          [[maybe_unused]] const uint64_t sb = kFp8 ? __shfl_sync(0xffffffffu, scaleBase, k0 + q) : 0;
          wq[q] = __shfl_sync(0xffffffffu, weight, k0 + q);
          used[q] = rb != 0;
#pragma unroll
          for (int j = 0; j < kWords; j++) {
            const int w = w0 + j * 32;
            v[q][j] = make_uint4(0, 0, 0, 0);
            sc[q][j] = 0.f;
            if (used[q] && w < words) {
              v[q][j] = ptx::ld_weak_v4(reinterpret_cast<const void*>(rb + static_cast<uint64_t>(w) * 16));
              if constexpr (kFp8) sc[q][j] = __uint_as_float(ptx::ld_weak_u32(reinterpret_cast<const uint32_t*>(sb) + w / 8));
            }
          }
        }
#pragma unroll
        for (int q = 0; q < kRows; q++) {
          if (!used[q]) continue;
#pragma unroll
          for (int j = 0; j < kWords; j++) {
            float f[kElems];
            float m = wq[q];
            if constexpr (kFp8) {
              // the 8 lanes of a 128-element group share one scale
              e4m3x16ToFloat(v[q][j], f);
              m *= sc[q][j];
            } else {
              Vec16<bf16>::toFloat(v[q][j], f);
            }
#pragma unroll
            for (int i = 0; i < kElems; i++) acc[j][i] += m * f[i];
          }
        }
      }
      uint4* dst = reinterpret_cast<uint4*>(y + static_cast<size_t>(t) * a.hidden);
#pragma unroll
      for (int j = 0; j < kWords; j++) {
        const int w = w0 + j * 32;
        if (w >= words) continue;
#pragma unroll
        for (int h = 0; h < kElems / 8; h++) {
          float part[8];
#pragma unroll
          for (int i = 0; i < 8; i++) part[i] = acc[j][8 * h + i];
          dst[w * (kElems / 8) + h] = Vec16<bf16>::fromFloat(part);
        }
      }
    }
  }
  if constexpr (!kOne) {
    // my reads are done: the peers may overwrite their expert outputs after this
    if (healthy) rankBarrier(c, rank, 1, blockIdx.x, epoch);
    finishLaunch(c, rank, epoch);
  }
}

// One warp per row: the dispatch's quantiser as a stand-alone pass (for expert outputs that are to be combined as fp8).
__global__ void __launch_bounds__(kThreads) moeQuantizeRowsKernel(const bf16* x, uint8_t* q, float* scales, int rows, int hidden) {
  const int lane = threadIdx.x & 31;
  const int warpsPerBlock = blockDim.x >> 5;
  const int words = hidden / 8;
  const int scalesPerRow = hidden / kMoeScaleGroup;
  for (int r = blockIdx.x * warpsPerBlock + (threadIdx.x >> 5); r < rows; r += gridDim.x * warpsPerBlock) {
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(r) * hidden);
#pragma unroll 1
    for (int w0 = 0; w0 < words; w0 += 32 * 8) {
      uint4 v[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int w = w0 + j * 32 + lane;
        v[j] = w < words ? src[w] : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int w = w0 + j * 32 + lane;
        float f[8];
        Vec16<bf16>::toFloat(v[j], f);
        float scale;
        const uint2 packed = quantizeWordE4m3(f, scale);
        if (w < words) {
          *reinterpret_cast<uint2*>(q + static_cast<size_t>(r) * hidden + static_cast<size_t>(w) * 8) = packed;
          if ((lane & 15) == 0) scales[static_cast<size_t>(r) * scalesPerRow + w / 16] = scale;
        }
      }
    }
  }
}

template <typename Kernel, typename Args>
cudaError_t launchCoop(Kernel kernel, const Args& args, int nBlocks, int emu, cudaStream_t stream) {
  dim3 grid(nBlocks, emu > 1 ? emu : 1, 1);
  dim3 block(kThreads, 1, 1);
  Args copy = args;
  void* params[] = {&copy};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), grid, block, params, 0, stream);
}

template <int kWords, int kRows, bool kFp8>
cudaError_t launchCombine(const MoeCombineArgs& args, int nBlocks, int emu, cudaStream_t stream) {
  MoeCombineArgs copy = args;
  const int words = args.hidden / (kFp8 ? 16 : 8);
  const int64_t units = static_cast<int64_t>(args.tokens) * ((words + 32 * kWords - 1) / (32 * kWords)), warps = static_cast<int64_t>(nBlocks) * (kThreads / 32);
  // With few rounds the units go round the blocks first: those of the last round, when not every warp has one, are spread over all SMs. With
  // more, neighbouring warps take neighbouring pieces of a row. One B200, dispatch and combine, us in neighbouring pieces / round the
  // blocks: 4096 bf16, top-2 (long pieces), 1.7 rounds 17.8 / 17.2, 2.0 23.1 / 22.4, 2.2 24.2 / 23.3, 2.4 25.7 / 26.0, 2.6 27.7 / 28.8, 2.8 29.6 / 30.8;
  // 8192 bf16, top-2, and 4096, top-1, cross at the same place: two or fewer rows leave little else to do than to read pieces in order.
  // 7168 fp8, top-8, 2.2 rounds 25.8 / 24.5, 2.6 27.5 / 27.1, 3.0 63.2 / 63.1, 3.5 46.9 / 46.9; top-4 2.8 rounds 20.1 / 18.9; 4096 bf16, top-4, 2.6
  // rounds 55.1 / 54.5, top-8 93.0 / 91.8; eight emulated ranks within 1 % but for 4096 fp8, top-8, 2.1 rounds 42.7 / 40.7.
  // (The kernel compares with three rounds itself; only the long pieces, whose line depends on topk, are told. Two strides in place of the flag
  // cost 0.4 % at 4096 tokens, the flag in all forms 1 % at 777 x 7168 fp8.)
  copy.roundTheBlocks = args.topk <= 2 ? 3 * units < 7 * warps : units < 3 * warps;
  if (args.comm.world > 1) return launchCoop(moeCombineKernel<kWords, kRows, kFp8, false>, copy, nBlocks, emu, stream);
  void* params[] = {&copy};
  return gemm::launchOverlapped(reinterpret_cast<const void*>(moeCombineKernel<kWords, kRows, kFp8, true>), dim3(nBlocks), dim3(kThreads), 0, params, stream);
}

int defaultBlocks(int emu, int world) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) (void)cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int n = sms / (emu > 1 ? emu : 1);
  // several GPUs: bound by NVLink, 64 blocks keep several MB in flight. One rank: bound by HBM, which takes every SM
  if (world > 1 && n > 64) n = 64;
  return n < 1 ? 1 : n;
}

bool validCommon(const DeviceComm& c, int tokens, int hidden, int topk, int numExperts, int emu) {
  if (tokens < 0 || tokens >= (1 << 24) || hidden <= 0 || hidden % 256 != 0 || hidden > 32 * kMaxWordsPerLane * 8) return false;
  if (topk < 1 || topk > kMoeMaxTopk || numExperts < c.world || numExperts > kMoeMaxExperts || numExperts % c.world != 0) return false;
  if (emu > 1 && emu != c.world) return false;
  return true;
}

}  // namespace

cudaError_t launchMoeDispatch(const MoeDispatchArgs& args, int nBlocks, cudaStream_t stream) {
  const int emu = args.emuRanks > 1 ? args.emuRanks : 1;
  if (!validCommon(args.comm, args.tokens, args.hidden, args.topk, args.numExperts, emu)) return cudaErrorInvalidValue;
  if (args.capacity <= 0 || (args.fp8 && args.recvScales == nullptr)) return cudaErrorInvalidValue;
  if (nBlocks <= 0) nBlocks = defaultBlocks(emu, args.comm.world);
  if (nBlocks > kBarrierSlots) return cudaErrorInvalidValue;
  if (!moeCountsAlone(args.comm.world, args.tokens, args.topk)) return launchCoop(moeDispatchKernel<false>, args, nBlocks, emu, stream);
  MoeDispatchArgs copy = args;
  void* params[] = {&copy};
  return gemm::launchOverlapped(reinterpret_cast<const void*>(moeDispatchKernel<true>), dim3(nBlocks), dim3(kThreads), 0, params, stream);
}

cudaError_t launchMoeQuantizeRows(const __nv_bfloat16* x, void* q, float* scales, int rows, int hidden, cudaStream_t stream) {
  if (rows < 0 || hidden <= 0 || hidden % 256 != 0) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  const int warpsPerBlock = kThreads / 32;
  int blocks = (rows + warpsPerBlock - 1) / warpsPerBlock;
  if (blocks > 148 * 4) blocks = 148 * 4;
  moeQuantizeRowsKernel<<<blocks, kThreads, 0, stream>>>(x, static_cast<uint8_t*>(q), scales, rows, hidden);
  return cudaGetLastError();
}

cudaError_t launchMoeCombine(const MoeCombineArgs& args, int nBlocks, cudaStream_t stream) {
  const int emu = args.emuRanks > 1 ? args.emuRanks : 1;
  if (!validCommon(args.comm, args.tokens, args.hidden, args.topk, args.numExperts, emu)) return cudaErrorInvalidValue;
  if (args.fp8 && args.outScales == nullptr) return cudaErrorInvalidValue;
  if (nBlocks <= 0) nBlocks = defaultBlocks(emu, args.comm.world);
  if (nBlocks > kBarrierSlots) return cudaErrorInvalidValue;
  // How much of a row a warp takes at a time. Long pieces of one or two rows stream best: a word costs about a fifth more in
  // the next shorter form. They leave warps idle where there are few of them, or where most warps have no unit in the last
  // round. The form is the one with the smallest product of that cost and the busiest warp's words (units x words per unit).
  // One B200, eight ranks, microseconds by form (words x rows):
  //   256 tokens x 8192 bf16, top-8: 8x1 56, 4x2 63, 2x4 65, 1x8 90;  2048 tokens, top-1: 102, 116, 176, 338
  //   256 tokens x 7168 fp8, top-8: 8x1 70 (no registers left for loads), 4x2 42, 2x4 44, 1x8 49
  //   86 tokens x 8192 fp8, top-4 (1.2 units of four words per warp): 4x2 21.8, 2x4 20.9;  115 x 1024, top-8: 18.4, 16.2, 1x8 13.6
  // Forms of more rows than there are experts per token only keep fewer loads in flight.
  const int words = args.hidden / (args.fp8 ? 16 : 8);
  const int64_t warps = static_cast<int64_t>(nBlocks) * (kThreads / 32);
  auto cost = [&](int wordsPerLane) {
    const int64_t units = static_cast<int64_t>(args.tokens) * ((words + 32 * wordsPerLane - 1) / (32 * wordsPerLane));
    const int perWord = wordsPerLane == 8 ? 100 : (wordsPerLane == 4 ? 120 : (wordsPerLane == 2 ? 135 : 165));
    return (units + warps - 1) / warps * wordsPerLane * perWord;
  };
  int form = args.fp8 ? 4 : 8;
  const int shortest = args.topk <= 2 ? 4 : (args.topk <= 4 ? 2 : 1);
  for (int w = form / 2; w >= shortest; w /= 2) {
    if (cost(w) < cost(form)) form = w;
  }
  switch (form) {
    case 8:
      return launchCombine<8, 1, false>(args, nBlocks, emu, stream);
    case 4:
      return args.fp8 ? launchCombine<4, 2, true>(args, nBlocks, emu, stream)
                      : launchCombine<4, 2, false>(args, nBlocks, emu, stream);
    case 2:
      return args.fp8 ? launchCombine<2, 4, true>(args, nBlocks, emu, stream)
                      : launchCombine<2, 4, false>(args, nBlocks, emu, stream);
    default:
      return args.fp8 ? launchCombine<1, 8, true>(args, nBlocks, emu, stream)
                      : launchCombine<1, 8, false>(args, nBlocks, emu, stream);
  }
}

}  // namespace mscclpp
