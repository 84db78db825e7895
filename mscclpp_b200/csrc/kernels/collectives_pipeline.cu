// Allreduce for buffers that are NOT in the symmetric heap (ordinary cudaMalloc / framework tensors), in ONE kernel.
//
// Peers cannot address such buffers, so the data takes a detour through heap scratch; what matters is that the three
// legs overlap instead of running as copy-in -> collective -> copy-out launches. Every thread block owns one slice
// (sliceBytes) of each "round" of the message and runs, per round,
//
//   1. copy-in     user input  -> its slice of the local scratch-in            (local stores)
//   2. barrier A   with the blocks of the same index on every rank            (all slices of this index are staged)
//   3. reduce      this rank's 1/world of the slice: multimem.ld_reduce through the NVSwitch, result to EVERY rank's scratch-out
//                  (multimem.st), or peer loads with an fp32 accumulator, result to every rank's scratch-out (peer stores) or, see
//                  pipelineFetches, to its own
//   4. barrier B   (every rank's part of the slice is reduced)
//   5. copy-out    scratch-out -> user output: the local one, or each part from the rank that has reduced it
//
// The barriers are split into a signal and a wait, and the copy-in of round r + 1 (with its signal) sits between round r's
// reduction and its wait for barrier B, so a block copies while its peers reduce. Blocks never wait for other blocks of
// their own rank, so while one block sits in a barrier the others copy and reduce as well: with a few blocks per SM the
// NVLink transfers, the local copies and the barrier latencies overlap. Scratch is double buffered per block (round
// parity), which is what makes two barriers per round enough.
// With all ranks on one GPU (four ranks, 32 MB bf16 each, one B200): 256 MB are stored and 320 MB read, the detour included, in 97-118 us on different
// boxes, 4.9-5.9 TB/s together; a plain copy reads and writes 8.1 TB/s of 32 MB (inside L2) and 6.4 of 256 MB. A round costs 9-10 us however
// little it moves - slices of 32 KB, 14 rounds 177 us, 48 KB, 10 rounds 138, 64 KB, 7 rounds 111, 96 KB, 5 rounds 106 on one box: its two waits and the
// round trips on either side of them, which only the SM's other block covers. So with slices that fill the scratch neither the bytes nor
// the waits alone bound it. On one box each, us: reduced parts stored to every peer's scratch 110, to the own one and fetched from there 100; both
// changes together, with 5 rounds instead of 7, 106 -> 99 and 107 -> 102; a rank's own part through the scratch as well 121; one copy load in
// flight per thread, system-scope accesses, the barriers unsplit and 16 blocks per rank instead of the 74 that fit 629. Tried instead: a warp
// for each copy and the others reducing, with three flags a round, 139; all three legs in one step with a single barrier 119; evict-first and
// evict-last accesses, which take a third of the DRAM writes away (265 -> 182 MB), 1 %.
// One round that covers the whole message is the un-pipelined "reduce-scatter + all-gather through scratch" form.
//
// Role of the reference's allreduce_nvls_block_pipeline.cu:16-147 / allreduce_nvls_warp_pipeline.cu:14-112 (NVLS) and
// allreduce_rsag_pipeline.cu:85-221 / allreduce_rsag.cu:33-128 (peer loads). Those specialise warps or blocks per leg
// and chain them with device semaphores; here every block runs all legs on its own slice and the overlap comes from
// the blocks being out of step with one another.
#include "collectives.cuh"

#include <type_traits>

namespace mscclpp {

namespace {

// Barrier words of this kernel live in the aux flag region behind those of the fused tensor-parallel kernels:
// u64 flags[2 phases][kBarrierSlots][kMaxRanks], value = (launch epoch << 32) | round + 1.
constexpr uint64_t kPipeFlagByteOffset = (4096ull * (kMaxRanks + 1) + 4096ull) * 4ull;
static_assert(kPipeFlagByteOffset % 8 == 0, "u64 flags");
static_assert(kPipeFlagByteOffset + 2ull * kBarrierSlots * kMaxRanks * 8ull <= kAuxFlagBytes, "aux flag region too small");

MSCCLPP_DEVICE_INLINE uint64_t* pipeFlag(const DeviceComm& c, int owner, int phase, int slot, int src) {
  return reinterpret_cast<uint64_t*>(c.peerBase[owner] + c.auxFlagsOff + kPipeFlagByteOffset) +
         ((static_cast<uint64_t>(phase) * kBarrierSlots + slot) * kMaxRanks + src);
}

// The two halves of a barrier with the blocks of the same slot on every rank; all threads of the block call both. What the
// block stored before pipeSignal is visible to a peer's block of this slot after its pipeWait for the same token. As in
// rankBarrier, one fence and a relaxed flag store publish, and one acquire follows relaxed polls.
MSCCLPP_DEVICE_INLINE void pipeSignal(const DeviceComm& c, int rank, int phase, int slot, uint64_t token) {
  __syncthreads();
  const int t = threadIdx.x;
  if (t < c.world && t != rank) {
    ptx::fence_acq_rel_sys();
    ptx::st_relaxed_sys(pipeFlag(c, t, phase, slot, rank), token);
  }
}
// (A flag per phase: no barrier stands between a round's last wait and the next round's first one, which could otherwise clear
// the flag before a slow warp has read it for the wait before.)
MSCCLPP_DEVICE_INLINE bool pipeWait(const DeviceComm& c, int rank, int phase, int slot, uint64_t token, int* okSmem) {
  const int t = threadIdx.x;
  if (t < c.world && t != rank) {
    const uint64_t* mine = pipeFlag(c, rank, phase, slot, t);
    SpinGuard g(c.status, c.timeoutNs);
    uint64_t v;
    bool here = true;
    while ((v = ptx::ld_relaxed_sys(mine)) < token) {
      if (!g.keepSpinning()) {
        g.report(kDevTimeoutBarrier, rank, 20000 + phase * 1000 + slot, t, token, v);
        here = false;
        break;
      }
    }
    if (here) (void)ptx::ld_acquire_sys(mine);
    else okSmem[phase] = 0;
  }
  __syncthreads();
  return okSmem[phase] != 0;
}

// 16-byte units [first, n) from src to dst, kCopyUnroll loads in flight per thread.
constexpr uint32_t kCopyUnroll = 4;
MSCCLPP_DEVICE_INLINE void copyUnits(char* dst, const char* src, uint32_t first, uint32_t n) {
  for (uint32_t u0 = first + threadIdx.x; u0 < n; u0 += blockDim.x * kCopyUnroll) {
    uint4 v[kCopyUnroll];
#pragma unroll
    for (uint32_t k = 0; k < kCopyUnroll; k++) {
      const uint32_t u = u0 + k * blockDim.x;  // (loads beyond the end repeat the last unit: no branch around them)
      v[k] = ptx::ld_weak_v4(src + static_cast<uint64_t>(u < n ? u : n - 1) * 16);
    }
#pragma unroll
    for (uint32_t k = 0; k < kCopyUnroll; k++) {
      const uint32_t u = u0 + k * blockDim.x;
      if (u < n) ptx::st_weak_v4(dst + static_cast<uint64_t>(u) * 16, v[k]);
    }
  }
}
// The last bytes of a message whose size is not a multiple of 16: one thread, byte by byte; the scratch unit is padded
// with zeros.
MSCCLPP_DEVICE_INLINE void copyTail(char* dst, const char* src, uint32_t n, uint32_t padTo) {
  if (threadIdx.x != 0) return;
#pragma unroll 1
  for (uint32_t i = 0; i < n; i++) *reinterpret_cast<volatile char*>(dst + i) = *reinterpret_cast<const volatile char*>(src + i);
#pragma unroll 1
  for (uint32_t i = n; i < padTo; i++) *reinterpret_cast<volatile char*>(dst + i) = 0;
}

template <typename T, ReduceOp Op>
MSCCLPP_DEVICE_INLINE uint4 switchReduce(const void* mc) {
  if constexpr (__is_same(T, __half)) {
    if constexpr (Op == SUM) return ptx::multimem_ld_reduce_add_f16x2_acc32(mc);
    else return ptx::multimem_ld_reduce_min_f16x2(mc);
  } else if constexpr (__is_same(T, __nv_bfloat16)) {
    if constexpr (Op == SUM) return ptx::multimem_ld_reduce_add_bf16x2_acc32(mc);
    else return ptx::multimem_ld_reduce_min_bf16x2(mc);
  } else if constexpr (__is_same(T, f8e4m3)) {
    return ptx::multimem_ld_reduce_add_e4m3x4(mc);
  } else if constexpr (__is_same(T, f8e5m2)) {
    return ptx::multimem_ld_reduce_add_e5m2x4(mc);
  } else {
    return ptx::multimem_ld_reduce_add_f32(mc);
  }
}

template <typename T, ReduceOp Op>
constexpr bool switchReducible() {
  if (__is_same(T, __half) || __is_same(T, __nv_bfloat16)) return true;
  if (Op != SUM) return false;
  return __is_same(T, float) || __is_same(T, f8e4m3) || __is_same(T, f8e5m2);
}

template <typename T, ReduceOp Op, bool kFloat = IsFloatLike<T>::value>
struct PipeAccum;
template <typename T, ReduceOp Op>
struct PipeAccum<T, Op, true> {
  float acc[Vec16<T>::kElems];
  MSCCLPP_DEVICE_INLINE void init(uint4 v) { Vec16<T>::toFloat(v, acc); }
  MSCCLPP_DEVICE_INLINE void add(uint4 v) { accumulate16<T, Op>(acc, v); }
  MSCCLPP_DEVICE_INLINE uint4 result() const { return Vec16<T>::fromFloat(acc); }
};
template <typename T, ReduceOp Op>
struct PipeAccum<T, Op, false> {
  uint4 acc;
  MSCCLPP_DEVICE_INLINE void init(uint4 v) { acc = v; }
  MSCCLPP_DEVICE_INLINE void add(uint4 v) { acc = reduce16<T, Op>(acc, v); }
  MSCCLPP_DEVICE_INLINE uint4 result() const { return acc; }
};

// kFetch (peer loads): a rank's sums stay in its own scratch, from which the peers fetch them, instead of going to every peer's
template <typename T, ReduceOp Op, bool kNvls, bool kFetch>
__global__ void __launch_bounds__(512, 2) pipelineAllreduceKernel(PipeArgs a) {
  const DeviceComm& c = a.comm;
  const int rank = deviceRank(c);
  const int world = c.world;
  const uint32_t epoch = launchEpoch(c, rank);
  const int slot = blockIdx.x;
  const uint64_t emu = static_cast<uint64_t>(blockIdx.y) * a.emuStride;
  const char* in = reinterpret_cast<const char*>(a.in) + emu;
  char* out = reinterpret_cast<char*>(a.out) + emu;
  const uint64_t bytes = a.bytes;
  const uint64_t nunits = (bytes + 15) / 16;
  const uint64_t sliceUnits = a.sliceBytes / 16;  // a multiple of `world`
  const uint64_t subUnits = sliceUnits / world;
  const uint64_t roundUnits = sliceUnits * gridDim.x;
  const uint64_t rounds = (nunits + roundUnits - 1) / roundUnits;
  // scratch (heap offset, equal on every rank): [in | out][parity][slot][sliceBytes]. A rank that is through with a launch may copy in
  // for its next one, with other slices, while its peers still fetch reduced parts of this one from it, so where `out` begins
  // must not change from launch to launch.
  const uint64_t scratchOff = reinterpret_cast<uint64_t>(a.scratch) - c.peerBase[c.rank];
  const uint64_t local = c.peerBase[rank];
  __shared__ int okSmem[2];
  __shared__ uint64_t heaps[8];  // (in shared memory: as kernel parameters their sums with the slices live in registers all along)
  if (threadIdx.x < 8) heaps[threadIdx.x] = c.peerBase[threadIdx.x];
  if (threadIdx.x < 2) okSmem[threadIdx.x] = 1;
  __syncthreads();

  const uint64_t parityBytes = static_cast<uint64_t>(gridDim.x) * a.sliceBytes;
  const uint32_t tailBytes = static_cast<uint32_t>(bytes & 15);   // of the message's last unit, 0 = it is whole
  auto inSliceOf = [&](uint64_t r) { return scratchOff + (r & 1) * parityBytes + static_cast<uint64_t>(slot) * a.sliceBytes; };
  auto firstOf = [&](uint64_t r) { return r * roundUnits + static_cast<uint64_t>(slot) * sliceUnits; };  // first global unit of my slice
  auto haveOf = [&](uint64_t r) {  // units of my slice that exist, the last of them possibly not whole
    const uint64_t first = firstOf(r);
    return static_cast<uint32_t>(first < nunits ? (nunits - first < sliceUnits ? nunits - first : sliceUnits) : 0);
  };
  auto tailOf = [&](uint64_t r, uint32_t have) { return have != 0 && firstOf(r) + have == nunits ? tailBytes : 0u; };
  // The part of a slice that this rank reduces is read by nobody else, and nobody else writes its result: with peer loads
  // its whole units skip the scratch both ways (1 / world of the copies).
  const uint32_t ownBegin = static_cast<uint32_t>(rank) * static_cast<uint32_t>(subUnits), ownEnd = ownBegin + static_cast<uint32_t>(subUnits);
  auto copyOthers = [&](char* dst, const char* src, uint32_t whole) {
    if constexpr (kNvls) {
      copyUnits(dst, src, 0, whole);
    } else {
      copyUnits(dst, src, 0, ownBegin < whole ? ownBegin : whole);
      copyUnits(dst, src, ownEnd, whole);
    }
  };
  // 1. copy-in (nothing to do for a slice beyond the end of the message, but the barriers still run: peers may not know)
  auto copyIn = [&](uint64_t r) {
    const uint32_t have = haveOf(r), tail = tailOf(r, have), whole = have - (tail != 0 ? 1 : 0);
    const char* src = in + firstOf(r) * 16;
    char* dst = reinterpret_cast<char*>(local + inSliceOf(r));
    copyOthers(dst, src, whole);
    if (tail != 0) copyTail(dst + static_cast<uint64_t>(whole) * 16, src + static_cast<uint64_t>(whole) * 16, tail, 16);
  };
  auto tokenOf = [&](uint64_t r) { return (static_cast<uint64_t>(epoch) << 32) | (r + 1); };

  bool healthy = true;
  if (rounds > 0) {
    copyIn(0);
    pipeSignal(c, rank, 0, slot, tokenOf(0));
  }
#pragma unroll 1
  for (uint64_t r = 0; r < rounds; r++) {
    const uint64_t inSlice = inSliceOf(r);
    const uint64_t outSlice = inSlice + a.outOffset;
    const uint32_t have = haveOf(r);
    // 2. every rank has staged its slice of this index
    healthy = pipeWait(c, rank, 0, slot, tokenOf(r), okSmem);
    if (!healthy) break;
    // 3. reduce my part of the slice, result to everybody's scratch-out
    {
      const uint32_t begin = ownBegin;
      const uint32_t end = ownEnd < have ? ownEnd : have;
      [[maybe_unused]] const uint32_t direct = have - (tailOf(r, have) != 0 ? 1 : 0);  // units below it are whole
      [[maybe_unused]] const uint64_t inDirect = reinterpret_cast<uint64_t>(in) + firstOf(r) * 16;
      [[maybe_unused]] const uint64_t outDirect = reinterpret_cast<uint64_t>(out) + firstOf(r) * 16;
      // eight loads in flight per thread: kUnroll units of up to kSources ranks each (with the switch, four sums)
      auto sweep = [&](auto unrollTag, auto sourcesTag) {
        constexpr int kUnroll = decltype(unrollTag)::value, kSources = decltype(sourcesTag)::value;
#pragma unroll 1
        for (uint32_t u0 = begin + threadIdx.x; u0 < end; u0 += blockDim.x * kUnroll) {
          uint4 v[kUnroll];
          if constexpr (kNvls) {
#pragma unroll
            for (int k = 0; k < kUnroll; k++) {
              const uint32_t u = u0 + k * blockDim.x;
              if (u < end) v[k] = switchReduce<T, Op>(reinterpret_cast<const void*>(c.mcBase + inSlice + static_cast<uint64_t>(u) * 16));
            }
          } else {
            uint4 w[kUnroll][kSources];
#pragma unroll
            for (int k = 0; k < kUnroll; k++) {
              const uint32_t u = u0 + k * blockDim.x;
              const uint32_t uc = u < end ? u : end - 1;
              const uint64_t off = static_cast<uint64_t>(uc) * 16;
              const uint64_t own = (uc < direct ? inDirect : local + inSlice) + off;
#pragma unroll
              for (int p = 0; p < kSources; p++)  // (slots beyond the last rank read local memory and are not added)
                w[k][p] = ptx::ld_weak_v4(reinterpret_cast<const void*>(p < world && p != rank ? heaps[p] + inSlice + off : own));
            }
#pragma unroll
            for (int k = 0; k < kUnroll; k++) {
              PipeAccum<T, Op> acc;
              acc.init(w[k][0]);
#pragma unroll
              for (int p = 1; p < kSources; p++)
                if (p < world) acc.add(w[k][p]);
              v[k] = acc.result();
            }
          }
#pragma unroll
          for (int k = 0; k < kUnroll; k++) {
            const uint32_t u = u0 + k * blockDim.x;
            if (u >= end) continue;
            const uint64_t off = outSlice + static_cast<uint64_t>(u) * 16;
            if constexpr (kNvls) {
              ptx::multimem_st_v4(reinterpret_cast<void*>(c.mcBase + off), v[k]);
            } else {
              if constexpr (!kFetch) {
#pragma unroll 1
                for (int i = 1; i < world; i++) {
                  const int p = rank + i < world ? rank + i : rank + i - world;
                  ptx::st_weak_v4(reinterpret_cast<void*>(heaps[p] + off), v[k]);
                }
                ptx::st_weak_v4(reinterpret_cast<void*>(u < direct ? outDirect + static_cast<uint64_t>(u) * 16 : local + off), v[k]);
              } else {
                ptx::st_weak_v4(reinterpret_cast<void*>(local + off), v[k]);
                if (u < direct) ptx::st_weak_v4(reinterpret_cast<void*>(outDirect + static_cast<uint64_t>(u) * 16), v[k]);
              }
            }
          }
        }
      };
      using std::integral_constant;
      if constexpr (kNvls) {
        sweep(integral_constant<int, 4>{}, integral_constant<int, 1>{});
      } else {
        if (world <= 2) sweep(integral_constant<int, 4>{}, integral_constant<int, 2>{});
        else if (world <= 4) sweep(integral_constant<int, 2>{}, integral_constant<int, 4>{});
        else sweep(integral_constant<int, 1>{}, integral_constant<int, 8>{});
      }
    }
    pipeSignal(c, rank, 1, slot, tokenOf(r));
    // the next round's copy-in, under the peers' reductions. Its scratch was last read in round r - 1, and the end of that
    // round told this block that every rank had reduced it.
    if (r + 1 < rounds) {
      copyIn(r + 1);
      pipeSignal(c, rank, 0, slot, tokenOf(r + 1));
    }
    // 4. every rank's part of my scratch-out slice has landed
    healthy = pipeWait(c, rank, 1, slot, tokenOf(r), okSmem);
    if (!healthy) break;
    // 5. copy-out
    const uint32_t tail = tailOf(r, have), whole = have - (tail != 0 ? 1 : 0);
    char* dst = out + firstOf(r) * 16;
    if constexpr (!kFetch) {
      copyOthers(dst, reinterpret_cast<const char*>(local + outSlice), whole);
    } else {
      const uint32_t sub = static_cast<uint32_t>(subUnits), mineBegin = ownBegin < whole ? ownBegin : whole, mineEnd = ownEnd < whole ? ownEnd : whole;
      const uint32_t n = whole - (mineEnd - mineBegin);
      for (uint32_t i0 = threadIdx.x; i0 < n; i0 += blockDim.x * kCopyUnroll) {
        uint4 v[kCopyUnroll];
        uint32_t at[kCopyUnroll];
#pragma unroll
        for (uint32_t k = 0; k < kCopyUnroll; k++) {
          uint32_t u = i0 + k * blockDim.x < n ? i0 + k * blockDim.x : n - 1;
          if (u >= mineBegin) u += mineEnd - mineBegin;
          at[k] = u;
          v[k] = ptx::ld_weak_v4(reinterpret_cast<const void*>(heaps[u / sub] + outSlice + static_cast<uint64_t>(u) * 16));
        }
#pragma unroll
        for (uint32_t k = 0; k < kCopyUnroll; k++)
          if (i0 + k * blockDim.x < n) ptx::st_weak_v4(dst + static_cast<uint64_t>(at[k]) * 16, v[k]);
      }
    }
    if (tail != 0) {
      const uint64_t from = !kFetch ? local : heaps[whole / static_cast<uint32_t>(subUnits)];
      copyTail(dst + static_cast<uint64_t>(whole) * 16, reinterpret_cast<const char*>(from + outSlice) + static_cast<uint64_t>(whole) * 16, tail, 0);
    }
  }
  if constexpr (kFetch) {  // the next launch may have its halves elsewhere: nobody goes on while a peer fetches
    if (a.scratchBytes == 0 && healthy) {
      pipeSignal(c, rank, 1, slot, tokenOf(rounds));
      pipeWait(c, rank, 1, slot, tokenOf(rounds), okSmem);
    }
  }
  finishLaunch(c, rank, epoch);
}

template <typename T, ReduceOp Op>
cudaError_t launchPipeTyped(const PipeArgs& a, int nBlocks, int nThreads, cudaStream_t stream) {
  dim3 grid(nBlocks, a.emuRanks > 1 ? a.emuRanks : 1, 1);
  dim3 block(nThreads, 1, 1);
  const void* kernel = pipelineFetches(a.fetch, a.comm.world, a.emuRanks) ? reinterpret_cast<const void*>(pipelineAllreduceKernel<T, Op, false, true>)
                                                                          : reinterpret_cast<const void*>(pipelineAllreduceKernel<T, Op, false, false>);
  if constexpr (switchReducible<T, Op>()) {  // (other types: peer loads)
    if (a.nvls) kernel = reinterpret_cast<const void*>(pipelineAllreduceKernel<T, Op, true, false>);
  }
  PipeArgs copy = a;
  copy.outOffset = a.scratchBytes != 0 ? a.scratchBytes / 32 * 16 : pipelineScratchBytes(nBlocks, a.sliceBytes) / 2;
  void* params[] = {&copy};
  if (a.emuRanks > 1) return launchEmulatedRanks(kernel, grid, block, params, 2, stream);
  return cudaLaunchKernel(kernel, grid, block, params, 0, stream);
}

}  // namespace

size_t pipelineScratchBytes(int nBlocks, uint64_t sliceBytes) { return 4ull * static_cast<size_t>(nBlocks) * sliceBytes; }

cudaError_t launchPipelineAllreduce(const PipeArgs& args, DataType dtype, ReduceOp op, int nBlocks, int nThreads, cudaStream_t stream) {
  const int world = args.comm.world;
  if (args.bytes == 0 || world < 1 || world > 8) return cudaErrorInvalidValue;
  if (nBlocks < 1 || nBlocks > kBarrierSlots || nThreads < 32 || nThreads > 512 || nThreads < world) return cudaErrorInvalidValue;
  if (args.sliceBytes == 0 || args.sliceBytes % (16ull * world) != 0) return cudaErrorInvalidValue;
  if (args.scratchBytes != 0 && args.scratchBytes < pipelineScratchBytes(nBlocks, args.sliceBytes)) return cudaErrorInvalidValue;
  if (args.scratch == nullptr || (reinterpret_cast<uintptr_t>(args.scratch) & 15) != 0) return cudaErrorInvalidValue;
  if (args.nvls && args.comm.mcBase == 0) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(args.in) & 15) != 0 || (reinterpret_cast<uintptr_t>(args.out) & 15) != 0) return cudaErrorInvalidValue;
  const bool isMin = op == MIN;
  switch (dtype) {
    case DataType::FLOAT16:
      return isMin ? launchPipeTyped<__half, MIN>(args, nBlocks, nThreads, stream) : launchPipeTyped<__half, SUM>(args, nBlocks, nThreads, stream);
    case DataType::BFLOAT16:
      return isMin ? launchPipeTyped<__nv_bfloat16, MIN>(args, nBlocks, nThreads, stream)
                   : launchPipeTyped<__nv_bfloat16, SUM>(args, nBlocks, nThreads, stream);
    case DataType::FLOAT32:
      return isMin ? launchPipeTyped<float, MIN>(args, nBlocks, nThreads, stream) : launchPipeTyped<float, SUM>(args, nBlocks, nThreads, stream);
    case DataType::INT32:
      return isMin ? launchPipeTyped<int32_t, MIN>(args, nBlocks, nThreads, stream) : launchPipeTyped<int32_t, SUM>(args, nBlocks, nThreads, stream);
    case DataType::UINT32:
      return isMin ? launchPipeTyped<uint32_t, MIN>(args, nBlocks, nThreads, stream) : launchPipeTyped<uint32_t, SUM>(args, nBlocks, nThreads, stream);
    case DataType::UINT8:
      return isMin ? launchPipeTyped<uint8_t, MIN>(args, nBlocks, nThreads, stream) : launchPipeTyped<uint8_t, SUM>(args, nBlocks, nThreads, stream);
    case DataType::FLOAT8_E4M3:
      return isMin ? launchPipeTyped<f8e4m3, MIN>(args, nBlocks, nThreads, stream) : launchPipeTyped<f8e4m3, SUM>(args, nBlocks, nThreads, stream);
    case DataType::FLOAT8_E5M2:
      return isMin ? launchPipeTyped<f8e5m2, MIN>(args, nBlocks, nThreads, stream) : launchPipeTyped<f8e5m2, SUM>(args, nBlocks, nThreads, stream);
    case DataType::FLOAT8_E4M3B15:
      return isMin ? launchPipeTyped<f8e4m3b15, MIN>(args, nBlocks, nThreads, stream)
                   : launchPipeTyped<f8e4m3b15, SUM>(args, nBlocks, nThreads, stream);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace mscclpp
