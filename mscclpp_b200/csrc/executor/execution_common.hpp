// Device-side representation of an execution plan: what the host resolves per (plan, message size)
// and the interpreter kernel consumes.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstdlib>

#include <mscclpp/device/symm.cuh>
#include <mscclpp/fifo_device.hpp>

#include <mscclpp/npkit/npkit_struct.hpp>

namespace mscclpp {

enum class OpType : uint8_t {
  NOP = 0,
  BARRIER,
  SIGNAL,
  RELAXED_SIGNAL,
  WAIT,
  RELAXED_WAIT,
  FLUSH,
  PUT,
  PUT_WITH_SIGNAL,
  PUT_WITH_SIGNAL_AND_FLUSH,
  GET,
  COPY,
  REDUCE,
  REDUCE_SEND,
  READ_REDUCE,
  READ_REDUCE_SEND,
  PUT_PACKETS,
  READ_PUT_PACKETS,
  COPY_PACKETS,
  UNPACK_PACKETS,
  REDUCE_PACKETS,
  REDUCE_SEND_PACKETS,
  REDUCE_COPY_PACKETS,
  REDUCE_COPY_SEND_PACKETS,
  GROUP_LOAD_REDUCE_STORE,
  GROUP_STORE,
  GROUP_STORE_PACKETS,
  SEM_ACQUIRE,
  SEM_RELEASE,
  PIPELINE_BEGIN,
  PIPELINE_END,
};

constexpr int kExecMaxOperands = 16;
constexpr int kExecMaxIds = 16;
constexpr int kExecMaxThreadBlocks = 128;
constexpr int kExecMaxChannels = 256;     // per channel type and rank
constexpr int kExecMaxSemaphores = 64;
constexpr int kExecMaxBarriers = 32;
constexpr int kExecMaxRanksInGroup = 16;

// One buffer range. `offset` is a HEAP offset (payload space); packet-space operands are expanded by the
// kernel (scratch base + 2 x payload offset, for LL16 and LL8 alike).
struct DevOperand {
  uint64_t offset;      // heap offset of the first byte (payload space)
  uint64_t size;        // bytes (payload space)
  int16_t rank;         // owning rank (local operands: the executing rank)
  uint8_t isScratch;    // scratch buffer: packet ops address it in packet space
  uint8_t isSwitch;     // multimem operand: address through mcBase (group = all ranks of switchGroup)
  uint16_t switchGroup; // index into DevPlan::groups
  uint16_t pad;
};

struct DevOp {
  uint8_t type;         // OpType
  uint8_t nSrc;
  uint8_t nDst;
  uint8_t nIds;
  uint8_t channelType;  // 0 memory, 1 port
  uint8_t inPipeline;   // operands are sliced per pipeline iteration
  uint16_t pad;
  uint32_t arg0;        // BARRIER: number of thread blocks; PIPELINE_BEGIN: iterations
  uint32_t arg1;        // PIPELINE_BEGIN: unit size in bytes; BARRIER: barrier id
  uint16_t ids[kExecMaxIds];  // channel ids (rank-level) or semaphore ids
  DevOperand src[kExecMaxOperands];
  DevOperand dst[kExecMaxOperands];
};

struct DevChannel {
  int16_t peer;       // rank at the other end
  int16_t mate;       // index of the paired channel on the peer
};

struct DevGroup {
  int16_t nRanks;
  int16_t ranks[kExecMaxRanksInGroup];
};

struct DevThreadBlock {
  uint32_t opBegin;
  uint32_t opEnd;
};

// Per-rank state kept in the heap (same offset on every rank): channel semaphores are written by peers.
struct ExecState {
  uint64_t inbound[2][kExecMaxChannels];   // [memory/port][channel]: signals received
  uint64_t expected[2][kExecMaxChannels];  // private: signals consumed
  int32_t semaphores[kExecMaxSemaphores];  // device semaphores of the plan (reset to init values per launch by block 0)
  uint32_t barriers[kExecMaxBarriers];     // grid barrier counters (monotonic)
  uint32_t barrierGen[kExecMaxBarriers];   // completed barrier generations (written by the last launch's end)
  uint32_t semInit;                        // launch epoch for which `semaphores` has been initialised
};

struct DevPlan {
  uint32_t nThreadBlocks;
  uint32_t nOps;
  DevThreadBlock tbs[kExecMaxThreadBlocks];
  DevChannel channels[2][kExecMaxChannels];
  DevGroup groups[8];
  int32_t semInit[kExecMaxSemaphores];
  uint32_t nSemaphores;
  uint32_t pad;
  const DevOp* ops;       // device array
};

// Request of a port-channel operation to the executor's host proxy (one 16-byte FIFO trigger):
//   fst: source heap offset [0,40) | size low 20 bits [40,60) | issuing rank [60,64)
//   snd: destination heap offset [0,40) | size high 8 bits [40,48) | channel id [48,56) | kind [56,59) | context [59,63)
// (bit 63 of snd belongs to the FIFO). Sizes are bytes, at most kPortMaxBytes per request.
constexpr uint64_t kPortMaxBytes = (1ull << 28) - 16;
constexpr uint32_t kPortData = 1, kPortSignal = 2, kPortSync = 4;
struct PortRequest {
  uint64_t srcOff, dstOff, size;
  uint32_t rank, channel, kind, context;
};
MSCCLPP_HOST_DEVICE_INLINE ProxyTrigger encodePortRequest(const PortRequest& r) {
  ProxyTrigger t;
  t.fst = (r.srcOff & ((1ull << 40) - 1)) | ((r.size & 0xfffffull) << 40) | (static_cast<uint64_t>(r.rank & 15u) << 60);
  t.snd = (r.dstOff & ((1ull << 40) - 1)) | (((r.size >> 20) & 0xffull) << 40) | (static_cast<uint64_t>(r.channel & 255u) << 48) |
          (static_cast<uint64_t>(r.kind & 7u) << 56) | (static_cast<uint64_t>(r.context & 15u) << 59);
  return t;
}
MSCCLPP_HOST_DEVICE_INLINE PortRequest decodePortRequest(const ProxyTrigger& t) {
  PortRequest r;
  r.srcOff = t.fst & ((1ull << 40) - 1);
  r.size = ((t.fst >> 40) & 0xfffffull) | (((t.snd >> 40) & 0xffull) << 20);
  r.rank = static_cast<uint32_t>(t.fst >> 60) & 15u;
  r.dstOff = t.snd & ((1ull << 40) - 1);
  r.channel = static_cast<uint32_t>(t.snd >> 48) & 255u;
  r.kind = static_cast<uint32_t>(t.snd >> 56) & 7u;
  r.context = static_cast<uint32_t>(t.snd >> 59) & 15u;
  return r;
}

// What a thread block's operations take, in us, on `team` CTAs of nThreads threads (see executionKernel): only as much of it as depends on the
// team. It shares the words of one source of one operation at a time - in a pipeline, of one iteration - so a source with few of them keeps
// few CTAs busy; and wherever a thread block meets, the barrier is one of the cluster. What the host proxy moves is shared by nobody. < 0: the
// block has packet operations, whose CTAs would all wait by themselves.
// The rates are those of one CTA of 1024 threads and the 0.55 us those of a cluster's barrier, one B200, all ranks on it. Plans of one thread
// block per rank, us on 1 / 2 / 4 / 8 CTAs: all-gather over eight ranks (seven puts), 32 KB each 24.4 / 26.9 / 26.9 / 26.8, 64 KB 28.9 / 28.9 / 26.8 / 26.8,
// 512 KB 104 / 66 / 44 / 35; reduce-scatter over two ranks, 128 KB 19.5 / 22.2 / 20.8 / 20.8, 512 KB 31.6 / 27.4 / 23.1 / 21.7; 64 puts of 128 KB with
// signal and wait 612 / 715 / 687 / 666, 8 of 256 KB 104 / 105 / 95 / 91. (By the bytes of all its operations together, whatever they are, the
// first and the last two of these got eight CTAs each, and 64 puts of 4 KB 574 us instead of 372.)
inline float execBlockUs(const DevOp* ops, size_t nOps, int nThreads, int team) {
  float us = 0.f, iterations = 1.f;
  uint64_t unit = 0;
  for (size_t i = 0; i < nOps; i++) {
    const DevOp& op = ops[i];
    const bool port = op.channelType == 1;
    float rate = 48.f;  // KB per us and CTA: copies
    int syncs = 0;
    switch (static_cast<OpType>(op.type)) {
      case OpType::PIPELINE_BEGIN:
        iterations = static_cast<float>(op.arg0);
        unit = op.arg1;
        continue;
      case OpType::PIPELINE_END:
        iterations = 1.f;
        unit = 0;
        continue;
      case OpType::NOP:
        syncs = 1;
        break;
      case OpType::BARRIER:
      case OpType::WAIT:
      case OpType::RELAXED_WAIT:
      case OpType::SEM_ACQUIRE:
      case OpType::SEM_RELEASE:
        syncs = 2;
        break;
      case OpType::SIGNAL:
      case OpType::RELAXED_SIGNAL:
      case OpType::FLUSH:
        syncs = port ? 2 : 0;
        break;
      case OpType::PUT:
        syncs = port ? 2 : 0;
        break;
      case OpType::PUT_WITH_SIGNAL:
      case OpType::PUT_WITH_SIGNAL_AND_FLUSH:
        syncs = port ? 2 : 1;
        break;
      case OpType::GET:
      case OpType::COPY:
        break;
      case OpType::REDUCE:
      case OpType::REDUCE_SEND:
      case OpType::READ_REDUCE:
      case OpType::READ_REDUCE_SEND:
        rate = op.nSrc > 2 ? 80.f : 64.f;
        break;
      case OpType::GROUP_LOAD_REDUCE_STORE:
      case OpType::GROUP_STORE:
        break;
      default:
        return -1.f;
    }
    if (team > 1) us += 0.55f * iterations * static_cast<float>(syncs);
    if (port) continue;
    for (int k = 0; k < op.nSrc; k++) {
      const uint64_t size = op.src[k].size, atOnce = unit != 0 && op.inPipeline && size > unit ? unit : size;
      const float busy = static_cast<float>(atOnce) / 16.f / static_cast<float>(nThreads);  // CTAs whose threads have a word each
      const float ctas = busy < 1.f ? 1.f : busy < static_cast<float>(team) ? busy : static_cast<float>(team);
      us += static_cast<float>(size) / 1000.f / (rate * static_cast<float>(nThreads) / 1024.f * ctas);
    }
  }
  return us;
}

// The CTAs per thread block that pay: at most and at least (1 and 1: none do), from blocksUs[k], the longest of the plan's thread blocks on 2^k of
// them. The launch takes as many of these as there are SMs for.
struct ExecTeam {
  int most = 1, least = 1;
};
inline ExecTeam execTeam(const float (&blocksUs)[4], int allowed = 8) {
  ExecTeam t;
  for (int k = 1; k < 4 && (1 << k) <= allowed; k++) {
    if (blocksUs[k] + 0.5f >= blocksUs[0]) continue;  // (half a microsecond: what the model is off by)
    if (t.most == 1) t.least = 1 << k;
    if (t.most == 1 || blocksUs[k] + 0.05f < blocksUs[k - 1]) t.most = 1 << k;
  }
  return t;
}

// How many CTAs an executor allows per thread block: what MSCCLPP_EXECUTOR_TEAM says (`setting`, null or empty where it is not set; rounded down to a
// power of two), else eight where all ranks are in the launch, and one where there are others. A plan's author counts on one SM for each
// thread block. Launches of ranks on several GPUs wait for one another: two plans on two streams that fit a GPU side by side finish in
// whatever order the ranks start them, but where a team of the one has taken the SMs of the other, ranks that start them in different
// orders wait until their time limit. Nor does a plan of few blocks leave SMs to the kernel that it is to run beside.
inline int execAllowedTeam(const char* setting, bool allRanksHere) {
  const int byDefault = allRanksHere ? 8 : 1;
  if (setting == nullptr || setting[0] == '\0') return byDefault;
  const int wanted = std::atoi(setting);
  int team = wanted < 1 ? 0 : 1;
  while (team != 0 && team < 8 && 2 * team <= wanted) team *= 2;
  return team != 0 ? team : byDefault;
}

struct ExecArgs {
  DeviceComm comm;
  const DevPlan* plans[kMaxRanks];  // [emulated rank]; real mode uses entry 0
  uint64_t stateOff;     // heap offset of ExecState
  uint64_t scratchOff;   // heap offset of the scratch buffer (first half when double buffered)
  uint64_t scratchHalf;  // bytes of one scratch half (0 = no double buffering)
  int emuRanks;
  int team;              // CTAs of a cluster that share a plan thread block (1, 2, 4 or 8; see executionKernel)
  int leastTeam;         // host: the fewest that pay (see execTeam)
  int packetLL8;         // packet ops use 8-byte LL8 packets instead of 16-byte LL16 ones
  int portContext;       // index of this plan context in the host proxy's table
  FifoDeviceHandle portFifo;  // request queue of the executor's host proxy (triggers == nullptr: the plan has no port ops)
  NpKitEventCollectContext* npkit;  // tracer buffers, nullptr = tracing off
};

}  // namespace mscclpp
