// sm_100a kernels of the device-to-device channel. See push.h for the interface.
//
// tpb_push_pack is ONE persistent launch (at most one CTA per SM) that serves a whole message:
//
//   * Warp 0 is a copy engine. Its elected lane drives a multi-stage pipeline of TMA bulk copies:
//     global -> shared (completion on an mbarrier) and shared -> global (bulk groups), for every
//     entry whose source, destination and size are 16-byte multiples. The loads only ever read
//     THIS GPU's memory; the stores may target a peer GPU's memory mapped over NVLink. No thread
//     touches the bytes. Tile size and depth are run-time parameters (PushTuning).
//   * The other warps handle what the bulk path cannot, one "warp tile" of up to 8 KiB at a time and
//     without CTA-wide barriers: ragged heads and tails, relatively misaligned buffers, dtype
//     conversion (fp32 <-> bf16/fp16), views whose rows are contiguous (copied as the runs they
//     are), and other 2-D strided sources, which a warp transposes through
//     its private padded shared-memory tile so that both the strided reads and the packed writes
//     are coalesced (32x32 elements; 64x64 moved as 32-bit words for 2-byte elements; 32 whole
//     packed rows written as one contiguous run for matrices of at most 64 columns bound for
//     another GPU). A warp makes one call per tensor for all of its tiles.
//   * Large transposed matrices may move as "block tiles" instead, which eight warps share behind a
//     barrier of their own: 128 bulk loads, sent for by as many threads, fill a stage of shared
//     memory, and the warps write it out transposed.
//   * Tiles are dealt round-robin (bulk and block tile t to CTA t mod gridDim.x, warp tile t to warp
//     t mod #warps), so no scheduling state lives in global memory.
//   * Completion: every CTA makes its writes visible system-wide, then arrives on a counter;
//     the last CTA resets the counter and publishes the flag with a release store at system
//     scope. The flag lives in the receiver's memory; its stream waits on it.
//
// A "light" instantiation (256 threads, no bulk copy engine, shared memory only when a tensor is
// staged through it) serves messages without bulk work, where launch latency matters most. Both
// come with the code for contiguous tensors only, for views moved by single warps too, and for all.
//
// Built with -DTPB_DEBUG_KERNELS the copy paths check every address against its table entry,
// skip what lies outside and count it (boundsViolations()); nothing in here can trap.
//
// Every wait in here is bounded: a bulk load that does not complete within the limit makes the
// CTA record kStatusBarrierTimeout, drain its own outstanding stores (the block tiles: wait, again
// within the limit, for their loads in flight) and fall through to the completion protocol, so the
// kernel always terminates.
#include "kernels/push.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common/cuda.h"
#include "common/trace.h"
#include "kernels/block_pipe.h"
#include "kernels/run_copy.cuh"
#include "kernels/smem_limit.h"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>

namespace tpb {
namespace kernels {

namespace {

std::atomic<uint64_t> gLaunches{0};
std::mutex gTuningMutex;
PushTuning initialTuning() {
  PushTuning t;
  if (const char* e = std::getenv("TPB_PUSH_BAND")) {
    if (e[0] >= '0' && e[0] <= '2' && e[1] == 0) t.bandRows = static_cast<uint32_t>(e[0] - '0');
  }
  if (const char* e = std::getenv("TPB_PUSH_NARROW")) {
    if (e[0] >= '0' && e[0] <= '2' && e[1] == 0) t.narrowRows = static_cast<uint32_t>(e[0] - '0');
  }
  if (const char* e = std::getenv("TPB_PUSH_BLOCK")) {
    if (e[0] >= '0' && e[0] <= '2' && e[1] == 0) t.blockForm = static_cast<uint32_t>(e[0] - '0');
  }
  // The shape of the bulk pipeline can be tried out without rebuilding; values that setPushTuning
  // would refuse are ignored.
  auto number = [](const char* name, uint32_t fallback) {
    const char* e = std::getenv(name);
    if (!e || !*e) return fallback;
    char* end = nullptr;
    const unsigned long v = std::strtoul(e, &end, 0);
    return end && *end == 0 ? static_cast<uint32_t>(v) : fallback;
  };
  const uint32_t tile = number("TPB_PUSH_TILE_BYTES", t.bulkTileBytes);
  const uint32_t stages = number("TPB_PUSH_STAGES", t.bulkStages);
  if (tile % 1024 == 0 && tile > 0 && stages >= 2 && stages <= static_cast<uint32_t>(kMaxBulkStages) &&
      static_cast<size_t>(tile) * stages <= 160 * 1024) {
    t.bulkTileBytes = tile;
    t.bulkStages = stages;
  }
  t.bulkMinBytes = number("TPB_PUSH_BULK_MIN_BYTES", t.bulkMinBytes);
  return t;
}
PushTuning gTuning = initialTuning();

constexpr uint32_t kWarpTileBytes = kStridedTile * (kStridedTile / 2 + 1) * 8;  // 4352 B per warp: 32 x 17 x 8-byte, or 32 x 33 x 4-byte
constexpr int kWidePitch = kWideTile + 2;                                        // 2-byte elements per staged column
constexpr uint32_t kWideWarpTileBytes = kWideTile * kWidePitch * 2;              // 8448 B per warp
constexpr size_t kMaxSmemPerCta = 227 * 1024;

// ---- PTX wrappers -----------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smemAddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbarInit(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbarExpectTx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddr(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbarTryWait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smemAddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: ~2^22 polls, each of which may block for the hardware's time slice.
__device__ __forceinline__ bool mbarWaitBounded(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < (1u << 22); ++i) {
    if (mbarTryWait(bar, parity)) return true;
    if (i > 64) __nanosleep(64);
  }
  return false;
}
// Non-multicast bulk copy global -> this CTA's shared memory, completion on an mbarrier.
__device__ __forceinline__ void bulkLoad(void* smemDst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smemAddr(smemDst)),
      "l"(gsrc), "r"(bytes), "r"(smemAddr(bar))
      : "memory");
}
// Bulk copy this CTA's shared memory -> global (local or peer), tracked by bulk groups.
__device__ __forceinline__ void bulkStore(void* gdst, const void* smemSrc, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst),
               "r"(smemAddr(smemSrc)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulkCommit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulkWaitRead() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulkWaitAll() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fenceProxyAsync() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void storeReleaseSys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t loadAcquireSys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t globalTimerNs() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// ---- self-checking build ------------------------------------------------------------------------
// With -DTPB_DEBUG_KERNELS every address the copy paths compute is compared with the byte range
// its table entry declares before it is used; an address outside is counted and the access is
// skipped, so a wrong index shows up as a number the host can read (boundsViolations()) and never
// as a fault. compute-sanitizer plays this role elsewhere; here the kernel checks itself.
#ifdef TPB_DEBUG_KERNELS
__device__ unsigned long long gBoundsViolations = 0;
__device__ __forceinline__ bool dbgInside(const void* p, uint64_t n, const void* base, uint64_t span) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(base);
  if (a >= b && a - b <= span && n <= span - (a - b)) return true;
  atomicAdd(&gBoundsViolations, 1ull);
  return false;
}
#define TPB_DBG_INSIDE(p, n, base, span) dbgInside(p, n, base, span)
#else
#define TPB_DBG_INSIDE(p, n, base, span) true
#endif

// ---- parameters ---------------------------------------------------------------------------------
template <int N>
struct PushParams {
  PushEntry entries[N];
  uint32_t numEntries;
  uint32_t bulkTiles;
  uint32_t plainTiles;
  uint32_t blockTiles;
  uint32_t* flag;
  uint32_t* counter;
  uint32_t* status;
  uint32_t bulkTileBytes;
  uint32_t bulkStages;
  uint32_t warpTileBytes;  // shared memory per register-path warp (0 when no entry needs staging)
  uint32_t flagValue;
  // Optional: nothing is read before *waitFlag has reached waitValue (cyclic comparison) or the
  // time limit has passed; used by a receiver that unpacks what another GPU is still delivering.
  const uint32_t* waitFlag;
  uint32_t waitValue;
  uint64_t waitTimeoutNs;
  // Optional: a word (mapped host memory) that receives doneValue once every CTA of the launch
  // has finished, whether the launch succeeded or gave up: the host's cheap way to learn that a
  // launch is over without an event.
  uint32_t* doneSlot;
  uint32_t doneValue;
  // When the kernel behind this one on the stream may be let go (see letDependentsLaunch):
  // 0 = at the start, 1 = when this CTA has issued all its work and is about to report in.
  uint32_t lateTrigger;
};
// Handing the parameters over is part of every launch's cost, in steps: with 752 bytes instead of 736, messages of 4 KiB
// streamed through a pipe on one GPU took 7.2 us each instead of 6.4, half a round trip 18.9 instead of 18.4.
static_assert(sizeof(PushParams<kMaxEntriesSmall>) <= 736, "the small parameter block");

// The arrive counter of a launch doubles as its failure latch: the low half counts CTAs that
// have reported in, every CTA that gave up adds one to the high half.
constexpr uint32_t kArriveMask = 0xffffu;
constexpr uint32_t kArriveFailed = 0x10000u;

__device__ __forceinline__ void reportStatus(uint32_t* status, uint32_t code) {
  // The word may live in mapped host memory, where only a plain store is certain to be seen
  // by the CPU; codes are never cleared by a kernel, so the order of racing writers is moot.
  if (status) {
    *reinterpret_cast<volatile uint32_t*>(status) = code;
    __threadfence_system();
  }
}

template <int N>
__device__ __forceinline__ const PushEntry* findEntry(const PushParams<N>& p, uint32_t tile, TileClass wanted) {
  // Entries of one class have increasing tileStart; a linear scan over <=96 entries in the
  // constant bank (uniform across the warp) costs less than the tile it locates.
  for (uint32_t i = 0; i < p.numEntries; ++i) {
    const PushEntry& e = p.entries[i];
    if (tileClassOf(e.kind) != wanted) continue;
    if (tile - e.tileStart < e.numTiles) return &e;
  }
  return nullptr;
}

// ---- conversions --------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float toFloat(T v);
template <>
__device__ __forceinline__ float toFloat<float>(float v) { return v; }
template <>
__device__ __forceinline__ float toFloat<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float toFloat<__half>(__half v) { return __half2float(v); }
template <typename T>
__device__ __forceinline__ T fromFloat(float v);
template <>
__device__ __forceinline__ float fromFloat<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 fromFloat<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half fromFloat<__half>(float v) { return __float2half_rn(v); }

// ---- plain contiguous copy: one warp, one 8 KiB tile ----------------------------------------------
// Bound by memory. The two ends of a tile may lie at any alignment relative to each other (a slice of
// a flat buffer sent into a fresh allocation): warpCopyRun moves it with 16-byte loads and stores all
// the same. Tiles meet on 16-byte boundaries of the destination, so only an entry's own ends are
// ragged. (Five bf16 slices at odd offsets, 238 MB: 142 us with loads as wide as both ends' common
// alignment, 78 us now.)
template <bool kShifted>
__device__ __forceinline__ void copyPlainTilesTyped(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  const uint8_t* from = static_cast<const uint8_t*>(e.src);
  uint8_t* to = static_cast<uint8_t*>(e.dst);
  const uint64_t count = e.count;
  const uint32_t numTiles = e.numTiles, skew = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(to) & 15);
#pragma unroll 1
  for (uint32_t t = first; t < numTiles; t += step) {
    const uint64_t off = t == 0 ? 0 : static_cast<uint64_t>(t) * kPlainTileBytes - skew;
    const uint64_t end = t + 1 == numTiles ? count : (static_cast<uint64_t>(t) + 1) * kPlainTileBytes - skew;
    const uint32_t bytes = static_cast<uint32_t>(end - off);
    if (!TPB_DBG_INSIDE(from + off, bytes, e.src, count) || !TPB_DBG_INSIDE(to + off, bytes, e.dst, count)) return;
    warpCopyRun<kShifted>(from + off, to + off, bytes, lane);
  }
}

// The shifted form is a function of its own: it needs more registers than the rest of the kernel,
// and a small aligned message should not fetch its instructions.
__device__ __noinline__ void copyShiftedTiles(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  copyPlainTilesTyped<true>(e, first, step, lane);
}
__device__ __forceinline__ void copyPlainTiles(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  if ((reinterpret_cast<uintptr_t>(e.src) ^ reinterpret_cast<uintptr_t>(e.dst)) & 15) copyShiftedTiles(e, first, step, lane);
  else copyPlainTilesTyped<false>(e, first, step, lane);
}

// ---- contiguous conversion ----------------------------------------------------------------------
// Bound by memory. A lane's unit is as many elements as fill 16 bytes of the wider type, so that every
// load and every store of a warp covers one contiguous stretch (512 bytes on the wide side, 256 or 512 on the
// narrow one), and eight loads per lane are in flight before the first unit is converted.
// (A transformer layer of width 4096, 12 tensors, 201 M elements: fp32 -> bf16 255 us with one 32-byte load per
// lane and step, 195 us now; bf16 -> fp32 307 us with one 16-byte load, 200 us now; the HBM floor is 184.)
template <typename S, typename D>
__device__ __forceinline__ void castUnits(const S* s, D* d, uint32_t units, int lane) {
  constexpr int kUnit = 16 / (sizeof(S) > sizeof(D) ? sizeof(S) : sizeof(D));
  constexpr int U = 8;
  struct alignas(kUnit * sizeof(S)) In { S v[kUnit]; };
  struct alignas(kUnit * sizeof(D)) Out { D v[kUnit]; };
  const In* in = reinterpret_cast<const In*>(s);
  Out* out = reinterpret_cast<Out*>(d);
  auto converted = [](const In& x) {
    Out o;
#pragma unroll
    for (int k = 0; k < kUnit; ++k) o.v[k] = fromFloat<D>(toFloat<S>(x.v[k]));
    return o;
  };
  uint32_t i = lane;
#pragma unroll 1
  for (; i + (U - 1) * 32 < units; i += U * 32) {
    In r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) r[u] = in[i + u * 32];
#pragma unroll
    for (int u = 0; u < U; ++u) out[i + u * 32] = converted(r[u]);
  }
#pragma unroll 1
  for (; i < units; i += 32) out[i] = converted(in[i]);
}

// Element by element, for ends that no unit fills and for sources and destinations that are not both
// aligned to a unit; eight loads in flight per lane.
template <typename S, typename D>
__device__ __forceinline__ void castElements(const S* s, D* d, uint32_t n, int lane) {
  constexpr int U = 8;
  uint32_t i = lane;
#pragma unroll 1
  for (; i + (U - 1) * 32 < n; i += U * 32) {
    S r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) r[u] = s[i + u * 32];
#pragma unroll
    for (int u = 0; u < U; ++u) d[i + u * 32] = fromFloat<D>(toFloat<S>(r[u]));
  }
#pragma unroll 1
  for (; i < n; i += 32) d[i] = fromFloat<D>(toFloat<S>(s[i]));
}

template <typename S, typename D>
__device__ __noinline__ void castTilesTyped(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  constexpr uint32_t perTile = kPlainTileBytes / sizeof(D);  // a tile is kPlainTileBytes of DESTINATION bytes
  constexpr int kUnit = 16 / (sizeof(S) > sizeof(D) ? sizeof(S) : sizeof(D));
  const S* const from = static_cast<const S*>(e.src);
  D* const to = static_cast<D*>(e.dst);
  const uint64_t count = e.count;
  const uint32_t numTiles = e.numTiles;
  const bool aligned = reinterpret_cast<uintptr_t>(from) % (kUnit * sizeof(S)) == 0 &&
      reinterpret_cast<uintptr_t>(to) % (kUnit * sizeof(D)) == 0;
#pragma unroll 1
  for (uint32_t t = first; t < numTiles; t += step) {
    const uint64_t at = static_cast<uint64_t>(t) * perTile;
    const uint32_t n = count - at > perTile ? perTile : static_cast<uint32_t>(count - at);
    const S* s = from + at;
    D* d = to + at;
    if (!TPB_DBG_INSIDE(s, uint64_t(n) * sizeof(S), e.src, count * sizeof(S)) ||
        !TPB_DBG_INSIDE(d, uint64_t(n) * sizeof(D), e.dst, count * sizeof(D)))
      return;
    const uint32_t units = aligned ? n / kUnit : 0;
    castUnits<S, D>(s, d, units, lane);
    castElements<S, D>(s + units * kUnit, d + units * kUnit, n - units * kUnit, lane);
  }
}

__device__ __forceinline__ void castTiles(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  const uint32_t key = (static_cast<uint32_t>(e.srcDtype) << 8) | e.dstDtype;
  constexpr uint32_t F32 = static_cast<uint32_t>(DType::kF32), BF = static_cast<uint32_t>(DType::kBF16),
                     F16 = static_cast<uint32_t>(DType::kF16);
  switch (key) {
    case (F32 << 8) | BF: castTilesTyped<float, __nv_bfloat16>(e, first, step, lane); break;
    case (F32 << 8) | F16: castTilesTyped<float, __half>(e, first, step, lane); break;
    case (BF << 8) | F32: castTilesTyped<__nv_bfloat16, float>(e, first, step, lane); break;
    case (F16 << 8) | F32: castTilesTyped<__half, float>(e, first, step, lane); break;
    case (BF << 8) | F16: castTilesTyped<__nv_bfloat16, __half>(e, first, step, lane); break;
    case (F16 << 8) | BF: castTilesTyped<__half, __nv_bfloat16>(e, first, step, lane); break;
    default: break;  // rejected on the host
  }
}

// ---- 2-D source whose rows are contiguous (a column shard of a row-major matrix) ---------------------
// Bound by memory. The packed result is one contiguous run, so it is cut into 8 KiB tiles that meet on
// 16-byte boundaries of the destination, whatever the length of a row, and every lane finds the source of its
// 16-byte vector: one row's bytes as a rule, the end of one row and the start of the next where a vector
// straddles them. Nothing goes through shared memory. (Four shards of 16384 x 2048 bf16 out of
// rows of 8192, 537 MB: 457 us as 32x32 tiles of 2-byte accesses, 87 us now, 0.94 of the HBM rate; 2047 columns out
// of 8191: 452 -> 132 us; fp32 -> bf16: 476 -> 131 us.)
struct RowCursor {
  const uint8_t* row;  // start of the row
  uint32_t at;         // bytes (or elements) into it
};

// 16 bytes from `p`, of which only bytes [from, to) are needed: aligned chunks without a needed byte are not
// touched, and what stands in the other bytes is unspecified.
__device__ __forceinline__ uint4 loadBytes16(const uint8_t* p, uint32_t from, uint32_t to) {
  const uint32_t d = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p) & 15);
  const uint4* c = reinterpret_cast<const uint4*>(p - d);
  uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
  if (from + d < 16) lo = c[0];
  if (to + d > 16) hi = c[1];
  uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  if (d & 8) {
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = w[k + 2];
  }
  if (d & 4) {
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] = w[k + 1];
  }
  const uint32_t bits = (d & 3) * 8;
  return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits), __funnelshift_r(w[2], w[3], bits),
                    __funnelshift_r(w[3], w[4], bits));
}
__device__ __forceinline__ uint32_t mergeWord(uint32_t first, uint32_t rest, int bytesOfFirst) {
  if (bytesOfFirst >= 4) return first;
  if (bytesOfFirst <= 0) return rest;
  const uint32_t mask = (1u << (8 * bytesOfFirst)) - 1;
  return (first & mask) | (rest & ~mask);
}

// kAligned: source, destination, pitch and row length are multiples of 16 bytes.
template <bool kAligned>
__device__ __noinline__ void rowCopyTiles(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  const uint8_t* const src = static_cast<const uint8_t*>(e.src);
  uint8_t* const dst = static_cast<uint8_t*>(e.dst);
  const uint32_t rowBytes = static_cast<uint32_t>(e.cols) * e.srcElemSize;  // the host keeps it below 2^31
  const int64_t pitch = e.rowStride * e.srcElemSize;
  const uint64_t total = static_cast<uint64_t>(e.rows) * rowBytes;
  [[maybe_unused]] const uint64_t span = static_cast<uint64_t>(e.rows - 1) * pitch + rowBytes;
  const uint32_t numTiles = e.numTiles, tileBytes = e.rowTileBytes, skew = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(dst) & 15);
  const uint32_t stepRows = 512 / rowBytes, stepBytes = 512 - stepRows * rowBytes;  // 32 lanes x 16 bytes further on
  const int64_t stepPitch = pitch * stepRows;
  auto cursorAt = [&](uint64_t x) {
    const uint64_t r = total >> 32 ? x / rowBytes : static_cast<uint32_t>(x) / rowBytes;
    return RowCursor{src + static_cast<int64_t>(r) * pitch, static_cast<uint32_t>(x - r * rowBytes)};
  };
  auto advance = [&](RowCursor& c) {
    c.row += stepPitch;
    c.at += stepBytes;
    if (c.at >= rowBytes) {
      c.at -= rowBytes;
      c.row += pitch;
    }
  };
#pragma unroll 1
  for (uint32_t t = first; t < numTiles; t += step) {
    const uint64_t off = t == 0 ? 0 : static_cast<uint64_t>(t) * tileBytes - skew;
    const uint64_t end = t + 1 == numTiles ? total : (static_cast<uint64_t>(t) + 1) * tileBytes - skew;
    const uint32_t bytes = static_cast<uint32_t>(end - off);
    uint32_t head = t == 0 ? (16 - skew) & 15 : 0;
    if (head > bytes) head = bytes;
    const uint32_t vectors = (bytes - head) / 16, done = head + vectors * 16;
    if (!kAligned) {  // the ragged ends of the whole result
      if (static_cast<uint32_t>(lane) < head) {
        const RowCursor c = cursorAt(off + lane);
        if (TPB_DBG_INSIDE(dst + off + lane, 1, dst, total)) dst[off + lane] = c.row[c.at];
      }
      if (done + lane < bytes) {
        const RowCursor c = cursorAt(off + done + lane);
        if (TPB_DBG_INSIDE(dst + off + done + lane, 1, dst, total)) dst[off + done + lane] = c.row[c.at];
      }
    }
    if (vectors == 0) continue;
    RowCursor c = cursorAt(off + head + static_cast<uint64_t>(lane) * 16);
    uint4* out = reinterpret_cast<uint4*>(dst + off + head);
    uint32_t i = lane;
    // What is left of a vector in its row: below 16 it straddles into the next row.
    auto finish = [&](uint4 v, const RowCursor& from) {
      const int left = static_cast<int>(rowBytes - from.at);
      if (left < 16 && TPB_DBG_INSIDE(from.row + pitch, 16 - left, src, span)) {
        const uint4 n = loadBytes16(from.row + pitch - left, left, 16);
        v = make_uint4(mergeWord(v.x, n.x, left), mergeWord(v.y, n.y, left - 4), mergeWord(v.z, n.z, left - 8),
                       mergeWord(v.w, n.w, left - 12));
      }
      return v;
    };
    auto load = [&](const RowCursor& from) {
      const uint32_t left = rowBytes - from.at, n = left < 16 ? left : 16;
      if (!TPB_DBG_INSIDE(from.row + from.at, n, src, span)) return make_uint4(0, 0, 0, 0);
      if constexpr (kAligned) return *reinterpret_cast<const uint4*>(from.row + from.at);
      else return loadBytes16(from.row + from.at, 0, n);
    };
    auto batches = [&](auto size) {  // as many whole batches of vectors i, i + 32, ... as there are
      constexpr int U = decltype(size)::value;
#pragma unroll 1
      for (; i + (U - 1) * 32 < vectors; i += U * 32) {
        uint4 v[U];
        RowCursor from[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          from[u] = c;
          v[u] = load(c);
          advance(c);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if constexpr (!kAligned) v[u] = finish(v[u], from[u]);
          if (TPB_DBG_INSIDE(out + i + u * 32, 16, dst, total)) out[i + u * 32] = v[u];
        }
      }
    };
    batches(std::integral_constant<int, kAligned ? 8 : 4>());
    batches(std::integral_constant<int, 2>());
    batches(std::integral_constant<int, 1>());
  }
}

// The same with a conversion: kUnit elements per lane where rows and addresses are multiples of that
// unit, else element by element.
template <typename S, typename D, int kUnit>
__device__ __forceinline__ void rowCastTiles(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  struct alignas(kUnit * sizeof(S)) In { S v[kUnit]; };
  struct alignas(kUnit * sizeof(D)) Out { D v[kUnit]; };
  const uint32_t perTile = e.rowTileBytes / static_cast<uint32_t>(sizeof(D));
  const S* const src = static_cast<const S*>(e.src);
  D* const dst = static_cast<D*>(e.dst);
  const uint32_t cols = static_cast<uint32_t>(e.cols), numTiles = e.numTiles;
  const int64_t rowStride = e.rowStride;
  const uint64_t count = e.count;
  const uint32_t stepRows = 32 * kUnit / cols, stepCols = 32 * kUnit - stepRows * cols;
  const int64_t stepStride = rowStride * stepRows;
  [[maybe_unused]] const uint64_t span = (static_cast<uint64_t>(e.rows - 1) * rowStride + cols) * sizeof(S);
#pragma unroll 1
  for (uint32_t t = first; t < numTiles; t += step) {
    const uint64_t at = static_cast<uint64_t>(t) * perTile;
    const uint32_t units = static_cast<uint32_t>(count - at > perTile ? perTile : count - at) / kUnit;
    const uint64_t x = at + static_cast<uint64_t>(lane) * kUnit;
    const uint64_t r = count >> 32 ? x / cols : static_cast<uint32_t>(x) / cols;
    const S* row = src + static_cast<int64_t>(r) * rowStride;
    uint32_t c = static_cast<uint32_t>(x - r * cols);
    Out* out = reinterpret_cast<Out*>(dst + at);
    auto load = [&]() {
      In v = {};
      if (TPB_DBG_INSIDE(row + c, sizeof(In), src, span)) v = *reinterpret_cast<const In*>(row + c);
      row += stepStride;
      c += stepCols;
      if (c >= cols) {
        c -= cols;
        row += rowStride;
      }
      return v;
    };
    auto storeConverted = [&](const In& v, uint32_t i) {
      Out o;
#pragma unroll
      for (int k = 0; k < kUnit; ++k) o.v[k] = fromFloat<D>(toFloat<S>(v.v[k]));
      if (TPB_DBG_INSIDE(out + i, sizeof(Out), dst, count * sizeof(D))) out[i] = o;
    };
    uint32_t i = lane;
    auto batches = [&](auto size) {
      constexpr int U = decltype(size)::value;
#pragma unroll 1
      for (; i + (U - 1) * 32 < units; i += U * 32) {
        In v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = load();
#pragma unroll
        for (int u = 0; u < U; ++u) storeConverted(v[u], i + u * 32);
      }
    };
    batches(std::integral_constant<int, 8>());
    batches(std::integral_constant<int, 2>());
    batches(std::integral_constant<int, 1>());
  }
}
template <typename S, typename D>
__device__ __noinline__ void rowCastTilesTyped(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  constexpr int kUnit = 16 / (sizeof(S) > sizeof(D) ? sizeof(S) : sizeof(D));
  const bool units = e.cols % kUnit == 0 && e.rowStride % kUnit == 0 &&
      reinterpret_cast<uintptr_t>(e.src) % (kUnit * sizeof(S)) == 0 && reinterpret_cast<uintptr_t>(e.dst) % (kUnit * sizeof(D)) == 0;
  if (units) rowCastTiles<S, D, kUnit>(e, first, step, lane);
  else rowCastTiles<S, D, 1>(e, first, step, lane);
}

__device__ __forceinline__ void rowTiles(const PushEntry& e, uint32_t first, uint32_t step, int lane) {
  if (e.srcDtype == e.dstDtype) {
    const uint64_t all = reinterpret_cast<uintptr_t>(e.src) | reinterpret_cast<uintptr_t>(e.dst) |
        static_cast<uint64_t>(e.cols * e.srcElemSize) | static_cast<uint64_t>(e.rowStride * e.srcElemSize);
    if (all & 15) rowCopyTiles<false>(e, first, step, lane);
    else rowCopyTiles<true>(e, first, step, lane);
    return;
  }
  const uint32_t key = (static_cast<uint32_t>(e.srcDtype) << 8) | e.dstDtype;
  constexpr uint32_t F32 = static_cast<uint32_t>(DType::kF32), BF = static_cast<uint32_t>(DType::kBF16),
                     F16 = static_cast<uint32_t>(DType::kF16);
  switch (key) {
    case (F32 << 8) | BF: rowCastTilesTyped<float, __nv_bfloat16>(e, first, step, lane); break;
    case (F32 << 8) | F16: rowCastTilesTyped<float, __half>(e, first, step, lane); break;
    case (BF << 8) | F32: rowCastTilesTyped<__nv_bfloat16, float>(e, first, step, lane); break;
    case (F16 << 8) | F32: rowCastTilesTyped<__half, float>(e, first, step, lane); break;
    case (BF << 8) | F16: rowCastTilesTyped<__nv_bfloat16, __half>(e, first, step, lane); break;
    case (F16 << 8) | BF: rowCastTilesTyped<__half, __nv_bfloat16>(e, first, step, lane); break;
    default: break;
  }
}

// ---- 2-D strided source through a per-warp shared-memory tile ------------------------------------
// A warp stages TR x 32 raw source elements as tile[c][r] (row stride TR+1 words keeps both access
// patterns free of bank conflicts for 4-byte elements), reading along whichever source dimension is
// contiguous, then writes rows of the packed destination: 32 consecutive elements per store.
// The entry lives in the kernel's parameter block and is reached through a generic pointer inside
// the tile routines: its fields are read once per call into this pack, or every use inside the
// loops would become a load behind the tile stores.
struct StridedArgs {
  const void* src;
  void* dst;
  int64_t rows, cols, rowStride, colStride;
  uint32_t numTiles;
#ifdef TPB_DEBUG_KERNELS
  uint64_t srcSpan, dstSpan;  // bytes the view covers from src / the packed result covers from dst
#endif
};
__device__ __forceinline__ StridedArgs loadStridedArgs(const PushEntry& e) {
  StridedArgs a{e.src, e.dst, e.rows, e.cols, e.rowStride, e.colStride, e.numTiles};
#ifdef TPB_DEBUG_KERNELS
  // Views with non-negative strides only (what the host accepts): the last element is the farthest.
  a.srcSpan = static_cast<uint64_t>((e.rows - 1) * e.rowStride + (e.cols - 1) * e.colStride + 1) * e.srcElemSize;
  a.dstSpan = static_cast<uint64_t>(e.rows) * e.cols * e.dstElemSize;
#endif
  return a;
}
#ifdef TPB_DEBUG_KERNELS
#define TPB_DBG_SRC(a, p, n) dbgInside(p, n, (a).src, (a).srcSpan)
#define TPB_DBG_DST(a, p, n) dbgInside(p, n, (a).dst, (a).dstSpan)
#else
#define TPB_DBG_SRC(a, p, n) true
#define TPB_DBG_DST(a, p, n) true
#endif

template <typename S, typename D, bool kConvert>
__device__ __forceinline__ void stridedTileTyped(const StridedArgs& a, uint32_t localTile, int lane, uint8_t* tileMem) {
  constexpr int TC = kStridedTile;                                 // columns per tile
  constexpr int TR = sizeof(S) == 8 ? kStridedTile / 2 : kStridedTile;  // rows per tile
  S* tile = reinterpret_cast<S*>(tileMem);
  const int64_t rows = a.rows, cols = a.cols, rowStride = a.rowStride, colStride = a.colStride;
  const S* src = static_cast<const S*>(a.src);
  D* dst = static_cast<D*>(a.dst);
  const uint32_t tilesPerRow = static_cast<uint32_t>((cols + TC - 1) / TC);  // the tile count fits 32 bits
  const int64_t r0 = static_cast<int64_t>(localTile / tilesPerRow) * TR;
  const int64_t c0 = static_cast<int64_t>(localTile % tilesPerRow) * TC;
  const int nr = static_cast<int>(rows - r0 < TR ? rows - r0 : TR);
  const int nc = static_cast<int>(cols - c0 < TC ? cols - c0 : TC);
  const bool rowsFast = (rowStride == 1 || rows == 1) && colStride != 1;
  if (rowsFast && rowStride == 1 && nr == TR && nc == TC) {
    // Full tile of a transposed matrix: no predicates, pointers stepped instead of recomputed,
    // sixteen loads in flight per lane.
    constexpr int kWide = 16;
    const bool act = lane < TR;
    const S* colPtr = src + (r0 + lane) + c0 * colStride;
#pragma unroll 1
    for (int c = 0; c < TC; c += kWide) {
      S v[kWide];
#pragma unroll
      for (int k = 0; k < kWide; ++k)
        if (act && TPB_DBG_SRC(a, colPtr + k * colStride, sizeof(S))) v[k] = colPtr[k * colStride];
      colPtr += kWide * colStride;
#pragma unroll
      for (int k = 0; k < kWide; ++k)
        if (act) tile[(c + k) * (TR + 1) + lane] = v[k];
    }
    __syncwarp();
    D* outPtr = dst + r0 * cols + c0 + lane;
    const S* mine = tile + lane * (TR + 1);
#pragma unroll 1
    for (int r = 0; r < TR; r += kWide) {
      S v[kWide];
#pragma unroll
      for (int k = 0; k < kWide; ++k) v[k] = mine[r + k];
#pragma unroll
      for (int k = 0; k < kWide; ++k) {
        D out;
        if constexpr (kConvert) out = fromFloat<D>(toFloat<S>(v[k]));
        else out = v[k];
        if (TPB_DBG_DST(a, outPtr + k * cols, sizeof(D))) outPtr[k * cols] = out;
      }
      outPtr += kWide * cols;
    }
    __syncwarp();
    return;
  }
  constexpr int kBatch = 4;  // independent loads issued before their results are parked in the tile
  if (rowsFast) {
    // lanes walk down a source column: coalesced reads when the source is a transposed matrix
    for (int rb = 0; rb < nr; rb += 32) {
      const int r = rb + lane;
      const S* colPtr = src + (r0 + r) * rowStride + c0 * colStride;
      for (int c = 0; c < nc; c += kBatch) {
        S v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
          if (r < nr && c + k < nc && TPB_DBG_SRC(a, colPtr + static_cast<int64_t>(c + k) * colStride, sizeof(S)))
            v[k] = colPtr[static_cast<int64_t>(c + k) * colStride];
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
          if (r < nr && c + k < nc) tile[(c + k) * (TR + 1) + r] = v[k];
      }
    }
  } else {
    for (int cb = 0; cb < nc; cb += 32) {
      const int c = cb + lane;
      const S* rowPtr = src + r0 * rowStride + (c0 + c) * colStride;
      for (int r = 0; r < nr; r += kBatch) {
        S v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
          if (c < nc && r + k < nr && TPB_DBG_SRC(a, rowPtr + static_cast<int64_t>(r + k) * rowStride, sizeof(S)))
            v[k] = rowPtr[static_cast<int64_t>(r + k) * rowStride];
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
          if (c < nc && r + k < nr) tile[c * (TR + 1) + r + k] = v[k];
      }
    }
  }
  __syncwarp();
  {
    const int c = lane;  // TC == 32: one column per lane
    D* rowPtr = dst + r0 * cols + c0 + c;
    for (int r = 0; r < nr; r += kBatch) {
      S v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (c < nc && r + k < nr) v[k] = tile[c * (TR + 1) + r + k];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (c < nc && r + k < nr) {
          D out;
          if constexpr (kConvert) out = fromFloat<D>(toFloat<S>(v[k]));
          else out = v[k];
          if (TPB_DBG_DST(a, rowPtr + static_cast<int64_t>(r + k) * cols, sizeof(D)))
            rowPtr[static_cast<int64_t>(r + k) * cols] = out;
        }
      }
    }
  }
  __syncwarp();  // the tile is reused by this warp's next strided tile
}

// Not inlined, one function per element type: inlined they would set the register budget of the
// whole kernel, including the copy loops that want many loads in flight. One call covers all
// of this warp's tiles of the entry (first, first + step, ...): a call saves and restores the
// registers it uses, which per tile would cost more local-memory traffic than the tile's payload.
template <typename S, typename D, bool kConvert>
__device__ __noinline__ void stridedTilesTyped(const PushEntry& a_, uint32_t first, uint32_t step, int lane,
                                               uint8_t* tileMem) {
  const StridedArgs a = loadStridedArgs(a_);
#pragma unroll 1
  for (uint32_t t = first; t < a.numTiles; t += step) stridedTileTyped<S, D, kConvert>(a, t, lane, tileMem);
}

__device__ __forceinline__ void stridedTiles(const PushEntry& a, uint32_t first, uint32_t step, int lane, uint8_t* tileMem) {
  const PushEntry& e = a;
  if (e.srcDtype == e.dstDtype || e.dstDtype == static_cast<uint8_t>(DType::kBytes)) {
    switch (e.srcElemSize) {
      case 1: stridedTilesTyped<uint8_t, uint8_t, false>(a, first, step, lane, tileMem); break;
      case 2: stridedTilesTyped<uint16_t, uint16_t, false>(a, first, step, lane, tileMem); break;
      case 4: stridedTilesTyped<uint32_t, uint32_t, false>(a, first, step, lane, tileMem); break;
      default: stridedTilesTyped<uint64_t, uint64_t, false>(a, first, step, lane, tileMem); break;
    }
    return;
  }
  const uint32_t key = (static_cast<uint32_t>(e.srcDtype) << 8) | e.dstDtype;
  constexpr uint32_t F32 = static_cast<uint32_t>(DType::kF32), BF = static_cast<uint32_t>(DType::kBF16),
                     F16 = static_cast<uint32_t>(DType::kF16);
  switch (key) {
    case (F32 << 8) | BF: stridedTilesTyped<float, __nv_bfloat16, true>(a, first, step, lane, tileMem); break;
    case (F32 << 8) | F16: stridedTilesTyped<float, __half, true>(a, first, step, lane, tileMem); break;
    case (BF << 8) | F32: stridedTilesTyped<__nv_bfloat16, float, true>(a, first, step, lane, tileMem); break;
    case (F16 << 8) | F32: stridedTilesTyped<__half, float, true>(a, first, step, lane, tileMem); break;
    case (BF << 8) | F16: stridedTilesTyped<__nv_bfloat16, __half, true>(a, first, step, lane, tileMem); break;
    case (F16 << 8) | BF: stridedTilesTyped<__half, __nv_bfloat16, true>(a, first, step, lane, tileMem); break;
    default: break;
  }
}

// Transposed matrix with few columns (cols <= 64, rowStride == 1): a tile is 32 whole rows of the
// packed result, i.e. ONE contiguous run of 32 * cols elements in the destination. Lanes read down
// the source columns as usual and park the (already converted) values in 32-bit slots tile[c][r];
// then every lane gathers the 16 bytes of its chunk of the run and stores them as one vector, so a
// warp writes 512 contiguous bytes per instruction instead of one 128-byte row segment. That is
// what a remote GPU's memory wants to see over NVLink. Needs cols * sizeof(D) to be a multiple of
// 16 and a 16-byte aligned destination.
template <typename S, typename D, bool kConvert>
__device__ __forceinline__ void stridedNarrowTile(const StridedArgs& a, uint32_t localTile, int lane, uint8_t* tileMem) {
  constexpr int TR = 32, P = TR + 1;
  constexpr int K = 16 / sizeof(D);  // destination elements per 16-byte chunk
  uint32_t* tile = reinterpret_cast<uint32_t*>(tileMem);
  const int64_t rows = a.rows, colStride = a.colStride;
  const int cols = static_cast<int>(a.cols);
  const S* src = static_cast<const S*>(a.src);
  D* dst = static_cast<D*>(a.dst);
  const int64_t r0 = static_cast<int64_t>(localTile) * TR;
  const int nr = static_cast<int>(rows - r0 < TR ? rows - r0 : TR);
  constexpr int kBatch = 16;
  {
    const bool act = lane < nr;
    const S* colPtr = src + (r0 + lane);
    for (int c = 0; c < cols; c += kBatch) {
      S v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (act && c + k < cols && TPB_DBG_SRC(a, colPtr + static_cast<int64_t>(c + k) * colStride, sizeof(S)))
          v[k] = colPtr[static_cast<int64_t>(c + k) * colStride];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (act && c + k < cols) {
          D out;
          if constexpr (kConvert) out = fromFloat<D>(toFloat<S>(v[k]));
          else out = v[k];
          uint32_t bits = 0;
          if constexpr (sizeof(D) == 4) bits = *reinterpret_cast<const uint32_t*>(&out);
          else if constexpr (sizeof(D) == 2) bits = *reinterpret_cast<const uint16_t*>(&out);
          else bits = *reinterpret_cast<const uint8_t*>(&out);
          tile[(c + k) * P + lane] = bits;
        }
      }
    }
  }
  __syncwarp();
  {
    const int chunksPerRow = cols / K;
    const int chunks = nr * chunksPerRow;
    uint4* out = reinterpret_cast<uint4*>(dst + r0 * cols);
    // (r, c) of chunk q, advanced by 32 chunks per step without dividing in the loop.
    int r = lane / chunksPerRow;
    int cc = lane - r * chunksPerRow;  // chunk index within its row
    const int stepRows = 32 / chunksPerRow, stepChunks = 32 - stepRows * chunksPerRow;
    for (int q = lane; q < chunks; q += 32) {
      const int c = cc * K;
      alignas(16) D vals[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const uint32_t bits = tile[(c + k) * P + r];
        if constexpr (sizeof(D) == 4) vals[k] = *reinterpret_cast<const D*>(&bits);
        else if constexpr (sizeof(D) == 2) {
          const uint16_t h = static_cast<uint16_t>(bits);
          vals[k] = *reinterpret_cast<const D*>(&h);
        } else {
          const uint8_t b = static_cast<uint8_t>(bits);
          vals[k] = *reinterpret_cast<const D*>(&b);
        }
      }
      if (TPB_DBG_DST(a, out + q, 16)) out[q] = *reinterpret_cast<const uint4*>(vals);
      r += stepRows;
      cc += stepChunks;
      if (cc >= chunksPerRow) {
        cc -= chunksPerRow;
        ++r;
      }
    }
  }
  __syncwarp();
}

template <typename S, typename D, bool kConvert>
__device__ __noinline__ void stridedNarrowTilesTyped(const PushEntry& e, uint32_t first, uint32_t step, int lane,
                                                     uint8_t* tileMem) {
  const StridedArgs a = loadStridedArgs(e);
#pragma unroll 1
  for (uint32_t t = first; t < a.numTiles; t += step) stridedNarrowTile<S, D, kConvert>(a, t, lane, tileMem);
}

__device__ __forceinline__ void stridedNarrowTiles(const PushEntry& e, uint32_t first, uint32_t step, int lane,
                                                   uint8_t* tileMem) {
  if (e.srcDtype == e.dstDtype || e.dstDtype == static_cast<uint8_t>(DType::kBytes)) {
    switch (e.srcElemSize) {
      case 1: stridedNarrowTilesTyped<uint8_t, uint8_t, false>(e, first, step, lane, tileMem); break;
      case 2: stridedNarrowTilesTyped<uint16_t, uint16_t, false>(e, first, step, lane, tileMem); break;
      default: stridedNarrowTilesTyped<uint32_t, uint32_t, false>(e, first, step, lane, tileMem); break;
    }
    return;
  }
  const uint32_t key = (static_cast<uint32_t>(e.srcDtype) << 8) | e.dstDtype;
  constexpr uint32_t F32 = static_cast<uint32_t>(DType::kF32), BF = static_cast<uint32_t>(DType::kBF16),
                     F16 = static_cast<uint32_t>(DType::kF16);
  switch (key) {
    case (F32 << 8) | BF: stridedNarrowTilesTyped<float, __nv_bfloat16, true>(e, first, step, lane, tileMem); break;
    case (F32 << 8) | F16: stridedNarrowTilesTyped<float, __half, true>(e, first, step, lane, tileMem); break;
    case (BF << 8) | F32: stridedNarrowTilesTyped<__nv_bfloat16, float, true>(e, first, step, lane, tileMem); break;
    case (F16 << 8) | F32: stridedNarrowTilesTyped<__half, float, true>(e, first, step, lane, tileMem); break;
    case (BF << 8) | F16: stridedNarrowTilesTyped<__nv_bfloat16, __half, true>(e, first, step, lane, tileMem); break;
    case (F16 << 8) | BF: stridedNarrowTilesTyped<__half, __nv_bfloat16, true>(e, first, step, lane, tileMem); break;
    default: break;
  }
}

// Transposed matrix (rowStride == 1) whose packed rows are at most 8 KiB, for destinations that
// want long contiguous writes (another GPU's memory over NVLink, where a 64-byte or misaligned
// 128-byte row segment costs a whole packet): a tile is a band of whole rows, as many as fit in
// 8 KiB. The band's elements are gathered down the source columns (consecutive rows of one column
// are adjacent in the source: coalesced, the more so the more rows a band has), converted, and laid
// out in shared memory exactly as the destination wants them, at the destination's own alignment
// modulo 16; the band then leaves as ONE contiguous run: bytes up to the first 16-byte boundary,
// 16-byte vectors, bytes after the last one. No alignment or divisibility is asked of anything.
template <typename S, typename D, bool kConvert>
__device__ __forceinline__ void stridedBandTile(const StridedArgs& a, uint32_t band, uint32_t bandRowsCount, int lane,
                                                uint8_t* tileMem) {
  const int64_t rows = a.rows, colStride = a.colStride;
  const uint32_t cols = static_cast<uint32_t>(a.cols);
  const S* src = static_cast<const S*>(a.src);
  const int64_t r0 = static_cast<int64_t>(band) * bandRowsCount;
  const uint32_t nr = static_cast<uint32_t>(rows - r0 < bandRowsCount ? rows - r0 : bandRowsCount);
  uint8_t* out = static_cast<uint8_t*>(a.dst) + static_cast<uint64_t>(r0) * cols * sizeof(D);
  const uint32_t skew = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(out) & 15);  // a multiple of sizeof(D)
  D* stage = reinterpret_cast<D*>(tileMem + skew);
  const uint32_t n = nr * cols;  // elements of this band
  // Gather: element q of the (c-major, r-minor) enumeration is (c, r) = (q / nr, q % nr); lanes take
  // q = lane, lane + 32, ... and keep (c, r) up to date without dividing in the loop.
  {
    constexpr int kBatch = 8;
    uint32_t c = lane / nr, r = lane - c * nr;
    const uint32_t stepC = 32 / nr, stepR = 32 - stepC * nr;
    for (uint32_t q = lane; q < n; q += 32 * kBatch) {
      S v[kBatch];
      uint32_t cs[kBatch], rs[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        cs[k] = c;
        rs[k] = r;
        if (q + 32 * k < n && TPB_DBG_SRC(a, src + static_cast<int64_t>(c) * colStride + r0 + r, sizeof(S)))
          v[k] = src[static_cast<int64_t>(c) * colStride + r0 + r];
        c += stepC;
        r += stepR;
        if (r >= nr) {
          r -= nr;
          ++c;
        }
      }
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (q + 32 * k < n) {
          D o;
          if constexpr (kConvert) o = fromFloat<D>(toFloat<S>(v[k]));
          else o = v[k];
          stage[rs[k] * cols + cs[k]] = o;
        }
      }
    }
  }
  __syncwarp();
  {
    const uint32_t bytes = n * static_cast<uint32_t>(sizeof(D));
    const uint8_t* from = tileMem + skew;
    // head: up to the first 16-byte boundary of the destination (and of the staging area: same skew)
    const uint32_t head = skew == 0 ? 0 : (16 - skew < bytes ? 16 - skew : bytes);
    if (static_cast<uint32_t>(lane) < head && TPB_DBG_DST(a, out + lane, 1)) out[lane] = from[lane];
    const uint32_t vectors = (bytes - head) / 16;
    const uint4* vfrom = reinterpret_cast<const uint4*>(from + head);
    uint4* vout = reinterpret_cast<uint4*>(out + head);
    for (uint32_t i = lane; i < vectors; i += 32)
      if (TPB_DBG_DST(a, vout + i, 16)) vout[i] = vfrom[i];
    const uint32_t done = head + vectors * 16;
    if (done + lane < bytes && TPB_DBG_DST(a, out + done + lane, 1)) out[done + lane] = from[done + lane];
  }
  __syncwarp();  // the staging area is reused by this warp's next band
}

template <typename S, typename D, bool kConvert>
__device__ __noinline__ void stridedBandTilesTyped(const PushEntry& e, uint32_t first, uint32_t step, int lane,
                                                   uint8_t* tileMem) {
  const StridedArgs a = loadStridedArgs(e);
  const uint32_t rowsPerBand = bandRows(static_cast<uint64_t>(e.cols), sizeof(D));
#pragma unroll 1
  for (uint32_t t = first; t < a.numTiles; t += step) stridedBandTile<S, D, kConvert>(a, t, rowsPerBand, lane, tileMem);
}

__device__ __forceinline__ void stridedBandTiles(const PushEntry& e, uint32_t first, uint32_t step, int lane,
                                                 uint8_t* tileMem) {
  if (e.srcDtype == e.dstDtype || e.dstDtype == static_cast<uint8_t>(DType::kBytes)) {
    switch (e.srcElemSize) {
      case 1: stridedBandTilesTyped<uint8_t, uint8_t, false>(e, first, step, lane, tileMem); break;
      case 2: stridedBandTilesTyped<uint16_t, uint16_t, false>(e, first, step, lane, tileMem); break;
      case 4: stridedBandTilesTyped<uint32_t, uint32_t, false>(e, first, step, lane, tileMem); break;
      default: stridedBandTilesTyped<uint64_t, uint64_t, false>(e, first, step, lane, tileMem); break;
    }
    return;
  }
  const uint32_t key = (static_cast<uint32_t>(e.srcDtype) << 8) | e.dstDtype;
  constexpr uint32_t F32 = static_cast<uint32_t>(DType::kF32), BF = static_cast<uint32_t>(DType::kBF16),
                     F16 = static_cast<uint32_t>(DType::kF16);
  switch (key) {
    case (F32 << 8) | BF: stridedBandTilesTyped<float, __nv_bfloat16, true>(e, first, step, lane, tileMem); break;
    case (F32 << 8) | F16: stridedBandTilesTyped<float, __half, true>(e, first, step, lane, tileMem); break;
    case (BF << 8) | F32: stridedBandTilesTyped<__nv_bfloat16, float, true>(e, first, step, lane, tileMem); break;
    case (F16 << 8) | F32: stridedBandTilesTyped<__half, float, true>(e, first, step, lane, tileMem); break;
    case (BF << 8) | F16: stridedBandTilesTyped<__nv_bfloat16, __half, true>(e, first, step, lane, tileMem); break;
    case (F16 << 8) | BF: stridedBandTilesTyped<__half, __nv_bfloat16, true>(e, first, step, lane, tileMem); break;
    default: break;
  }
}

// Transposed matrix of 2-byte elements (rowStride == 1), with the source, the destination, both
// extents and the column stride all even: a warp moves a 64x64 tile, reading 32-bit words down the
// source columns (128 B per instruction instead of 64) and writing 32-bit words along the packed
// rows. Staged as tile[c][r] with an even pitch, so a word of two rows lands on an aligned word.
__device__ __forceinline__ void stridedWide16Tile(const StridedArgs& a, uint32_t localTile, int lane, uint8_t* tileMem) {
  constexpr int T = kWideTile, P = kWidePitch;
  const uint16_t* tile = reinterpret_cast<const uint16_t*>(tileMem);
  uint32_t* tileWords = reinterpret_cast<uint32_t*>(tileMem);
  const int64_t rows = a.rows, cols = a.cols, colStride = a.colStride;
  const uint16_t* src = static_cast<const uint16_t*>(a.src);
  uint16_t* dst = static_cast<uint16_t*>(a.dst);
  const uint32_t tilesPerRow = static_cast<uint32_t>((cols + T - 1) / T);
  const int64_t r0 = static_cast<int64_t>(localTile / tilesPerRow) * T;
  const int64_t c0 = static_cast<int64_t>(localTile % tilesPerRow) * T;
  const int nr = static_cast<int>(rows - r0 < T ? rows - r0 : T);  // even
  const int nc = static_cast<int>(cols - c0 < T ? cols - c0 : T);  // even
  constexpr int kBatch = 16;
  const uint16_t* colPtr = src + (r0 + 2 * lane) + c0 * colStride;
  uint32_t* rowPtr = reinterpret_cast<uint32_t*>(dst + r0 * cols + c0) + lane;
  const int64_t rowWords = cols / 2;
  const uint16_t* lo = tile + (2 * lane) * P;
  const uint16_t* hi = lo + P;
  if (nr == T && nc == T) {
    // Full tile: no predicates, constant trip counts.
#pragma unroll 1
    for (int c = 0; c < T; c += kBatch) {
      uint32_t v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (TPB_DBG_SRC(a, colPtr + k * colStride, 4)) v[k] = *reinterpret_cast<const uint32_t*>(colPtr + k * colStride);
      colPtr += kBatch * colStride;
#pragma unroll
      for (int k = 0; k < kBatch; ++k) tileWords[(c + k) * (P / 2) + lane] = v[k];
    }
    __syncwarp();
#pragma unroll 1
    for (int r = 0; r < T; r += kBatch) {
      uint32_t v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) v[k] = static_cast<uint32_t>(lo[r + k]) | (static_cast<uint32_t>(hi[r + k]) << 16);
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (TPB_DBG_DST(a, rowPtr + k * rowWords, 4)) rowPtr[k * rowWords] = v[k];
      rowPtr += kBatch * rowWords;
    }
    __syncwarp();
    return;
  }
  {
    const bool active = 2 * lane < nr;
    for (int c = 0; c < nc; c += kBatch) {
      uint32_t v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (active && c + k < nc && TPB_DBG_SRC(a, colPtr + static_cast<int64_t>(c + k) * colStride, 4))
          v[k] = *reinterpret_cast<const uint32_t*>(colPtr + static_cast<int64_t>(c + k) * colStride);
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (active && c + k < nc) tileWords[(c + k) * (P / 2) + lane] = v[k];
    }
  }
  __syncwarp();
  {
    const bool active = 2 * lane < nc;
    for (int r = 0; r < nr; r += kBatch) {
      uint32_t v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (active && r + k < nr) v[k] = static_cast<uint32_t>(lo[r + k]) | (static_cast<uint32_t>(hi[r + k]) << 16);
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (active && r + k < nr && TPB_DBG_DST(a, rowPtr + static_cast<int64_t>(r + k) * rowWords, 4))
          rowPtr[static_cast<int64_t>(r + k) * rowWords] = v[k];
    }
  }
  __syncwarp();
}

__device__ __noinline__ void stridedWide16Tiles(const PushEntry& e, uint32_t first, uint32_t step, int lane,
                                                uint8_t* tileMem) {
  const StridedArgs a = loadStridedArgs(e);
#pragma unroll 1
  for (uint32_t t = first; t < a.numTiles; t += step) stridedWide16Tile(a, t, lane, tileMem);
}

// ---- large transposed matrices (rowStride 1): one tile per CTA, fetched by bulk copies -----------------
// Bound by memory, which runs at its rate only when what it is asked for comes in long pieces and enough of it is
// under way. Eight warps share a tile of 128 slots; a slot is 256 bytes down a source column (128, 64 or 32 rows of
// 2-, 4- or 8-byte elements) and arrives as ONE bulk copy of the 16-byte chunks that hold it, whatever its
// alignment: no registers, no conditions, and two tiles ahead of the one being written. A matrix of more than 64
// columns fills the slots with adjacent columns, and a warp writes its rows in runs of 128 elements; a narrower one
// fills them with several chunks of rows of all its columns, and the tile leaves as one contiguous run.
//
// A slot takes 272 bytes in shared memory: with 16-byte reads the slots of eight consecutive lanes then lie in
// different banks. A lane reads 16 bytes of its own column (8, 4 or 2 rows), shifts them into place if the column
// did not start on a 16-byte boundary, and the warp stores them row by row. For 2-byte destinations a lane takes
// two adjacent columns, so that it stores words; rows off the word grid are shifted on by a shuffle.
// (Kernel times, warp tiles before / now: 2 x 8192 x 8192 fp32 222 / 182 us, 0.90 of the HBM rate; 4 x 8191 x 4097 bf16
// 177 / 122; 2 x 8192 x 4096 int64 231 / 184; fp32 -> bf16 98 / 82; 2 x 4 M x 8 fp32 475 / 97; 2 x 1 M x 50 bf16 363 / 108.)
constexpr int kBlockThreads = 256;  // the warps that share a tile: all of the light kernel, 8 of the full one
constexpr uint32_t kSlotPitch = 272;
constexpr uint32_t kBlockTileBytes = kBlockSlots * kSlotPitch;
constexpr uint32_t kBlockStagesLight = 3;  // 102 KiB: two CTAs on an SM
static_assert(kBlockTileBytes + 64 <= 8 * kWideWarpTileBytes, "one tile fits the eight warps' own staging areas");

__device__ __forceinline__ void blockBarrier() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// The same barrier; tells whether any of the threads came with `bad`.
__device__ __forceinline__ bool blockBarrierAny(bool bad) {
  uint32_t any;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "bar.red.or.pred q, 1, 256, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(any)
      : "r"(static_cast<uint32_t>(bad))
      : "memory");
  return any != 0;
}

template <typename S, typename D, bool kConvert>
__device__ __forceinline__ D convertOne(S v) {
  if constexpr (kConvert) return fromFloat<D>(toFloat<S>(v));
  else return v;
}
template <typename To, typename From>
__device__ __forceinline__ To bitsAs(From v) {
  static_assert(sizeof(To) == sizeof(From), "same size");
  return *reinterpret_cast<const To*>(&v);
}
template <typename D>
__device__ __forceinline__ uint32_t packPair(D lo, D hi) {
  return __byte_perm(bitsAs<uint16_t>(lo), bitsAs<uint16_t>(hi), 0x5410);
}

// The stages of a CTA's block tiles: where they lie and how many tiles have gone through them.
struct BlockPipe {
  uint8_t* buffers;
  uint64_t* full;  // one barrier per stage, kBlockSlots arrivals each
  TileRing ring;
};

template <typename S, typename D, bool kConvert, bool kNarrow>
struct BlockTransposer {
  static constexpr int kRows = 256 / sizeof(S);  // rows of a slot
  static constexpr bool kPairs = sizeof(D) == 2 && !kNarrow;

  const StridedArgs& a;
  BlockPipe& pipe;
  int tid, lane, warp;
  uint32_t n, chunks, tilesC;
  uint32_t myChunk, myColumn;  // what this thread's slot holds
  uint32_t skew[2];            // wide: where in their first 16 bytes this lane's columns start (even, odd of a pair)
  bool anySkew;                // the same for all lanes: some column is off the 16-byte grid

  __device__ __forceinline__ BlockTransposer(const StridedArgs& args, BlockPipe& p, int tid_)
      : a(args), pipe(p), tid(tid_), lane(tid_ & 31), warp(tid_ >> 5) {
    n = static_cast<uint32_t>(a.cols);
    chunks = kNarrow ? kBlockSlots / n : 1;
    tilesC = kNarrow ? 1 : static_cast<uint32_t>((a.cols + kBlockSlots - 1) / kBlockSlots);
    myChunk = kNarrow ? tid / n : 0;
    myColumn = kNarrow ? tid - myChunk * n : tid;
    // Tiles start multiples of 256 bytes down and of 32 columns across: the same in each.
    const uint32_t origin = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(a.src));
    const uint32_t stride = static_cast<uint32_t>(a.colStride) * static_cast<uint32_t>(sizeof(S));
    skew[0] = (origin + (kPairs ? 2 * lane : lane) * stride) & 15;
    skew[1] = (origin + (kPairs ? 2 * lane + 1 : lane) * stride) & 15;
    anySkew = ((origin | stride) & 15) != 0;
  }

  struct Place {
    int64_t r0, c0;
    int nr, nc;  // rows and columns that exist
  };
  __device__ __forceinline__ Place place(uint32_t t) const {
    Place p;
    const int rows = static_cast<int>(chunks) * kRows;
    p.r0 = static_cast<int64_t>(t / tilesC) * rows;
    p.c0 = kNarrow ? 0 : static_cast<int64_t>(t % tilesC) * kBlockSlots;
    p.nr = static_cast<int>(a.rows - p.r0 < rows ? a.rows - p.r0 : rows);
    p.nc = kNarrow ? static_cast<int>(n) : static_cast<int>(a.cols - p.c0 < kBlockSlots ? a.cols - p.c0 : kBlockSlots);
    return p;
  }

  // One copy per thread of the first kBlockSlots. Every one of them arrives, with the bytes it sends for.
  __device__ __forceinline__ void issue(uint32_t t, uint32_t stage) {
    if (tid >= kBlockSlots) return;
    fenceProxyAsync();  // the stage may have been read until the barrier before this
    const Place p = place(t);
    const int left = p.nr - static_cast<int>(myChunk) * kRows, nr = left < kRows ? left : kRows;
    uint32_t bytes = 0;
    const S* from = static_cast<const S*>(a.src) + p.r0 + static_cast<int64_t>(myChunk) * kRows + (p.c0 + myColumn) * a.colStride;
    const uintptr_t begin = reinterpret_cast<uintptr_t>(from) & ~static_cast<uintptr_t>(15);
    if (static_cast<int>(myColumn) < p.nc && myChunk < chunks && nr > 0 && TPB_DBG_SRC(a, from, nr * sizeof(S)))
      bytes = static_cast<uint32_t>(((reinterpret_cast<uintptr_t>(from + nr) + 15) & ~static_cast<uintptr_t>(15)) - begin);
    // In pairs, the even columns of a group of 64 lie before the odd ones.
    const uint32_t at = kPairs ? (tid & ~63u) + ((tid & 63u) >> 1) + 32 * (tid & 1u) : tid;
    mbarExpectTx(&pipe.full[stage], bytes);
    if (bytes)
      bulkLoad(pipe.buffers + stage * kBlockTileBytes + at * kSlotPitch, reinterpret_cast<const void*>(begin), bytes, &pipe.full[stage]);
  }

  // 16 bytes of a slot, `by` bytes (a multiple of the element size, below 16) behind the 16-byte boundary `chunk`.
  __device__ __forceinline__ void window(const uint4* chunk, uint32_t by, uint32_t (&w)[4]) const {
    const uint4 lo = chunk[0];
    w[0] = lo.x, w[1] = lo.y, w[2] = lo.z, w[3] = lo.w;
    if (!anySkew) return;
    const uint4 hi = chunk[1];
    uint32_t x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int k = 0; k < 6; ++k) x[k] = by & 8 ? x[k + 2] : x[k];
    if constexpr (sizeof(S) <= 4) {
#pragma unroll
      for (int k = 0; k < 5; ++k) x[k] = by & 4 ? x[k + 1] : x[k];
    }
    const uint32_t bits = (by & 2) * 8;
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = sizeof(S) == 2 ? __funnelshift_r(x[k], x[k + 1], bits) : x[k];
  }

  // Up to 128 columns of one packed row: v[i] is column 32 i + lane, at `mine` + 32 i.
  template <bool kFull>
  __device__ __forceinline__ void storeRow(D* mine, const D (&v)[4], int nc) const {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if ((kFull || 32 * i + lane < nc) && TPB_DBG_DST(a, mine + 32 * i, sizeof(D))) mine[32 * i] = v[i];
  }
  // The same for 2-byte elements: w[i] is columns 64 i + 2 lane and the next, at `mine` + 64 i.
  template <bool kFull>
  __device__ __forceinline__ void storeRowPairs(uint16_t* mine, const uint32_t (&w)[2], int nc) const {
    if ((reinterpret_cast<uintptr_t>(mine) & 2) == 0) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int c = 64 * i + 2 * lane;
        if (kFull || c + 1 < nc) {
          if (TPB_DBG_DST(a, mine + 64 * i, 4)) *reinterpret_cast<uint32_t*>(mine + 64 * i) = w[i];
        } else if (c < nc) {
          if (TPB_DBG_DST(a, mine + 64 * i, 2)) mine[64 * i] = static_cast<uint16_t>(w[i]);
        }
      }
      return;
    }
    // Off the word grid: columns c + 1 and c + 2 make a word (the second comes from the next lane, behind lane 31
    // from lane 0's next group), the first and the last column of the segment go alone.
    const uint32_t behind[2] = {__shfl_sync(0xffffffffu, lane == 0 ? w[1] : w[0], (lane + 1) & 31), __shfl_down_sync(0xffffffffu, w[1], 1)};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = 64 * i + 2 * lane + 1, end = kFull ? kBlockSlots : nc;
      if ((kFull && i == 0) || c + 1 < end) {
        if (TPB_DBG_DST(a, mine + 64 * i + 1, 4)) *reinterpret_cast<uint32_t*>(mine + 64 * i + 1) = __funnelshift_r(w[i], behind[i], 16);
      } else if (c < end) {
        if (TPB_DBG_DST(a, mine + 64 * i + 1, 2)) mine[64 * i + 1] = static_cast<uint16_t>(w[i] >> 16);
      }
    }
    if (lane == 0 && TPB_DBG_DST(a, mine, 2)) *mine = static_cast<uint16_t>(w[0]);
  }

  // Wide: a slot is sixteen windows long, a warp takes two of them across all slots.
  template <bool kFull>
  __device__ __forceinline__ void writeRows(const uint8_t* buffer, const Place& p) const {
    constexpr int kWindowRows = 16 / sizeof(S);  // rows that a lane reads at once
    const int64_t cols = a.cols;
    D* mine = static_cast<D*>(a.dst) + (p.r0 + 2 * warp * kWindowRows) * cols + p.c0 + (kPairs ? 2 * lane : lane);
    const uint4* slot = reinterpret_cast<const uint4*>(buffer + lane * kSlotPitch) + 2 * warp;
    int left = p.nr - 2 * warp * kWindowRows;
#pragma unroll 1
    for (int q = 0; q < 2; ++q, ++slot, left -= kWindowRows) {
      if (!kFull && left <= 0) return;
      uint32_t w[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) window(slot + i * 32 * (kSlotPitch / 16), skew[kPairs ? i & 1 : 0], w[i]);
#pragma unroll
      for (int k = 0; k < kWindowRows; ++k) {
        if (kFull || k < left) {
          auto value = [&](int i) {  // row k of this lane's i-th column
            if constexpr (sizeof(S) == 8) return bitsAs<S>(static_cast<uint64_t>(w[i][2 * k]) | (static_cast<uint64_t>(w[i][2 * k + 1]) << 32));
            else if constexpr (sizeof(S) == 4) return bitsAs<S>(w[i][k]);
            else return bitsAs<S>(static_cast<uint16_t>(w[i][k >> 1] >> (16 * (k & 1))));
          };
          if constexpr (kPairs) {
            uint32_t pairs[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if constexpr (sizeof(S) == 2 && !kConvert) pairs[i] = __byte_perm(w[2 * i][k >> 1], w[2 * i + 1][k >> 1], k & 1 ? 0x7632 : 0x5410);
              else pairs[i] = packPair(convertOne<S, D, kConvert>(value(2 * i)), convertOne<S, D, kConvert>(value(2 * i + 1)));
            }
            storeRowPairs<kFull>(reinterpret_cast<uint16_t*>(mine), pairs, p.nc);
          } else {
            D v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = convertOne<S, D, kConvert>(value(i));
            storeRow<kFull>(mine, v, p.nc);
          }
        }
        mine += cols;
      }
    }
  }

  // Narrow: the tile is one contiguous run of the packed result.
  __device__ __forceinline__ void writeRun(const uint8_t* buffer, const Place& p) const {
    const uint32_t total = static_cast<uint32_t>(p.nr) * n;
    D* out = static_cast<D*>(a.dst) + p.r0 * a.cols;
    uint32_t r = 0, c = 0;
    const uint32_t origin = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(a.src));
    const uint32_t stride = static_cast<uint32_t>(a.colStride) * static_cast<uint32_t>(sizeof(S));
    auto element = [&](uint32_t column) {
      const uint32_t slot = (r / kRows) * n + column;  // tiles and chunks are whole 256 bytes: the same alignment in each
      const uint8_t* at = buffer + slot * kSlotPitch + ((origin + column * stride) & 15) + (r % kRows) * sizeof(S);
      return convertOne<S, D, kConvert>(*reinterpret_cast<const S*>(at));
    };
    if constexpr (sizeof(D) == 2) {
      if (n % 2 == 0 && (reinterpret_cast<uintptr_t>(out) & 3) == 0) {  // two adjacent columns leave as one word
        storeRun<2>(reinterpret_cast<uint32_t*>(out), total / 2, r, c, [&]() { return packPair(element(c), element(c + 1)); });
        return;
      }
    }
    storeRun<1>(out, total, r, c, [&]() { return element(c); });
  }
  // `count` items of kColumns adjacent columns each, one per thread in turn; (r, c) follow.
  template <int kColumns, typename T, typename F>
  __device__ __forceinline__ void storeRun(T* out, uint32_t count, uint32_t& r, uint32_t& c, F&& item) const {
    const uint32_t stepR = kColumns * kBlockThreads / n, stepC = kColumns * kBlockThreads - stepR * n;
    r = kColumns * tid / n;
    c = kColumns * tid - r * n;
    auto next = [&]() {
      const T v = item();
      r += stepR;
      c += stepC;
      if (c >= n) {
        c -= n;
        ++r;
      }
      return v;
    };
    constexpr int U = 8;
    uint32_t q = tid;
#pragma unroll 1
    for (; q + (U - 1) * kBlockThreads < count; q += U * kBlockThreads) {
      T v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = next();
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (TPB_DBG_DST(a, out + q + u * kBlockThreads, sizeof(T))) out[q + u * kBlockThreads] = v[u];
    }
#pragma unroll 1
    for (; q < count; q += kBlockThreads) {
      const T v = next();
      if (TPB_DBG_DST(a, out + q, sizeof(T))) out[q] = v;
    }
  }

  // A warp whose lanes do not all see the tile writes none of it: rows are put together across the lanes.
  __device__ __forceinline__ bool arrived(uint32_t stage, uint32_t parity) {
    return __all_sync(0xffffffffu, mbarWaitBounded(&pipe.full[stage], parity)) != 0;
  }
  // The steps of takeTiles (block_pipe.h), in its order: what holds for a copy that does not arrive is said and tested
  // there. Written out, because called through it the kernel took 2 to 3 % longer (64 MiB of bf16 in 31 columns 45 us
  // instead of 42).
  __device__ __forceinline__ void run(uint32_t first, uint32_t step) {
    uint32_t ahead = first;  // next tile to send for
    for (uint32_t s = 0; s < pipe.ring.stages && ahead < a.numTiles; ++s, ahead += step)
      if (!pipe.ring.failed) issue(ahead, pipe.ring.issued++ % pipe.ring.stages);
#pragma unroll 1
    for (uint32_t t = first; t < a.numTiles; t += step) {
      const uint32_t stage = pipe.ring.taken % pipe.ring.stages;
      if (!pipe.ring.failed) pipe.ring.failed = !arrived(stage, (pipe.ring.taken / pipe.ring.stages) & 1);
      const uint8_t* buffer = pipe.buffers + stage * kBlockTileBytes;
      if (!pipe.ring.failed) {
        ++pipe.ring.taken;
        const Place p = place(t);
        if constexpr (kNarrow) writeRun(buffer, p);
        else if (p.nr == kRows && p.nc == kBlockSlots) writeRows<true>(buffer, p);
        else writeRows<false>(buffer, p);
      }
      blockBarrier();  // everybody is through with this stage
      if (ahead < a.numTiles) {
        if (!pipe.ring.failed) issue(ahead, pipe.ring.issued++ % pipe.ring.stages);
        ahead += step;
      }
    }
  }
};

template <typename S, typename D, bool kConvert, bool kNarrow>
__device__ __noinline__ void blockTilesOfForm(const PushEntry& e, uint32_t first, uint32_t step, int tid, BlockPipe& pipe) {
  const StridedArgs a = loadStridedArgs(e);
  BlockPipe mine = pipe;
  BlockTransposer<S, D, kConvert, kNarrow>(a, mine, tid).run(first, step);
  pipe = mine;
}
template <typename S, typename D, bool kConvert>
__device__ __forceinline__ void blockTilesTyped(const PushEntry& e, uint32_t first, uint32_t step, int tid, BlockPipe& pipe) {
  if (e.cols <= kBlockNarrowCols) blockTilesOfForm<S, D, kConvert, true>(e, first, step, tid, pipe);
  else blockTilesOfForm<S, D, kConvert, false>(e, first, step, tid, pipe);
}

// Block tiles first, first + step, ... of the block class; the kBlockThreads threads of `tid` take part. False,
// for all of them alike, if a copy never completed: not everything was written, the launch reports it, and the memory
// of the stages is not to be used again.
template <int N>
__device__ __forceinline__ bool runBlockTiles(const PushParams<N>& p, uint32_t first, uint32_t step, int tid, uint8_t* mem) {
  constexpr uint32_t F32 = static_cast<uint32_t>(DType::kF32), BF = static_cast<uint32_t>(DType::kBF16),
                     F16 = static_cast<uint32_t>(DType::kF16);
  const uint32_t stages = p.bulkTiles == 0 ? kBlockStagesLight : 1;  // beside the bulk pipeline there is room for one
  BlockPipe pipe{mem, reinterpret_cast<uint64_t*>(mem + stages * kBlockTileBytes), TileRing{stages, 0, 0, false}};
  if (tid == 0) {
    for (uint32_t s = 0; s < stages; ++s) mbarInit(&pipe.full[s], kBlockSlots);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  blockBarrier();
  uint32_t t = first;
  while (t < p.blockTiles) {
    const PushEntry& e = *findEntry(p, t, kBlockClass);
    const uint32_t local = t - e.tileStart;
    if (e.srcDtype == e.dstDtype) {
      switch (e.srcElemSize) {
        case 2: blockTilesTyped<uint16_t, uint16_t, false>(e, local, step, tid, pipe); break;
        case 4: blockTilesTyped<uint32_t, uint32_t, false>(e, local, step, tid, pipe); break;
        default: blockTilesTyped<uint64_t, uint64_t, false>(e, local, step, tid, pipe); break;
      }
    } else {
      switch ((static_cast<uint32_t>(e.srcDtype) << 8) | e.dstDtype) {
        case (F32 << 8) | BF: blockTilesTyped<float, __nv_bfloat16, true>(e, local, step, tid, pipe); break;
        case (F32 << 8) | F16: blockTilesTyped<float, __half, true>(e, local, step, tid, pipe); break;
        case (BF << 8) | F32: blockTilesTyped<__nv_bfloat16, float, true>(e, local, step, tid, pipe); break;
        case (F16 << 8) | F32: blockTilesTyped<__half, float, true>(e, local, step, tid, pipe); break;
        case (BF << 8) | F16: blockTilesTyped<__nv_bfloat16, __half, true>(e, local, step, tid, pipe); break;
        case (F16 << 8) | BF: blockTilesTyped<__half, __nv_bfloat16, true>(e, local, step, tid, pipe); break;
        default: break;
      }
    }
    t += (e.numTiles - local + step - 1) / step * step;
  }
  if (blockBarrierAny(pipe.ring.failed)) {
    if (tid < kBlockSlots)
      waitForCopiesUnderWay(pipe.ring.taken, pipe.ring.issued, pipe.ring.stages,
                            [&](uint32_t stage, uint32_t parity) { mbarWaitBounded(&pipe.full[stage], parity); });
    if (tid == 0) reportStatus(p.status, kStatusBarrierTimeout);
    blockBarrier();
    return false;
  }
  // The memory goes back to the warps' own tiles, behind the copies that were written there.
  if (tid == 0)
    for (uint32_t s = 0; s < stages; ++s) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smemAddr(&pipe.full[s])) : "memory");
  blockBarrier();
  return true;
}

// What a kernel has code for: contiguous copies and conversions; 2-D views moved by single warps too; block tiles too.
enum Forms : int { kContiguousForms = 0, kWarpForms = 1, kAllForms = 2 };

// Warp tiles t = firstWarp, firstWarp + totalWarps, ... of the plain class.
template <int N, int kForms>
__device__ __forceinline__ void runPlainWarp(const PushParams<N>& p, uint32_t firstWarp, uint32_t totalWarps, int lane,
                                             uint8_t* tileMem) {
  uint32_t t = firstWarp;
  while (t < p.plainTiles) {
    const PushEntry* e = findEntry(p, t, kPlainClass);
    const uint32_t local = t - e->tileStart;
    // One call handles every tile of this entry that falls to this warp.
    if (e->kind == kCopyPlain) {
      copyPlainTiles(*e, local, totalWarps, lane);
    } else if (kForms == kContiguousForms || e->kind == kCastPlain) {
      castTiles(*e, local, totalWarps, lane);
    } else if constexpr (kForms != kContiguousForms) {
      if (e->kind == kRows) rowTiles(*e, local, totalWarps, lane);
      else if (e->kind == kStridedWide16) stridedWide16Tiles(*e, local, totalWarps, lane, tileMem);
      else if (e->kind == kStridedNarrow) stridedNarrowTiles(*e, local, totalWarps, lane, tileMem);
      else if (e->kind == kStridedBand) stridedBandTiles(*e, local, totalWarps, lane, tileMem);
      else stridedTiles(*e, local, totalWarps, lane, tileMem);
    }
    t += (e->numTiles - local + totalWarps - 1) / totalWarps * totalWarps;
  }
}

// One lane polls, the CTA learns the outcome. Bounded by the timer and by an iteration cap.
template <int N>
__device__ __forceinline__ bool waitForProducer(const PushParams<N>& p) {
  if (p.waitFlag == nullptr) return true;
  bool arrived = true;
  if (threadIdx.x == 0) {
    arrived = false;
    const uint64_t start = globalTimerNs();
    uint32_t backoff = 32;
    for (uint64_t i = 0; i < (1ull << 32); ++i) {
      if (static_cast<int32_t>(loadAcquireSys(p.waitFlag) - p.waitValue) >= 0) {
        arrived = true;
        break;
      }
      if (globalTimerNs() - start > p.waitTimeoutNs) break;
      __nanosleep(backoff);
      if (backoff < 1024) backoff <<= 1;
    }
    if (!arrived) reportStatus(p.status, kStatusWaitTimeout);
  }
  return __syncthreads_and(arrived) != 0;
}

// Last step of every launch. A launch that gave up anywhere (a bulk load that never completed,
// a producer that never arrived) does NOT publish its flag: whoever waits for it runs into its
// own time limit instead of reading half-written data.
// Programmatic dependent launch: a push kernel lets the kernel queued behind it on the stream start
// right away (its own blocks are on the SMs within microseconds, so "when every block has got
// going" is the moment), and itself waits for the kernel before it only where it first touches
// memory that kernel may have written. Two pushes queued back to back thus overlap the launch
// latency and the prologue of the second with the tail of the first; a kernel that is not launched
// with the attribute (anything of the user's) is serialised as always.
__device__ __forceinline__ void letDependentsLaunch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void waitForEarlierKernels() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void publish(const PushParams<N>& p, bool failedHere) {
  if (p.lateTrigger) letDependentsLaunch();
  if (p.flag == nullptr && p.doneSlot == nullptr) return;
  // Make this thread's writes visible system-wide before the CTA reports in.
  __threadfence_system();
  const bool ctaFailed = __syncthreads_or(failedHere) != 0;
  if (threadIdx.x == 0) {
    bool last = true, anyFailed = ctaFailed;
    if (gridDim.x > 1) {
      const uint32_t mine = 1u + (ctaFailed ? kArriveFailed : 0u);
      const uint32_t before = atomicAdd(p.counter, mine);
      last = (before & kArriveMask) == gridDim.x - 1;
      anyFailed = ((before + mine) & ~kArriveMask) != 0;
      if (last) {
        *p.counter = 0;  // ready for the next launch that is given this counter
        __threadfence_system();
      }
    }
    // With one CTA the barrier above already ordered every write of the launch before this.
    if (last) {
      if (p.flag != nullptr && !anyFailed) storeReleaseSys(p.flag, p.flagValue);
      if (p.doneSlot != nullptr) {
        *reinterpret_cast<volatile uint32_t*>(p.doneSlot) = p.doneValue;
        __threadfence_system();
      }
    }
  }
}

// ---- the kernels --------------------------------------------------------------------------------
template <int N, int kForms>
__global__ void __launch_bounds__(kThreads, 1) tpb_push_pack(const __grid_constant__ PushParams<N> p) {
  extern __shared__ uint8_t smemRaw[];
  // Layout: [bulk stages][warp tiles][mbarriers]; dynamic shared memory is only guaranteed to be
  // 16-byte aligned, the bulk stages want 128.
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 127) & ~static_cast<uintptr_t>(127));
  uint8_t* stages = base;
  uint8_t* warpTiles = base + static_cast<size_t>(p.bulkStages) * p.bulkTileBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(warpTiles + (kThreads / 32 - 1) * p.warpTileBytes);

  const int tid = threadIdx.x;
  const int S = static_cast<int>(p.bulkStages);
  const bool haveBulk = p.bulkTiles > blockIdx.x;
  bool failed = false;

  if (!p.lateTrigger) letDependentsLaunch();
  if (tid == 0 && haveBulk) {
    for (int s = 0; s < S; ++s) mbarInit(&full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  waitForEarlierKernels();  // from here on memory is read and written
  if (!waitForProducer(p)) {
    publish(p, true);
    return;
  }

  if (tid < 32) {
    // ---- warp 0: the bulk copy pipeline, driven by one elected lane ----
    if (tid == 0 && haveBulk) {
      const uint32_t first = blockIdx.x, step = gridDim.x;
      const uint32_t mine = (p.bulkTiles - first + step - 1) / step;  // tiles this CTA owns
      const uint32_t tileBytes = p.bulkTileBytes;
#ifdef TPB_DEBUG_KERNELS
      // A bulk copy off the 16-byte grid is an illegal instruction: check the whole table first
      // and leave the pipeline alone if any entry is wrong.
      bool tableOk = true;
      for (uint32_t i = 0; i < p.numEntries; ++i) {
        const PushEntry& e = p.entries[i];
        if (e.kind != kCopyBulk) continue;
        if ((reinterpret_cast<uintptr_t>(e.src) | reinterpret_cast<uintptr_t>(e.dst) | e.count) & 15) {
          atomicAdd(&gBoundsViolations, 1ull);
          tableOk = false;
        }
      }
#else
      constexpr bool tableOk = true;
#endif
      auto describe = [&](uint32_t i, const uint8_t*& src, uint8_t*& dst, uint32_t& bytes) {
        const uint32_t t = first + i * step;
        const PushEntry* e = findEntry(p, t, kBulkClass);
        const uint64_t off = static_cast<uint64_t>(t - e->tileStart) * tileBytes;
        const uint64_t left = e->count - off;
        bytes = left < tileBytes ? static_cast<uint32_t>(left) : tileBytes;
        src = static_cast<const uint8_t*>(e->src) + off;
        dst = static_cast<uint8_t*>(e->dst) + off;
      };
      auto issueLoad = [&](uint32_t i) {
        const uint8_t* src;
        uint8_t* dst;
        uint32_t bytes;
        describe(i, src, dst, bytes);
        const int s = i % S;
        mbarExpectTx(&full[s], bytes);
        bulkLoad(stages + static_cast<size_t>(s) * tileBytes, src, bytes, &full[s]);
      };
      const uint32_t prologue = !tableOk ? 0 : mine < static_cast<uint32_t>(S) ? mine : S;
      for (uint32_t i = 0; i < prologue; ++i) issueLoad(i);
      for (uint32_t c = 0; tableOk && c < mine; ++c) {
        const int s = c % S;
        if (!mbarWaitBounded(&full[s], (c / S) & 1)) {
          failed = true;
          break;
        }
        const uint8_t* src;
        uint8_t* dst;
        uint32_t bytes;
        describe(c, src, dst, bytes);
        fenceProxyAsync();
        bulkStore(dst, stages + static_cast<size_t>(s) * tileBytes, bytes);
        bulkCommit();
        // Refill the stage whose store was issued one iteration ago: by now it has most likely
        // finished reading shared memory, so this wait rarely stalls the pipeline.
        if (c >= 1 && (c - 1) + S < mine) {
          bulkWaitRead<1>();
          issueLoad((c - 1) + S);
        }
      }
      bulkWaitAll();  // stores are complete (not merely read out of shared memory)
      if (failed) reportStatus(p.status, kStatusBarrierTimeout);
    }
  } else {
    // ---- warps 1..: everything that needs registers ----
    constexpr uint32_t kPlainWarps = kThreads / 32 - 1;
    const uint32_t warp = tid / 32 - 1;
    // Eight of these warps share the block tiles; the others go straight to the tiles a warp does alone.
    if constexpr (kForms == kAllForms) {
      if (p.blockTiles > 0 && warp < kBlockThreads / 32) failed = !runBlockTiles(p, blockIdx.x, gridDim.x, tid - 32, warpTiles);
    }
    if (!failed)
      runPlainWarp<N, kForms>(p, blockIdx.x * kPlainWarps + warp, gridDim.x * kPlainWarps, tid & 31,
                              warpTiles + warp * p.warpTileBytes);
  }
  publish(p, failed);
}

template <int N, int kForms>
__global__ void __launch_bounds__(kLightThreads, 2) tpb_push_pack_light(const __grid_constant__ PushParams<N> p) {
  extern __shared__ __align__(16) uint8_t lightTiles[];  // kWarps * p.warpTileBytes, none for plain copies
  constexpr uint32_t kWarps = kLightThreads / 32;
  const uint32_t warp = threadIdx.x / 32;
  if (!p.lateTrigger) letDependentsLaunch();
  waitForEarlierKernels();
  if (!waitForProducer(p)) {
    publish(p, true);
    return;
  }
  static_assert(kLightThreads == kBlockThreads, "the whole light CTA shares a block tile");
  bool failed = false;
  if constexpr (kForms == kAllForms) {
    if (p.blockTiles > 0) failed = !runBlockTiles(p, blockIdx.x, gridDim.x, threadIdx.x, lightTiles);
  }
  if (!failed)
    runPlainWarp<N, kForms>(p, blockIdx.x * kWarps + warp, gridDim.x * kWarps, threadIdx.x & 31,
                            lightTiles + warp * p.warpTileBytes);
  publish(p, failed);
}

__global__ void tpb_wait_flag(const uint32_t* flag, uint32_t value, uint64_t timeoutNs, uint32_t* status) {
  if (threadIdx.x != 0) return;
  const uint64_t start = globalTimerNs();
  uint32_t backoff = 32;
  // Both limits bound the loop: the timer deadline and an iteration cap.
  for (uint64_t i = 0; i < (1ull << 32); ++i) {
    const uint32_t v = loadAcquireSys(flag);
    if (static_cast<int32_t>(v - value) >= 0) return;
    if (globalTimerNs() - start > timeoutNs) break;
    __nanosleep(backoff);
    if (backoff < 1024) backoff <<= 1;
  }
  // Only a failure is written: the word is shared with other waits and an earlier failure must
  // not be wiped out by a later success.
  reportStatus(status, kStatusWaitTimeout);
}

__global__ void tpb_delay(uint32_t* buf, size_t words, uint64_t ns) {
  const uint64_t start = globalTimerNs();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  // Bounded by the deadline and by an iteration cap.
  for (uint32_t it = 0; it < (1u << 24); ++it) {
    for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += stride) buf[i] = buf[i] * 1664525u + it;
    if (globalTimerNs() - start > ns) break;
    __nanosleep(1000);
  }
}

__host__ __device__ __forceinline__ uint32_t patternWord(uint64_t seed, uint64_t wordIndex) {
  // splitmix-style hash: cheap, seedable, identical on host and device
  uint64_t z = seed + (wordIndex + 1) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return static_cast<uint32_t>(z ^ (z >> 31));
}

__global__ void tpb_fill(uint8_t* buf, size_t bytes, uint64_t seed) {
  const size_t words = bytes / 4;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  uint32_t* w = reinterpret_cast<uint32_t*>(buf);
  for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += stride) w[i] = patternWord(seed, i);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (size_t b = words * 4; b < bytes; ++b) buf[b] = static_cast<uint8_t>(patternWord(seed, words) >> (8 * (b & 3)));
  }
}

__global__ void tpb_verify(const uint8_t* buf, size_t bytes, uint64_t seed, unsigned long long* mismatches) {
  const size_t words = bytes / 4;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  const uint32_t* w = reinterpret_cast<const uint32_t*>(buf);
  unsigned long long bad = 0;
  for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += stride) {
    const uint32_t x = w[i] ^ patternWord(seed, i);
    if (x) bad += ((x & 0xff) != 0) + ((x & 0xff00) != 0) + ((x & 0xff0000) != 0) + ((x & 0xff000000u) != 0);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (size_t b = words * 4; b < bytes; ++b)
      bad += buf[b] != static_cast<uint8_t>(patternWord(seed, words) >> (8 * (b & 3)));
  }
  if (bad) atomicAdd(mismatches, bad);
}

void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

// Launches with the programmatic-stream-serialization attribute (see letDependentsLaunch) where
// that pays: small launches that publish or await a flag, i.e. the eager pushes and unpacks
// between processes, which follow each other on a stream with no other work in between (measured
// across two GPUs: 9.1-10.9 us per message instead of 10.8-12.9 from 4 to 64 KiB; from 128 KiB
// to 4 MiB the attribute cost 2 us per message, beyond that it made no difference).
// TPB_PUSH_PDL=0 turns it off.
constexpr uint64_t kDependentLaunchMaxBytes = 64 * 1024;
// Larger launches up to TPB_PUSH_PDL_LATE_MAX_BYTES (default 0: none) are launched as dependents
// too, but let their own dependents go only when their work has been issued.
uint64_t lateDependentMaxBytes() {
  static const uint64_t v = [] {
    const char* e = std::getenv("TPB_PUSH_PDL_LATE_MAX_BYTES");
    return e && *e ? std::strtoull(e, nullptr, 0) : 0ull;
  }();
  return v;
}
bool programmaticLaunches() {
  static const bool on = [] {
    const char* e = std::getenv("TPB_PUSH_PDL");
    return !(e && e[0] == '0' && e[1] == 0);
  }();
  return on;
}

template <typename Kernel, typename Params>
void launchMaybeDependent(Kernel kernel, uint32_t grid, uint32_t threads, size_t smem, cudaStream_t stream, const Params& p,
                          bool dependent) {
  if (!dependent || !programmaticLaunches()) {
    kernel<<<grid, threads, smem, stream>>>(p);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, p);
}

template <typename Kernel>
void allowSmem(Kernel kernel, size_t bytes) {
  check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)),
        "cudaFuncSetAttribute");
}

template <int N, int kForms>
void launchForm(const PushEntry* entries, uint32_t n, uint32_t bulkTiles, uint32_t plainTiles, uint32_t blockTiles,
               uint32_t bulkTileBytes, uint32_t bulkStages, cudaStream_t stream, int maxCtas, uint32_t* flag, uint32_t flagValue,
               uint32_t* counter, uint32_t* status, const WaitBefore& wait, const DoneSlot& done, uint64_t bytesOut) {
  const bool publishes = flag != nullptr || wait.flag != nullptr || done.slot != nullptr;
  const bool early = bytesOut <= kDependentLaunchMaxBytes;
  const bool dependent = publishes && (early || bytesOut <= lateDependentMaxBytes());
  PushParams<N> p;
  p.lateTrigger = early ? 0 : 1;
  for (uint32_t i = 0; i < n; ++i) p.entries[i] = entries[i];
  p.numEntries = n;
  p.bulkTiles = bulkTiles;
  p.plainTiles = plainTiles;
  p.blockTiles = blockTiles;
  p.flagValue = flagValue;
  p.flag = flag;
  p.counter = counter;
  p.status = status;
  p.waitFlag = wait.flag;
  p.waitValue = wait.value;
  p.waitTimeoutNs = wait.timeoutNs;
  p.doneSlot = done.slot;
  p.doneValue = done.value;
  p.bulkTileBytes = bulkTileBytes;
  p.bulkStages = bulkStages;
  p.warpTileBytes = 0;
  for (uint32_t i = 0; i < n; ++i) {
    const uint32_t need = entries[i].kind == kStridedWide16 || entries[i].kind == kTransposed || entries[i].kind == kStridedNarrow ||
            entries[i].kind == kStridedBand
        ? kWideWarpTileBytes
        : entries[i].kind == kStrided                                                            ? kWarpTileBytes
                                                                                                 : 0;
    if (need > p.warpTileBytes) p.warpTileBytes = need;
  }
  int dev = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  if (bulkTiles == 0) {
    // Light kernel: 8 warps per CTA, shared memory only when an entry is staged through it.
    constexpr uint32_t kWarps = kLightThreads / 32;
    uint32_t grid = (plainTiles + kWarps - 1) / kWarps;
    if (blockTiles > grid) grid = blockTiles;
    if (grid > static_cast<uint32_t>(maxCtas) * 2) grid = static_cast<uint32_t>(maxCtas) * 2;
    if (grid == 0) grid = 1;
    size_t lightSmem = static_cast<size_t>(kWarps) * p.warpTileBytes;
    if (blockTiles > 0) lightSmem = std::max<size_t>(lightSmem, kBlockStagesLight * (kBlockTileBytes + sizeof(uint64_t)));
    static SmemLimit lightLimit;
    if (lightSmem > 48 * 1024) lightLimit.raise(dev, lightSmem, [](size_t most) { allowSmem(tpb_push_pack_light<N, kForms>, most); });
    launchMaybeDependent(tpb_push_pack_light<N, kForms>, grid, kLightThreads, lightSmem, stream, p, dependent);
    check(cudaGetLastError(), "tpb_push_pack_light launch");
    ++gLaunches;
    return;
  }
  const size_t smem = static_cast<size_t>(bulkStages) * bulkTileBytes + (kThreads / 32 - 1) * p.warpTileBytes +
      kMaxBulkStages * sizeof(uint64_t) + 128;
  if (smem > kMaxSmemPerCta) throw std::runtime_error("push plan needs more shared memory than a CTA has");
  static SmemLimit limit;
  limit.raise(dev, smem, [](size_t most) { allowSmem(tpb_push_pack<N, kForms>, most); });
  constexpr uint32_t kPlainWarps = kThreads / 32 - 1;
  uint32_t want = bulkTiles;
  const uint32_t plainCtas = (plainTiles + kPlainWarps - 1) / kPlainWarps;
  if (plainCtas > want) want = plainCtas;
  if (blockTiles > want) want = blockTiles;
  uint32_t grid = want < static_cast<uint32_t>(maxCtas) ? want : static_cast<uint32_t>(maxCtas);
  if (grid == 0) grid = 1;
  launchMaybeDependent(tpb_push_pack<N, kForms>, grid, kThreads, smem, stream, p, dependent);
  check(cudaGetLastError(), "tpb_push_pack launch");
  ++gLaunches;
}

// A message runs a kernel that has no code for forms it does not hold. Messages of one contiguous tensor are the
// most frequent ones and mostly overhead, and what the forms of views keep across calls costs every launch of a
// kernel that holds them. (Kernel times on one B200, everything in one kernel / this: 64 KiB copied 5.15 / 4.6 us, 1000
// elements fp32 -> bf16 8.6 / 6.9; half a round trip of 4 KiB through a pipe 18.9 / 17.6.)
template <int N, typename... Rest>
void launchOne(const PushEntry* entries, uint32_t n, const Rest&... rest) {
  int forms = kContiguousForms;
  for (uint32_t i = 0; i < n; ++i) {
    if (entries[i].kind == kTransposed) forms = kAllForms;
    else if (isView(entries[i].kind) && forms == kContiguousForms) forms = kWarpForms;
  }
  if (forms == kAllForms) launchForm<N, kAllForms>(entries, n, rest...);
  else if (forms == kWarpForms) launchForm<N, kWarpForms>(entries, n, rest...);
  else launchForm<N, kContiguousForms>(entries, n, rest...);
}

}  // namespace

void setPushTuning(const PushTuning& t) {
  if (t.bulkStages < 2 || t.bulkStages > static_cast<uint32_t>(kMaxBulkStages) || t.bulkTileBytes % 1024 != 0 ||
      t.bulkTileBytes == 0 || static_cast<size_t>(t.bulkStages) * t.bulkTileBytes > 160 * 1024)
    throw std::runtime_error("invalid bulk pipeline tuning");
  std::unique_lock<std::mutex> l(gTuningMutex);
  gTuning = t;
}
PushTuning getPushTuning() {
  std::unique_lock<std::mutex> l(gTuningMutex);
  return gTuning;
}

// ---- host-side planning -------------------------------------------------------------------------
bool castSupported(DType s, DType d) {
  auto isFloat = [](DType t) { return t == DType::kF32 || t == DType::kBF16 || t == DType::kF16; };
  return s == d || (isFloat(s) && isFloat(d));
}

uint64_t convertedBytes(uint64_t srcBytes, DType s, DType d) {
  if (s == d || d == DType::kBytes) return srcBytes;
  return srcBytes / dtypeSize(s) * dtypeSize(d);
}

namespace {
uint32_t tilesOf(const PushEntry& e, uint32_t bulkTileBytes) {
  auto over = [](uint64_t n, uint64_t tile) { return (n + tile - 1) / tile; };
  uint64_t tiles = 0;
  switch (e.kind) {
    case kCopyBulk: tiles = over(e.count, bulkTileBytes); break;
    case kCopyPlain: tiles = over(e.count, kPlainTileBytes); break;
    case kCastPlain: tiles = over(e.count, kPlainTileBytes / e.dstElemSize); break;
    case kRows: tiles = over(e.count * e.dstElemSize, e.rowTileBytes); break;
    case kStridedBand: tiles = over(e.rows, bandRows(static_cast<uint64_t>(e.cols), e.dstElemSize)); break;
    case kStridedNarrow: tiles = over(e.rows, kStridedTile); break;
    case kTransposed: {
      const bool narrow = e.cols <= kBlockNarrowCols;
      const uint64_t rows = 256 / e.srcElemSize * (narrow ? kBlockSlots / e.cols : 1);
      tiles = over(e.rows, rows) * (narrow ? 1 : over(e.cols, kBlockSlots));
      break;
    }
    case kStridedWide16: tiles = over(e.rows, kWideTile) * over(e.cols, kWideTile); break;
    default: tiles = over(e.rows, e.srcElemSize == 8 ? kStridedTile / 2 : kStridedTile) * over(e.cols, kStridedTile); break;
  }
  return static_cast<uint32_t>(tiles);
}
void pushEntry(PushPlan& plan, PushEntry e) {
  if (e.count == 0) return;
  uint32_t* const totals[kTileClasses] = {&plan.plainTiles, &plan.bulkTiles, &plan.blockTiles};
  uint32_t& total = *totals[tileClassOf(e.kind)];
  e.numTiles = tilesOf(e, plan.bulkTileBytes);
  e.tileStart = total;
  total += e.numTiles;
  plan.entries.push_back(e);
}

}  // namespace

// Why the lines lie where they do. (Launches back to back on one B200, us each, warp form / block form; they end on steps
// of about 2 us, so less than that is a tie.)
//   * Few columns leave most lanes of a 32x32 warp tile idle, and a tile that is not quite full takes the warps' predicated
//     path: 64 MiB of fp32 in 5 columns 178 / 32, 31 columns 77 / 33, 63 columns 78 / 31, 127 columns 72 / 28.
//   * Where all warp tiles are full the block form only wins by its longer pieces, once there are tiles enough: fp32 in 128
//     columns 8 MiB 8.3 / 10.3, 16 MiB 12.3 / 12.3, 64 MiB 35 / 27; in 64 columns 16 MiB 12.3 / 13.4, 64 MiB 34 / 31.
//   * A last tile of few columns costs nearly a full one, most of all where the warp form writes less than it reads:
//     64 MiB of fp32 -> bf16 in 65 columns 40 / 51, 129 columns 36 / 45, 160 columns 33 / 39, 257 columns 33 / 35.
//   * Beside the bulk pipeline it has one stage and eight warps of one CTA an SM, and loses what it wins by overlap:
//     64 MiB of fp32 beside 1 MiB, 64 columns 37 / 53, 130 columns 41 / 82, 1000 columns 39 / 53, but 5 columns 189 / 55,
//     63 columns 82 / 56, 127 columns 82 / 51, 383 columns 77 / 51. The more the bulk pipeline has to do, the less it
//     matters, and wide 2-byte matrices then gain: 16 MiB in 130 columns beside 16 MiB 29 / 31, beside 64 MiB 42 / 39.
bool blockFormPays(const PushEntry& e, uint64_t bulkBytes) {
  constexpr uint64_t MiB = 1 << 20, kNever = ~0ull;
  const uint64_t bytes = e.count * e.srcElemSize;
  const int64_t cols = e.cols;
  const bool narrow = cols < kBlockNarrowCols, converts = e.srcElemSize != e.dstElemSize, widens = e.dstElemSize > e.srcElemSize;
  // The share of a block tile's slots that hold a column; how many columns lie in a warp tile that is not full.
  const double filled = cols <= kBlockNarrowCols ? static_cast<double>(kBlockSlots / cols * cols) / kBlockSlots
                                                 : static_cast<double>(cols) / ((cols + kBlockSlots - 1) / kBlockSlots * kBlockSlots);
  const int64_t ragged = cols % kStridedTile;
  if (!widens && static_cast<uint64_t>(e.rows) * e.srcElemSize <= kBlockMinRowBytes) return false;

  if (bulkBytes > 0) {
    if ((cols > kBlockSlots || (cols > kBlockNarrowCols && filled >= 0.75)) && e.srcElemSize == 2 && !converts && bulkBytes >= 2 * bytes) return true;
    if (ragged == 0) return false;
    if (narrow) return e.srcElemSize == 2 || ragged > 2 || bytes >= 12 * MiB;
    if (ragged > 24) return widens || !converts || filled >= 0.9;
    return (filled >= 0.9 && bytes < 6 * MiB) || (widens && filled >= 0.75);
  }

  uint64_t least = 0;  // the plan has its own least size
  if (cols == kStridedTile || cols == kBlockNarrowCols) {  // one or two warp tiles, all full
    if (e.srcElemSize != 2) least = (e.srcElemSize == 8 ? 12 : converts ? 48 : 24) * MiB;
    else least = widens ? 6 * MiB : cols == kBlockNarrowCols ? 48 * MiB : 0;
  } else if (!narrow && e.srcElemSize != 2 && ragged < kStridedTile / 2) {
    const bool full = ragged == 0 && (e.rows % kStridedTile == 0 || e.rows >= 10 * kStridedTile), several = cols > kBlockSlots;
    if (converts && filled < (full ? 0.8 : several ? 0.7 : 0.6)) least = kNever;
    else if (full) least = (filled < 0.66 ? 48 : 12) * MiB;
    else if (several && filled < 0.6) least = e.srcElemSize == 8 ? 24 * MiB : kNever;
    else if (several && filled < 0.7) least = 6 * MiB;
  }
  return bytes >= least;
}

std::vector<PushEntry> entriesOfLaunch(const PushEntry* entries, size_t n, uint32_t bulkTileBytes, uint32_t (&tiles)[kTileClasses]) {
  std::vector<PushEntry> part(entries, entries + n);
  const uint32_t blockForm = getPushTuning().blockForm;
  uint64_t bulkBytes = 0;
  for (const auto& e : part)
    if (e.kind == kCopyBulk) bulkBytes += e.count;
  for (auto& e : part) {
    if (e.kind == kTransposed && (blockForm == 0 || (blockForm == 1 && !blockFormPays(e, bulkBytes)))) {
      e.kind = e.warpForm;
      e.numTiles = tilesOf(e, bulkTileBytes);
    }
    uint32_t& next = tiles[tileClassOf(e.kind)];
    e.tileStart = next;
    next += e.numTiles;
  }
  return part;
}

namespace {
// Memory that the driver places on another GPU than the current one, or on the host.
bool sourceIsForeign(const void* src) {
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return cudaIsForeignMemory(src, device);
}
}  // namespace

void chooseBulkTile(PushPlan& plan, uint64_t bulkBytes, int ctas) {
  const PushTuning t = getPushTuning();
  plan.bulkStages = t.bulkStages;
  plan.bulkTileBytes = t.bulkTileBytes;
  if (!plan.entries.empty() || bulkBytes == 0 || ctas <= 0) return;
  const uint64_t perWave = static_cast<uint64_t>(ctas) * t.bulkTileBytes;
  const uint64_t waves = (bulkBytes + perWave - 1) / perWave;
  uint64_t tile = (bulkBytes + waves * ctas - 1) / (waves * ctas);
  tile = (tile + 1023) / 1024 * 1024;
  if (tile < 4096) tile = 4096;
  if (tile > t.bulkTileBytes) tile = t.bulkTileBytes;
  plan.bulkTileBytes = static_cast<uint32_t>(tile);
}

void appendToPlan(PushPlan& plan, const CopyItem& item, bool useBulk) {
  if (plan.bulkTileBytes == 0) {
    const PushTuning t = getPushTuning();
    plan.bulkTileBytes = t.bulkTileBytes;
    plan.bulkStages = t.bulkStages;
  }
  PushEntry e{};
  e.srcDtype = static_cast<uint8_t>(item.srcDtype);
  const DType dstDtype = item.dstDtype == DType::kBytes ? item.srcDtype : item.dstDtype;
  e.dstDtype = static_cast<uint8_t>(dstDtype);
  e.srcElemSize = static_cast<uint8_t>(dtypeSize(item.srcDtype));
  e.dstElemSize = static_cast<uint8_t>(dtypeSize(dstDtype));
  const bool convert = dstDtype != item.srcDtype;
  if (convert && !castSupported(item.srcDtype, dstDtype)) throw std::runtime_error("unsupported dtype conversion");
  plan.totalBytesOut += convertedBytes(item.srcBytes, item.srcDtype, dstDtype);

  if (item.strided) {
    const StridedView& v = item.view;
    if (static_cast<uint64_t>(v.rows) * v.cols * dtypeSize(v.dtype) != item.srcBytes)
      throw std::runtime_error("strided view does not match the tensor length");
    e.srcDtype = static_cast<uint8_t>(v.dtype);
    e.srcElemSize = static_cast<uint8_t>(dtypeSize(v.dtype));
    if (!convert) {
      e.dstDtype = e.srcDtype;
      e.dstElemSize = e.srcElemSize;
    }
    e.src = item.src;
    e.dst = item.dst;
    e.kind = kStrided;
    {
      // The word-wide variant needs even everything; it also needs its larger staging area to fit
      // next to the bulk stages this plan was sized with.
      const uintptr_t both = reinterpret_cast<uintptr_t>(item.src) | reinterpret_cast<uintptr_t>(item.dst);
      const size_t smemWithWide = static_cast<size_t>(plan.bulkStages) * plan.bulkTileBytes +
          (kThreads / 32 - 1) * kWideWarpTileBytes + kMaxBulkStages * sizeof(uint64_t) + 128;
      if (!convert && e.srcElemSize == 2 && v.rowStride == 1 && v.colStride != 1 && v.rows >= kWideTile &&
          v.cols >= kWideTile && v.rows % 2 == 0 && v.cols % 2 == 0 && v.colStride % 2 == 0 && (both & 3) == 0 &&
          smemWithWide <= kMaxSmemPerCta)
        e.kind = kStridedWide16;
      // Few columns: whole packed rows per tile, written as one contiguous run (wins over the above).
      const uint64_t dstRowBytes = static_cast<uint64_t>(v.cols) * e.dstElemSize;
      const uint32_t narrowRows = getPushTuning().narrowRows;
      if ((narrowRows == 2 || (narrowRows == 1 && item.remote)) && v.rowStride == 1 && v.colStride != 1 &&
          v.cols <= kNarrowMaxCols && e.srcElemSize <= 4 && e.dstElemSize <= 4 &&
          dstRowBytes % 16 == 0 && (reinterpret_cast<uintptr_t>(item.dst) & 15) == 0 && v.rows > 1 &&
          smemWithWide <= kMaxSmemPerCta)
        e.kind = kStridedNarrow;
      // Any other transposed matrix with rows of at most 8 KiB: bands of whole rows, each written
      // as one contiguous run whatever its alignment.
      const uint32_t bands = getPushTuning().bandRows;
      if (e.kind != kStridedNarrow && (bands == 2 || (bands == 1 && item.remote)) && v.rowStride == 1 &&
          v.colStride != 1 && v.rows > 1 && dstRowBytes <= kBandBytes && smemWithWide <= kMaxSmemPerCta)
        e.kind = kStridedBand;
      // Large transposed matrices that none of the forms above for another GPU takes: one tile per CTA. The tiles are
      // fetched by bulk copies, which read the launching GPU's own memory only.
      if (useBulk && e.kind != kStridedNarrow && e.kind != kStridedBand && e.srcElemSize >= 2 && v.rowStride == 1 &&
          v.colStride != 1 && v.cols >= 2 && static_cast<uint64_t>(v.rows) * e.srcElemSize >= kBlockMinRowBytes &&
          item.srcBytes >= blockMinBytes(v.cols, e.srcElemSize) && smemWithWide <= kMaxSmemPerCta && !sourceIsForeign(item.src))
        e.warpForm = e.kind, e.kind = kTransposed;
      // Rows that are contiguous in the source are copied as the runs they are. Shorter than a vector they
      // would straddle more than two rows per vector: those, and rows whose length does not fit the
      // kernel's 32-bit offsets, stay with the element-wise tiles.
      const uint64_t srcRowBytes = static_cast<uint64_t>(v.cols) * e.srcElemSize;
      if (v.rows > 1 && v.colStride == 1 && srcRowBytes >= 16 && srcRowBytes < (1u << 31) && (!convert || v.cols >= 16)) {
        e.kind = kRows;
        e.rowTileBytes = rowTileBytes(static_cast<uint64_t>(v.rows) * dstRowBytes);
      }
    }
    e.rows = v.rows;
    e.cols = v.cols;
    e.rowStride = v.rowStride;
    e.colStride = v.colStride;
    e.count = static_cast<uint64_t>(v.rows) * v.cols;
    pushEntry(plan, e);
    return;
  }
  if (convert) {
    e.src = item.src;
    e.dst = item.dst;
    e.kind = kCastPlain;
    e.count = item.srcBytes / dtypeSize(item.srcDtype);
    pushEntry(plan, e);
    return;
  }
  // Contiguous copy: aligned body on the bulk path, ragged head and tail on the plain path.
  const uint8_t* src = static_cast<const uint8_t*>(item.src);
  uint8_t* dst = static_cast<uint8_t*>(item.dst);
  uint64_t bytes = item.srcBytes;
  const uintptr_t sa = reinterpret_cast<uintptr_t>(src), da = reinterpret_cast<uintptr_t>(dst);
  const bool sameSkew = ((sa ^ da) & 15) == 0;
  if (useBulk && sameSkew && bytes >= getPushTuning().bulkMinBytes) {
    // Bulk (TMA) loads read the launching GPU's own memory only. Whatever the caller asked for, a
    // source that the driver places on another GPU or in host memory goes through plain loads.
    if (sourceIsForeign(src)) useBulk = false;
  }
  if (!useBulk || !sameSkew || bytes < getPushTuning().bulkMinBytes) {
    e.src = src;
    e.dst = dst;
    e.kind = kCopyPlain;
    e.count = bytes;
    pushEntry(plan, e);
    return;
  }
  const uint64_t head = (16 - (sa & 15)) & 15;
  if (head) {
    PushEntry h = e;
    h.src = src;
    h.dst = dst;
    h.kind = kCopyPlain;
    h.count = head;
    pushEntry(plan, h);
    src += head;
    dst += head;
    bytes -= head;
  }
  const uint64_t body = bytes & ~static_cast<uint64_t>(15);
  PushEntry b = e;
  b.src = src;
  b.dst = dst;
  b.kind = kCopyBulk;
  b.count = body;
  pushEntry(plan, b);
  if (bytes - body) {
    PushEntry t = e;
    t.src = src + body;
    t.dst = dst + body;
    t.kind = kCopyPlain;
    t.count = bytes - body;
    pushEntry(plan, t);
  }
}

int launchPush(const PushPlan& plan, cudaStream_t stream, int maxCtas, uint32_t* flag, uint32_t flagValue,
               uint32_t* counter, uint32_t* status, WaitBefore wait, DoneSlot done) {
  if ((flag != nullptr || done.slot != nullptr) && counter == nullptr && maxCtas > 1)
    throw std::runtime_error("a launch that publishes a flag or a completion word from several CTAs needs an arrive counter");
  const size_t n = plan.entries.size();
  trace::Scope traced("tpb_push_pack launch", plan.totalBytesOut);
  if (maxCtas <= 0) maxCtas = 1;
  const uint32_t tileBytes = plan.bulkTileBytes ? plan.bulkTileBytes : 32768;
  const uint32_t stages = plan.bulkStages ? plan.bulkStages : 4;
  if (n <= static_cast<size_t>(kMaxEntriesLarge)) {
    const PushEntry* entries = plan.entries.data();
    uint32_t tiles[kTileClasses] = {plan.plainTiles, plan.bulkTiles, plan.blockTiles};
    std::vector<PushEntry> part;
    if (plan.blockTiles > 0) {
      for (uint32_t& t : tiles) t = 0;
      part = entriesOfLaunch(entries, n, tileBytes, tiles);
      entries = part.data();
    }
    if (n <= static_cast<size_t>(kMaxEntriesSmall))
      launchOne<kMaxEntriesSmall>(entries, static_cast<uint32_t>(n), tiles[kBulkClass], tiles[kPlainClass], tiles[kBlockClass],
                                  tileBytes, stages, stream, maxCtas, flag, flagValue, counter, status, wait, done,
                                  plan.totalBytesOut);
    else
      launchOne<kMaxEntriesLarge>(entries, static_cast<uint32_t>(n), tiles[kBulkClass], tiles[kPlainClass], tiles[kBlockClass],
                                  tileBytes, stages, stream, maxCtas, flag, flagValue, counter, status, wait, done,
                                  plan.totalBytesOut);
    return 1;
  }
  // More entries than one parameter block holds: several launches on the same stream, each with
  // its own tile numbering; only the last publishes the flag (stream order covers the others).
  int launches = 0;
  for (size_t first = 0; first < n; first += kMaxEntriesLarge) {
    const size_t cnt = n - first < static_cast<size_t>(kMaxEntriesLarge) ? n - first : kMaxEntriesLarge;
    uint32_t tiles[kTileClasses] = {};
    const std::vector<PushEntry> part = entriesOfLaunch(plan.entries.data() + first, cnt, tileBytes, tiles);
    const bool last = first + cnt == n;
    // Only the first launch waits for the producer; stream order covers the rest.
    launchOne<kMaxEntriesLarge>(part.data(), static_cast<uint32_t>(cnt), tiles[kBulkClass], tiles[kPlainClass],
                                tiles[kBlockClass], tileBytes, stages, stream,
                                maxCtas, last ? flag : nullptr, flagValue, counter, status,
                                first == 0 ? wait : WaitBefore(), last ? done : DoneSlot(), plan.totalBytesOut);
    ++launches;
  }
  return launches;
}

void launchWaitFlag(cudaStream_t stream, const uint32_t* flag, uint32_t value, uint64_t timeoutNs, uint32_t* status) {
  tpb_wait_flag<<<1, 32, 0, stream>>>(flag, value, timeoutNs, status);
  check(cudaGetLastError(), "tpb_wait_flag launch");
  ++gLaunches;
}

void launchDelay(cudaStream_t stream, void* buf, size_t bytes, uint32_t microseconds) {
  uint64_t ns = static_cast<uint64_t>(microseconds) * 1000;
  if (ns > 2'000'000'000ull) ns = 2'000'000'000ull;
  tpb_delay<<<8, 128, 0, stream>>>(static_cast<uint32_t*>(buf), bytes / 4, ns);
  check(cudaGetLastError(), "tpb_delay launch");
  ++gLaunches;
}

void launchFill(cudaStream_t stream, void* buf, size_t bytes, uint64_t seed) {
  if (bytes == 0) return;
  size_t blocks = (bytes / 4 + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks == 0) blocks = 1;
  tpb_fill<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(static_cast<uint8_t*>(buf), bytes, seed);
  check(cudaGetLastError(), "tpb_fill launch");
  ++gLaunches;
}

void launchVerify(cudaStream_t stream, const void* buf, size_t bytes, uint64_t seed, unsigned long long* mismatches) {
  if (bytes == 0) return;
  size_t blocks = (bytes / 4 + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks == 0) blocks = 1;
  tpb_verify<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(static_cast<const uint8_t*>(buf), bytes, seed,
                                                                mismatches);
  check(cudaGetLastError(), "tpb_verify launch");
  ++gLaunches;
}

uint8_t patternByte(uint64_t seed, uint64_t index) {
  return static_cast<uint8_t>(patternWord(seed, index / 4) >> (8 * (index & 3)));
}

uint64_t launchCount() { return gLaunches.load(); }

bool debugKernels() {
#ifdef TPB_DEBUG_KERNELS
  return true;
#else
  return false;
#endif
}

uint64_t boundsViolations() {
#ifdef TPB_DEBUG_KERNELS
  // Summed over the devices this process has a context on (and only those: asking a device
  // without one would create it).
  unsigned long long total = 0;
  const int n = cudaDeviceCountNoThrow();
  for (int d = 0; d < n; ++d) {
    if (cudaPrimaryContextActive(d) != 1) continue;
    CudaDeviceGuard g(d);
    unsigned long long v = 0;
    check(cudaMemcpyFromSymbol(&v, gBoundsViolations, sizeof(v)), "reading the violation counter");
    total += v;
  }
  return total;
#else
  return 0;
#endif
}

}  // namespace kernels
}  // namespace tpb
