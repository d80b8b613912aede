// Allocation-free variant of the push kernel: see include/tpb/noalloc.h for who needs it and the
// rules for using it. The table of copies travels as the kernel's parameter; the arrive counter, which an
// ordinary launch gets from its caller, lives here in a file-scope device array.
#include <tpb/noalloc.h>

#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <string>

#include "kernels/run_copy.cuh"

namespace {

using tpb::kernels::warpCopyRun;

constexpr uint32_t kTileBytes = 8 * 1024;  // one warp's unit of work, as in the ordinary kernel
constexpr int kThreads = 256;
constexpr int kCtasPerSm = 2;
constexpr size_t kCounterBytes = 256;
constexpr int kMaxDevices = 64;

struct alignas(16) TableEntry {
  const void* src;
  void* dst;
  uint64_t bytes;
  uint32_t tileStart;
  uint32_t numTiles;
};
static_assert(sizeof(TableEntry) == 32, "table entry layout");

template <int N>
struct Table {
  TableEntry entries[N];
};
constexpr uint32_t kSmallTable = 16;  // most calls: 0.5 KiB of parameters to hand over instead of 8

// Arrive counters, zero between calls; calls take them in turn, so that one that is still running
// (on another stream, against the rules) does not see its counter moved by the next. Every GPU that loads
// this library holds this array until the process exits. In HOST code the name is only a stand-in for the symbol; the
// device address comes from cudaGetSymbolAddress (see lookupScratch).
static __device__ __align__(256) unsigned char g_scratch[kCounterBytes];
std::atomic<uint32_t> g_nextCounter{0};

// Bound by memory: one warp per 8 KiB tile, 4 KiB of loads in flight per warp, 16 warps per SM; tiles meet
// on 16-byte boundaries of the destination, so that only a range's own ends are ragged. (192 records of 1 MiB + 6
// bytes packed densely, 201 MB: 508 us when ranges of different alignment went byte by byte, 70 us now; the call
// 515 -> 76 us.)
// `counter` is one word of g_scratch; the host looks its address up.
template <int N>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    tpb_noalloc_push_kernel(const __grid_constant__ Table<N> table, uint32_t* counter, uint32_t count, uint32_t totalTiles,
                            uint32_t* flag, uint32_t flagValue) {
  const uint32_t warpsPerCta = kThreads / 32;
  const uint32_t warp = blockIdx.x * warpsPerCta + threadIdx.x / 32;
  const uint32_t totalWarps = gridDim.x * warpsPerCta;
  const int lane = threadIdx.x & 31;
  for (uint32_t t = warp; t < totalTiles; t += totalWarps) {
    uint32_t e = 0;  // the last entry that starts at or before tile t
#pragma unroll
    for (uint32_t half = N / 2; half > 0; half /= 2)
      if (e + half < count && table.entries[e + half].tileStart <= t) e += half;
    const TableEntry& entry = table.entries[e];
    const uint32_t local = t - entry.tileStart;
    const uint32_t skew = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(entry.dst) & 15);
    const uint64_t off = local == 0 ? 0 : static_cast<uint64_t>(local) * kTileBytes - skew;
    const uint64_t end = local + 1 == entry.numTiles ? entry.bytes : (static_cast<uint64_t>(local) + 1) * kTileBytes - skew;
    warpCopyRun<true>(static_cast<const uint8_t*>(entry.src) + off, static_cast<uint8_t*>(entry.dst) + off,
                      static_cast<uint32_t>(end - off), lane);
  }
  if (flag == nullptr) return;
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int arrived = atomicAdd(counter, 1u);
    if (arrived == gridDim.x - 1) {
      *counter = 0;  // ready for the next call
      __threadfence_system();
      asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(flagValue) : "memory");
    }
  }
}

template <int N>
cudaError_t launch(const TableEntry* entries, uint32_t n, uint32_t tiles, uint32_t grid, uint32_t* counter, uint32_t* flag,
                   uint32_t flagValue, cudaStream_t stream) {
  Table<N> table;  // entries behind the n-th are never read
  for (uint32_t i = 0; i < n; ++i) table.entries[i] = entries[i];
  tpb_noalloc_push_kernel<N><<<grid, kThreads, 0, stream>>>(table, counter, n, tiles, flag, flagValue);
  return cudaGetLastError();
}

thread_local std::string t_lastCudaError;

// Device address of g_scratch for the current device and that device's SM count; both resolved
// once per device, when the kernel is loaded there too.
int lookupScratch(unsigned char** out, int* smCount) {
  static std::mutex mu;
  static unsigned char* perDevice[kMaxDevices] = {};
  static int smsOf[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    t_lastCudaError = e != cudaSuccess ? cudaGetErrorString(e) : "device index out of range";
    return TPB_NOALLOC_CUDA_ERROR;
  }
  std::unique_lock<std::mutex> lock(mu);
  if (perDevice[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_scratch);
    if (e != cudaSuccess || p == nullptr) {
      t_lastCudaError = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e);
      cudaGetLastError();
      return TPB_NOALLOC_CUDA_ERROR;
    }
    // Both forms of the kernel are loaded now. Where modules load lazily, the first launch of a form would load it,
    // which may allocate and synchronise, and may happen inside a capture that began after the caller's first call.
    for (const void* form : {reinterpret_cast<const void*>(&tpb_noalloc_push_kernel<kSmallTable>),
                             reinterpret_cast<const void*>(&tpb_noalloc_push_kernel<TPB_NOALLOC_MAX_ITEMS>)}) {
      cudaFuncAttributes attributes;
      e = cudaFuncGetAttributes(&attributes, form);
      if (e != cudaSuccess) {
        t_lastCudaError = std::string("loading the kernel: ") + cudaGetErrorString(e);
        cudaGetLastError();
        return TPB_NOALLOC_CUDA_ERROR;
      }
    }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
      cudaGetLastError();
      sms = 1;
    }
    smsOf[dev] = sms;
    perDevice[dev] = static_cast<unsigned char*>(p);
  }
  *out = perDevice[dev];
  *smCount = smsOf[dev];
  return TPB_NOALLOC_OK;
}

}  // namespace

extern "C" int tpb_noalloc_push(const tpb_noalloc_item* items, size_t count, uint32_t* flag, uint32_t flag_value,
                                void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (count > TPB_NOALLOC_MAX_ITEMS) return TPB_NOALLOC_TOO_MANY;
  if (count > 0 && items == nullptr) return TPB_NOALLOC_BAD_ARGUMENT;

  // The table is built on the stack: no host allocation either.
  TableEntry table[TPB_NOALLOC_MAX_ITEMS];
  uint32_t n = 0, tiles = 0;
  for (size_t i = 0; i < count; ++i) {
    if (items[i].bytes == 0) continue;
    if (items[i].src == nullptr || items[i].dst == nullptr) return TPB_NOALLOC_BAD_ARGUMENT;
    if (items[i].bytes > UINT64_MAX - kTileBytes) return TPB_NOALLOC_BAD_ARGUMENT;  // rounding up would wrap
    const uint64_t t = (items[i].bytes + kTileBytes - 1) / kTileBytes;
    if (t > 0xffffffffull - tiles) return TPB_NOALLOC_BAD_ARGUMENT;
    table[n].src = items[i].src;
    table[n].dst = items[i].dst;
    table[n].bytes = items[i].bytes;
    table[n].tileStart = tiles;
    table[n].numTiles = static_cast<uint32_t>(t);
    tiles += static_cast<uint32_t>(t);
    ++n;
  }

  unsigned char* scratch = nullptr;
  int sms = 1;
  int rc = lookupScratch(&scratch, &sms);
  if (rc != TPB_NOALLOC_OK) return rc;

  const uint32_t warpsPerCta = kThreads / 32;
  uint32_t grid = (tiles + warpsPerCta - 1) / warpsPerCta;
  if (grid > static_cast<uint32_t>(sms) * kCtasPerSm) grid = static_cast<uint32_t>(sms) * kCtasPerSm;
  if (grid == 0) grid = 1;
  uint32_t* counter = reinterpret_cast<uint32_t*>(scratch) + g_nextCounter.fetch_add(1) % (kCounterBytes / sizeof(uint32_t));
  const cudaError_t e = n <= kSmallTable
      ? launch<kSmallTable>(table, n, tiles, grid, counter, flag, flag_value, stream)
      : launch<TPB_NOALLOC_MAX_ITEMS>(table, n, tiles, grid, counter, flag, flag_value, stream);
  if (e != cudaSuccess) {
    t_lastCudaError = cudaGetErrorString(e);
    return TPB_NOALLOC_CUDA_ERROR;
  }
  return TPB_NOALLOC_OK;
}

extern "C" const char* tpb_noalloc_strerror(int code) {
  switch (code) {
    case TPB_NOALLOC_OK: return "ok";
    case TPB_NOALLOC_TOO_MANY: return "more items than TPB_NOALLOC_MAX_ITEMS (256): split the request";
    case TPB_NOALLOC_BAD_ARGUMENT: return "null pointer for a non-empty item, or sizes that overflow";
    case TPB_NOALLOC_CUDA_ERROR: return t_lastCudaError.c_str();
    default: return "unknown code";
  }
}
