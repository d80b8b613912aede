// GPU tests of the push kernel's copy paths over alignments, extents, strides and element types,
// against an element-by-element CPU gather. Every destination is fenced by canary bytes. Values are
// random bits (NaNs, infinities and denormals among them); conversions are compared with the
// compiler's own _Float16 and with round-to-nearest-even on the bits for bfloat16: one right answer,
// except that any NaN stands for any other.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <random>

#include "common/cuda.h"
#include "kernels/push.h"
#include "test_util.h"

using namespace tpb;
using namespace tpb::kernels;

namespace {

#define CK(x) TPB_CUDA_CHECK(x)

struct Spec {
  DType from = DType::kU8, to = DType::kU8;
  int64_t rows = 1, cols = 0, rowStride = 0, colStride = 1;  // elements; a contiguous run is one row
  bool strided = false;
  size_t srcOff = 0, dstOff = 0;  // bytes past a 256-byte boundary
  bool remote = false;
};

float bitsToFloat(uint32_t b) {
  float f;
  std::memcpy(&f, &b, 4);
  return f;
}
float valueOf(const uint8_t* p, DType t) {
  uint32_t b = 0;
  if (t == DType::kF32) {
    std::memcpy(&b, p, 4);
    return bitsToFloat(b);
  }
  uint16_t h;
  std::memcpy(&h, p, 2);
  if (t == DType::kBF16) return bitsToFloat(static_cast<uint32_t>(h) << 16);
  _Float16 x;
  std::memcpy(&x, &h, 2);
  return static_cast<float>(x);
}
void store(uint8_t* p, DType t, float v) {
  uint32_t b;
  std::memcpy(&b, &v, 4);
  if (t == DType::kF32) {
    std::memcpy(p, &b, 4);
  } else if (t == DType::kBF16) {
    const uint16_t h = std::isnan(v) ? 0x7fff : static_cast<uint16_t>((b + 0x7fffu + ((b >> 16) & 1)) >> 16);
    std::memcpy(p, &h, 2);
  } else {
    const _Float16 x = static_cast<_Float16>(v);
    std::memcpy(p, &x, 2);
  }
}
bool isNan(const uint8_t* p, DType t) {
  return (t == DType::kF32 || t == DType::kBF16 || t == DType::kF16) && std::isnan(valueOf(p, t));
}

std::string describe(const Spec& s) {
  return std::to_string(s.rows) + "x" + std::to_string(s.cols) + " strides " + std::to_string(s.rowStride) + "," +
      std::to_string(s.colStride) + " type " + std::to_string(int(s.from)) + "->" + std::to_string(int(s.to)) +
      " offsets " + std::to_string(s.srcOff) + "," + std::to_string(s.dstOff) + (s.remote ? " remote" : "");
}

struct DeviceMem {
  uint8_t* p = nullptr;
  explicit DeviceMem(size_t n) { CK(cudaMalloc(&p, n)); }
  ~DeviceMem() { cudaFree(p); }
};

// All specs as one message: one plan, checked element by element; gaps must keep their canaries.
void checkMessage(const std::vector<Spec>& specs, bool bulk = true, int ctas = 148, bool publish = false) {
  std::mt19937 rng(static_cast<uint32_t>(specs.size() * 977 + specs[0].cols * 31 + specs[0].srcOff));
  size_t srcBytes = 256, dstBytes = 256;
  std::vector<size_t> srcAt, dstAt;
  for (const Spec& s : specs) {
    const size_t span = s.strided
        ? static_cast<size_t>((s.rows - 1) * s.rowStride + (s.cols - 1) * s.colStride + 1) * dtypeSize(s.from)
        : static_cast<size_t>(s.rows * s.cols) * dtypeSize(s.from);
    srcAt.push_back(srcBytes + s.srcOff);
    dstAt.push_back(dstBytes + s.dstOff);
    srcBytes += (s.srcOff + span + 511) / 256 * 256;
    dstBytes += (s.dstOff + static_cast<size_t>(s.rows * s.cols) * dtypeSize(s.to) + 511) / 256 * 256;
  }
  std::vector<uint8_t> src(srcBytes + 256), want(dstBytes + 256, 0xCD), got(dstBytes + 256);
  for (size_t i = 0; i + 4 <= src.size(); i += 4) {
    const uint32_t r = rng();
    std::memcpy(&src[i], &r, 4);
  }
  DeviceMem dsrc(src.size()), ddst(want.size());
  CK(cudaMemcpy(dsrc.p, src.data(), src.size(), cudaMemcpyHostToDevice));
  CK(cudaMemset(ddst.p, 0xCD, want.size()));
  PushPlan plan;
  for (size_t i = 0; i < specs.size(); ++i) {
    const Spec& s = specs[i];
    const size_t es = dtypeSize(s.from), ed = dtypeSize(s.to);
    CopyItem it;
    it.src = dsrc.p + srcAt[i];
    it.dst = ddst.p + dstAt[i];
    it.srcBytes = static_cast<uint64_t>(s.rows * s.cols) * es;
    it.srcDtype = s.from;
    it.dstDtype = s.to;
    it.remote = s.remote;
    if (s.strided) {
      it.strided = true;
      it.view = StridedView{s.from, s.rows, s.cols, s.rowStride, s.colStride};
    }
    appendToPlan(plan, it, bulk);
    for (int64_t r = 0; r < s.rows; ++r)
      for (int64_t c = 0; c < s.cols; ++c) {
        const uint8_t* from = &src[srcAt[i] + (s.strided ? r * s.rowStride + c * s.colStride : r * s.cols + c) * es];
        uint8_t* to = &want[dstAt[i] + (r * s.cols + c) * ed];
        if (s.from == s.to) std::memcpy(to, from, es);
        else store(to, s.to, valueOf(from, s.from));
      }
  }
  if (publish) {
    DeviceMem words(256);  // flag, arrive counter, status
    CK(cudaMemset(words.p, 0, 256));
    uint32_t* w = reinterpret_cast<uint32_t*>(words.p);
    launchPush(plan, nullptr, ctas, w, 77, w + 8, w + 16);
    uint32_t after[64];
    CK(cudaMemcpy(after, words.p, 256, cudaMemcpyDeviceToHost));
    EXPECT_EQ(after[0], uint32_t(77));
    EXPECT_EQ(after[8], uint32_t(0));
    EXPECT_EQ(after[16], uint32_t(kStatusOk));
  } else if (!plan.entries.empty()) {
    launchPush(plan, nullptr, ctas, nullptr, 0, nullptr, nullptr);
  }
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(got.data(), ddst.p, got.size(), cudaMemcpyDeviceToHost));
  if (got != want) {
    std::vector<bool> inside(got.size(), false);
    for (size_t i = 0; i < specs.size(); ++i) {
      const Spec& s = specs[i];
      const size_t ed = dtypeSize(s.to);
      for (int64_t q = 0; q < s.rows * s.cols; ++q) {
        const size_t at = dstAt[i] + q * ed;
        std::fill(inside.begin() + at, inside.begin() + at + ed, true);
        if (std::memcmp(&got[at], &want[at], ed) == 0) continue;
        if (s.from != s.to && isNan(&got[at], s.to) && isNan(&want[at], s.to)) continue;
        throw tpbtest::TestFailure("element " + std::to_string(q) + " of " + describe(s) + " differs");
      }
    }
    for (size_t i = 0; i < got.size(); ++i)
      if (!inside[i] && got[i] != 0xCD) throw tpbtest::TestFailure("canary at " + std::to_string(i) + " overwritten");
  }
}

Spec run(size_t bytes, size_t srcOff, size_t dstOff) {
  Spec s;
  s.cols = static_cast<int64_t>(bytes);
  s.srcOff = srcOff;
  s.dstOff = dstOff;
  return s;
}

}  // namespace

// Byte runs whose two ends are aligned differently: every pair of alignments modulo 16, at sizes
// around a vector, a batch of vectors (4 KiB) and a tile (8 KiB).
TPB_GPU_TEST(Kernel, RunsOfEveryRelativeAlignment, 1) {
  for (size_t bytes : {size_t(1), size_t(15), size_t(16), size_t(17), size_t(31), size_t(33), size_t(511), size_t(527),
                       size_t(4095), size_t(4111), size_t(4129), size_t(8191), size_t(8192), size_t(8207), size_t(8209),
                       size_t(16384 + 1), size_t(3 * 8192 + 30), size_t(70001)}) {
    std::vector<Spec> specs;
    for (size_t so = 0; so < 16; ++so)
      for (size_t d = 0; d < 16; ++d) {
        specs.push_back(run(bytes, so, d));
        if (specs.size() == 64) {  // one parameter block holds 96 entries
          checkMessage(specs);
          specs.clear();
        }
      }
  }
  checkMessage({run((9u << 20) + 5, 3, 0), run((3u << 20) + 1, 0, 7), run((1u << 20), 9, 9)});
  checkMessage({run((2u << 20) + 5, 13, 6)}, true, 3);  // fewer warps than tiles
}

// Conversions of contiguous tensors: every pair of types, aligned and not, at sizes around a unit, a
// batch and a tile (8 KiB of destination).
TPB_GPU_TEST(Kernel, ConversionsAtTileEdgesAndAlignments, 1) {
  const DType types[] = {DType::kF32, DType::kBF16, DType::kF16};
  for (DType from : types)
    for (DType to : types) {
      if (from == to) continue;
      const int64_t tile = 8192 / static_cast<int64_t>(dtypeSize(to));
      for (int64_t n : {int64_t(1), int64_t(3), int64_t(4), int64_t(7), int64_t(9), int64_t(127), int64_t(129), int64_t(1023),
                        int64_t(1025), tile - 1, tile, tile + 1, 3 * tile + 5, int64_t(200001)}) {
        std::vector<Spec> specs;
        for (size_t so : {size_t(0), size_t(1), size_t(2), size_t(4)})
          for (size_t d : {size_t(0), size_t(1), size_t(4), size_t(5)}) {
            Spec s;
            s.from = from;
            s.to = to;
            s.cols = n;
            s.srcOff = so * dtypeSize(from);
            s.dstOff = d * dtypeSize(to);
            specs.push_back(s);
          }
        checkMessage(specs);
      }
    }
}

// Views whose rows are contiguous: row lengths from one vector to more than a tile, every mix of
// alignments of source, destination, pitch and length, overlapping rows (stride 0) and conversions.
TPB_GPU_TEST(Kernel, ViewsWithContiguousRows, 1) {
  struct Shape {
    int64_t rows, bytes, gap;
  };
  for (Shape shape : {Shape{1, 16, 0}, Shape{700, 16, 16}, Shape{700, 17, 1}, Shape{700, 31, 2}, Shape{513, 32, 32},
                      Shape{300, 100, 28}, Shape{130, 512, 64}, Shape{130, 520, 1}, Shape{33, 4096, 4096}, Shape{33, 4099, 5},
                      Shape{5, 8192, 16}, Shape{3, 20000, 33}, Shape{2, 100001, 7}, Shape{40, 333, -333}}) {
    std::vector<Spec> specs;
    for (size_t so : {size_t(0), size_t(1), size_t(6), size_t(16)})
      for (size_t d : {size_t(0), size_t(3), size_t(15)}) {
        Spec s;
        s.rows = shape.rows;
        s.cols = shape.bytes;
        s.strided = true;
        s.rowStride = shape.bytes + shape.gap;
        s.srcOff = so;
        s.dstOff = d;
        specs.push_back(s);
      }
    checkMessage(specs);
    checkMessage({specs[3]}, true, 1);
  }
  const DType types[] = {DType::kF32, DType::kBF16, DType::kF16};
  for (DType from : types)
    for (DType to : types)
      for (int64_t cols : {int64_t(16), int64_t(17), int64_t(64), int64_t(100), int64_t(1000), int64_t(4097), int64_t(9000)}) {
        std::vector<Spec> specs;
        for (int64_t gap : {int64_t(0), int64_t(1), int64_t(8)})
          for (size_t off : {size_t(0), size_t(1), size_t(8)}) {
            Spec s;
            s.from = from;
            s.to = to;
            s.rows = 20000 / cols + 2;
            s.cols = cols;
            s.strided = true;
            s.rowStride = cols + gap;
            s.srcOff = off * dtypeSize(from);
            s.dstOff = (off & 1) * dtypeSize(to);
            specs.push_back(s);
          }
        checkMessage(specs);
      }
  // Rows too short for a vector, 8-byte elements, another GPU as the destination.
  Spec narrow;
  narrow.rows = 1000;
  narrow.cols = 7;
  narrow.strided = true;
  narrow.rowStride = 9;
  Spec wide;
  wide.from = wide.to = DType::kI64;
  wide.rows = 77;
  wide.cols = 129;
  wide.strided = true;
  wide.rowStride = 200;
  wide.srcOff = 8;
  wide.remote = true;
  checkMessage({narrow, wide});
}

// The same at every size of tile that a result of such rows is cut into, and at the edges between them.
TPB_GPU_TEST(Kernel, ViewsWithContiguousRowsAtEveryTileSize, 1) {
  const int64_t warps = 148 * 16;
  for (int64_t tile : {512, 1024, 2048, 4608, 7680, 8192})
    for (int64_t cols : {4, 5, 16, 33}) {
      const int64_t rows = warps * tile / (cols * 4);  // the last row at which this tile is taken, or next to it
      std::vector<Spec> specs;
      for (int64_t more : {-1, 0, 1}) {
        Spec s;
        s.from = s.to = DType::kF32;
        s.rows = rows + more;
        s.cols = cols;
        s.strided = true;
        s.rowStride = cols + (more < 0 ? 4 : 1);
        s.srcOff = more < 0 ? 0 : 4;
        s.dstOff = more > 0 ? 4 : 0;
        specs.push_back(s);
      }
      if (cols >= 16) specs[0].to = specs[2].to = DType::kBF16, specs[2].dstOff = 2;
      checkMessage(specs);
    }
}

// Large transposed matrices, which a CTA transposes tile by tile: extents around the tiles (128 columns; 128,
// 64 or 32 rows), narrow matrices whose tiles hold several chunks of rows, odd column strides and addresses,
// every element size, every conversion; alone and beside a tensor on the bulk path.
namespace {
Spec transposed(DType from, DType to, int64_t rows, int64_t cols, int64_t pad, size_t so, size_t d) {
  Spec s;
  s.from = from;
  s.to = to;
  s.rows = rows;
  s.cols = cols;
  s.strided = true;
  s.rowStride = 1;
  s.colStride = rows + pad;
  s.srcOff = so * dtypeSize(from);
  s.dstOff = d * dtypeSize(to);
  return s;
}
uint32_t kindOf(const Spec& s) {
  PushPlan plan;
  CopyItem it;
  it.src = reinterpret_cast<void*>(uintptr_t(0x10000000) + s.srcOff);
  it.dst = reinterpret_cast<void*>(uintptr_t(0x70000000) + s.dstOff);
  it.srcDtype = s.from;
  it.dstDtype = s.to;
  it.srcBytes = static_cast<uint64_t>(s.rows * s.cols) * dtypeSize(s.from);
  it.strided = true;
  it.view = StridedView{s.from, s.rows, s.cols, s.rowStride, s.colStride};
  appendToPlan(plan, it, true);
  return plan.entries.back().kind;
}
std::vector<std::pair<DType, DType>> transposableTypes() {
  std::vector<std::pair<DType, DType>> types = {{DType::kI64, DType::kI64}, {DType::kI32, DType::kI32}, {DType::kI16, DType::kI16}};
  for (DType from : {DType::kF32, DType::kBF16, DType::kF16})
    for (DType to : {DType::kF32, DType::kBF16, DType::kF16})
      if (from != to) types.emplace_back(from, to);
  return types;
}
}  // namespace

TPB_GPU_TEST(Kernel, LargeTransposedMatrices, 1) {
  int turn = 0;
  for (auto [from, to] : transposableTypes()) {
    const int64_t least = static_cast<int64_t>(blockMinBytes(65, dtypeSize(from)) / dtypeSize(from));
    for (int64_t cols : {65, 127, 128, 129, 130, 319, 512})
      for (int64_t extra : {0, 1, 63}) {
        const int64_t rows = (least + cols - 1) / cols / 128 * 128 + 128 + extra;
        const Spec s = transposed(from, to, rows, cols, turn & 1, (turn >> 1) & 1, (turn >> 2) & 1);
        ++turn;
        EXPECT_EQ(int(kindOf(s)), int(kTransposed));
        checkMessage({s});
      }
    const int64_t shortest = static_cast<int64_t>(kBlockMinRowBytes / dtypeSize(from));  // long rows, short columns
    const Spec flat = transposed(from, to, shortest + turn % 3, least / shortest + 1, 0, 0, turn & 1);
    EXPECT_EQ(int(kindOf(flat)), int(kTransposed));
    checkMessage({flat});
  }
}

TPB_GPU_TEST(Kernel, LargeNarrowTransposedMatrices, 1) {
  int turn = 0;
  for (auto [from, to] : transposableTypes()) {
    const int64_t least = static_cast<int64_t>(blockMinBytes(2, dtypeSize(from)) / dtypeSize(from));
    for (int64_t cols : {2, 3, 5, 8, 12, 17, 31, 32, 33, 43, 50, 63, 64}) {
      const int64_t rows = least / cols + 1 + turn % 3;
      const Spec s = transposed(from, to, rows, cols, turn & 1, (turn >> 1) & 1, (turn >> 2) & 1);
      ++turn;
      EXPECT_EQ(int(kindOf(s)), int(kTransposed));
      checkMessage({s});
    }
  }
}

TPB_GPU_TEST(Kernel, LargeTransposedMatricesInOneMessage, 1) {
  const Spec bulk = run(3 << 20, 0, 0);
  std::vector<Spec> specs = {transposed(DType::kBF16, DType::kBF16, 4097, 1027, 0, 0, 1),
                             transposed(DType::kF32, DType::kBF16, 3000, 515, 3, 1, 1),
                             transposed(DType::kI64, DType::kI64, 70001, 9, 0, 0, 1),
                             transposed(DType::kF32, DType::kF32, 40, 30, 0, 0, 0),
                             run(100001, 3, 0),
                             transposed(DType::kF16, DType::kF32, 2048, 2048, 0, 0, 0)};
  checkMessage(specs);           // the light kernel
  checkMessage(specs, true, 3);  // few CTAs
  checkMessage(specs, false);    // no bulk copies: the warp tiles
  specs.push_back(bulk);         // the full one: eight of its warps share the block tiles
  checkMessage(specs);
  checkMessage(specs, true, 3);
}

// More entries than one launch takes: both sides of the cut hold transposed matrices, contiguous rows and plain runs, and
// the tiles of each launch are numbered anew. The flag is published once, behind all of them.
TPB_GPU_TEST(Kernel, MessagesOfMoreThanOneLaunch, 1) {
  for (bool withBulk : {false, true}) {
    std::vector<Spec> specs;
    for (int i = 0; i < 130; ++i) {
      if (i == 3 || i == 95 || i == 96 || i == 120) {
        specs.push_back(transposed(DType::kF32, i == 96 ? DType::kBF16 : DType::kF32, i == 3 ? 180001 : 4099, i == 3 ? 7 : 259 + i, 1, 0, i & 1));
      } else if (i % 10 == 5) {
        Spec s;
        s.from = s.to = DType::kI64;
        s.rows = 100 + i;
        s.cols = 5 + i % 3;
        s.strided = true;
        s.rowStride = s.cols + 2;
        specs.push_back(s);
      } else if (withBulk && (i == 50 || i == 110)) {
        specs.push_back(run(1 << 20, 0, 0));
      } else {
        specs.push_back(run(1000 + 37 * i, i % 16, (i * 7) % 16));
      }
    }
    checkMessage(specs, true, 148, true);
    checkMessage(specs, true, 5, true);
  }
}

// A column that stands for all (stride 0), as an expanded tensor has it.
TPB_GPU_TEST(Kernel, TransposedMatricesOfOneRepeatedColumn, 1) {
  for (int64_t cols : {3, 64, 129}) {
    Spec s = transposed(DType::kF32, DType::kF32, (5 << 20) / 4 / cols, cols, 0, 1, 0);
    s.colStride = 0;
    EXPECT_EQ(int(kindOf(s)), int(kTransposed));
    checkMessage({s});
    s.to = DType::kBF16;
    checkMessage({s, run(1 << 20, 0, 0)});
  }
}
