// Copies whole pages (or state slots) inside a pool: what a forked request
// needs of its parent's partly filled last page, and the zeros a new request's
// state starts from. The reference copies a shared partial block before a
// sequence writes into it (crates/core/engine/src/manager.rs:749-763, the copy
// itself being the caller's); here all copies of a fork are one launch.
//
// Bound by how many bytes are in flight: a block moves one piece of 16 KB,
// each thread four 16-byte words that are all asked for before the first is
// stored, and a unit is cut into as many pieces as it has. One block per unit
// left a request's recurrence state (2 to 4 MB) to a single SM: 0.06 TB/s read
// and written, 985 us for a fork's seven copies. Sixteen such forks and four
// decode steps behind them took 22.7 ms that way, 6.1 ms in pieces.
#include "common.cuh"

namespace mxb {

constexpr int kCopyThreads = 256;
constexpr int kCopyWords = 4;                                        // 16-byte words a thread has in flight
constexpr long long kCopyPiece = 16LL * kCopyThreads * kCopyWords;   // bytes a block moves
constexpr int kMaxSpans = 32;                                        // spans a launch takes (in its parameters)

// `entries` runs of `bytes`, `stride` apart on both sides; no source: zeros.
struct CopySpan {
  unsigned char* to;
  const unsigned char* from;
  long long bytes, stride;
  int entries;
  int first_block;   // of the launch
};
struct CopySpans {
  CopySpan span[kMaxSpans];
  int count;
};

template <typename Word>
__device__ __forceinline__ void copy_piece(unsigned char* to, const unsigned char* from, long long bytes, long long piece) {
  const long long words = bytes / static_cast<long long>(sizeof(Word));
  const long long per_piece = kCopyPiece / static_cast<long long>(sizeof(Word));
  const long long begin = piece * per_piece, end = begin + per_piece < words ? begin + per_piece : words;
  Word* target = reinterpret_cast<Word*>(to);
  const Word* source = reinterpret_cast<const Word*>(from);
  for (long long base = begin + threadIdx.x; base < end; base += kCopyThreads * kCopyWords) {
    Word held[kCopyWords];
#pragma unroll
    for (int i = 0; i < kCopyWords; ++i) {
      const long long at = base + i * kCopyThreads;
      held[i] = source != nullptr && at < end ? source[at] : Word{};
    }
#pragma unroll
    for (int i = 0; i < kCopyWords; ++i) {
      const long long at = base + i * kCopyThreads;
      if (at < end) target[at] = held[i];
    }
  }
}

__device__ __forceinline__ void copy_widest(unsigned char* to, const unsigned char* from, long long bytes, long long piece) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(to) | reinterpret_cast<uintptr_t>(from) | static_cast<uintptr_t>(bytes);
  if (all % 16 == 0) copy_piece<uint4>(to, from, bytes, piece);
  else if (all % 4 == 0) copy_piece<uint32_t>(to, from, bytes, piece);
  else copy_piece<unsigned char>(to, from, bytes, piece);
}

// Block (pair, entry, piece) copies a piece of unit pairs[pair].x to unit
// pairs[pair].y of one entry, in the widest words the addresses allow.
__global__ void __launch_bounds__(kCopyThreads) copy_units_kernel(
    unsigned char* __restrict__ pool, const int2* __restrict__ pairs, long long unit_bytes, int units,
    int* __restrict__ status) {
  const int2 pair = pairs[blockIdx.x];
  if (pair.x < 0 || pair.x >= units || pair.y < 0 || pair.y >= units) {
    if (threadIdx.x == 0) atomicOr(status, kStatusBadPage);
    return;
  }
  if (pair.x == pair.y) return;
  unsigned char* entry = pool + static_cast<size_t>(blockIdx.y) * units * unit_bytes;
  const long long pieces = (unit_bytes + kCopyPiece - 1) / kCopyPiece;
  for (long long piece = blockIdx.z; piece < pieces; piece += gridDim.z)
    copy_widest(entry + static_cast<size_t>(pair.y) * unit_bytes, entry + static_cast<size_t>(pair.x) * unit_bytes,
                unit_bytes, piece);
}

__global__ void __launch_bounds__(kCopyThreads) copy_spans_kernel(const __grid_constant__ CopySpans list) {
  int at = 0;
  while (at + 1 < list.count && static_cast<int>(blockIdx.x) >= list.span[at + 1].first_block) ++at;
  const CopySpan& span = list.span[at];
  const int pieces = static_cast<int>((span.bytes + kCopyPiece - 1) / kCopyPiece);
  const int block = static_cast<int>(blockIdx.x) - span.first_block;
  const long long offset = static_cast<long long>(block / pieces) * span.stride;
  copy_widest(span.to + offset, span.from == nullptr ? nullptr : span.from + offset, span.bytes, block % pieces);
}

}  // namespace mxb

using namespace mxb;

// pool: [entries, units, unit_bytes] bytes on the device; pairs: [count] (source
// unit, target unit) on the device. Source and target units of one call must
// not overlap each other's targets (a target is never another pair's source).
MXB_API int mxb_copy_units(void* pool, int entries, int units, long long unit_bytes, const void* pairs,
                           int count, int* status, cudaStream_t stream) {
  if (count <= 0 || entries <= 0 || unit_bytes <= 0) return 0;
  if (entries > 65535) return static_cast<int>(cudaErrorInvalidValue);
  const long long pieces = (unit_bytes + kCopyPiece - 1) / kCopyPiece;
  const dim3 grid(static_cast<unsigned>(count), static_cast<unsigned>(entries),
                  static_cast<unsigned>(pieces < 65535 ? pieces : 65535));
  copy_units_kernel<<<grid, kCopyThreads, 0, stream>>>(static_cast<unsigned char*>(pool), static_cast<const int2*>(pairs),
                                                       unit_bytes, units, status);
  return static_cast<int>(cudaGetLastError());
}

// spans: on the host, [count][5] of (target address, source address or 0 for
// zeros, bytes, stride, entries): `entries` runs of `bytes` on the device,
// `stride` bytes from one to the next on both sides. No target may overlap
// another span's source. The list travels in the kernel's parameters, so the
// host neither waits for a copy of it nor keeps it.
MXB_API int mxb_copy_spans(const long long* spans, int count, cudaStream_t stream) {
  CopySpans list;
  list.count = 0;
  long long blocks = 0;
  for (int i = 0; i <= count; ++i) {
    const long long* s = spans + 5 * static_cast<size_t>(i);
    const bool some = i < count && s[2] > 0 && s[4] > 0;
    const long long more = some ? s[4] * ((s[2] + kCopyPiece - 1) / kCopyPiece) : 0;
    if (more > 0x7fffffffLL) return static_cast<int>(cudaErrorInvalidValue);
    if (list.count > 0 && (i == count || list.count == kMaxSpans || blocks + more > 0x7fffffffLL)) {
      copy_spans_kernel<<<static_cast<unsigned>(blocks), kCopyThreads, 0, stream>>>(list);
      const cudaError_t error = cudaGetLastError();
      if (error != cudaSuccess) return static_cast<int>(error);
      list.count = 0;
      blocks = 0;
    }
    if (!some) continue;
    list.span[list.count++] = {reinterpret_cast<unsigned char*>(s[0]), reinterpret_cast<const unsigned char*>(s[1]), s[2],
                               s[3], static_cast<int>(s[4]), static_cast<int>(blocks)};
    blocks += more;
  }
  return 0;
}
