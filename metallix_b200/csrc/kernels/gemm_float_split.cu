// C[M, N] = A[M, K] * W[N, K]^T of float32 operands on the fifth-generation tensor cores, with float32's precision.
//
// A float32 number is the sum of three bfloat16 numbers, x = x1 + x2 + x3, each the rounding of what the ones before
// left: 8 bits each, 24 together (Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for
// higher-precision computations", ARITH 2019). Of the nine products of two such numbers six are made: x1 y1, x1 y2, x2 y1, x2 y2, x1 y3
// and x3 y1; what is left out is at most 2^-24 of |x y|, and 2^-27 on average. Products of bfloat16 are exact; what
// limits the result is how they are added up. The tensor core cuts sums off where it aligns them, so x1 y1 is summed
// over 64 k at a time and these sums are added up in registers, rounded to nearest; the five small products have an
// accumulator of their own, whose errors are 2^-8 of the large one's. Against 64 bits the result is closer than a
// float32 sum in ascending k: 1.0e-7 and 5.7e-7 at k = 1,024, 1.2e-7 and 9.9e-7 at 3,072 (normal numbers; positive ones 1.0e-7 and 4.9e-7).
//
// What bounds it: the tensor core, 6 x 64 cycles per 16 k of a 128 x 128 tile. The operands are read as float32 and
// split by eight warps (5.5 instructions a value) on their way to shared memory: no pass over W beforehand and no room for
// it. 917 rows (us, against the CUDA cores' kernel): 4096 x 1024 77 and 213, 6144 x 1024 110 and 261, 1024 x 2048 50 and 128, 1024 x
// 3072 65 and 188, 4096 x 12288 745 and 2,465: 77 to 124 TFLOP/s of float32, 460 to 740 of the tensor core's. Without the
// splitters' arithmetic the first of these took 50 us of 70, without their loads 55: a load has two steps to arrive in (with one
// 72 us), and they are volatile because the compiler moved them down to their use (100 us).
//
// A row's bits do not depend on what other rows there are: how the sums over k are grouped follows from n and k alone. Few
// rows give each group to a block of its own and add the groups up in a second kernel; with many, a tile's block takes
// its groups one after the other, and their sum stays in tensor memory, in the same order. (With as many parts of k as the
// rows left room for, 917 rows took 70, 105, 43 and 58 us of the first four.)
//
// A number that is not finite, or too near the largest, has no such parts (infinity minus infinity), and leaves an output that is
// not finite. A number below 2^-102 has parts that bfloat16 holds with fewer bits or not at all, which leaves up to 2^-126 of it
// out: 2^-24 of an output from 2^-60 on, as long as the other operands add up to no more than 2^42. Outputs that are not finite, or nearer 0 but
// not 0, are made again in float32 and ascending k, with the general product's bits, tile by tile, by the
// adders of a block once it has walked all of its tiles (nobody waits for them any more), or by the kernel that adds the groups up.
// 917 rows x 4096 x 1024: 77 us, some 90 more with a row of NaN, 680 more with nothing else (the CUDA cores' kernel 213).
//
// Every wait on a barrier is bounded: if it runs out, the status word gets a bit and the block stops, frees its tensor
// memory and leaves.
#include <cfloat>

#include "tcgen05.cuh"

namespace mxb {

constexpr int kSplitTile = 128;          // rows of A and of W a tile
constexpr int kSplitStep = 32;           // k that are handed over at once, half a 128-byte row of bfloat16
constexpr int kSplitChunk = 64;          // k that the tensor core sums up
constexpr int kSplitSlots = 4;           // steps in shared memory: two stages of 64 k, each in halves
constexpr int kSplitPlaneBytes = kSplitTile * kSplitChunk * 2;
constexpr int kSplitStageBytes = 6 * kSplitPlaneBytes;   // three parts of A, three of W
constexpr int kSplitAdders = 8, kSplitSplitters = 8;     // warps
constexpr int kSplitPutPitch = 20;       // floats: eight rows' 16 bytes in different banks
constexpr int kSplitPutBytes = kSplitAdders * 32 * kSplitPutPitch * 4;   // where the adders turn their results around
constexpr int kSplitSharedBytes = 2 * kSplitStageBytes + kSplitPutBytes + 1024;
constexpr int kSplitThreads = 32 * (4 + kSplitAdders + kSplitSplitters);   // warpgroups: one that issues, two and two
constexpr int kSplitTmemColumns = 512;   // large sums twice, then small sums twice, or once and the sum of the groups so far

constexpr float kSplitLeast = 8.67361738e-19f;   // 2^-60

// An output that the parts cannot be trusted with: not finite, or so near 0 (but not 0, which rows of zeros give) that it may
// be made of numbers whose smallest parts bfloat16 does not reach.
__device__ __forceinline__ bool is_doubtful(float x) { return !(fabsf(x) <= FLT_MAX) || (fabsf(x) < kSplitLeast && x != 0.0f); }

// Two numbers' leading bfloat16 parts, packed; the numbers become what that left.
__device__ __forceinline__ uint32_t split_pair(float& x, float& y) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(x, y);
  const uint32_t packed = *reinterpret_cast<const uint32_t*>(&pair);
  x -= __uint_as_float(packed << 16);
  y -= __uint_as_float(packed & 0xffff0000u);
  return packed;
}

// The products that are made again: tiles of 32 x 128 by 256 threads, each 2 rows x two times 4 columns.
constexpr int kAgainRows = 32, kAgainColumns = 128, kAgainK = 16, kAgainThreads = 256;
constexpr int kAgainShared = kAgainK * (kAgainRows + 4 + kAgainColumns + 4);   // floats
static_assert(kAgainThreads == 32 * kSplitAdders, "a block's adders make them");

// Where the 256 threads meet: whether one of them says yes.
__device__ __forceinline__ bool again_any(bool mine) {
  int any;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.s32 p, %1, 0;\n"
      "barrier.cta.red.or.pred q, 1, 256, p;\n"
      "selp.s32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(any) : "r"(static_cast<int>(mine)) : "memory");
  return any != 0;
}
__device__ __forceinline__ int again_row(int t, int i) { return (t >> 4) * 2 + i; }
__device__ __forceinline__ int again_column(int t, int j) { return (t & 15) * 4 + (j >> 2) * 64 + (j & 3); }

// The tile's doubtful outputs, as sums in ascending k; v are this thread's. False where there are none.
__device__ __forceinline__ bool make_again(float (&v)[2][8], float* shared, int t, int row0, int col0, const float* __restrict__ a,
                                           const float* __restrict__ w, int m, int n, int k, long long lda, long long ldw) {
  bool odd = false;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) odd = odd || is_doubtful(v[i][j]);
  if (!again_any(odd)) return false;
  float* sA = shared;                                  // [kAgainK][kAgainRows + 4]
  float* sW = shared + kAgainK * (kAgainRows + 4);     // [kAgainK][kAgainColumns + 4]
  float acc[2][8] = {};
  for (int k0 = 0; k0 < k; k0 += kAgainK) {
    auto bring = [&](float* to, int pitch, const float* from, long long ld, int rows, int first, int e) {   // k is a multiple of 4
      const int row = e >> 2, at = (e & 3) * 4;
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (first + row < rows && k0 + at < k) x = *reinterpret_cast<const float4*>(from + (first + row) * ld + k0 + at);
      to[at * pitch + row] = x.x;
      to[(at + 1) * pitch + row] = x.y;
      to[(at + 2) * pitch + row] = x.z;
      to[(at + 3) * pitch + row] = x.w;
    };
    if (t < kAgainRows * 4) bring(sA, kAgainRows + 4, a, lda, m, row0, t);
#pragma unroll
    for (int e = 0; e < 2; ++e) bring(sW, kAgainColumns + 4, w, ldw, n, col0, t + e * kAgainThreads);
    again_any(false);
#pragma unroll 4
    for (int kk = 0; kk < kAgainK; ++kk) {
      const float2 x = *reinterpret_cast<const float2*>(sA + kk * (kAgainRows + 4) + again_row(t, 0));
      const float4 y = *reinterpret_cast<const float4*>(sW + kk * (kAgainColumns + 4) + again_column(t, 0));
      const float4 z = *reinterpret_cast<const float4*>(sW + kk * (kAgainColumns + 4) + again_column(t, 4));
      const float rows[2] = {x.x, x.y}, columns[8] = {y.x, y.y, y.z, y.w, z.x, z.y, z.z, z.w};
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(rows[i], columns[j], acc[i][j]);
    }
    again_any(false);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (is_doubtful(v[i][j])) v[i][j] = acc[i][j];
  return true;
}

__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_float_split_kernel(float* __restrict__ c, const float* __restrict__ a, const float* __restrict__ w, int m, int n, int k,
                        long long lda, long long ldw, long long ldc, int groups, int slices, float* __restrict__ scratch, int* status) {
  extern __shared__ unsigned char split_shared_raw[];
  __shared__ __align__(8) uint64_t step_full[kSplitSlots], step_empty[kSplitSlots];
  __shared__ __align__(8) uint64_t large_full[2], large_empty[2], small_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int failed_slot;
  volatile int& failed = failed_slot;
  unsigned char* stages = split_shared_raw + ((1024 - (shared_address(split_shared_raw) & 1023)) & 1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tiles = ceil_div(m, kSplitTile), n_tiles = ceil_div(n, kSplitTile);
  const int chunks = ceil_div(k, kSplitChunk);
  const int units = m_tiles * n_tiles * slices;   // (tile, slice: some groups of k side by side), the row tile fastest

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSplitSlots; ++s) {
      barrier_init(&step_full[s], kSplitSplitters);
      barrier_init(&step_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      barrier_init(&large_full[b], 1);
      barrier_init(&large_empty[b], kSplitAdders);
      barrier_init(&small_empty[b], kSplitAdders);
    }
    barrier_init_fence();
    failed = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                 ::"r"(shared_address(&tmem_base_slot)), "r"(kSplitTmemColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  auto first_group = [&](int unit, int after) { return (unit / m_tiles % slices + after) * groups / slices; };   // after 1: of the next slice
  // All groups of a tile one after the other in one block: their sum lies in tensor memory meanwhile, where else the second
  // accumulator of small sums is.
  const bool chained = slices == 1 && groups > 1;
  auto small_of = [&](int local) { return chained ? 0 : local & 1; };
  auto small_turn = [&](int local) { return static_cast<uint32_t>(chained ? local & 1 : (local >> 1) & 1); };
  auto first_chunk = [&](int group) { return static_cast<int>(static_cast<long long>(group) * chunks / groups); };

  // 640 threads start with 96 registers each; the adders' 64 sums want more and the issuing warps need few.
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n");
    // ---- one thread issues every MMA
    if (warp == 0) {
      constexpr uint32_t idesc = tc_instruction_descriptor(kSplitTile, kSplitTile);
      const uint64_t desc = tc_smem_descriptor(shared_address(stages));
      int step = 0, chunk_count = 0, local = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < units && ok && !given_up(failed); unit += gridDim.x) {
        for (int group = first_group(unit, 0), last = first_group(unit, 1); group < last && ok; ++group, ++local) {
          const int begin = first_chunk(group), end = first_chunk(group + 1);
          const uint32_t tmem_small = tmem_base + (2 + small_of(local)) * kSplitTile;
          ok = barrier_wait_warp(&small_empty[small_of(local)], small_turn(local) ^ 1, status);
          for (int chunk = begin; chunk < end && ok; ++chunk, ++chunk_count) {
            const int buffer = chunk_count & 1;
            ok = barrier_wait_warp(&large_empty[buffer], ((chunk_count >> 1) & 1) ^ 1, status);
            const uint32_t tmem_large = tmem_base + buffer * kSplitTile;
#pragma unroll
            for (int half = 0; half < 2; ++half, ++step) {
              const int slot = step % kSplitSlots;
              ok = ok && barrier_wait_warp(&step_full[slot], (step / kSplitSlots) & 1, status);
              if (!ok) break;
              tc_fence_after_sync();
              if (elect_one()) {
                const uint64_t at = desc + (((slot >> 1) * kSplitStageBytes + half * kSplitStep * 2) >> 4);
                constexpr uint64_t plane = kSplitPlaneBytes >> 4;
#pragma unroll
                for (int kk = 0; kk < kSplitStep / 16; ++kk) {
                  const uint64_t x = at + kk * 2, y = x + 3 * plane;
                  tc_mma(tmem_small, x, y + 2 * plane, idesc, chunk > begin || half > 0 || kk > 0 ? 1u : 0u);
                  tc_mma(tmem_small, x + 2 * plane, y, idesc, 1u);
                  tc_mma(tmem_small, x + plane, y + plane, idesc, 1u);
                  tc_mma(tmem_small, x, y + plane, idesc, 1u);
                  tc_mma(tmem_small, x + plane, y, idesc, 1u);
                  tc_mma(tmem_large, x, y, idesc, half > 0 || kk > 0 ? 1u : 0u);
                }
                tc_commit(&step_empty[slot]);
                if (half == 1) tc_commit(&large_full[buffer]);   // the last one of a tile covers its small sums too
              }
            }
          }
        }
      }
      if (!ok) failed = 1;
    }
  } else if (warp < 4 + kSplitAdders) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n");   // 128 x 32 + 256 x 112 + 256 x 112 = 640 x 96 at most
    // ---- adders: two warps per 32 rows, 64 columns each
    const int lane_base = (warp & 3) * 32, columns = ((warp - 4) >> 2) * 64;
    const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(lane_base) << 16) + columns;
    float* turned = reinterpret_cast<float*>(stages + 2 * kSplitStageBytes) + (warp - 4) * 32 * kSplitPutPitch;
    int chunk_count = 0, local = 0;
    bool ok = true, odd = false;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
      for (int group = first_group(unit, 0), last = first_group(unit, 1); group < last; ++group, ++local) {
        const int begin = first_chunk(group), end = first_chunk(group + 1);
        float acc[64];
#pragma unroll
        for (int i = 0; i < 64; ++i) acc[i] = 0.0f;
        for (int chunk = begin; chunk < end; ++chunk, ++chunk_count) {
          const int buffer = chunk_count & 1;
          if (!barrier_wait_warp(&large_full[buffer], (chunk_count >> 1) & 1, status) || given_up(failed)) { ok = false; break; }
          tc_fence_after_sync();
#pragma unroll
          for (int part = 0; part < 4; ++part) {
            uint32_t sum[16];
            tc_load_16(tmem_lane + buffer * kSplitTile + part * 16, sum);
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[part * 16 + i] += __uint_as_float(sum[i]);
          }
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) barrier_arrive(&large_empty[buffer]);
        }
        if (!ok) break;
#pragma unroll
        for (int part = 0; part < 4; ++part) {
          uint32_t sum[16];
          tc_load_16(tmem_lane + (2 + small_of(local)) * kSplitTile + part * 16, sum);
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[part * 16 + i] += __uint_as_float(sum[i]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) barrier_arrive(&small_empty[small_of(local)]);
        if (chained && group > 0) {   // eight columns at a time: sixteen did not leave the other roles their registers
#pragma unroll
          for (int part = 0; part < 64; part += 8) {
            uint32_t sum[8];
            tc_load_8(tmem_lane + 3 * kSplitTile + part, sum);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[part + i] += __uint_as_float(sum[i]);
          }
        }
        if (chained && group + 1 < last) {
#pragma unroll
          for (int part = 0; part < 64; part += 8) {
            uint32_t sum[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) sum[i] = __float_as_uint(acc[part + i]);
            tc_store_8(tmem_lane + 3 * kSplitTile + part, sum);
          }
          tc_store_wait();
        } else {
          const int row0 = unit % m_tiles * kSplitTile + lane_base, column0 = unit / m_tiles / slices * kSplitTile + columns;
          float* to = slices > 1 ? scratch + static_cast<long long>(group) * m * n : c;
          const long long ld = slices > 1 ? n : ldc;
          const bool quads = (reinterpret_cast<uintptr_t>(to) & 15) == 0 && ld % 4 == 0;
          // 16 columns at a time by way of shared memory, so that a store takes 64 bytes of eight rows and not 16 of all 32,
          // which kept the adders some 4 us a tile.
#pragma unroll
          for (int part = 0; part < 4; ++part) {
#pragma unroll
            for (int i = 0; i < 16; i += 4)
              *reinterpret_cast<float4*>(turned + lane * kSplitPutPitch + i) =
                  make_float4(acc[part * 16 + i], acc[part * 16 + i + 1], acc[part * 16 + i + 2], acc[part * 16 + i + 3]);
            __syncwarp();
            const int column = column0 + part * 16 + (lane & 3) * 4;
#pragma unroll 1
            for (int r = lane >> 2; r < 32; r += 8) {
              const float4 x = *reinterpret_cast<const float4*>(turned + r * kSplitPutPitch + (lane & 3) * 4);
              if (row0 + r < m) {
                odd = odd || is_doubtful(x.x) || is_doubtful(x.y) || is_doubtful(x.z) || is_doubtful(x.w);
                float* at = to + (row0 + r) * ld + column;
                if (quads && column + 4 <= n) {
                  *reinterpret_cast<float4*>(at) = x;
                } else {
                  if (column < n) at[0] = x.x;
                  if (column + 1 < n) at[1] = x.y;
                  if (column + 2 < n) at[2] = x.z;
                  if (column + 3 < n) at[3] = x.w;
                }
              }
            }
            __syncwarp();   // the next 16 columns go where these were; tensor memory is loaded by the warp as a whole
          }
        }
      }
    }
    if (!ok) failed = 1;
    // Every product of the block's is finished where all of these waits ended: nothing reads or writes the stages any more.
    if (slices == 1 && again_any(odd) && !again_any(!ok)) {
      const int t = threadIdx.x - 4 * 32;
      for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int col0 = unit / m_tiles * kSplitTile;
        for (int row0 = unit % m_tiles * kSplitTile; row0 < (unit % m_tiles + 1) * kSplitTile && row0 < m; row0 += kAgainRows) {
          float v[2][8];
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int row = row0 + again_row(t, i), column = col0 + again_column(t, j);
              v[i][j] = row < m && column < n ? c[row * ldc + column] : 0.0f;
            }
          if (!make_again(v, reinterpret_cast<float*>(stages), t, row0, col0, a, w, m, n, k, lda, ldw)) continue;
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int row = row0 + again_row(t, i), column = col0 + again_column(t, j);
              if (row < m && column < n) c[row * ldc + column] = v[i][j];
            }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n");
    // ---- splitters: float32 from memory, two steps ahead in registers, to three bfloat16 tiles each in shared memory
    const int t = threadIdx.x - 32 * (4 + kSplitAdders);
    // Eight lanes bring a row's 128 bytes. A half-warp's two rows are four apart, so that the swizzle puts their 64 bytes a
    // part into different banks.
    const int quad = t & 7, eight = t >> 3;
    const int row_in = (eight & ~7) | ((eight & 1) << 2) | ((eight >> 1) & 3);   // of 32 rows a pass
    const float* rows[8];   // of A and of W that this thread brings; rows behind the last one bring that one again
    int unit = blockIdx.x, at = 0, last = 0;   // the step that is fetched next
    auto open = [&]() {
      at = first_chunk(first_group(unit, 0)) * 2, last = first_chunk(first_group(unit, 1)) * 2;
      const int rows_a = unit % m_tiles * kSplitTile + row_in, rows_w = unit / m_tiles / slices * kSplitTile + row_in;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        rows[i] = a + min(rows_a + i * 32, m - 1) * lda;
        rows[4 + i] = w + min(rows_w + i * 32, n - 1) * ldw;
      }
    };
    auto fetch = [&](int i) {   // volatile: a load that the compiler moves down to its use is waited for there
      const float* from = rows[i] + min(at * kSplitStep + quad * 4, k - 4);
      float4 v;
      asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(from));
      return v;
    };
    bool more = unit < units;   // a step is left to be fetched
    if (more) open();
    auto advance = [&]() {
      if (++at == last) {
        unit += gridDim.x;
        more = unit < units;
        if (more) open();
      }
    };
    struct Fetched {
      float4 four[8];
      bool held, beyond;   // there is one; it lies behind the end of k
    } first, second;       // two steps under way
    auto fill = [&](Fetched& f) {
      f.held = more;
      if (!more) return;
      f.beyond = at * kSplitStep + quad * 4 >= k;
#pragma unroll
      for (int i = 0; i < 8; ++i) f.four[i] = fetch(i);
      advance();
    };
    fill(first);
    fill(second);
    int step = 0;
    bool ok = true;
    auto split_step = [&](Fetched& f) {
      if (!f.held) return false;
      const int slot = step % kSplitSlots;
      ok = barrier_wait_warp(&step_empty[slot], ((step / kSplitSlots) & 1) ^ 1, status);
      if (!ok || given_up(failed)) return false;
      unsigned char* stage = stages + (slot >> 1) * kSplitStageBytes;
      const int piece = (slot & 1) * 4 + (quad >> 1);   // of 16 bytes in the row of 128
      const bool beyond = f.beyond;
      f.held = more;
      f.beyond = at * kSplitStep + quad * 4 >= k;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float4 now = f.four[i];
        if (more) f.four[i] = fetch(i);   // has two steps' time to arrive
        if (beyond) now = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const int row = (i & 3) * 32 + row_in;
        unsigned char* to = stage + (i < 4 ? 0 : 3) * kSplitPlaneBytes + row * 128 + ((piece ^ (row & 7)) << 4) + (quad & 1) * 8;
#pragma unroll
        for (int part = 0; part < 3; ++part) {
          const uint32_t low = split_pair(now.x, now.y), high = split_pair(now.z, now.w);
          *reinterpret_cast<uint2*>(to + part * kSplitPlaneBytes) = make_uint2(low, high);
        }
      }
      if (more) advance();
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // before the tensor core reads them
      __syncwarp();
      if (lane == 0) barrier_arrive(&step_full[slot]);
      ++step;
      return true;
    };
    while (split_step(first) && split_step(second)) {
    }
    if (!ok) failed = 1;
  }

  tc_fence_before_sync();
  __syncthreads();
  if (failed && threadIdx.x == 0) {
    // A wait ran out somewhere. Give products that may still be under way a
    // millisecond before the block's memory goes back.
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kSplitTmemColumns) : "memory");
}

// The groups of k, in order: a block a tile of 32 x 128.
__global__ void __launch_bounds__(kAgainThreads)
gemm_float_groups_kernel(float* __restrict__ c, const float* __restrict__ scratch, const float* __restrict__ a,
                        const float* __restrict__ w, int m, int n, int k, long long lda, long long ldw, long long ldc, int groups) {
  __shared__ __align__(16) float shared[kAgainShared];
  const int t = threadIdx.x, row0 = blockIdx.x * kAgainRows, col0 = blockIdx.y * kAgainColumns;
  const size_t all = static_cast<size_t>(m) * n;
  const bool quads = n % 4 == 0;
  float v[2][8] = {};
#pragma unroll 4
  for (int s = 0; s < groups; ++s)   // the loads of several groups are under way at once
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const int row = row0 + again_row(t, i), column = col0 + again_column(t, j);
        const float* from = scratch + s * all + static_cast<size_t>(row) * n + column;
        if (quads) {
          const float4 x = row < m && column < n ? *reinterpret_cast<const float4*>(from) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          v[i][j] += x.x, v[i][j + 1] += x.y, v[i][j + 2] += x.z, v[i][j + 3] += x.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) v[i][j + e] += row < m && column + e < n ? from[e] : 0.0f;
        }
      }
  make_again(v, shared, t, row0, col0, a, w, m, n, k, lda, ldw);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      const int row = row0 + again_row(t, i), column = col0 + again_column(t, j);
      if (row >= m || column >= n) continue;
      float* to = c + row * ldc + column;
      if (quads && (reinterpret_cast<uintptr_t>(to) & 15) == 0) {
        *reinterpret_cast<float4*>(to) = make_float4(v[i][j], v[i][j + 1], v[i][j + 2], v[i][j + 3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (column + e < n) to[e] = v[i][j + e];
      }
    }
}

}  // namespace mxb

using namespace mxb;

// Into how many groups the sums over k are cut: by n and k alone, so that a row of A has the same bits whatever else is in the
// batch. As many as one round of 148 blocks takes where there is one tile of rows, none shorter than four chunks.
MXB_API int mxb_gemm_float_split_groups(int n, int k) {
  const int chunks = ceil_div(k, kSplitChunk), fitting = 148 / ceil_div(n, kSplitTile);
  const int most = chunks / 4 < 8 ? chunks / 4 : 8;
  const int groups = fitting < most ? fitting : most;
  return groups > 1 ? groups : 1;
}

// How the groups are dealt out: all to the block of their tile, which adds them up as it goes (1), or in slices to several
// blocks, which leave each group's sums in scratch for a second kernel. The fewest rounds of 148 blocks, each with a start
// worth about two chunks (a chunk is 2.1 us); with several slices the second kernel (worth three) and the sums' way through
// memory, 30 MB a chunk. us with one slice and with the best number: 917 rows x 1024 x 2048 74 and 50 (2 slices), x 1024 x 3072
// 104 and 65 (2), x 4096 x 1024 77 and 77 (1); 8 rows 75 and 20 (8), 106 and 24 (8), 42 and 19 (4).
MXB_API int mxb_gemm_float_split_slices(int m, int n, int k) {
  const long long tiles = static_cast<long long>(ceil_div(m, kSplitTile)) * ceil_div(n, kSplitTile);
  const int chunks = ceil_div(k, kSplitChunk), groups = mxb_gemm_float_split_groups(n, k);
  int best = 1;
  long long least = 0;
  for (int slices = 1; slices <= groups; ++slices) {
    const long long through_memory = slices > 1 ? 3 + 8LL * groups * m * n / 30000000 : 0;
    const long long cost = (tiles * slices + 147) / 148 * (ceil_div(ceil_div(groups, slices) * chunks, groups) + 2) + through_memory;
    if (slices == 1 || cost < least) least = cost, best = slices;
  }
  return best;
}

// c, a, w float32; k and the row strides of a and w multiples of 4, a and w on 16 bytes; scratch: groups * m * n float32 where
// slices > 1.
MXB_API int mxb_gemm_float_split(void* c, const void* a, const void* w, int m, int n, int k, long long lda, long long ldw,
                                 long long ldc, int groups, int slices, float* scratch, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0 || k % 4 != 0 || lda % 4 != 0 || ldw % 4 != 0 || ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) != 0 ||
      groups < 1 || groups > ceil_div(k, kSplitChunk) || slices < 1 || slices > groups || (slices > 1 && scratch == nullptr))
    return static_cast<int>(cudaErrorInvalidValue);
  const long long units = static_cast<long long>(ceil_div(m, kSplitTile)) * ceil_div(n, kSplitTile) * slices;
  if (units > 0x7fffffffLL) return static_cast<int>(cudaErrorInvalidValue);
  int device = 0, sms = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaError_t e = cudaFuncSetAttribute(gemm_float_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSharedBytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  float* to = static_cast<float*>(c);
  const float *x = static_cast<const float*>(a), *weight = static_cast<const float*>(w);
  gemm_float_split_kernel<<<static_cast<int>(units < sms ? units : sms), kSplitThreads, kSplitSharedBytes, stream>>>(
      to, x, weight, m, n, k, lda, ldw, ldc, groups, slices, scratch, status);
  e = cudaGetLastError();
  if (e != cudaSuccess || slices == 1) return static_cast<int>(e);
  gemm_float_groups_kernel<<<dim3(ceil_div(m, kAgainRows), ceil_div(n, kAgainColumns)), kAgainThreads, 0, stream>>>(
      to, scratch, x, weight, m, n, k, lda, ldw, ldc, groups);
  return static_cast<int>(cudaGetLastError());
}
