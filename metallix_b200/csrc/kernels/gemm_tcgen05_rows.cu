// C[M, N] = A[M, K] * W[N, K]^T in bfloat16 for up to 64 rows of A, one matrix or (grouped) an expert's matrix for each of
// several tiles of up to 64 rows: steps of single tokens over wide layers.
//
// What bounds it: reading W once. The tensor core multiplies 128 rows whatever M is, at a hundredth of its rate, so all
// that counts is how much of W is on its way: each block keeps up to 24 stages of 128 k under way by TMA, of which A's part
// is its few rows only (the instruction reads 128 rows from there on: what it finds behind them makes accumulator rows
// that nobody stores), and W's rows are dealt out so that one round of 148 blocks, or several full ones, takes them all.
// An instruction takes 40 cycles however narrow its tile is, so a block of 128 k takes some 450: tiles of a few rows of W
// are bound by that (4096 x 4096 at 8 rows 15.8 us, 12.3 in the load-based kernel), tall matrices by W, and so are
// experts: 16 tokens over 13 of 6144 x 4096 136 -> 117 us (5.6 TB/s), 3 tokens over 1536 x 1024 18.4 ->
// 10.3, where tiles of 128 rows and 256 columns leave SMs idle in the last round.
//
// Warp 0 feeds the stages, warp 1 issues the MMAs, warps 2..9 run the epilogues of gemm_tcgen05_kernel (the accumulators'
// bits are the same: k in the same order). Two accumulators in tensor memory, tiles in turn. Every wait on a
// barrier is bounded: if it runs out, the status word gets a bit, the block stops issuing work, frees its tensor memory
// and leaves.
#include "tc_epilogue.cuh"

namespace mxb {

constexpr int kRowsK = 128;                 // k per stage: two boxes of 64
constexpr int kRowsThreads = 64 + 32 * 8;
constexpr int kRowsStages = 24;             // at most
constexpr int kRowsColumns = 256;           // rows of W a tile, at most
constexpr int kRowsTilesBytes = 200 * 1024;

template <int EPI>
__global__ void __launch_bounds__(kRowsThreads, 1)
gemm_tcgen05_rows_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         void* __restrict__ out, int m, int n, int k, long long ldo, const int* __restrict__ tile_group,
                         int group_rows, int m_tiles, int tile_stride, int tile_rows, int a_rows, int w_rows, int stages,
                         float limit, const float* __restrict__ row_scale, int* status) {
  extern __shared__ unsigned char rows_shared_raw[];
  __shared__ __align__(8) uint64_t full_barrier[kRowsStages], empty_barrier[kRowsStages];
  __shared__ __align__(8) uint64_t accumulator_full[2], accumulator_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int failed_slot;
  volatile int& failed = failed_slot;
  const int out_columns = tc_gated(EPI) ? w_rows / 2 : w_rows;
  // A's stages ahead of W's: the 128 rows that an instruction reads end within the stages either way.
  const int a_half = a_rows * 128, w_half = w_rows * 128;   // bytes of a box of 64 k
  unsigned char* a_tiles = rows_shared_raw + ((1024 - (shared_address(rows_shared_raw) & 1023)) & 1023);
  unsigned char* w_tiles = a_tiles + stages * 2 * a_half;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = (n + out_columns - 1) / out_columns;
  const int total_tiles = m_tiles * n_tiles;
  const int k_blocks = (k + kRowsK - 1) / kRowsK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      barrier_init(&full_barrier[s], 1);
      barrier_init(&empty_barrier[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      barrier_init(&accumulator_full[b], 1);
      barrier_init(&accumulator_empty[b], 8);   // a lane of every epilogue warp
    }
    barrier_init_fence();
    failed = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                 ::"r"(shared_address(&tmem_base_slot)), "r"(2 * kRowsColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;

  if (warp == 0) {
    int stage = 0;
    uint32_t parity = 1;
    for (int tile = blockIdx.x; tile < total_tiles && !given_up(failed); tile += gridDim.x) {
      const int m_tile = tile / n_tiles;
      int n0 = tile % n_tiles * out_columns;
      if (tile_group != nullptr) {
        const int group = tile_group[m_tile];
        if (group < 0) continue;
        n0 += group * group_rows;   // the rows of this group's matrix
      }
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!barrier_wait_warp(&empty_barrier[stage], parity, status)) { failed = 1; break; }
        if (elect_one()) {
          unsigned char *a_tile = a_tiles + stage * 2 * a_half, *w_tile = w_tiles + stage * 2 * w_half;
          barrier_arrive_expect(&full_barrier[stage], 2 * (a_half + w_half));
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int x = kb * kRowsK + half * kTmaColumns;
            if (tc_gated(EPI)) {
              tma_load_2d(w_tile + half * w_half, &map_b, x, n0, &full_barrier[stage]);                    // gate rows
              tma_load_2d(w_tile + half * w_half + w_half / 2, &map_b, x, n + n0, &full_barrier[stage]);   // up rows
            } else {
              tma_load_2d(w_tile + half * w_half, &map_b, x, n0, &full_barrier[stage]);
            }
            tma_load_2d(a_tile + half * a_half, &map_a, x, m_tile * tile_stride, &full_barrier[stage]);
          }
        }
        if (++stage == stages) stage = 0, parity ^= 1;
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = tc_instruction_descriptor(128, w_rows);
    const uint64_t a_desc = tc_smem_descriptor(shared_address(a_tiles)), w_desc = tc_smem_descriptor(shared_address(w_tiles));
    const uint32_t a_step = a_half >> 4, w_step = w_half >> 4;
    int stage = 0, local = 0;
    uint32_t parity = 0;
    for (int tile = blockIdx.x; tile < total_tiles && !given_up(failed); tile += gridDim.x) {
      if (tile_group != nullptr && tile_group[tile / n_tiles] < 0) continue;
      const int buffer = local & 1;
      if (!barrier_wait_warp(&accumulator_empty[buffer], ((local >> 1) & 1) ^ 1, status)) { failed = 1; break; }
      tc_fence_after_sync();
      const uint32_t tmem_d = tmem_base + buffer * kRowsColumns;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!barrier_wait_warp(&full_barrier[stage], parity, status)) { failed = 1; break; }
        tc_fence_after_sync();
        if (elect_one()) {
          const uint64_t a_at = a_desc + stage * 2 * a_step, w_at = w_desc + stage * 2 * w_step;
#pragma unroll
          for (int kk = 0; kk < kRowsK / 16; ++kk)   // 16 k: 32 bytes further along the swizzled row, then the next box
            tc_mma(tmem_d, a_at + kk / 4 * a_step + kk % 4 * 2, w_at + kk / 4 * w_step + kk % 4 * 2, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          tc_commit(&empty_barrier[stage]);
          if (kb + 1 == k_blocks) tc_commit(&accumulator_full[buffer]);
        }
        if (++stage == stages) stage = 0, parity ^= 1;
      }
      ++local;
    }
  } else {
    const int lane_base = (warp & 3) * 32, half = (warp - 2) >> 2;
    int local = 0;
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
      const int m_tile = tile / n_tiles, n0 = tile % n_tiles * out_columns;
      if (tile_group != nullptr && tile_group[m_tile] < 0) continue;
      const int buffer = local & 1;
      if (!barrier_wait_warp(&accumulator_full[buffer], (local >> 1) & 1, status)) { failed = 1; break; }
      if (given_up(failed)) break;
      tc_fence_after_sync();
      if (lane_base < tile_rows) {
        const int row = m_tile * tile_stride + lane_base + lane;
        const bool stored = lane_base + lane < tile_rows && row < m;
        const float scale = EPI == kTcGelu && row_scale != nullptr && stored ? row_scale[row] : 1.0f;
        const uint32_t tmem_row = tmem_base + buffer * kRowsColumns + (static_cast<uint32_t>(lane_base) << 16);
#pragma unroll 1
        for (int c = half * 16; c < out_columns; c += 32)
          tc_epilogue<EPI, 16>(tmem_row + c, tmem_row + out_columns + c, out, row, stored, n0 + c, n, ldo, limit, scale);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) barrier_arrive(&accumulator_empty[buffer]);
      ++local;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (failed && threadIdx.x == 0) {
    // A wait ran out somewhere. Give loads that may still be in flight a
    // millisecond before the block's shared memory goes back.
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(2 * kRowsColumns) : "memory");
}

template <int EPI>
static int launch_rows(const TcProduct& p, cudaStream_t stream) {
  int device = 0, sms = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const bool grouped = p.tile_group != nullptr;
  const int tile_stride = grouped ? 128 : p.m;             // rows of A from one tile to the next
  const int tile_rows = grouped ? p.tile_rows : p.m;
  const int a_rows = (tile_rows + 7) / 8 * 8;
  const int m_tiles = grouped ? (p.m + 127) / 128 : 1;
  // Columns a tile: for one matrix what gives every SM the same number of tiles; experts come in a number that only the GPU
  // knows, so their tiles are small.
  const int unit = tc_gated(EPI) ? 32 : 16, per_unit = 16;   // a gated tile holds as many up rows
  int columns = 64;
  if (!grouped) {
    const int most = tc_gated(EPI) ? kRowsColumns / 2 : kRowsColumns;
    const int rounds = ceil_div(p.n, sms * most);
    columns = ceil_div(ceil_div(p.n, sms * rounds), per_unit) * per_unit;
  } else if (tc_gated(EPI)) {
    columns = 32;
  }
  const int w_rows = columns / per_unit * unit;
  const int stage_bytes = 2 * 128 * (a_rows + w_rows);
  const int stages = kRowsTilesBytes / stage_bytes < kRowsStages ? kRowsTilesBytes / stage_bytes : kRowsStages;
  CUtensorMap map_a, map_b;
  if (!make_map(&map_a, p.a, p.m, p.k, p.lda, a_rows) || !make_map(&map_b, p.w, p.w_rows, p.k, p.ldw, tc_gated(EPI) ? w_rows / 2 : w_rows))
    return static_cast<int>(cudaErrorInvalidValue);
  auto kernel = gemm_tcgen05_rows_kernel<EPI>;
  constexpr int shared_bytes = kRowsTilesBytes + 16 * 1024 + 1024;   // an instruction's 128 rows of A may reach past the last stage
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shared_bytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  const long long tiles = static_cast<long long>(m_tiles) * ceil_div(p.n, columns);
  kernel<<<static_cast<int>(tiles < sms ? tiles : sms), kRowsThreads, shared_bytes, stream>>>(
      map_a, map_b, p.out, p.m, p.n, p.k, p.ldo, p.tile_group, p.group_rows, m_tiles, tile_stride, tile_rows, a_rows, w_rows, stages,
      p.limit, p.row_scale, p.status);
  return static_cast<int>(cudaGetLastError());
}

int launch_tc_rows(const TcProduct& p, int epilogue, cudaStream_t stream) {
  switch (epilogue) {
    case kTcStoreBf16: return launch_rows<kTcStoreBf16>(p, stream);
    case kTcStoreF32: return launch_rows<kTcStoreF32>(p, stream);
    case kTcSwiGLU: return launch_rows<kTcSwiGLU>(p, stream);
    case kTcReluSquared: return launch_rows<kTcReluSquared>(p, stream);
    case kTcGeGLU: return launch_rows<kTcGeGLU>(p, stream);
    case kTcClampedGLU: return launch_rows<kTcClampedGLU>(p, stream);
    case kTcGelu: return launch_rows<kTcGelu>(p, stream);
  }
  return static_cast<int>(cudaErrorInvalidValue);
}

}  // namespace mxb
