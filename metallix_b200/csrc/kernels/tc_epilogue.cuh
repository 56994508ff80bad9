// What the tcgen05 products do with finished columns of the accumulator, one thread per row.
#pragma once

#include "tcgen05.cuh"

namespace mxb {

enum TcEpilogue : int { kTcStoreBf16 = 0, kTcStoreF32 = 1, kTcSwiGLU = 2, kTcReluSquared = 3, kTcGeGLU = 4, kTcClampedGLU = 5, kTcGelu = 6 };
// the epilogues that take a tile of gate rows beside a tile of up rows: act(gate) * up (silu, or the tanh form of gelu), or the product of clamped halves
__host__ __device__ constexpr bool tc_gated(int epilogue) { return epilogue == kTcSwiGLU || epilogue == kTcGeGLU || epilogue == kTcClampedGLU; }

// WIDE (16 or 32) columns of row `row` from `column` on, from tensor memory at `taddr` (a gated epilogue's up columns at
// `taddr_up`) through the epilogue to `out`; columns from n on are left out, and the row altogether unless `stored`. All
// lanes of a warp call it.
template <int EPI, int WIDE>
__device__ __forceinline__ void tc_epilogue(uint32_t taddr, uint32_t taddr_up, void* out, int row, bool stored, int column,
                                            int n, long long ldo, float limit, float scale) {
  uint32_t acc[WIDE];
  __syncwarp();   // lanes that stored nothing of the columns before are back ahead of the others
  tc_load(taddr, acc);
  float values[WIDE];
  if (tc_gated(EPI)) {
    uint32_t up[WIDE];
    tc_load(taddr_up, up);
#pragma unroll
    for (int i = 0; i < WIDE; ++i) {
      // gate and up take the rounding to bfloat16 they would get on their way through memory
      const float gate = to_float(from_float<__nv_bfloat16>(__uint_as_float(acc[i])));
      const float u = to_float(from_float<__nv_bfloat16>(__uint_as_float(up[i])));
      values[i] = gated_product(gate, u, EPI == kTcGeGLU ? kActGeluTanh : (EPI == kTcClampedGLU ? kActClamped : kActSilu), limit);  // rounded to bfloat16 anyway
    }
  } else if (EPI == kTcReluSquared) {
#pragma unroll
    for (int i = 0; i < WIDE; ++i) {
      const float u = fmaxf(__uint_as_float(acc[i]), 0.0f);
      values[i] = u * u;
    }
  } else if (EPI == kTcGelu) {
#pragma unroll
    for (int i = 0; i < WIDE; ++i) values[i] = gelu_of(scale * __uint_as_float(acc[i]));
  } else {
#pragma unroll
    for (int i = 0; i < WIDE; ++i) values[i] = __uint_as_float(acc[i]);
  }
  if (!stored) return;
  if (EPI == kTcStoreF32) {
    float* dst = static_cast<float*>(out) + static_cast<long long>(row) * ldo + column;
    if (column + WIDE <= n && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
      for (int i = 0; i < WIDE; i += 4)
        *reinterpret_cast<float4*>(dst + i) = make_float4(values[i], values[i + 1], values[i + 2], values[i + 3]);
    } else {
      for (int i = 0; i < WIDE; ++i)
        if (column + i < n) dst[i] = values[i];
    }
  } else {
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(out) + static_cast<long long>(row) * ldo + column;
    if (column + WIDE <= n && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
      for (int i = 0; i < WIDE; i += 8) {
        uint32_t packed[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          __nv_bfloat162 pair = __floats2bfloat162_rn(values[i + 2 * j], values[i + 2 * j + 1]);
          packed[j] = *reinterpret_cast<uint32_t*>(&pair);
        }
        *reinterpret_cast<uint4*>(dst + i) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
      }
    } else {
      for (int i = 0; i < WIDE; ++i)
        if (column + i < n) dst[i] = from_float<__nv_bfloat16>(values[i]);
    }
  }
}

// A product's operands, as mxb_gemm_tcgen05 and its grouped form hand them on.
struct TcProduct {
  void* out;
  const void* a;
  const void* w;
  int m, n, k, w_rows;
  long long lda, ldw, ldo;
  const int* tile_group;   // null: one matrix
  int group_rows, tile_rows;
  float limit;
  const float* row_scale;
  int* status;
};

// Products of few rows, bound by reading W (gemm_tcgen05_rows.cu).
constexpr int kTcFewRows = 64;
// Gated experts only up to here: a tile holds 32 gate and 32 up rows, and wide ones fill the SMs in tiles of 128 and 128 anyway. us in
// few rows and in whole tiles, 12 experts, two or three a token: 4096 x 4096 with 16 tokens 174 and 146, 4 tokens 94 and 86; 2048 x 4096
// 83 and 86, but 65 and 49 with 3 tokens; 1536 x 1024 23 and 27; 768 x 2048 19 and 23. Not gated: 6144 x 4096, 3, 16 and 64 tokens
// 59 and 63, 120 and 139, 129 and 138; 1024 x 3072 15 and 29, 26 and 33, 27 and 33; the exceptions are counts whose narrow
// tiles just open another round (7 experts of 4096 x 4096 57 and 53).
constexpr int kTcFewGatedColumns = 2048;
int launch_tc_rows(const TcProduct& p, int epilogue, cudaStream_t stream);

}  // namespace mxb
