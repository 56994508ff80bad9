// The matrix-memory recurrence (mlstm.cu states it) over portions of prompts, all chunks of 64 tokens at once.
//
// The chunkwise kernel of mlstm.cu walks a head's chunks one after another, on few blocks, with a shared-memory read
// for every multiply-add; what a chunk adds to the state, and its outputs once the state ahead of it is known, need no
// such order. So, in float32 throughout:
//   1. gates    per request and head: in each chunk the sums F_t of the log forget gates and the running maximum
//               M_t = max_(s <= t) (F_t - F_s + i_s), then m_t = max(F_t + m0, M_t) with m0 walked over the chunks.
//               F is summed and subtracted in 64 bits: a chunk of 64 tokens whose gates nearly close has an F of some
//               hundreds, which 32 bits would leave with an error of 1e-5 in every weight.
//   2. parts    per chunk and head: S = sum_s e^(F_L - F_s + i_s - m_L) k_s v_s^T, and
//               P_ts = e^(F_t - F_s + i_s - m_t) (k_s . q_t) for s <= t with its sums over s.
//   3. pass     C <- e^(F_L + m0 - m_L) C + S over the chunks, value by value; S is replaced by the C ahead of its chunk.
//   4. outputs  per chunk, head and 128 columns: [e^(F_t + m0 - m_t) q_t | P_t] times [C ; V], over the normaliser.
// 2 and 4 are products of 64 x 128 tiles, 64 outputs a thread, and take nearly all the time: bound by the multiply-adds
// and the shared-memory reads they need. 2,048 tokens, 8 heads of 128 x 512: 1,205 us in mlstm.cu, 348 here.
// What a window of chunks needs of scratch is bounded; longer steps go window by window, the state carried in its slot.
#include <type_traits>

#include "common.cuh"

namespace mxb {

constexpr int kTokens = 64;          // of a chunk
constexpr int kColumns = 128;        // of a tile of S or of the outputs
constexpr int kStep = 16;            // k per stage of a product
constexpr int kTileThreads = 128;
constexpr int kGateWarps = 8;
constexpr int kHeadSlice = 32;       // columns of C that share a copy of n and m in the state (mlstm.cu)
constexpr long long kScratchBytes = 128ll << 20;   // for S and P of a window

__device__ __forceinline__ float chunk_log_sigmoid(float z) {
  return z >= 0.0f ? -log1pf(expf(-z)) : z - log1pf(expf(z));
}

struct ChunkScratch {
  int* total;        // [1] chunks of the step
  int2* table;       // [chunks] (row, first token of the chunk within the row)
  double* F;         // [chunks][heads][64]
  float* i;          // [chunks][heads][64], -inf behind the row's last token
  float* m;          // [chunks][heads][64], that of the last token from there on
  float* m0;         // [chunks][heads]
  float* P;          // [window][heads][64 (s)][64 (t)]
  float* sums;       // [window][heads][64 (t)]
  float* S;          // [window][heads][dim * vdim + dim]: S or C, then n
  int chunks, window;
};

struct ChunkArgs {
  const void* proj;
  long long ld;
  int q_off, k_off, v_off, i_off, f_off;
  const float *i_bias, *f_bias;
  float cap, q_scale;
  float* state;
  long long slot_stride;
  int num_slots;
  const int *row_start, *row_length, *request_slots;
  float* out;
  int rows, heads, dim, vdim;
  int* status;
  ChunkScratch s;
};

__device__ __forceinline__ int chunks_of_row(const ChunkArgs& a, int row) {
  const int length = a.row_length[row], slot = a.request_slots[row];
  return length > 0 && slot >= 0 && slot < a.num_slots ? (length + kTokens - 1) / kTokens : 0;
}

// One block per (request, head).
template <typename T>
__global__ void __launch_bounds__(kGateWarps * 32)
mlstm_gates_kernel(ChunkArgs a) {
  __shared__ int s_base;
  __shared__ double s_F[kGateWarps], s_M[kGateWarps];
  __shared__ float s_m0[kGateWarps + 1];
  const int row = blockIdx.x, head = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    int before = 0;
    for (int r = lane; r < row; r += 32) before += chunks_of_row(a, r);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(0xffffffffu, before, d);
    if (lane == 0) s_base = before;
  }
  __syncthreads();
  const int base = s_base, chunks = chunks_of_row(a, row), length = a.row_length[row];
  const bool fits = base + chunks <= a.s.chunks;   // rows that overlap could bring more than the step's tokens
  if (head == 0 && threadIdx.x == 0) {
    if (length > 0 && (chunks == 0 || !fits)) atomicOr(a.status, kStatusBadSlot);
    if (row == a.rows - 1) a.s.total[0] = fits ? base + chunks : a.s.chunks;
  }
  if (chunks == 0) return;
  if (!fits) {   // its chunks, as far as there is room for them, are no row's
    if (head == 0)
      for (int c = threadIdx.x; base + c < a.s.chunks; c += kGateWarps * 32) a.s.table[base + c] = make_int2(-1, 0);
    return;
  }
  const int slices = (a.vdim + kHeadSlice - 1) / kHeadSlice, first = a.row_start[row];
  const long long head_stride = static_cast<long long>(a.dim) * a.vdim + static_cast<long long>(slices) * (a.dim + 1);
  float* m_state = a.state + a.request_slots[row] * a.slot_stride + head * head_stride +
                   static_cast<long long>(a.dim) * a.vdim + static_cast<long long>(slices) * a.dim;
  const float bi = a.i_bias[head], bf = a.f_bias[head];
  if (threadIdx.x == 0) s_m0[kGateWarps] = m_state[0];
  for (int group = 0; group < chunks; group += kGateWarps) {
    const int c = group + warp;
    double F[2] = {0.0, 0.0}, M[2];
    float ig[2];
    if (c < chunks) {
      float f[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = c * kTokens + 2 * lane + j;
        ig[j] = -INFINITY;
        f[j] = 0.0f;
        if (t < length) {
          const T* x = static_cast<const T*>(a.proj) + static_cast<long long>(first + t) * a.ld;
          ig[j] = a.cap * tanhf((to_float(x[a.i_off + head]) + bi) / a.cap);
          f[j] = chunk_log_sigmoid(a.cap * tanhf((to_float(x[a.f_off + head]) + bf) / a.cap));
        }
      }
      F[0] = f[0];
      F[1] = F[0] + f[1];
      double sum = F[1];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += other;
      }
      double ahead = __shfl_up_sync(0xffffffffu, sum, 1);
      if (lane == 0) ahead = 0.0;
      F[0] += ahead;
      F[1] += ahead;
      double best[2];
      best[0] = ig[0] - F[0];
      best[1] = fmax(best[0], ig[1] - F[1]);
      double run = best[1];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, run, d);
        if (lane >= d) run = fmax(run, other);
      }
      double earlier = __shfl_up_sync(0xffffffffu, run, 1);
      if (lane == 0) earlier = -INFINITY;
      M[0] = F[0] + fmax(best[0], earlier);
      M[1] = F[1] + fmax(best[1], earlier);
      if (lane == 31) {
        s_F[warp] = F[1];
        s_M[warp] = M[1];
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      float m = s_m0[kGateWarps];
      for (int w = 0; w < kGateWarps; ++w) {
        s_m0[w] = m;
        if (group + w < chunks) m = static_cast<float>(fmax(s_F[w] + m, s_M[w]));
      }
      s_m0[kGateWarps] = m;
    }
    __syncthreads();
    if (c < chunks) {
      const size_t at = static_cast<size_t>(base + c) * a.heads + head;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const size_t t = at * kTokens + 2 * lane + j;
        a.s.F[t] = F[j];
        a.s.i[t] = ig[j];
        a.s.m[t] = static_cast<float>(fmax(F[j] + s_m0[warp], M[j]));
      }
      if (lane == 0) {
        a.s.m0[at] = s_m0[warp];
        if (head == 0) a.s.table[base + c] = make_int2(row, c * kTokens);
      }
    }
    __syncthreads();   // the walk's numbers are read before the next group's overwrite them
  }
  for (int slice = threadIdx.x; slice < slices; slice += kGateWarps * 32) m_state[slice] = s_m0[kGateWarps];
}

// Four neighbours of a row of the projection's output, or of scratch; QUADS: they lie on a boundary that takes one load.
template <bool QUADS>
__device__ __forceinline__ float4 four_of(const float* p, int count) {
  if (QUADS) return count > 0 ? *reinterpret_cast<const float4*>(p) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  return make_float4(count > 0 ? p[0] : 0.0f, count > 1 ? p[1] : 0.0f, count > 2 ? p[2] : 0.0f, count > 3 ? p[3] : 0.0f);
}
template <bool QUADS>
__device__ __forceinline__ float4 four_of(const __nv_bfloat16* p, int count) {
  if (QUADS) {
    if (count <= 0) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                       __uint_as_float(raw.y & 0xffff0000u));
  }
  return make_float4(count > 0 ? to_float(p[0]) : 0.0f, count > 1 ? to_float(p[1]) : 0.0f, count > 2 ? to_float(p[2]) : 0.0f,
                     count > 3 ? to_float(p[3]) : 0.0f);
}
template <bool QUADS>
__device__ __forceinline__ void put_four(float* to, int count, const float* four) {
  if (QUADS) {
    if (count > 0) *reinterpret_cast<float4*>(to) = make_float4(four[0], four[1], four[2], four[3]);
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (i < count) to[i] = four[i];
}
__device__ __forceinline__ float4 times(float4 x, float f) { return make_float4(f * x.x, f * x.y, f * x.z, f * x.w); }

// acc[8][N] += sum over k < count of A[k][row] B[k][column]: a tile of 64 x 16 N outputs by 8 x 16 threads. load_a(k,
// row) and load_b(k, column) give four neighbours of the operands (0 beyond what they have): of k from there on where
// A_ALONG_K (B_ALONG_K), else of rows (columns). Loads of one value each took as long as the
// multiply-adds: 2,048 tokens, 8 heads of 128 x 512, the whole recurrence 476 us, 348 with four a load.
template <int N, bool A_ALONG_K, bool B_ALONG_K, typename LoadA, typename LoadB>
__device__ __forceinline__ void tile_product(float (&acc)[8][N], float* shared, int count, LoadA load_a, LoadB load_b) {
  constexpr int BN = 16 * N, PITCH_A = kTokens + 4, PITCH_B = BN + 4;
  constexpr int A_EACH = kTokens * kStep / 4 / kTileThreads, B_EACH = BN * kStep / 4 / kTileThreads;
  float* sA = shared;                          // [2][kStep][PITCH_A]
  float* sB = shared + 2 * kStep * PITCH_A;    // [2][kStep][PITCH_B]
  const int tid = threadIdx.x;
  const int ty = (tid >> 6) * 4 + ((tid >> 3) & 3), tx = ((tid >> 5) & 1) * 8 + (tid & 7);
  float4 next_a[A_EACH], next_b[B_EACH];
  auto place = [](int e, int rows, bool along_k, int& k, int& row) {
    k = along_k ? e % (kStep / 4) * 4 : e / (rows / 4);
    row = along_k ? e / (kStep / 4) : e % (rows / 4) * 4;
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int x = 0; x < A_EACH; ++x) {
      int k, row;
      place(tid + x * kTileThreads, kTokens, A_ALONG_K, k, row);
      next_a[x] = k0 + k < count ? load_a(k0 + k, row) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int x = 0; x < B_EACH; ++x) {
      int k, row;
      place(tid + x * kTileThreads, BN, B_ALONG_K, k, row);
      next_b[x] = k0 + k < count ? load_b(k0 + k, row) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  };
  auto put = [](float* at, int pitch, bool along_k, float4 four) {
    if (along_k) at[0] = four.x, at[pitch] = four.y, at[2 * pitch] = four.z, at[3 * pitch] = four.w;
    else *reinterpret_cast<float4*>(at) = four;
  };
  auto store = [&](int stage) {
#pragma unroll
    for (int x = 0; x < A_EACH; ++x) {
      int k, row;
      place(tid + x * kTileThreads, kTokens, A_ALONG_K, k, row);
      put(sA + (stage * kStep + k) * PITCH_A + row, PITCH_A, A_ALONG_K, next_a[x]);
    }
#pragma unroll
    for (int x = 0; x < B_EACH; ++x) {
      int k, row;
      place(tid + x * kTileThreads, BN, B_ALONG_K, k, row);
      put(sB + (stage * kStep + k) * PITCH_B + row, PITCH_B, B_ALONG_K, next_b[x]);
    }
  };
  const int stages = (count + kStep - 1) / kStep;
  __syncthreads();   // whoever used this shared memory before is done
  if (stages > 0) fetch(0);
  if (stages > 0) store(0);
  __syncthreads();
  for (int s = 0; s < stages; ++s) {
    if (s + 1 < stages) fetch((s + 1) * kStep);
    const float* ra = sA + (s & 1) * kStep * PITCH_A + ty * 4;
    const float* rb = sB + (s & 1) * kStep * PITCH_B + tx * 4;
#pragma unroll
    for (int kk = 0; kk < kStep; ++kk) {
      __align__(16) float av[8], bv[N];
#pragma unroll
      for (int x = 0; x < 8; x += 4) *reinterpret_cast<float4*>(av + x) = *reinterpret_cast<const float4*>(ra + kk * PITCH_A + x * 8);
#pragma unroll
      for (int x = 0; x < N; x += 4) *reinterpret_cast<float4*>(bv + x) = *reinterpret_cast<const float4*>(rb + kk * PITCH_B + x * 16);
#pragma unroll
      for (int x = 0; x < 8; ++x)
#pragma unroll
        for (int y = 0; y < N; ++y) acc[x][y] = fmaf(av[x], bv[y], acc[x][y]);
    }
    if (s + 1 < stages) store((s + 1) & 1);   // last read a stage ago, behind that stage's barrier
    __syncthreads();
  }
}
template <int N>
__host__ __device__ constexpr int tile_shared() { return 2 * kStep * (kTokens + 4 + 16 * N + 4); }
__device__ __forceinline__ int tile_row(int x) {
  const int tid = threadIdx.x, ty = (tid >> 6) * 4 + ((tid >> 3) & 3);
  return ty * 4 + x / 4 * 32 + x % 4;
}
__device__ __forceinline__ int tile_column(int y) {
  const int tid = threadIdx.x, tx = ((tid >> 5) & 1) * 8 + (tid & 7);
  return tx * 4 + y / 4 * 64 + y % 4;
}

// Block (chunk of the window, head, piece): the pieces are S in tiles of 64 of its rows x 128 columns, then P.
template <typename T, bool QUADS>
__global__ void __launch_bounds__(kTileThreads, 3)
mlstm_parts_kernel(ChunkArgs a, int from) {
  __shared__ __align__(16) float tiles[tile_shared<8>()];
  __shared__ double sF[kTokens];
  __shared__ float s_i[kTokens], s_m[kTokens], take[kTokens], column_sums[8][kTokens];
  const int chunk = from + blockIdx.x, head = blockIdx.y, dim = a.dim, vdim = a.vdim;
  if (chunk >= a.s.total[0]) return;
  const int2 where = a.s.table[chunk];
  if (where.x < 0) return;
  const int len = min(kTokens, a.row_length[where.x] - where.y);
  const T* x0 = static_cast<const T*>(a.proj) + static_cast<long long>(a.row_start[where.x] + where.y) * a.ld;
  const size_t at = static_cast<size_t>(chunk) * a.heads + head, in_window = static_cast<size_t>(blockIdx.x) * a.heads + head;
  if (threadIdx.x < kTokens) {
    const int t = threadIdx.x;
    sF[t] = a.s.F[at * kTokens + t];
    s_i[t] = a.s.i[at * kTokens + t];
    s_m[t] = a.s.m[at * kTokens + t];
    take[t] = expf(static_cast<float>(a.s.F[at * kTokens + kTokens - 1] - sF[t] + s_i[t] - a.s.m[at * kTokens + kTokens - 1]));
  }
  __syncthreads();
  const int across = (vdim + kColumns - 1) / kColumns, down = (dim + kTokens - 1) / kTokens;
  const int piece = blockIdx.z;
  if (piece < across * down) {
    const int d0 = piece / across * kTokens, v0 = piece % across * kColumns;
    float acc[8][8] = {};
    tile_product<8, false, false>(
        acc, tiles, len,
        [&](int s, int d) { return times(four_of<QUADS>(x0 + s * a.ld + a.k_off + head * dim + d0 + d, dim - d0 - d), take[s]); },
        [&](int s, int v) { return four_of<QUADS>(x0 + s * a.ld + a.v_off + head * vdim + v0 + v, vdim - v0 - v); });
    float* S = a.s.S + in_window * (static_cast<size_t>(dim) * vdim + dim);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const int d = d0 + tile_row(x);
#pragma unroll
      for (int y = 0; y < 8; y += 4)
        if (d < dim) put_four<QUADS>(S + static_cast<size_t>(d) * vdim + v0 + tile_column(y), vdim - v0 - tile_column(y), acc[x] + y);
    }
    if (v0 == 0 && threadIdx.x < kTokens && d0 + threadIdx.x < dim) {
      const int d = d0 + threadIdx.x;
      float sum = 0.0f;
      for (int s = 0; s < len; ++s) sum = fmaf(take[s], to_float(x0[s * a.ld + a.k_off + head * dim + d]), sum);
      S[static_cast<size_t>(dim) * vdim + d] = sum;
    }
    return;
  }
  float acc[8][4] = {};   // rows s, columns t
  tile_product<4, true, true>(
      acc, tiles, dim,
      [&](int d, int s) { return four_of<QUADS>(x0 + s * a.ld + a.k_off + head * dim + d, s < len ? dim - d : 0); },
      [&](int d, int t) { return times(four_of<QUADS>(x0 + t * a.ld + a.q_off + head * dim + d, t < len ? dim - d : 0), a.q_scale); });
  float* P = a.s.P + in_window * kTokens * kTokens;
  float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int x = 0; x < 8; ++x) {
    const int s = tile_row(x);
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int t = tile_column(y);
      const float p = s <= t && t < len ? expf(static_cast<float>(sF[t] - sF[s] + s_i[s] - s_m[t])) * acc[x][y] : 0.0f;
      P[s * kTokens + t] = p;
      part[y] += p;
    }
  }
#pragma unroll
  for (int y = 0; y < 4; ++y) column_sums[tile_row(0) / 4][tile_column(y)] = part[y];
  __syncthreads();
  if (threadIdx.x < kTokens) {
    float sum = 0.0f;
#pragma unroll
    for (int p = 0; p < 8; ++p) sum += column_sums[p][threadIdx.x];
    a.s.sums[in_window * kTokens + threadIdx.x] = sum;
  }
}

// One thread per value of a head's C and n.
__global__ void __launch_bounds__(256)
mlstm_pass_kernel(ChunkArgs a, int from) {
  __shared__ float keep[256];
  const int head = blockIdx.y, dim = a.dim, vdim = a.vdim;
  const int matrix = dim * vdim, values = matrix + dim;
  const int e = blockIdx.x * 256 + threadIdx.x;
  const int until = min(a.s.total[0], from + a.s.window), count = until - from;
  for (int c = threadIdx.x; c < count; c += 256) {
    const size_t at = static_cast<size_t>(from + c) * a.heads + head;
    keep[c] = expf(static_cast<float>(a.s.F[at * kTokens + kTokens - 1] + a.s.m0[at] - a.s.m[at * kTokens + kTokens - 1]));
  }
  __syncthreads();
  if (e >= values) return;
  const int slices = (vdim + kHeadSlice - 1) / kHeadSlice;
  const long long head_stride = static_cast<long long>(matrix) + static_cast<long long>(slices) * (dim + 1);
  auto home = [&](int row) { return a.state + a.request_slots[row] * a.slot_stride + head * head_stride; };
  auto put = [&](int row, float value) {
    if (e < matrix) home(row)[e] = value;
    else for (int slice = 0; slice < slices; ++slice) home(row)[matrix + static_cast<long long>(slice) * dim + e - matrix] = value;
  };
  int row = -1;
  float c = 0.0f;
  float* S = a.s.S + static_cast<size_t>(head) * values + e;
  const size_t stride = static_cast<size_t>(a.heads) * values;
  constexpr int kAhead = 8;   // loads of S under way at once
  for (int at = 0; at < count; at += kAhead) {
    float s[kAhead];
#pragma unroll
    for (int x = 0; x < kAhead; ++x) s[x] = at + x < count ? S[(at + x) * stride] : 0.0f;
#pragma unroll
    for (int x = 0; x < kAhead; ++x) {
      if (at + x >= count) break;
      const int now = a.s.table[from + at + x].x;
      if (now != row) {
        if (row >= 0) put(row, c);
        row = now;
        if (row >= 0) c = home(row)[e];   // the first of the copies of n
      }
      if (row < 0) continue;
      S[(at + x) * stride] = c;
      c = fmaf(keep[at + x], c, s[x]);
    }
  }
  if (row >= 0) put(row, c);
}

template <typename T, bool QUADS>
__global__ void __launch_bounds__(kTileThreads, 3)
mlstm_outputs_kernel(ChunkArgs a, int from) {
  __shared__ __align__(16) float tiles[tile_shared<8>()];
  __shared__ float decay[kTokens], below[kTokens];
  const int chunk = from + blockIdx.x, head = blockIdx.y, dim = a.dim, vdim = a.vdim, v0 = blockIdx.z * kColumns;
  if (chunk >= a.s.total[0]) return;
  const int2 where = a.s.table[chunk];
  if (where.x < 0) return;
  const int len = min(kTokens, a.row_length[where.x] - where.y), first = a.row_start[where.x] + where.y;
  const T* x0 = static_cast<const T*>(a.proj) + static_cast<long long>(first) * a.ld;
  const size_t at = static_cast<size_t>(chunk) * a.heads + head, in_window = static_cast<size_t>(blockIdx.x) * a.heads + head;
  const float* C = a.s.S + in_window * (static_cast<size_t>(dim) * vdim + dim);
  const float* n = C + static_cast<size_t>(dim) * vdim;
  const float* P = a.s.P + in_window * kTokens * kTokens;
  if (threadIdx.x < kTokens) {
    const int t = threadIdx.x;
    decay[t] = expf(static_cast<float>(a.s.F[at * kTokens + t] + a.s.m0[at] - a.s.m[at * kTokens + t]));
  }
  // the normalisers: a warp a token, 16 tokens each
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  for (int t = warp; t < len; t += kTileThreads / 32) {
    float dot = 0.0f;
    for (int d = lane; d < dim; d += 32) dot = fmaf(n[d], to_float(x0[t * a.ld + a.q_off + head * dim + d]) * a.q_scale, dot);
    dot = fmaf(decay[t], warp_sum(dot), a.s.sums[in_window * kTokens + t]);
    if (lane == 0) below[t] = fmaxf(fabsf(dot), expf(-a.s.m[at * kTokens + t])) + 1.0e-6f;
  }
  bool finite = true;
  auto value = [&](int s, int v) { return v0 + v < vdim ? to_float(x0[s * a.ld + a.v_off + head * vdim + v0 + v]) : 0.0f; };
  float acc[8][8] = {};
  tile_product<8, false, false>(acc, tiles, len, [&](int s, int t) { return *reinterpret_cast<const float4*>(P + s * kTokens + t); },
                                [&](int s, int v) {
    const float4 f = four_of<QUADS>(x0 + s * a.ld + a.v_off + head * vdim + v0 + v, vdim - v0 - v);
    finite = finite && fmaxf(fmaxf(fabsf(f.x), fabsf(f.y)), fmaxf(fabsf(f.z), fabsf(f.w))) < INFINITY && f.x == f.x && f.y == f.y &&
             f.z == f.z && f.w == f.w;
    return f;
  });
  if (__syncthreads_or(!finite)) {   // 0 times what is not finite is no 0: a token takes only what is not behind it
#pragma unroll 1
    for (int s = 0; s < len; ++s)
#pragma unroll
      for (int x = 0; x < 8; ++x)
#pragma unroll
        for (int y = 0; y < 8; ++y) {
          if (s == 0) acc[x][y] = 0.0f;
          if (s <= tile_row(x)) acc[x][y] = fmaf(P[s * kTokens + tile_row(x)], value(s, tile_column(y)), acc[x][y]);
        }
  }
  tile_product<8, true, false>(
      acc, tiles, dim,
      [&](int d, int t) {
        return times(times(four_of<QUADS>(x0 + t * a.ld + a.q_off + head * dim + d, t < len ? dim - d : 0), a.q_scale), decay[t]);
      },
      [&](int d, int v) { return four_of<QUADS>(C + static_cast<size_t>(d) * vdim + v0 + v, vdim - v0 - v); });
#pragma unroll
  for (int x = 0; x < 8; ++x) {
    const int t = tile_row(x);
    if (t >= len) continue;
    float* out = a.out + (static_cast<long long>(first + t) * a.heads + head) * vdim;
#pragma unroll
    for (int y = 0; y < 8; y += 4) {
      const int v = v0 + tile_column(y);
      const float four[4] = {acc[x][y] / below[t], acc[x][y + 1] / below[t], acc[x][y + 2] / below[t], acc[x][y + 3] / below[t]};
      put_four<QUADS>(out + v, vdim - v, four);
    }
  }
}

// The scratch's places from `base` on (null: only the size is wanted).
static ChunkScratch chunk_scratch(unsigned char* base, long long tokens, int rows, int longest, int heads, int dim, int vdim,
                                  size_t* bytes) {
  ChunkScratch s;
  const long long by_rows = static_cast<long long>(rows) * ((longest + kTokens - 1) / kTokens), by_tokens = tokens / kTokens + rows;
  s.chunks = static_cast<int>(by_rows < by_tokens ? by_rows : by_tokens);
  const long long each = 4ll * heads * (static_cast<long long>(dim) * vdim + dim + kTokens * kTokens + kTokens);
  long long window = kScratchBytes / each;
  window = window < 16 ? 16 : (window > 256 ? 256 : window);
  s.window = static_cast<int>(window < s.chunks ? window : s.chunks);
  size_t cursor = 0;
  auto take = [&](size_t size) {
    unsigned char* p = base + cursor;
    cursor += (size + 255) / 256 * 256;
    return p;
  };
  const size_t all = static_cast<size_t>(s.chunks) * heads, some = static_cast<size_t>(s.window) * heads;
  s.total = reinterpret_cast<int*>(take(4));
  s.table = reinterpret_cast<int2*>(take(static_cast<size_t>(s.chunks) * 8));
  s.F = reinterpret_cast<double*>(take(all * kTokens * 8));
  s.i = reinterpret_cast<float*>(take(all * kTokens * 4));
  s.m = reinterpret_cast<float*>(take(all * kTokens * 4));
  s.m0 = reinterpret_cast<float*>(take(all * 4));
  s.P = reinterpret_cast<float*>(take(some * kTokens * kTokens * 4));
  s.sums = reinterpret_cast<float*>(take(some * kTokens * 4));
  s.S = reinterpret_cast<float*>(take(some * (static_cast<size_t>(dim) * vdim + dim) * 4));
  *bytes = cursor;
  return s;
}

}  // namespace mxb

using namespace mxb;

// How many KiB of scratch mxb_mlstm_chunks needs for a step of `tokens` tokens whose longest row brings `longest`; 0: the
// step does not take this way. It costs some 90 us, little for a chunk and as much for a row of one token as for a whole
// chunk; mlstm.cu's walk costs 0.4 to 0.6 us per token of the longest row, or the whole step's work where that is more. So
// it is taken where a row is long (a row of 256 tokens; of 192 where the step's work is much) and the rows beside it are few
// for that, and where a step brings 512 tokens in rows of 32 and more and much work. us, the walk first, heads x dim x vdim:
//   one row of 192 tokens      8 x 128 x 512  122 and 120   8 x 64 x 256   83 and  97   4 x 64 x 128   81 and  91
//   of 256                                    159 and 122                 108 and  97                 105 and  93
//   of 2,048                                1,205 and 450                 802 and 198                 787 and 108
//   192, 63 single tokens                     587 and 654                 260 and 243                 113 and 149
//   512, 127 single tokens                  1,306 and 1,248               584 and 417                 265 and 237
//   512, 255 single tokens                  2,162 and 2,311               932 and 755                 348 and 456
//   four rows of 128                          294 and 155                 109 and  98                  57 and  95
//   sixteen of 128                          1,017 and 486                 365 and 204                 108 and 112
//   eight of 64                               265 and 167                 110 and 104                  33 and  99
//   four of 64, 300 single tokens           2,169 and 2,692               872 and 843                 222 and 509
// The second figures are those of products that read one value at a time, when the lines were drawn. Since they read four,
// what is taken costs, walk first again: one row of 192 99 and 62; of 256 131 and 64, 90 and 47, 90 and 46; of 2,048 1,011 and 296,
// 688 and 120, 684 and 61; 512 beside 127 single tokens 1,235 and 1,009, 519 and 327, 243 and 172; four of 128 260 and 93; sixteen
// of 128 941 and 336, 312 and 124.
MXB_API int mxb_mlstm_chunks_scratch(long long tokens, int rows, int longest, int heads, int dim, int vdim) {
  const bool much = tokens * heads * dim * vdim > 1ll << 26;
  const bool few_beside_long = (longest >= 256 || (longest >= 192 && much)) && 3ll * rows <= longest - 128;
  const bool many = longest >= 64 && tokens >= 512 && tokens >= 32ll * rows && much;
  if (rows <= 0 || tokens <= 0 || !(few_beside_long || many)) return 0;
  if (heads <= 0 || heads > 65535 || dim <= 0 || dim > 256 || vdim <= 0 || vdim > 65536) return 0;
  size_t bytes = 0;
  chunk_scratch(nullptr, tokens, rows, longest, heads, dim, vdim, &bytes);
  return bytes >> 40 ? 0 : static_cast<int>((bytes + 1023) >> 10);
}

// As mxb_mlstm_scan, for steps that mxb_mlstm_chunks_scratch gives a size for; `scratch` lies on 16 bytes.
MXB_API int mxb_mlstm_chunks(const void* proj, long long ld, int q_off, int k_off, int v_off, int i_off, int f_off,
                             const float* i_bias, const float* f_bias, float cap, float q_scale, float* state,
                             long long slot_stride, int num_slots, const int* row_start, const int* row_length,
                             const int* request_slots, float* out, long long tokens, int rows, int heads, int dim, int vdim,
                             int dtype, int longest, void* scratch, int* status, cudaStream_t stream) {
  if (mxb_mlstm_chunks_scratch(tokens, rows, longest, heads, dim, vdim) == 0 || !(cap > 0.0f) || scratch == nullptr ||
      (reinterpret_cast<uintptr_t>(scratch) & 15) || (dtype != kF32 && dtype != kBF16))
    return static_cast<int>(cudaErrorInvalidValue);
  size_t bytes = 0;
  const ChunkArgs a = {proj, ld, q_off, k_off, v_off, i_off, f_off, i_bias, f_bias, cap, q_scale, state, slot_stride,
                       num_slots, row_start, row_length, request_slots, out, rows, heads, dim, vdim, status,
                       chunk_scratch(static_cast<unsigned char*>(scratch), tokens, rows, longest, heads, dim, vdim, &bytes)};
  const int across = ceil_div(vdim, kColumns), pieces = across * ceil_div(dim, kTokens) + 1;
  auto run = [&](auto type, auto quads) {
    using T = decltype(type);
    constexpr bool QUADS = decltype(quads)::value;
    mlstm_gates_kernel<T><<<dim3(rows, heads), kGateWarps * 32, 0, stream>>>(a);
    for (int from = 0; from < a.s.chunks; from += a.s.window) {
      const int here = a.s.chunks - from < a.s.window ? a.s.chunks - from : a.s.window;
      mlstm_parts_kernel<T, QUADS><<<dim3(here, heads, pieces), kTileThreads, 0, stream>>>(a, from);
      mlstm_pass_kernel<<<dim3(ceil_div(dim * vdim + dim, 256), heads), 256, 0, stream>>>(a, from);
      mlstm_outputs_kernel<T, QUADS><<<dim3(here, heads, across), kTileThreads, 0, stream>>>(a, from);
    }
  };
  // Four values a load where every head's part of a row starts on such a boundary.
  const bool quads = dim % 4 == 0 && vdim % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0 && ld % 4 == 0 &&
                     (reinterpret_cast<uintptr_t>(proj) & (dtype == kF32 ? 15 : 7)) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  if (dtype == kF32) quads ? run(float(), std::true_type()) : run(float(), std::false_type());
  else quads ? run(__nv_bfloat16(), std::true_type()) : run(__nv_bfloat16(), std::false_type());
  return static_cast<int>(cudaGetLastError());
}
