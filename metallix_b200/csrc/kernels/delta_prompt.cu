// The delta rule with a decay per channel (delta_rule.cu states it) over portions of prompts in bfloat16, and the steps of
// single tokens of all three recurrences there that keep a matrix per head.
//
// A token by itself is a chain of dependent steps (decay, a dot with the key over the lanes that share a column, the
// write), and delta_rule.cu pays that chain per token. Here eight tokens pay it once. With S the state ahead of eight
// tokens, g_t their decays and G_t = g_1 ... g_t (products of numbers of at most 1: nothing grows), unrolling gives
//   u_t = beta_t (v_t - (k_t G_t) . S - sum_(s < t) A_ts u_s),    A_ts = sum_d k_t k_s g_(s+1) ... g_t
//   o_t = (q_t G_t) . S + sum_(s <= t) P_ts u_s,                  P_ts = sum_d q_t k_s g_(s+1) ... g_t
//   S <- G_8 S + sum_s (k_s g_(s+1) ... g_8) u_s^T
// What does not depend on S or on the column, the three kinds of products with keys and queries, G_8, A and P, is made
// first, a block per (eight tokens, head), in the order in which the lanes will read it. Then a block of four warps walks
// a head's 32 columns, four columns and eight channels a thread: all 16 dots with S at once, their sums over the lanes
// together, a small triangular solve per column, one update of S. A fifth warp keeps the next eights on their way, one bulk
// copy each. Float32 throughout, as there. The sums run in another order than token by token, so a float32 step, whose
// results are the same however a prompt is cut, stays there.
// The walk is bound by its shared-memory reads and by what is left of the chain: 353 us with its records for 1,777 tokens
// of 32 heads of 128 x 128; delta_rule.cu takes 919. Token by token with four columns a thread it stayed at 480 to 530,
// whichever way the channels were shared out: the exchanges of every token were the chain.
// One decay per head and the dual stay with delta_rule.cu over prompts too, although eight tokens at a time took 341 us there
// for 725 (one row of 1,777 tokens, 32 heads), and the dual 314 for 853: their sums in another order moved the logits of a
// decoder whose routers stand close to a tie behind them by up to 0.05 of their size, one token's row by 0.28.
#include <type_traits>

#include "async_copy.cuh"
#include "common.cuh"

namespace mxb {

enum WalkMode : int { kWalkChannel = 0, kWalkHead = 1, kWalkDual = 2 };   // the numbers of delta_rule.cu
constexpr int kEight = 8;         // tokens of a stage
constexpr int kWalkStages = 4;
constexpr int kWalkCols = 4;      // columns of a thread
constexpr int kWalkPer = 8;       // channels of a lane
constexpr long long kWalkScratch = 128ll << 20;   // bytes of records ahead of the walk, at most

// float32 values of a record (eight tokens of a head, `width` channels): k_t G_t, q_t G_t and k_s g_(s+1) ... g_8 of the
// eight, G_8, A [8][8] (0 for s >= t), P [8][8] (0 for s > t), beta [8]. What a token that is not there leaves is 0.
__host__ __device__ constexpr int walk_record(int width) { return 25 * width + 136; }
// Where channel d of a vector lies: of the lanes' shares, the first four values of all lanes come first.
__device__ __forceinline__ int walk_slot(int d, int lanes) { return ((d % kWalkPer) / 4 * lanes + d / kWalkPer) * 4 + d % 4; }

__device__ __forceinline__ float walk_softplus(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

// Two channels per instruction.
using Pair = unsigned long long;
__device__ __forceinline__ Pair mul_pair(Pair a, Pair b) {
  Pair d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ Pair fma_pair(Pair a, Pair b, Pair c) {
  Pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ Pair make_pair(float x, float y) {
  return static_cast<Pair>(__float_as_uint(y)) << 32 | __float_as_uint(x);
}
__device__ __forceinline__ float first_of(Pair x) { return __uint_as_float(static_cast<unsigned>(x)); }
__device__ __forceinline__ float second_of(Pair x) { return __uint_as_float(static_cast<unsigned>(x >> 32)); }

struct WalkArgs {
  const void* qkv;
  long long ld;
  int q_off, k_off, v_off;
  const void* beta_pre;
  long long ldb;
  int b_off;
  const void* step_pre;
  long long lds;
  const float *step_bias, *rate, *skip;
  float* state;
  long long slot_stride;
  int num_slots;
  const int *row_start, *row_length, *request_slots;
  float* out;
  int rows, heads, groups, dim, vdim;
  int* status;
  float* records;        // [heads][eights][record]: the rows' eights one row after another
  int eights;            // at most
  long long from, to;    // the window: packed tokens from .. to - 1

  // A row's tokens inside the window.
  __device__ __forceinline__ long long first(int row) const { return max(static_cast<long long>(row_start[row]), from); }
  __device__ __forceinline__ int count(int row) const {
    const int length = row_length[row], slot = request_slots[row];
    if (length <= 0 || slot < 0 || slot >= num_slots) return 0;
    const long long end = min(static_cast<long long>(row_start[row]) + length, to);
    return static_cast<int>(max(end - first(row), 0ll));
  }
};

// One block per (eight tokens, head), a warp a token.
template <typename T, int LANES>
__global__ void __launch_bounds__(32 * kEight)
walk_records_kernel(WalkArgs a) {
  constexpr int WIDTH = LANES * kWalkPer, NL = WIDTH / 32;
  __shared__ float sq[kEight][WIDTH], sk[kEight][WIDTH], sg[kEight][WIDTH];
  __shared__ int s_row, s_ahead;
  const int head = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {   // whose eight this is
    int ahead = 0, row = -1;
    for (int r0 = 0; r0 < a.rows && row < 0; r0 += 32) {
      const int mine = r0 + lane < a.rows ? (a.count(r0 + lane) + kEight - 1) / kEight : 0;
      int sum = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += other;
      }
      const unsigned beyond = __ballot_sync(0xffffffffu, ahead + sum > static_cast<int>(blockIdx.x));
      if (beyond) {
        const int at = __ffs(beyond) - 1;
        row = r0 + at;
        ahead += __shfl_sync(0xffffffffu, sum - mine, at);
      } else {
        ahead += __shfl_sync(0xffffffffu, sum, 31);
      }
    }
    if (lane == 0) {
      s_row = row;
      s_ahead = ahead;
    }
  }
  __syncthreads();
  const int row = s_row;
  if (row < 0) return;
  const int t = (static_cast<int>(blockIdx.x) - s_ahead) * kEight + warp;   // of the row's tokens in the window
  const bool live = t < a.count(row);
  const long long token = a.first(row) + t;
  float* record = a.records + (static_cast<size_t>(head) * a.eights + blockIdx.x) * walk_record(WIDTH);
  float *const A = record + 25 * WIDTH, *const P = A + kEight * kEight, *const beta = P + kEight * kEight;
  const float rate = a.rate[head];
  float q[NL] = {}, k[NL] = {}, write = 0.0f, qq = 0.0f, kk = 0.0f;
  if (live) {
    const int group = head / (a.heads / a.groups);
    const T* x = static_cast<const T*>(a.qkv) + token * a.ld;
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      const int d = lane + 32 * i;
      q[i] = d < a.dim ? to_float(x[a.q_off + group * a.dim + d]) : 0.0f;
      k[i] = d < a.dim ? to_float(x[a.k_off + group * a.dim + d]) : 0.0f;
      qq = fmaf(q[i], q[i], qq);
      kk = fmaf(k[i], k[i], kk);
    }
    const float q_unit = rsqrtf(warp_sum(qq) + 1e-6f) * rsqrtf(static_cast<float>(a.dim)), k_unit = rsqrtf(warp_sum(kk) + 1e-6f);
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      q[i] *= q_unit;
      k[i] *= k_unit;
    }
    write = sigmoid_of(to_float(static_cast<const T*>(a.beta_pre)[token * a.ldb + a.b_off + head]));
  }
#pragma unroll
  for (int i = 0; i < NL; ++i) {
    const int d = lane + 32 * i;
    sq[warp][d] = q[i];
    sk[warp][d] = k[i];
    sg[warp][d] = live && d < a.dim ? expf(-rate * walk_softplus(static_cast<const float*>(a.step_pre)[token * a.lds + head * a.dim + d] +
                                                                 a.step_bias[head * a.dim + d]))
                                    : 1.0f;
  }
  if (lane == 0) beta[warp] = write;
  __syncthreads();
  // A and P of this warp's key against the queries and keys behind it.
  float after[NL];
#pragma unroll
  for (int i = 0; i < NL; ++i) after[i] = k[i];
#pragma unroll
  for (int later = 0; later < kEight; ++later) {
    float kd = 0.0f, qd = 0.0f;
    if (later >= warp) {
#pragma unroll
      for (int i = 0; i < NL; ++i) {
        const int d = lane + 32 * i;
        if (later > warp) after[i] *= sg[later][d];
        kd = fmaf(sk[later][d], after[i], kd);
        qd = fmaf(sq[later][d], after[i], qd);
      }
      kd = warp_sum(kd);
      qd = warp_sum(qd);
    }
    if (lane == 0) {
      A[later * kEight + warp] = later > warp ? kd : 0.0f;
      P[later * kEight + warp] = later >= warp ? qd : 0.0f;
    }
  }
  // what is left of this warp's key behind the eight, and its key and query on the state ahead of them
#pragma unroll
  for (int i = 0; i < NL; ++i) {
    const int d = lane + 32 * i, at = walk_slot(d, LANES);
    float before = 1.0f;
    for (int s = 0; s <= warp; ++s) before *= sg[s][d];
    record[warp * WIDTH + at] = k[i] * before;
    record[(kEight + warp) * WIDTH + at] = q[i] * before;
    record[(2 * kEight + warp) * WIDTH + at] = after[i];
    if (warp == kEight - 1) record[3 * kEight * WIDTH + at] = before;
  }
}

// LANES lanes share four columns, eight channels each. Block (request, head, columns): blockDim.x - 32 threads with
// columns and a warp that fetches. A thread counts its four columns from one of them on (column c of a lane is c ^ own),
// and tokens of the outputs likewise, so that an exchange which halves what a lane adds up needs no choosing.
template <typename T, int LANES>
__global__ void __launch_bounds__(160)
walk_kernel(WalkArgs a) {
  constexpr int WIDTH = LANES * kWalkPer, RECORD = walk_record(WIDTH), PAIRS = kWalkPer / 2;
  constexpr int SHARERS = LANES / 4;            // lanes that end with the same column
  constexpr int OWN = kEight / SHARERS;         // tokens of it whose output a lane writes
  extern __shared__ __align__(16) float stages[];   // [kWalkStages][RECORD]
  __shared__ __align__(8) uint64_t full[kWalkStages], empty[kWalkStages];
  __shared__ int s_ahead;
  const int row = blockIdx.x, head = blockIdx.y;
  const int length = a.row_length[row], slot = a.request_slots[row];
  if (length > 0 && (slot < 0 || slot >= a.num_slots)) {
    if (threadIdx.x == 0) atomicOr(a.status, kStatusBadSlot);
    return;
  }
  const int count = a.count(row), rounds = (count + kEight - 1) / kEight;
  if (count == 0) return;
  const int workers = blockDim.x - 32;   // threads with columns
  if (static_cast<int>(threadIdx.x) >= workers) {
    int ahead = 0;
    for (int r = threadIdx.x - workers; r < row; r += 32) ahead += (a.count(r) + kEight - 1) / kEight;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) ahead += __shfl_xor_sync(0xffffffffu, ahead, d);
    if (static_cast<int>(threadIdx.x) == workers) {
      s_ahead = ahead;
      for (int s = 0; s < kWalkStages; ++s) {
        barrier_init(&full[s], 1);
        barrier_init(&empty[s], workers / 32);
      }
      barrier_init_fence();
    }
  }
  __syncthreads();
  if (s_ahead + rounds > a.eights) {   // rows that overlap could bring more than the window's tokens
    if (threadIdx.x == 0) atomicOr(a.status, kStatusBadSlot);
    return;
  }
  const long long first = a.first(row);
  bool ok = true;
  if (static_cast<int>(threadIdx.x) >= workers) {   // ---- the warp that fetches
    if ((threadIdx.x & 31) == 0) {
      const float* records = a.records + (static_cast<size_t>(head) * a.eights + s_ahead) * RECORD;
      for (int r = 0; r < rounds && ok; ++r) {
        const int stage = r % kWalkStages;
        ok = barrier_wait(&empty[stage], ((r / kWalkStages) & 1) ^ 1, a.status);
        if (!ok) break;
        barrier_arrive_expect(&full[stage], RECORD * 4);
        bulk_copy(stages + stage * RECORD, records + static_cast<size_t>(r) * RECORD, RECORD * 4, &full[stage]);
      }
    }
  } else {
    const int part = threadIdx.x % LANES;
    const int own = (part & (LANES / 2) ? 2 : 0) + (part & (LANES / 4) ? 1 : 0);   // the column this lane ends with
    const int turned = part % SHARERS * OWN;                                        // the first token whose output it writes
    const int column = (blockIdx.z * (workers / LANES) + threadIdx.x / LANES) * kWalkCols;
    float* home = a.state + static_cast<long long>(slot) * a.slot_stride +
                  (static_cast<long long>(head) * a.vdim + column) * a.dim + part * kWalkPer;
    const bool whole = a.dim % kWalkPer == 0 && a.slot_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(a.state) & 15) == 0;
    Pair s[kWalkCols][PAIRS];
#pragma unroll
    for (int c = 0; c < kWalkCols; ++c) {
      const float* from = home + static_cast<long long>(c ^ own) * a.dim;
      const bool live = column + (c ^ own) < a.vdim;
#pragma unroll
      for (int i = 0; i < PAIRS; i += 2) {
        const int d = part * kWalkPer + 2 * i;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live && whole && d < a.dim) x = *reinterpret_cast<const float4*>(from + 2 * i);
        else if (live && !whole) {
          if (d < a.dim) x.x = from[2 * i];
          if (d + 1 < a.dim) x.y = from[2 * i + 1];
          if (d + 2 < a.dim) x.z = from[2 * i + 2];
          if (d + 3 < a.dim) x.w = from[2 * i + 3];
        }
        s[c][i] = make_pair(x.x, x.y);
        s[c][i + 1] = make_pair(x.z, x.w);
      }
    }
    // This lane's column of a stage's tokens, a stage ahead. The values stay as they come until they are used, and no
    // branch stands around a load (places outside repeat others): either would make each load wait for the one before.
    const T* values = static_cast<const T*>(a.qkv) + first * a.ld + a.v_off + head * a.vdim + min(column + own, a.vdim - 1);
    T next[kEight];
    auto fetch = [&](int t0) {
#pragma unroll
      for (int t = 0; t < kEight; ++t) next[t] = values[static_cast<long long>(min(t0 + t, count - 1)) * a.ld];
    };
    fetch(0);
    for (int r = 0; r < rounds; ++r) {
      const int stage = r % kWalkStages, tokens = min(kEight, count - r * kEight);
      T value[kEight];
#pragma unroll
      for (int t = 0; t < kEight; ++t) value[t] = next[t];
      if (!barrier_wait_warp(&full[stage], (r / kWalkStages) & 1, a.status)) { ok = false; break; }
      fetch((r + 1) * kEight);   // on their way while this stage is walked
      const float* record = stages + stage * RECORD;
      auto vector = [&](int index, Pair (&into)[PAIRS]) {
        const ulonglong2* from = reinterpret_cast<const ulonglong2*>(record + index * WIDTH) + part;
#pragma unroll
        for (int i = 0; i < PAIRS; i += 2) {
          const ulonglong2 x = from[i / 2 * LANES];
          into[i] = x.x;
          into[i + 1] = x.y;
        }
      };
      auto dots = [&](int index, float (&into)[kWalkCols]) {
        Pair x[PAIRS];
        vector(index, x);
#pragma unroll
        for (int c = 0; c < kWalkCols; ++c) {
          Pair sum = mul_pair(x[0], s[c][0]);
#pragma unroll
          for (int i = 1; i < PAIRS; ++i) sum = fma_pair(x[i], s[c][i], sum);
          into[c] = first_of(sum) + second_of(sum);
        }
      };
      // ---- (k_t G_t) . S of this lane's column, then what is written of every token
      float u[kEight][kWalkCols];
      {
        float kd[kEight][kWalkCols];
#pragma unroll
        for (int t = 0; t < kEight; ++t) dots(t, kd[t]);
#pragma unroll
        for (int t = 0; t < kEight; ++t) {
          kd[t][0] += __shfl_xor_sync(0xffffffffu, kd[t][2], LANES / 2);
          kd[t][1] += __shfl_xor_sync(0xffffffffu, kd[t][3], LANES / 2);
        }
#pragma unroll
        for (int t = 0; t < kEight; ++t) kd[t][0] += __shfl_xor_sync(0xffffffffu, kd[t][1], LANES / 4);
#pragma unroll
        for (int offset = SHARERS / 2; offset > 0; offset >>= 1)
#pragma unroll
          for (int t = 0; t < kEight; ++t) kd[t][0] += __shfl_xor_sync(0xffffffffu, kd[t][0], offset);
#pragma unroll
        for (int t = 0; t < kEight; ++t) u[t][0] = kd[t][0];
      }
      {
        const float* A = record + 25 * WIDTH;
        const float* beta = A + 2 * kEight * kEight;
        float b[kEight];
        *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(beta);
        *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(beta + 4);
#pragma unroll
        for (int t = 0; t < kEight; ++t) {
          // converted here and not behind the sum, which the schedule does not survive (1,777 tokens: 447 us for 353)
          float rest = to_float(value[t]), line[kEight], seen = u[t][0];
          *reinterpret_cast<float4*>(line) = *reinterpret_cast<const float4*>(A + t * kEight);
          *reinterpret_cast<float4*>(line + 4) = *reinterpret_cast<const float4*>(A + t * kEight + 4);
#pragma unroll
          for (int e = 0; e < t; ++e) seen = fmaf(line[e], u[e][0], seen);
          rest -= seen;
          u[t][0] = t < tokens ? b[t] * rest : 0.0f;
        }
      }
      // ---- (q_t G_t) . S, each lane's tokens counted from those whose outputs it writes
      float qd[kEight][kWalkCols];
#pragma unroll
      for (int t = 0; t < kEight; ++t) dots(kEight + (t ^ turned), qd[t]);
      // the other columns' u, from the lanes that have them
#pragma unroll
      for (int t = 0; t < kEight; ++t) u[t][1] = __shfl_xor_sync(0xffffffffu, u[t][0], LANES / 4);
#pragma unroll
      for (int t = 0; t < kEight; ++t) {
        u[t][2] = __shfl_xor_sync(0xffffffffu, u[t][0], LANES / 2);
        u[t][3] = __shfl_xor_sync(0xffffffffu, u[t][1], LANES / 2);
      }
      // ---- the state behind the eight
      {
        Pair g[PAIRS];
        vector(3 * kEight, g);
#pragma unroll
        for (int c = 0; c < kWalkCols; ++c)
#pragma unroll
          for (int i = 0; i < PAIRS; ++i) s[c][i] = mul_pair(s[c][i], g[i]);
#pragma unroll
        for (int t = 0; t < kEight; ++t) {
          Pair k[PAIRS];
          vector(2 * kEight + t, k);
#pragma unroll
          for (int c = 0; c < kWalkCols; ++c) {
            const Pair both = make_pair(u[t][c], u[t][c]);
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) s[c][i] = fma_pair(k[i], both, s[c][i]);
          }
        }
      }
      // ---- outputs
      float line[OWN][kEight];
      const float* P = record + 25 * WIDTH + kEight * kEight;
#pragma unroll
      for (int t = 0; t < OWN; ++t) {
        *reinterpret_cast<float4*>(line[t]) = *reinterpret_cast<const float4*>(P + (t ^ turned) * kEight);
        *reinterpret_cast<float4*>(line[t] + 4) = *reinterpret_cast<const float4*>(P + (t ^ turned) * kEight + 4);
      }
      __syncwarp();
      if ((threadIdx.x & 31) == 0) barrier_arrive(&empty[stage]);   // read: the stage may be fetched over
#pragma unroll
      for (int t = 0; t < kEight; ++t) {
        qd[t][0] += __shfl_xor_sync(0xffffffffu, qd[t][2], LANES / 2);
        qd[t][1] += __shfl_xor_sync(0xffffffffu, qd[t][3], LANES / 2);
      }
#pragma unroll
      for (int t = 0; t < kEight; ++t) qd[t][0] += __shfl_xor_sync(0xffffffffu, qd[t][1], LANES / 4);
      // `turned` sets the bits of a token's number from OWN on by the lane's bits from 1 on, in the same order
#pragma unroll
      for (int offset = SHARERS / 2, half = kEight / 2; offset > 0; offset >>= 1, half >>= 1)
#pragma unroll
        for (int t = 0; t < half; ++t) qd[t][0] += __shfl_xor_sync(0xffffffffu, qd[t + half][0], offset);
#pragma unroll
      for (int t = 0; t < OWN; ++t) {
        const int mine = t ^ turned;
        float o = qd[t][0];
#pragma unroll
        for (int e = 0; e < kEight; ++e)   // chosen, not weighed with 0: a later token's infinity stays out of this one
          o = e <= mine ? fmaf(line[t][e], u[e][0], o) : o;
        if (mine < tokens && column + own < a.vdim)
          a.out[(first + r * kEight + mine) * (static_cast<long long>(a.heads) * a.vdim) + static_cast<long long>(head) * a.vdim +
                column + own] = o;
      }
    }
    if (ok) {
#pragma unroll
      for (int c = 0; c < kWalkCols; ++c) {
        if (column + (c ^ own) >= a.vdim) continue;
        float* to = home + static_cast<long long>(c ^ own) * a.dim;
#pragma unroll
        for (int i = 0; i < PAIRS; i += 2) {
          const int d = part * kWalkPer + 2 * i;
          const float x[4] = {first_of(s[c][i]), second_of(s[c][i]), first_of(s[c][i + 1]), second_of(s[c][i + 1])};
          if (whole) {
            if (d < a.dim) *reinterpret_cast<float4*>(to + 2 * i) = make_float4(x[0], x[1], x[2], x[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (d + e < a.dim) to[2 * i + e] = x[e];
          }
        }
      }
    }
  }
  if (!ok)   // a wait ran out: give copies that may still be in flight a millisecond before the shared memory goes back
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  __syncthreads();
}

// A step of single tokens: bound by reading and writing the states. A warp has (LANES = 16) eight columns of a (request,
// head), four columns and eight channels a thread as above; every load, the state's and the token's, is on its way at
// once and no thread waits for another warp. Every sum has the terms and the order of delta_rule.cu, so that a token gets
// the same bits alone as among others of its request (delta_rule.cu: a trip to memory for the row's length, one for its slot, one
// for the state with 32 bytes a thread, two barriers). 16 requests, 32 heads of 128 x 128, a decay per channel: 47 -> 24 us,
// per head 41 -> 20, the dual with 128 heads of 128 x 64 56 -> 32 (their states' bytes take 10, 10 and 20); 64 requests,
// per head 137 -> 55.
template <typename T, int LANES, int MODE>
__global__ void __launch_bounds__(128)
step_kernel(WalkArgs a) {
  constexpr bool LOOKS = MODE != kWalkDual;
  constexpr int NL = LANES * kWalkPer / 32;   // channels a lane adds to the norms: those that delta_rule.cu gives it
  const int row = blockIdx.x, head = blockIdx.y, lane = threadIdx.x & 31;
  const int length = a.row_length[row], slot = a.request_slots[row];
  if (length <= 0) return;
  if (slot < 0 || slot >= a.num_slots) {
    if (threadIdx.x == 0) atomicOr(a.status, kStatusBadSlot);
    return;
  }
  const int part = threadIdx.x % LANES, d0 = part * kWalkPer;
  const int column = (blockIdx.z * (128 / LANES) + threadIdx.x / LANES) * kWalkCols;
  const bool has = d0 < a.dim;   // dim is a multiple of eight
  float* home = a.state + static_cast<long long>(slot) * a.slot_stride + (static_cast<long long>(head) * a.vdim + column) * a.dim + d0;
  float4 s[kWalkCols][2];
#pragma unroll
  for (int c = 0; c < kWalkCols; ++c)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      s[c][i] = has && column + c < a.vdim ? *reinterpret_cast<const float4*>(home + static_cast<long long>(c) * a.dim + 4 * i)
                                           : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  struct alignas(16) Eight { T v[16 / sizeof(T)]; };
  constexpr int PIECES = kWalkPer * sizeof(T) / 16, EACH = 16 / sizeof(T);
  const int group = head / (a.heads / a.groups);
  const long long first = a.row_start[row];
#pragma unroll 1
  for (long long token = first; token < first + length; ++token) {   // once, unless a row is longer than the caller said
    const T* x = static_cast<const T*>(a.qkv) + token * a.ld;
    const bool last = token + 1 == first + length;
    Eight raw_q[PIECES] = {}, raw_k[PIECES] = {};
    if (has)
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        raw_q[i] = *reinterpret_cast<const Eight*>(x + a.q_off + group * a.dim + d0 + i * EACH);
        raw_k[i] = *reinterpret_cast<const Eight*>(x + a.k_off + group * a.dim + d0 + i * EACH);
      }
    T norm_q[NL], norm_k[NL];
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      const int d = min(lane + 32 * i, a.dim - 1);
      norm_q[i] = x[a.q_off + group * a.dim + d];
      norm_k[i] = x[a.k_off + group * a.dim + d];
    }
    T raw_v[kWalkCols];
#pragma unroll
    for (int c = 0; c < kWalkCols; ++c) raw_v[c] = x[a.v_off + head * a.vdim + min(column + c, a.vdim - 1)];
    float pre[MODE == kWalkChannel ? kWalkPer : 1], bias[MODE == kWalkChannel ? kWalkPer : 1];
    if (MODE == kWalkChannel) {
#pragma unroll
      for (int i = 0; i < kWalkPer; ++i) {
        pre[i] = has ? static_cast<const float*>(a.step_pre)[token * a.lds + head * a.dim + d0 + i] : 0.0f;
        bias[i] = has ? a.step_bias[head * a.dim + d0 + i] : 0.0f;
      }
    } else {
      pre[0] = to_float(static_cast<const T*>(a.step_pre)[token * a.lds + head]);
      bias[0] = a.step_bias[head];
    }
    const float rate = a.rate[head], skip = MODE == kWalkDual ? a.skip[head] : 0.0f;
    float beta = LOOKS ? sigmoid_of(to_float(static_cast<const T*>(a.beta_pre)[token * a.ldb + a.b_off + head])) : 0.0f;

    float q[kWalkPer], k[kWalkPer], g[kWalkPer], qq = 0.0f, kk = 0.0f, qk = 0.0f;
#pragma unroll
    for (int i = 0; i < kWalkPer; ++i) {
      q[i] = to_float(raw_q[i / EACH].v[i % EACH]);
      k[i] = to_float(raw_k[i / EACH].v[i % EACH]);
    }
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      const bool there = lane + 32 * i < a.dim;
      const float qd = there ? to_float(norm_q[i]) : 0.0f, kd = there ? to_float(norm_k[i]) : 0.0f;
      qq = fmaf(qd, qd, qq);
      kk = fmaf(kd, kd, kk);
      qk = fmaf(qd, kd, qk);
    }
    qk = warp_sum(qk);
    if (LOOKS) {
      const float q_unit = rsqrtf(warp_sum(qq) + 1e-6f) * rsqrtf(static_cast<float>(a.dim)), k_unit = rsqrtf(warp_sum(kk) + 1e-6f);
#pragma unroll
      for (int i = 0; i < kWalkPer; ++i) {
        q[i] *= q_unit;
        k[i] *= k_unit;
      }
      qk = qk * q_unit * k_unit;
    }
    // over the lanes of a column: neighbours first where the column is looked at, the dual in the order of its exchanges
    auto over_lanes = [](float v) {
#pragma unroll
      for (int step = 1; step < LANES; step <<= 1) v += __shfl_xor_sync(0xffffffffu, v, LOOKS ? step : LANES / 2 / step);
      return v;
    };
    if (MODE == kWalkChannel) {
#pragma unroll
      for (int i = 0; i < kWalkPer; ++i) g[i] = expf(-rate * walk_softplus(pre[MODE == kWalkChannel ? i : 0] + bias[MODE == kWalkChannel ? i : 0]));
    } else {
      const float step = walk_softplus(pre[0] + bias[0]), decay = expf(-rate * step);
      if (!LOOKS) beta = step;
#pragma unroll
      for (int i = 0; i < kWalkPer; ++i) g[i] = decay;
    }
#pragma unroll
    for (int c = 0; c < kWalkCols; ++c) {
      float r[kWalkPer] = {s[c][0].x, s[c][0].y, s[c][0].z, s[c][0].w, s[c][1].x, s[c][1].y, s[c][1].z, s[c][1].w};
      float k_dot = 0.0f, q_dot = 0.0f;
#pragma unroll
      for (int i = 0; i < kWalkPer; ++i) {
        r[i] *= g[i];
        k_dot = fmaf(k[i], r[i], k_dot);
        q_dot = fmaf(q[i], r[i], q_dot);
      }
      if (LOOKS) k_dot = over_lanes(k_dot);
      q_dot = over_lanes(q_dot);
      const float v = to_float(raw_v[c]), u = beta * (LOOKS ? v - k_dot : v);
      if (column + c < a.vdim) {
        s[c][0] = make_float4(fmaf(k[0], u, r[0]), fmaf(k[1], u, r[1]), fmaf(k[2], u, r[2]), fmaf(k[3], u, r[3]));
        s[c][1] = make_float4(fmaf(k[4], u, r[4]), fmaf(k[5], u, r[5]), fmaf(k[6], u, r[6]), fmaf(k[7], u, r[7]));
        if (has && last) {
          float4* to = reinterpret_cast<float4*>(home + static_cast<long long>(c) * a.dim);
          to[0] = s[c][0];
          to[1] = s[c][1];
        }
        float o = fmaf(qk, u, q_dot);
        if (MODE == kWalkDual) o = fmaf(skip, v, o);
        if (part == 0)
          a.out[token * (static_cast<long long>(a.heads) * a.vdim) + static_cast<long long>(head) * a.vdim + column + c] = o;
      }
    }
  }
}

static int walk_lanes(int dim) { return dim <= 64 ? 8 : 16; }
// Tokens of a window; its rows' eights are at most window / 8 + rows.
static long long walk_window(long long tokens, int rows, int heads, int dim) {
  const long long eights = kWalkScratch / (4ll * heads * walk_record(walk_lanes(dim) * kWalkPer));
  long long window = (eights - rows) * kEight;
  if (window < 256) window = 256;
  return window < tokens ? window : tokens;
}

}  // namespace mxb

using namespace mxb;

// How many KiB of scratch mxb_delta_prompt needs for a step of `tokens` tokens whose longest row brings `longest` (0:
// unknown); 0: the step does not take this way. It does in bfloat16 with a decay per channel (mode 0) where a row brings 64
// tokens, or 32 and there is other work (us, delta_rule.cu first, heads of 128 x 128: 16 heads, one row of 24 tokens 17 and
// 17, of 32 20 and 25, of 56 29 and 30, of 64 33 and 32, of 1,777 672 and 304; 8 heads, four rows of 32 26 and 26; 16 heads,
// three 43 and 28; 24 heads, one row of 40 29 and 30, of 48 34 and 32; 32 heads, one row of 32 25 and 26, of 40 30 and 28;
// beside 31 single tokens 131 and 89; 128 heads, eight rows of 512 7,383 and 3,025, whose records come in several
// windows). Keys have 33 to 128 channels: narrower ones leave lanes without channels, wider ones do not fit a thread's registers.
MXB_API int mxb_delta_prompt_scratch(long long tokens, int rows, int longest, int mode, int heads, int dim, int dtype) {
  if (dtype != kBF16 || tokens <= 0 || rows <= 0 || longest < 32 || mode != kWalkChannel || heads <= 0 || heads > 65535 || dim <= 32 || dim > 128)
    return 0;
  if (longest < 64 && static_cast<long long>(heads) * rows < 40 && heads * tokens < 1152) return 0;
  const long long eights = walk_window(tokens, rows, heads, dim) / kEight + rows;
  const long long kib = (eights * 4 * heads * walk_record(walk_lanes(dim) * kWalkPer) + 1023) >> 10;
  return kib > 0x7fffffffLL ? 0 : static_cast<int>(kib);
}

// As mxb_delta_rule (mode 0), for steps that mxb_delta_prompt_scratch gives a size for; `scratch` lies on 16 bytes.
MXB_API int mxb_delta_prompt(const void* qkv, long long ld, int q_off, int k_off, int v_off, const void* beta_pre,
                             long long ldb, int b_off, const void* step_pre, long long lds, const float* step_bias,
                             const float* rate, const float* skip, int mode, float* state, long long slot_stride, int num_slots,
                             const int* row_start, const int* row_length, const int* request_slots, float* out,
                             long long tokens, int rows, int heads, int groups, int dim, int vdim, int dtype, int longest,
                             void* scratch, int* status, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (groups <= 0 || heads % groups != 0 || vdim <= 0 || skip != nullptr || scratch == nullptr ||
      (reinterpret_cast<uintptr_t>(scratch) & 15) ||
      mxb_delta_prompt_scratch(tokens, rows, longest, mode, heads, dim, dtype) == 0)
    return static_cast<int>(cudaErrorInvalidValue);
  const int lanes = walk_lanes(dim);
  const long long window = walk_window(tokens, rows, heads, dim);
  WalkArgs a = {qkv, ld, q_off, k_off, v_off, beta_pre, ldb, b_off, step_pre, lds, step_bias, rate, skip, state, slot_stride,
                num_slots, row_start, row_length, request_slots, out, rows, heads, groups, dim, vdim, status,
                static_cast<float*>(scratch), static_cast<int>(window / kEight + rows), 0, 0};
  // 32 columns a block, 16 where that leaves SMs without a block.
  const int columns = static_cast<long long>(rows) * heads * ceil_div(vdim, 32) < 120 ? 16 : 32;
  const int threads = ceil_div(columns / kWalkCols * lanes, 32) * 32 + 32;
  const int of_block = (threads - 32) / lanes * kWalkCols;
  auto run = [&](auto lanes_of) {
    using T = __nv_bfloat16;
    constexpr int LANES = decltype(lanes_of)::value;
    constexpr int shared = kWalkStages * walk_record(LANES * kWalkPer) * 4;
    const cudaError_t e = cudaFuncSetAttribute(walk_kernel<T, LANES>, cudaFuncAttributeMaxDynamicSharedMemorySize, shared);
    if (e != cudaSuccess) return static_cast<int>(e);
    for (a.from = 0; a.from < tokens; a.from += window) {
      a.to = a.from + window < tokens ? a.from + window : tokens;
      const int eights = static_cast<int>((a.to - a.from) / kEight + rows);
      walk_records_kernel<T, LANES><<<dim3(eights, heads), 32 * kEight, 0, stream>>>(a);
      walk_kernel<T, LANES><<<dim3(rows, heads, ceil_div(vdim, of_block)), threads, shared, stream>>>(a);
    }
    return static_cast<int>(cudaGetLastError());
  };
  return lanes == 8 ? run(std::integral_constant<int, 8>()) : run(std::integral_constant<int, 16>());
}

// Whether mxb_delta_step takes a step: single tokens (longest 1), keys of 40, 48 ... 128 channels whose rows and states
// start on 16 bytes. Other steps of single tokens stay with mxb_delta_rule.
MXB_API int mxb_delta_step_supported(const void* qkv, long long ld, int q_off, int k_off, int mode, const float* state,
                                     long long slot_stride, int heads, int dim, int dtype, int longest) {
  const int each = dtype == kF32 ? 4 : 8;   // values of 16 bytes
  return longest == 1 && mode >= kWalkChannel && mode <= kWalkDual && (dtype == kF32 || dtype == kBF16) && heads > 0 &&
                 heads <= 65535 && dim > 32 && dim <= 128 && dim % kWalkPer == 0 && ld % each == 0 && q_off % each == 0 &&
                 k_off % each == 0 && slot_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(qkv) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(state) & 15) == 0
             ? 1 : 0;
}

MXB_API int mxb_delta_step(const void* qkv, long long ld, int q_off, int k_off, int v_off, const void* beta_pre,
                           long long ldb, int b_off, const void* step_pre, long long lds, const float* step_bias,
                           const float* rate, const float* skip, int mode, float* state, long long slot_stride, int num_slots,
                           const int* row_start, const int* row_length, const int* request_slots, float* out, int rows,
                           int heads, int groups, int dim, int vdim, int dtype, int longest, int* status, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (groups <= 0 || heads % groups != 0 || vdim <= 0 || (mode == kWalkDual) != (skip != nullptr) ||
      !mxb_delta_step_supported(qkv, ld, q_off, k_off, mode, state, slot_stride, heads, dim, dtype, longest))
    return static_cast<int>(cudaErrorInvalidValue);
  const WalkArgs a = {qkv, ld, q_off, k_off, v_off, beta_pre, ldb, b_off, step_pre, lds, step_bias, rate, skip, state,
                      slot_stride, num_slots, row_start, row_length, request_slots, out, rows, heads, groups, dim, vdim, status,
                      nullptr, 0, 0, 0};
  const int lanes = walk_lanes(dim);
  const dim3 grid(rows, heads, ceil_div(vdim, 128 / lanes * kWalkCols));
  auto by_mode = [&](auto type, auto lanes_of) {
    using T = decltype(type);
    constexpr int LANES = decltype(lanes_of)::value;
    if (mode == kWalkChannel) step_kernel<T, LANES, kWalkChannel><<<grid, 128, 0, stream>>>(a);
    else if (mode == kWalkHead) step_kernel<T, LANES, kWalkHead><<<grid, 128, 0, stream>>>(a);
    else step_kernel<T, LANES, kWalkDual><<<grid, 128, 0, stream>>>(a);
    return static_cast<int>(cudaGetLastError());
  };
  auto by_lanes = [&](auto type) {
    return lanes == 8 ? by_mode(type, std::integral_constant<int, 8>()) : by_mode(type, std::integral_constant<int, 16>());
  };
  return dtype == kF32 ? by_lanes(float()) : by_lanes(__nv_bfloat16());
}
