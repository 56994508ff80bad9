// The selective state-space recurrence (Mamba's scan) over the packed tokens
// of a step, with the state kept per request.
//
// Per channel c and state n, with a step size d_t[c] = softplus(p_t[c] + b[c])
// that depends on the token:
//
//   S[c, n] <- exp(d_t[c] A[c, n]) S[c, n] + d_t[c] x_t[c] B_t[n]
//   y_t[c]  =  sum_n S[c, n] C_t[n] + D[c] x_t[c]
//   out_t[c] = y_t[c] * silu(z_t[c])
//
// Step sizes, decays, exponentials, the state and the sums are float32 in
// both precisions; x, B, C and z arrive in the compute type. Four lanes share
// a channel, each owning every fourth state in registers; a request row's
// tokens are walked in order, so what a position gets does not depend on how
// the sequence was cut into steps (float32 always; bfloat16 where no step took
// the chunks below, which agree with the walk to float32's rounding). `state` is
// [slots, channels, states] float32; a row of length 0 touches no slot.
//
// Prompts in bfloat16: one walk per channel over 1,201 tokens is a chain of 1,201 steps on few warps (that row and two of 700 and 800
// with 2,048 channels: 445 us). So their rows are cut into chunks of 64 tokens that run side by side, twice: once from a state of
// zeros for what a chunk adds and the sum of its step sizes, from which the state ahead of every chunk follows
// (S <- exp(A sum) S + added), then from that state for the outputs: 210 us.
#include <type_traits>

#include "common.cuh"

namespace mxb {

constexpr int kScanLanes = 4;          // lanes that share a channel
constexpr int kScanThreads = 128;      // 32 channels a block

__device__ __forceinline__ float softplus_of(float v) { return v > 20.0f ? v : log1pf(expf(v)); }

constexpr int kScanChunk = 64;         // tokens of a chunk of a prompt
constexpr long long kScanScratch = 256ll << 20;   // bytes that the states ahead of the chunks may take

enum ScanPart : int { kWholeRow = 0, kChunkAdds = 1, kChunkOutputs = 2 };

// Scratch of the chunks: states [rows][chunks][channels][states], then step sizes [rows][chunks][channels].
template <typename T, int PER, int AHEAD, int PART>
__global__ void __launch_bounds__(kScanThreads)
selective_scan_kernel(const T* __restrict__ x, long long ldx, const float* __restrict__ step, long long ld_step,
                      const float* __restrict__ step_bias, const float* __restrict__ a, const T* __restrict__ b,
                      const T* __restrict__ c, long long ldbc, const float* __restrict__ d, const T* __restrict__ z,
                      long long ldz, float* __restrict__ state, const int* __restrict__ row_start,
                      const int* __restrict__ row_length, const int* __restrict__ request_slots,
                      T* __restrict__ out, int channels, int states, int num_slots, float* __restrict__ chunk_states,
                      float* __restrict__ chunk_steps, int chunks, int* status) {
  const int row = blockIdx.y;
  const int all = row_length[row], begin = PART == kWholeRow ? 0 : static_cast<int>(blockIdx.z) * kScanChunk;
  if (all <= begin) return;
  const bool last = PART == kWholeRow || all - begin <= kScanChunk;
  if (PART == kChunkAdds && last) return;   // nothing follows it
  const int n = last ? all - begin : kScanChunk;
  const int slot = request_slots[row];
  // A row of more chunks than the caller said would reach beyond its part of the scratch: none of it is worked on.
  if (slot < 0 || slot >= num_slots || (PART != kWholeRow && all > chunks * kScanChunk)) {
    if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(status, kStatusBadSlot);
    return;
  }
  static_assert(PART == kWholeRow || AHEAD >= kScanLanes, "the chunks take the form with tokens side by side");
  const int lane = threadIdx.x & (kScanLanes - 1);
  const int ch = blockIdx.x * (kScanThreads / kScanLanes) + (threadIdx.x / kScanLanes);
  const bool live = ch < channels;
  const int cc = live ? ch : channels - 1;      // idle lanes of the last block shadow a real channel and write nothing
  const int start = row_start[row] + begin;
  float* held = state + (static_cast<size_t>(slot) * channels + cc) * states;
  const size_t of_chunk = PART == kWholeRow ? 0 : (static_cast<size_t>(row) * chunks + blockIdx.z) * channels + cc;
  const float* ahead_of_it = PART == kChunkOutputs ? chunk_states + of_chunk * states : held;
  float s[PER], decay[PER], steps = 0.0f;
  constexpr bool BESIDE = PART != kWholeRow;   // a lane's states lie side by side (else every fourth is its own)
  auto state_of = [&](int j) { return BESIDE ? lane * PER + j : lane + kScanLanes * j; };
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int k = state_of(j);
    s[j] = PART != kChunkAdds && k < states ? ahead_of_it[k] : 0.0f;
    decay[j] = k < states ? a[static_cast<size_t>(cc) * states + k] : 0.0f;
  }
  const float bias = step_bias[cc], skip = d[cc];
  // The recurrence ties a token to the one before it only through one
  // multiply-add per state; everything else about a token (its loads, step
  // size, decays, increments, gate) does not wait for the token before. So
  // AHEAD tokens are fetched and prepared side by side, then stepped through.
  // A token past the row's end repeats the last one's loads with a decay of
  // one and an increment of zero, which leaves the state as it is. A step of
  // single tokens (a decode step) takes AHEAD = 1.
  if constexpr (AHEAD >= kScanLanes) {
    // What belongs to a token and not to a state (its step size, its input
    // times the step size, its gate) is the same for the lanes that share a
    // channel: lane l works it out for the tokens l, l + 4, ... of the batch
    // and hands it round; it also writes those tokens' outputs.
    constexpr int OWN = AHEAD / kScanLanes;
    // B and C of a chunk, the same for every channel, as float32 in shared memory: a lane's states in one read instead
    // of two loads per state and token (three rows of 2,048 channels: 224 -> 210 us). A whole row keeps the loads: its
    // chain would wait at the barriers (192 tokens: 72 -> 78 us).
    struct alignas(4 * PER) States { float v[PER]; };
    constexpr int HELD = PART == kWholeRow ? 1 : kScanChunk;
    __shared__ States s_b[HELD][kScanLanes], s_c[PART == kChunkOutputs ? HELD : 1][kScanLanes];
    if constexpr (PART != kWholeRow) {
      for (int e = threadIdx.x; e < n * kScanLanes * PER; e += kScanThreads) {
        const int i = e / (kScanLanes * PER), k = e % (kScanLanes * PER);
        const size_t t = static_cast<size_t>(start + i);
        (&s_b[i][0].v[0])[k] = k < states ? to_float(b[t * ldbc + k]) : 0.0f;   // a state that is not there stays at zero
        if (PART == kChunkOutputs) (&s_c[i][0].v[0])[k] = k < states ? to_float(c[t * ldbc + k]) : 0.0f;
      }
      __syncthreads();
    }
    for (int i0 = 0; i0 < n; i0 += AHEAD) {
      T bs[AHEAD][PER], cs[AHEAD][PER];
      float own_dt[OWN], own_dx[OWN], own_x[OWN], own_gate[OWN];
#pragma unroll
      for (int h = 0; h < OWN; ++h) {
        const int i = i0 + lane + kScanLanes * h;
        const size_t t = static_cast<size_t>(start + (i < n ? i : n - 1));
        own_dt[h] = step[t * ld_step + cc];
        own_x[h] = to_float(x[t * ldx + cc]);
        own_gate[h] = PART == kChunkAdds ? 0.0f : to_float(z[t * ldz + cc]);
      }
      if (PART == kWholeRow) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          const size_t t = static_cast<size_t>(start + (i0 + u < n ? i0 + u : n - 1));
#pragma unroll
          for (int j = 0; j < PER; ++j) {
            const int k = state_of(j);
            bs[u][j] = k < states ? b[t * ldbc + k] : from_float<T>(0.0f);   // a state that is not there stays at zero
            cs[u][j] = k < states ? c[t * ldbc + k] : from_float<T>(0.0f);
          }
        }
      }
#pragma unroll
      for (int h = 0; h < OWN; ++h) {
        own_dt[h] = softplus_of(own_dt[h] + bias);
        own_dx[h] = own_dt[h] * own_x[h];
        own_gate[h] = own_gate[h] / (1.0f + expf(-own_gate[h]));
        if (PART == kChunkAdds && i0 + lane + kScanLanes * h < n) steps += own_dt[h];
      }
      float keep[AHEAD][PER], add[AHEAD][PER], y[AHEAD];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const bool valid = i0 + u < n;
        const float dt = __shfl_sync(0xffffffffu, own_dt[u / kScanLanes], u % kScanLanes, kScanLanes);
        const float dx = __shfl_sync(0xffffffffu, own_dx[u / kScanLanes], u % kScanLanes, kScanLanes);
        const States b4 = s_b[PART == kWholeRow ? 0 : min(i0 + u, n - 1)][lane];
#pragma unroll
        for (int j = 0; j < PER; ++j) {
          keep[u][j] = valid ? expf(dt * decay[j]) : 1.0f;
          add[u][j] = valid ? dx * (PART == kWholeRow ? to_float(bs[u][j]) : b4.v[j]) : 0.0f;
        }
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const States c4 = s_c[PART == kChunkOutputs ? min(i0 + u, n - 1) : 0][lane];
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
          s[j] = fmaf(keep[u][j], s[j], add[u][j]);
          if (PART != kChunkAdds) sum = fmaf(s[j], PART == kWholeRow ? to_float(cs[u][j]) : c4.v[j], sum);
        }
        y[u] = sum;
      }
      if constexpr (PART != kChunkAdds) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          y[u] += __shfl_xor_sync(0xffffffffu, y[u], 1);
          y[u] += __shfl_xor_sync(0xffffffffu, y[u], 2);
          if (lane == u % kScanLanes && live && i0 + u < n)
            out[static_cast<size_t>(start + i0 + u) * channels + cc] =
                from_float<T>(fmaf(skip, own_x[u / kScanLanes], y[u]) * own_gate[u / kScanLanes]);
        }
      }
    }
  } else {
    for (int i0 = 0; i0 < n; i0 += AHEAD) {
      float pv[AHEAD], xs[AHEAD], zs[AHEAD];
      T bs[AHEAD][PER], cs[AHEAD][PER];
  #pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const size_t t = static_cast<size_t>(start + (i0 + u < n ? i0 + u : n - 1));
        pv[u] = step[t * ld_step + cc];
        xs[u] = to_float(x[t * ldx + cc]);
        zs[u] = to_float(z[t * ldz + cc]);
  #pragma unroll
        for (int j = 0; j < PER; ++j) {
          const int k = lane + kScanLanes * j;
          bs[u][j] = k < states ? b[t * ldbc + k] : from_float<T>(0.0f);   // a state that is not there stays at zero
          cs[u][j] = k < states ? c[t * ldbc + k] : from_float<T>(0.0f);
        }
      }
      float keep[AHEAD][PER], add[AHEAD][PER], gate[AHEAD], y[AHEAD];
  #pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const bool valid = i0 + u < n;
        const float dt = softplus_of(pv[u] + bias);
        const float dx = dt * xs[u];
  #pragma unroll
        for (int j = 0; j < PER; ++j) {
          keep[u][j] = valid ? expf(dt * decay[j]) : 1.0f;
          add[u][j] = valid ? dx * to_float(bs[u][j]) : 0.0f;
        }
        gate[u] = zs[u] / (1.0f + expf(-zs[u]));
      }
  #pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        float sum = 0.0f;
  #pragma unroll
        for (int j = 0; j < PER; ++j) {
          s[j] = fmaf(keep[u][j], s[j], add[u][j]);
          sum = fmaf(s[j], to_float(cs[u][j]), sum);
        }
        y[u] = sum;
      }
  #pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        y[u] += __shfl_xor_sync(0xffffffffu, y[u], 1);
        y[u] += __shfl_xor_sync(0xffffffffu, y[u], 2);
        if (lane == 0 && live && i0 + u < n)
          out[static_cast<size_t>(start + i0 + u) * channels + cc] = from_float<T>(fmaf(skip, xs[u], y[u]) * gate[u]);
      }
    }
  }
  if (PART == kChunkAdds) {
    steps += __shfl_xor_sync(0xffffffffu, steps, 1);
    steps += __shfl_xor_sync(0xffffffffu, steps, 2);
    if (live && lane == 0) chunk_steps[of_chunk] = steps;
    held = chunk_states + of_chunk * states;
  }
  if (live && (PART == kChunkAdds || last)) {
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int k = state_of(j);
      if (k < states) held[k] = s[j];
    }
  }
}

// The state ahead of every chunk, in the place of what the chunk adds: one thread per (channel, state) of a row.
__global__ void __launch_bounds__(256)
selective_scan_states_kernel(const float* __restrict__ a, const float* __restrict__ state, const int* __restrict__ row_length,
                             const int* __restrict__ request_slots, float* __restrict__ chunk_states,
                             const float* __restrict__ chunk_steps, int channels, int states, int num_slots, int chunks) {
  const int row = blockIdx.y, n = row_length[row], slot = request_slots[row];
  const size_t values = static_cast<size_t>(channels) * states, e = blockIdx.x * size_t(256) + threadIdx.x;
  if (n <= 0 || n > chunks * kScanChunk || slot < 0 || slot >= num_slots || e >= values) return;
  const int used = ceil_div(n, kScanChunk);
  const float decay = a[e];
  float s = state[slot * values + e];
  float* at = chunk_states + static_cast<size_t>(row) * chunks * values + e;
  const float* steps = chunk_steps + static_cast<size_t>(row) * chunks * channels + e / states;
  constexpr int kAhead = 8;   // chunks whose loads are under way at once
  for (int c0 = 0; c0 < used; c0 += kAhead) {
    float added[kAhead], step[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int c = min(c0 + j, used - 1);
      added[j] = at[c * values];
      step[j] = steps[static_cast<size_t>(c) * channels];
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (c0 + j >= used) break;
      at[(c0 + j) * values] = s;
      s = fmaf(expf(step[j] * decay), s, added[j]);   // the last chunk's is not used
    }
  }
}

template <typename T, int PER>
static int launch_scan(const void* x, long long ldx, const float* step, long long ld_step, const float* step_bias,
                       const float* a, const void* b, const void* c, long long ldbc, const float* d, const void* z,
                       long long ldz, float* state, const int* row_start, const int* row_length,
                       const int* request_slots, void* out, int rows, int channels, int states, int num_slots,
                       int longest, float* scratch, int* status, cudaStream_t stream) {
  dim3 grid(ceil_div(channels, kScanThreads / kScanLanes), rows);
  constexpr int ahead = PER <= 4 ? 8 : (PER <= 16 ? 2 : 1);
  int chunks = 0;
  float* steps = nullptr;
#define SCAN(AHEAD, PART)                                                                                            \
  selective_scan_kernel<T, PER, AHEAD, PART><<<grid, kScanThreads, 0, stream>>>(                                    \
      static_cast<const T*>(x), ldx, step, ld_step, step_bias, a, static_cast<const T*>(b), static_cast<const T*>(c), \
      ldbc, d, static_cast<const T*>(z), ldz, state, row_start, row_length, request_slots, static_cast<T*>(out),    \
      channels, states, num_slots, scratch, steps, chunks, status)
  if constexpr (PER <= 4 && std::is_same_v<T, __nv_bfloat16>) {
    if (scratch != nullptr) {
      chunks = ceil_div(longest, kScanChunk);
      steps = scratch + static_cast<size_t>(rows) * chunks * channels * states;
      grid.z = chunks;
      SCAN(ahead, kChunkAdds);
      selective_scan_states_kernel<<<dim3(ceil_div(channels * states, 256), rows), 256, 0, stream>>>(
          a, state, row_length, request_slots, scratch, steps, channels, states, num_slots, chunks);
      SCAN(ahead, kChunkOutputs);
      return static_cast<int>(cudaGetLastError());
    }
  }
  if (longest == 1 || ahead == 1) SCAN(1, kWholeRow); else SCAN(ahead, kWholeRow);
#undef SCAN
  return static_cast<int>(cudaGetLastError());
}

}  // namespace mxb

using namespace mxb;

// How many float32 values of scratch mxb_selective_scan wants, to walk a step's rows in chunks: none (0) in float32, whose
// results are the same however a sequence is cut and whatever else a step brings, where the longest
// row is not known or short, or has more than 16 states, or where the step is wide: the chunks cost twice the arithmetic,
// which pays as long as a walk's chain of steps is what takes the time. The line lies at 6,000 (channel, token) pairs per
// token of the longest row (us, whole rows first): 4,600 pairs (2,048 channels, rows of 1,201, 700 and 800 tokens) 445 and
// 210, 2,140 (700 beside 31 single tokens) 245 and 122, 2,048 (one row of 256) 93 and 52; 6,144 (6,144 channels, one row of
// 192) 78 and 60, 8,192 (4,096 channels, two rows) 80 and 85, 18,400 618 and 730. And a row costs some 12 tokens' work and
// half a token's per chunk of the longest row however short it is, mostly its state's way to the scratch and back: beside
// a row of 256, 2,048 channels, 31 single tokens 96 and 83, 63 98 and 108, 400 166 and 415; beside one of 1,024, 63 360 and 192.
// The second line's numbers take the measured winners among 140 such steps and no loser.
MXB_API int mxb_selective_scan_scratch(long long tokens, int rows, int channels, int states, int longest, int dtype) {
  if (dtype != kBF16 || tokens <= 0 || rows <= 0 || channels <= 0 || states <= 0 || states > 4 * kScanLanes || longest < 3 * kScanChunk ||
      tokens * channels > 6000ll * longest)
    return 0;
  const long long chunks = ceil_div(longest, kScanChunk);
  if (channels * (tokens + rows * (24 + chunks)) > 18000ll * longest - 1600000ll) return 0;
  const long long each = static_cast<long long>(channels) * (states + 1);
  const long long values = chunks * rows * each;
  return chunks > 65535 || values * 4 > kScanScratch ? 0 : static_cast<int>(values);
}

// x, z: [tokens, channels] (row strides ldx, ldz); step: float32 [tokens, channels] ahead of its bias and softplus;
// a: float32 [channels, states] (negative); b, c: [tokens, states] with row stride ldbc; d: [channels];
// out: [tokens, channels] contiguous. Up to 256 states. longest: the most tokens of a row (0 if not known); with scratch,
// a row that brings more than `longest` rounded up to 64 sets the status word's bit for bad rows and is left out.
// scratch: as many float32 values as mxb_selective_scan_scratch says, or null: every row in one walk.
MXB_API int mxb_selective_scan(const void* x, long long ldx, const float* step, long long ld_step,
                               const float* step_bias, const float* a, const void* b, const void* c, long long ldbc,
                               const float* d, const void* z, long long ldz, float* state, const int* row_start,
                               const int* row_length, const int* request_slots, void* out, int rows, int channels,
                               int states, int num_slots, int longest, float* scratch, int dtype, int* status,
                               cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (channels <= 0 || states <= 0 || states > 64 * kScanLanes) return static_cast<int>(cudaErrorInvalidValue);
  if (scratch != nullptr && (dtype != kBF16 || states > 4 * kScanLanes || longest <= 0)) return static_cast<int>(cudaErrorInvalidValue);
  const int per = ceil_div(states, kScanLanes);
#define ARGS x, ldx, step, ld_step, step_bias, a, b, c, ldbc, d, z, ldz, state, row_start, row_length, request_slots, \
             out, rows, channels, states, num_slots, longest, scratch, status, stream
#define DISPATCH(T)                                    \
  if (per <= 1) return launch_scan<T, 1>(ARGS);        \
  if (per <= 2) return launch_scan<T, 2>(ARGS);        \
  if (per <= 4) return launch_scan<T, 4>(ARGS);        \
  if (per <= 8) return launch_scan<T, 8>(ARGS);        \
  if (per <= 16) return launch_scan<T, 16>(ARGS);      \
  if (per <= 32) return launch_scan<T, 32>(ARGS);      \
  return launch_scan<T, 64>(ARGS);
  if (dtype == kF32) { DISPATCH(float) }
  if (dtype == kBF16) { DISPATCH(__nv_bfloat16) }
#undef DISPATCH
#undef ARGS
  return static_cast<int>(cudaErrorInvalidValue);
}
