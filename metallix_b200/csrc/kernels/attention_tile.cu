// Attention over the paged cache for any mix of prompt portions and decoded
// tokens: the general kernel of both precisions.
//
// One block takes up to 16 consecutive query tokens of one request and one
// query head, walks the request's keys in tiles of 32 absolute positions
// through its block table, and keeps scores, running maximum, running sum and
// the output accumulator in float32. Key tiles start at multiples of 32 of the
// absolute position, and a row's arithmetic touches only its own keys in
// ascending order, so the result at a position is bit-identical however the
// tokens were cut into steps or batched.
//
// Replaces the reference's gather of the whole context plus
// fast::scaled_dot_product_attention (crates/models/qwen/src/forward/paged.rs:329-342,
// :1067-1076, :1176-1184): s = (q k^T) * scale, causal with the diagonal at the
// query's own position, optional window (key > position - window) and chunk (key >= position - position % chunk),
// both widened by the first `keep` positions, softmax over keys, query head j reads key/value head j / (heads / kv_heads).
//
// Further parameters, each off by default: `softcap` c bounds a score to
// (-c, c) ahead of the softmax, s <- c tanh(s / c); the pool may hold one plane
// per page instead of two (`planes` 1: the values are the first `value_dim`
// values of the key rows themselves, what attention through a shared latent
// needs); `value_dim` (at most head_dim) is how many values of a value row
// make up the output, out being [tokens, heads, value_dim]; the output gate
// may be one number per (token, head) (`gate_per_head`) instead of one per value;
// `has_sink` adds a key without a value whose score is `sink_score` to every
// query's softmax (with score 0: one more in the denominator); `sink_heads`, when
// given, holds one such score per query head (float32) and is used instead;
// `bias` adds a number per head and distance to every (capped) score.
#include "common.cuh"

namespace mxb {

constexpr int kTileQueries = 16;
constexpr int kTileKeys = 32;
constexpr int kTileThreads = 128;
constexpr int kScorePitch = kTileKeys + 4;   // floats; the four rows of a warp read 16 bytes each from banks of their own
constexpr float kMinusHuge = -1.0e30f;

struct TileArgs {
  const void* q;
  const void* cache;
  void* out;
  const int* block_tables;
  int max_pages;
  const int *tile_request, *tile_start, *tile_length, *positions;
  int tiles, heads, kv_heads, head_dim, page_tokens, num_pages, window, chunk, keep;
  float scale;
  const void* gate;
  long long gate_stride;
  int planes, value_dim;
  float softcap;
  int gate_per_head, has_sink;
  float sink_score;
  const float* sink_heads;
  ScoreBias bias;
  int stages;     // key tiles held at a time: 2 asks for the next one while this one is used (asynchronous copies)
  int vectors;    // rows of the cache may be read four values at a time
  int* status;
};

// Floats of a row of queries or keys in shared memory: an odd number of 16-byte words, so that eight keys or four
// query rows read at the same offset fall on different banks.
__host__ __device__ __forceinline__ int row_pitch(int dim) { return ((dim + 3) / 4 | 1) * 4; }

__device__ __forceinline__ float4 four_values(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 four_values(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                     __uint_as_float(raw.y & 0xffff0000u));
}
__device__ __forceinline__ void async_16(float* to, const float* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(to))), "l"(from)
               : "memory");
}

// Bound by the CUDA cores and by shared memory's bandwidth. G query heads of one key/value head share a block's keys
// and values: a thread scores its query row of each head against four keys (per four values 4 + G 16-byte reads for
// 16 G multiply-adds) and owns four neighbouring values of the output per VQ (4 + G reads for 16 G). One head a block with
// 4-byte reads, a page looked up for every value, took 842 us for two prompts of 517 and some 400 float32 tokens, 16 heads
// of 128 over 8; this form takes 153 us.
template <typename T, int G, int VQ>
__global__ void __launch_bounds__(kTileThreads)
paged_attention_tile_kernel(const __grid_constant__ TileArgs args) {
  extern __shared__ __align__(16) float shared[];
  const int head_dim = args.head_dim, value_dim = args.value_dim;
  const int pitch = row_pitch(head_dim), value_pitch = VQ * 32;
  float* sQ = shared;                                        // [G][16][pitch]
  float* sP = sQ + G * kTileQueries * pitch;                 // [G][16][kScorePitch]
  float* sKV = sP + G * kTileQueries * kScorePitch;          // [stages]([32][pitch] keys, [32][value_pitch] values)
  const int stage_floats = kTileKeys * (pitch + value_pitch);

  // blocks of the last tiles first: they walk over the most keys
  const int per_tile = args.heads / G;
  const int tile = args.tiles - 1 - static_cast<int>(blockIdx.x) / per_tile;
  const int head0 = static_cast<int>(blockIdx.x) % per_tile * G;
  const int kv = head0 / (args.heads / args.kv_heads);
  const int request = args.tile_request[tile];
  const int t0 = args.tile_start[tile];
  const int n = args.tile_length[tile];
  const int pos0 = args.positions[t0];
  const int last_pos = pos0 + n - 1;
  const int first_key = first_visible_key(pos0, args.window, args.chunk);
  const int tid = threadIdx.x;
  const int r = tid >> 3, lane8 = tid & 7;
  const int my_pos = pos0 + r;
  const int my_first = first_visible_key(my_pos, args.window, args.chunk);   // first key this row sees
  const bool row_valid = r < n;
  const bool warp_live = (r & ~3) < n;   // some row of this warp is valid
  const int* table = args.block_tables + static_cast<size_t>(request) * args.max_pages;
  const T* q = static_cast<const T*>(args.q);
  const T* cache = static_cast<const T*>(args.cache);
  const int page_tokens = args.page_tokens;
  const size_t plane = static_cast<size_t>(args.kv_heads) * page_tokens * head_dim;   // from a page's keys to its values

  for (int i = tid; i < G * kTileQueries * pitch; i += kTileThreads) {
    const int line = i / pitch, d = i - line * pitch, g = line / kTileQueries, row = line - g * kTileQueries;
    sQ[i] = row < n && d < head_dim
                ? to_float(q[(static_cast<size_t>(t0 + row) * args.heads + head0 + g) * head_dim + d]) : 0.0f;
  }

  // Brings the keys and values of a tile to shared memory; a thread has a quarter of one key's row.
  const KeyWalk walk = key_walk(first_key, last_pos, args.keep, kTileKeys);
  auto fetch = [&](int step, float* at) {
    const int kk = tid >> 2, sub = tid & 3;
    const int key = walk.tile(step) * kTileKeys + kk;
    float* sK = at + kk * pitch;
    float* sV = at + kTileKeys * pitch + kk * value_pitch;
    const T* from = nullptr;
    if (key_seen(key, last_pos, first_key, args.keep)) {
      const int page = table[key / page_tokens];
      if (page < 0 || page >= args.num_pages)
        atomicOr(args.status, kStatusBadPage);
      else
        from = cache + ((static_cast<size_t>(page) * args.planes * args.kv_heads + kv) * page_tokens + key % page_tokens) * head_dim;
    }
    const T* values = args.planes == 2 ? from + plane : from;
    if (from != nullptr && args.vectors) {
      for (int d = sub * 4; d < head_dim; d += 16) {
        if constexpr (sizeof(T) == 4) async_16(sK + d, from + d);
        else *reinterpret_cast<float4*>(sK + d) = four_values(from + d);
      }
      for (int d = sub * 4; d < value_pitch; d += 16) {
        if (d + 4 <= value_dim) {
          if constexpr (sizeof(T) == 4) async_16(sV + d, values + d);
          else *reinterpret_cast<float4*>(sV + d) = four_values(values + d);
        } else {
          for (int e = 0; e < 4; ++e) sV[d + e] = d + e < value_dim ? to_float(values[d + e]) : 0.0f;
        }
      }
    } else {
      for (int d = sub; d < pitch; d += 4) sK[d] = from != nullptr && d < head_dim ? to_float(from[d]) : 0.0f;
      for (int d = sub; d < value_pitch; d += 4) sV[d] = from != nullptr && d < value_dim ? to_float(values[d]) : 0.0f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float m[G], l[G];
  float4 acc[G][VQ];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = kMinusHuge, l[g] = 0.0f;
#pragma unroll
    for (int j = 0; j < VQ; ++j) acc[g][j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }

  const bool ahead = args.stages == 2;
  if (ahead) fetch(0, sKV);
  for (int step = 0; step < walk.count; ++step) {
    const float* sK = sKV + (ahead ? step % 2 : 0) * stage_floats;
    const float* sV = sK + kTileKeys * pitch;
    __syncthreads();  // the previous tile's keys, values and weights are no longer read
    if (ahead) {
      if (step + 1 < walk.count) fetch(step + 1, sKV + (step + 1) % 2 * stage_floats);
      else asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      fetch(step, sKV);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (!warp_live) continue;

    const int key0 = walk.tile(step) * kTileKeys;
    float s[G][4];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[g][j] = 0.0f;
    const float* qrow = sQ + r * pitch;
    const float* krow = sK + lane8 * pitch;
#pragma unroll 2
    for (int d = 0; d < head_dim; d += 4) {
      float4 kx[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) kx[j] = *reinterpret_cast<const float4*>(krow + 8 * j * pitch + d);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 x = *reinterpret_cast<const float4*>(qrow + g * kTileQueries * pitch + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[g][j] = fmaf(x.x, kx[j].x, s[g][j]);
          s[g][j] = fmaf(x.y, kx[j].y, s[g][j]);
          s[g][j] = fmaf(x.z, kx[j].z, s[g][j]);
          s[g][j] = fmaf(x.w, kx[j].w, s[g][j]);
        }
      }
    }
    float alpha[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      bool visible[4];
      float tile_max = kMinusHuge;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = key0 + lane8 + 8 * j;
        visible[j] = row_valid && key_seen(key, my_pos, my_first, args.keep);
        // rounded as written: every form of the kernel has to leave the compiler the same choice of joint roundings
        float dot = __fmul_rn(s[g][j], args.scale);
        if (args.softcap > 0.0f) dot = __fmul_rn(args.softcap, tanhf(dot / args.softcap));
        if (args.bias.table != nullptr) dot = __fadd_rn(dot, bias_at(args.bias.row(head0 + g), my_pos - key, args.bias.far));
        s[g][j] = visible[j] ? dot : kMinusHuge;
        tile_max = fmaxf(tile_max, s[g][j]);
      }
#pragma unroll
      for (int offset = 1; offset < 8; offset <<= 1)
        tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, offset));
      const float m_new = fmaxf(m[g], tile_max);
      alpha[g] = expf(m[g] - m_new);
      float psum = 0.0f;
      float* prow = sP + (g * kTileQueries + r) * kScorePitch;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = visible[j] ? expf(s[g][j] - m_new) : 0.0f;
        prow[lane8 + 8 * j] = p;
        psum += p;
      }
#pragma unroll
      for (int offset = 1; offset < 8; offset <<= 1) psum += __shfl_xor_sync(0xffffffffu, psum, offset);
      l[g] = fmaf(l[g], alpha[g], psum);
      m[g] = m_new;
    }
    __syncwarp();  // a row's 8 threads sit in one warp

#pragma unroll
    for (int j = 0; j < VQ; ++j) {
      float4 sum[G];
#pragma unroll
      for (int g = 0; g < G; ++g) sum[g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float* vcol = sV + lane8 * 4 + 32 * j;
      // unrolled by two quads of keys at most: the output's accumulators want the registers
#pragma unroll 2
      for (int k = 0; k < kTileKeys; k += 4) {
        float4 v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const float4*>(vcol + (k + e) * value_pitch);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float4 p = *reinterpret_cast<const float4*>(sP + (g * kTileQueries + r) * kScorePitch + k);
          const float weight[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            sum[g].x = fmaf(weight[e], v[e].x, sum[g].x);
            sum[g].y = fmaf(weight[e], v[e].y, sum[g].y);
            sum[g].z = fmaf(weight[e], v[e].z, sum[g].z);
            sum[g].w = fmaf(weight[e], v[e].w, sum[g].w);
          }
        }
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        acc[g][j].x = fmaf(acc[g][j].x, alpha[g], sum[g].x);
        acc[g][j].y = fmaf(acc[g][j].y, alpha[g], sum[g].y);
        acc[g][j].z = fmaf(acc[g][j].z, alpha[g], sum[g].z);
        acc[g][j].w = fmaf(acc[g][j].w, alpha[g], sum[g].w);
      }
    }
    __syncwarp();
  }

  if (row_valid) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int head = head0 + g;
      const float sink = args.sink_heads != nullptr ? args.sink_heads[head] : args.sink_score;
      const float inv = 1.0f / (args.has_sink ? l[g] + expf(sink - m[g]) : l[g]);
      T* dst = static_cast<T*>(args.out) + (static_cast<size_t>(t0 + r) * args.heads + head) * value_dim;
      const T* gate = static_cast<const T*>(args.gate);
      if (gate != nullptr)
        gate += (t0 + r) * args.gate_stride + static_cast<long long>(head) * (args.gate_per_head ? 1 : value_dim);
      const float whole = gate != nullptr && args.gate_per_head ? sigmoid_of(to_float(gate[0])) : 1.0f;
#pragma unroll
      for (int j = 0; j < VQ; ++j) {
        const float four[4] = {acc[g][j].x, acc[g][j].y, acc[g][j].z, acc[g][j].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int d = lane8 * 4 + 32 * j + e;
          if (d < value_dim)
            dst[d] = from_float<T>(four[e] * inv * (gate != nullptr && !args.gate_per_head ? sigmoid_of(to_float(gate[d])) : whole));
        }
      }
    }
  }
}

constexpr size_t kTileSharedMost = 227 * 1024;

// Bytes of queries and weights of G heads, and of a tile of keys and values.
static size_t tile_fixed(int head_dim, int G) { return sizeof(float) * G * kTileQueries * (row_pitch(head_dim) + kScorePitch); }
static size_t tile_stage(int head_dim, int VQ) { return sizeof(float) * kTileKeys * (row_pitch(head_dim) + VQ * 32); }

template <typename T, int G, int VQ>
static int launch_tile(TileArgs args, cudaStream_t stream) {
  const size_t fixed = tile_fixed(args.head_dim, G), stage = tile_stage(args.head_dim, VQ);
  const long long blocks = static_cast<long long>(args.tiles) * (args.heads / G);
  if (blocks > 0x7fffffffLL) return static_cast<int>(cudaErrorInvalidValue);
  // Two key tiles at a time where the blocks are too few to hide a tile's trip to memory behind one another (a decode
  // step); with more, twice the blocks on an SM hide it better (four of 55 KB at 128 values and two heads).
  args.stages = sizeof(T) == 4 && args.vectors && blocks <= 296 && fixed + 2 * stage <= kTileSharedMost ? 2 : 1;
  const size_t shared = fixed + args.stages * stage;
  auto kernel = paged_attention_tile_kernel<T, G, VQ>;
  if (shared > 48 * 1024) {
    // The limit is the function's, not the launch's: always the most, so that another thread's launch still fits it.
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTileSharedMost));
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  kernel<<<static_cast<unsigned>(blocks), kTileThreads, shared, stream>>>(args);
  return static_cast<int>(cudaGetLastError());
}

// How many query heads share a block: as many as the key/value head has, up to what the registers hold (`most`) and to
// what fits shared memory (four heads of more than 532 values whose outputs have 65 to 128 do not; one always does), as
// long as two blocks an SM are left.
static int shared_heads(const TileArgs& args, int most, int VQ) {
  const int group = args.heads / args.kv_heads;
  for (int g = most; g > 1; g /= 2)
    if (group % g == 0 && static_cast<long long>(args.tiles) * (args.heads / g) >= 296 &&
        tile_fixed(args.head_dim, g) + tile_stage(args.head_dim, VQ) <= kTileSharedMost)
      return g;
  return 1;
}

template <typename T, int VQ>
static int launch_heads(const TileArgs& args, cudaStream_t stream) {
  if constexpr (VQ <= 4) {
    const int g = shared_heads(args, 4, VQ);
    if (g == 4) return launch_tile<T, 4, VQ>(args, stream);
    if (g == 2) return launch_tile<T, 2, VQ>(args, stream);
  } else if constexpr (VQ <= 8) {
    if (shared_heads(args, 2, VQ) == 2) return launch_tile<T, 2, VQ>(args, stream);
  }
  return launch_tile<T, 1, VQ>(args, stream);
}

template <typename T>
static int launch_values(TileArgs args, cudaStream_t stream) {
  args.vectors = args.head_dim % 4 == 0 && reinterpret_cast<uintptr_t>(args.cache) % (4 * sizeof(T)) == 0;
  if (args.value_dim <= 32) return launch_heads<T, 1>(args, stream);
  if (args.value_dim <= 64) return launch_heads<T, 2>(args, stream);
  if (args.value_dim <= 128) return launch_heads<T, 4>(args, stream);
  if (args.value_dim <= 256) return launch_heads<T, 8>(args, stream);
  return launch_heads<T, 18>(args, stream);
}

}  // namespace mxb

using namespace mxb;

// Query tiles are listed by the caller: tile i covers tokens tile_start[i] ..
// tile_start[i] + tile_length[i] - 1 (at most 16, consecutive positions of
// request row tile_request[i]).
MXB_API int mxb_paged_attention_tile(const void* q, const void* cache, void* out,
                                     const int* block_tables, int max_pages,
                                     const int* tile_request, const int* tile_start,
                                     const int* tile_length, const int* positions, int tiles,
                                     int heads, int kv_heads, int head_dim, int page_tokens,
                                     int num_pages, int window, int chunk, int keep, float scale, int dtype, const void* gate,
                                     long long gate_stride, int planes, int value_dim, float softcap,
                                     int gate_per_head, int has_sink, float sink_score, const float* sink_heads,
                                     const float* bias_table, int bias_far, int* status, cudaStream_t stream) {
  if (tiles <= 0) return 0;
  if (head_dim <= 0 || head_dim > 576 || heads % kv_heads != 0) return static_cast<int>(cudaErrorInvalidValue);
  if (bias_table != nullptr && bias_far < 0) return static_cast<int>(cudaErrorInvalidValue);
  const ScoreBias bias = {bias_table, bias_far};
  if ((planes != 1 && planes != 2) || value_dim <= 0 || value_dim > head_dim) return static_cast<int>(cudaErrorInvalidValue);
  const TileArgs args = {q, cache, out, block_tables, max_pages, tile_request, tile_start, tile_length, positions, tiles, heads,
                         kv_heads, head_dim, page_tokens, num_pages, window, chunk, keep, scale, gate, gate_stride, planes,
                         value_dim, softcap, gate_per_head, has_sink, sink_score, sink_heads, bias, 1, 0, status};
  if (dtype == kF32) return launch_values<float>(args, stream);
  if (dtype == kBF16) return launch_values<__nv_bfloat16>(args, stream);
  return static_cast<int>(cudaErrorInvalidValue);
}
