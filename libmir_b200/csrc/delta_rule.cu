// The gated delta rule: a recurrent mixer whose state per head is a matrix S [key channels, value channels].
//
// Per token, with q and k already unit vectors (q also times key_dim^-1/2), v the value row, beta in (0, 1) and a
// decay g in (0, 1) per head or per key channel:
//     S <- diag(g) S ;  u = beta (v - S^T k) ;  S <- S + k u^T ;  o = S^T q
// so the read-out sees the write of its own token.  The state is 32-bit, lives in the request's state slot and is
// carried from step to step; everything that enters the recurrence is computed in 32-bit here: the unit norms, the
// sigmoid of beta, softplus, both exponentials of the decay.
//
// Kernels of this file:
//   delta_rule_prepare the short convolution (short_conv.cu), then what else the recurrence needs of a token: q and k as unit vectors,
//                     sigmoid(beta), the decay; all tokens in parallel.
//   delta_rule_scan   the recurrence: a few lanes per (request, head, value channel) hold one column of S in
//                     registers, walk over the request's tokens of this step, and write the column back.  The state is
//                     stored [head][value channel][key channel], so a column is one contiguous run.
//   delta_rule_step   the same for a step of single tokens, with nothing staged.
//   delta_rule_group  and the walk over its groups: the recurrence four tokens a step, for prompts of the bfloat16 engine.
//   gated_head_norm   out = o / rms(o) * weight * act(gate) per (token, head), act = silu or sigmoid.
// A row of a captured decode batch whose position is negative is padding: nothing of it is read or written.
#include "common.cuh"
#include "scan_pairs.cuh"
#include "short_conv.cuh"

using namespace mir;

namespace {

constexpr int kMaxPerLane = 8;          // key channels per lane: key_dim <= 256

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

// Everything the recurrence needs of a token, in 32-bit, one CTA per token: the short convolution and silu of
// q | k | v (as short_conv_silu), q and k made unit vectors per key head (q also times key_dim^-1/2),
// beta = sigmoid(beta_raw), decay = exp(-exp(a_log) * softplus(decay_raw + dt_bias)).  A warp takes a key head at a
// time and keeps its channels in registers between the convolution and the norm; the rest is elementwise.
//   x          packed projection rows, convolved channel c of token t at x[t * ldx + c]; w [channels, taps]
//   beta_raw   (t, h) at beta_raw[t * ld_beta + h];  decay_raw (t, j) at decay_raw[t * ld_decay + j], j < decay_width
//   qkv        out [tokens, channels]; beta out [tokens, heads]; decay out [tokens, decay_width]
__device__ __forceinline__ float2 pair_of(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 pair_of(const __nv_bfloat16* p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}

// PAIRED: every thread works on two neighbouring channels (4- or 8-byte loads of the inputs); needs an even head
// width, an even number of value channels, an even row stride and a pointer aligned to two elements.
template <typename T, typename TD, bool PAIRED>
__global__ void delta_rule_prepare_kernel(const T* __restrict__ x, long long ldx, const T* __restrict__ w,
                                          float* __restrict__ tail, const T* __restrict__ beta_raw,
                                          long long ld_beta, const TD* __restrict__ decay_raw, long long ld_decay,
                                          const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                                          const int* __restrict__ row_of_token, const int* __restrict__ query_starts,
                                          const int* __restrict__ state_slots, const int* __restrict__ positions,
                                          float* __restrict__ qkv, float* __restrict__ beta, float* __restrict__ decay,
                                          int heads, int kv_heads, int key_dim, int value_dim, int decay_width,
                                          int taps) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int token = blockIdx.x;
  if (positions[token] < 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int row = row_of_token[token];
  const int start = query_starts[row];
  const int local = token - start;
  const int channels = 2 * kv_heads * key_dim + heads * value_dim;
  float* old = tail + (size_t)state_slots[row] * (taps - 1) * channels;
  float* out = qkv + (size_t)token * channels;
  // A request that brings one token moves its tail on right here: a channel's tail is read by the one thread that
  // convolves the channel, which then shifts it and appends the token's input (short_conv_tail skips such rows).
  const bool alone = query_starts[row + 1] - start == 1;
  auto convolved = [&](int c) {
    float acc = 0.0f;
    for (int j = 0; j < taps; ++j) {
      const int src = local - (taps - 1) + j;
      const float value = src >= 0 ? to_float(x[(size_t)(start + src) * ldx + c])
                                   : old[(size_t)(taps - 1 + src) * channels + c];
      acc = fmaf(to_float(w[(size_t)c * taps + j]), value, acc);
    }
    if (alone) {
      for (int j = 0; j + 2 < taps; ++j) old[(size_t)j * channels + c] = old[(size_t)(j + 1) * channels + c];
      if (taps > 1) old[(size_t)(taps - 2) * channels + c] = to_float(x[(size_t)token * ldx + c]);
    }
    return silu(acc);
  };
  // q heads, then k heads: unit vectors
  const float q_scale = rsqrtf((float)key_dim);
  // the CTAs of a token (gridDim.y of them, more where a step has few tokens) share its heads and channels out
  const int part = blockIdx.y, parts = gridDim.y;
  const int index = part * blockDim.x + threadIdx.x, stride = parts * blockDim.x;
  auto convolved_pair = [&](int c) {                           // channels c and c + 1, c even
    float first = 0.0f, second = 0.0f;
    for (int j = 0; j < taps; ++j) {
      const int src = local - (taps - 1) + j;
      const float2 value = src >= 0 ? pair_of(x + (size_t)(start + src) * ldx + c)
                                    : pair_of(old + (size_t)(taps - 1 + src) * channels + c);
      first = fmaf(to_float(w[(size_t)c * taps + j]), value.x, first);
      second = fmaf(to_float(w[(size_t)(c + 1) * taps + j]), value.y, second);
    }
    if (alone) {
      for (int j = 0; j + 2 < taps; ++j)
        *reinterpret_cast<float2*>(old + (size_t)j * channels + c) = pair_of(old + (size_t)(j + 1) * channels + c);
      if (taps > 1) *reinterpret_cast<float2*>(old + (size_t)(taps - 2) * channels + c) = pair_of(x + (size_t)token * ldx + c);
    }
    return make_float2(silu(first), silu(second));
  };
  for (int unit = part * warps + warp; unit < 2 * kv_heads; unit += parts * warps) {
    float values[kMaxPerLane];
    float square = 0.0f;
    if (PAIRED) {
#pragma unroll
      for (int m = 0; m < kMaxPerLane; m += 2) {
        const int i = 2 * lane + 32 * m;
        const float2 both = i < key_dim ? convolved_pair(unit * key_dim + i) : make_float2(0.0f, 0.0f);
        values[m] = both.x;
        values[m + 1] = both.y;
        square = fmaf(both.x, both.x, fmaf(both.y, both.y, square));
      }
    } else {
#pragma unroll
      for (int m = 0; m < kMaxPerLane; ++m) {
        const int i = lane + 32 * m;
        values[m] = i < key_dim ? convolved(unit * key_dim + i) : 0.0f;
        square = fmaf(values[m], values[m], square);
      }
    }
    const float unit_scale = rsqrtf(warp_sum(square) + 1e-6f) * (unit < kv_heads ? q_scale : 1.0f);
    if (PAIRED) {
#pragma unroll
      for (int m = 0; m < kMaxPerLane; m += 2) {
        const int i = 2 * lane + 32 * m;
        if (i < key_dim)
          *reinterpret_cast<float2*>(out + unit * key_dim + i) = make_float2(values[m] * unit_scale, values[m + 1] * unit_scale);
      }
    } else {
#pragma unroll
      for (int m = 0; m < kMaxPerLane; ++m) {
        const int i = lane + 32 * m;
        if (i < key_dim) out[unit * key_dim + i] = values[m] * unit_scale;
      }
    }
  }
  if (PAIRED) {
    for (int c = 2 * kv_heads * key_dim + 2 * index; c < channels; c += 2 * stride)
      *reinterpret_cast<float2*>(out + c) = convolved_pair(c);
  } else {
    for (int c = 2 * kv_heads * key_dim + index; c < channels; c += stride) out[c] = convolved(c);
  }
  for (int h = index; h < heads; h += stride)
    beta[(size_t)token * heads + h] = sigmoid(to_float(beta_raw[(size_t)token * ld_beta + h]));
  const int per_head = decay_width / heads;
  for (int j = index; j < decay_width; j += stride)
    decay[(size_t)token * decay_width + j] =
        expf(-expf(a_log[j / per_head]) * softplus(to_float(decay_raw[(size_t)token * ld_decay + j]) + dt_bias[j]));
}

// The same for up to four taps and key heads of up to 128 channels in multiples of four (value channels likewise): a warp takes
// 128 neighbouring channels (a key head, or value channels, or decays, four channels a lane) and a run of RUN tokens.  The
// taps' weights and the decays' constants are read once for the run, an input once for all taps, and all inputs of the run
// are on their way before the first is used.  Bound by latency: 2,274 tokens of 4,096 channels 38 us (one token a CTA with every
// tap read anew: 58), 2 tokens of 6,144 channels and 2,048 decays 4.8 us (8.8).
__device__ __forceinline__ float4 quad_of(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 quad_of(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
template <typename T> struct Quad;
template <> struct Quad<float> { using Raw = uint4; };
template <> struct Quad<__nv_bfloat16> { using Raw = uint2; };

constexpr int kRunWarps = 4, kRunTaps = 4;
template <typename T, typename TD, int RUN>
__global__ void __launch_bounds__(kRunWarps * 32)
delta_rule_prepare_run_kernel(const T* __restrict__ x, long long ldx, const T* __restrict__ w, float* __restrict__ tail,
                              const T* __restrict__ beta_raw, long long ld_beta, const TD* __restrict__ decay_raw,
                              long long ld_decay, const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                              const int* __restrict__ row_of_token, const int* __restrict__ query_starts,
                              const int* __restrict__ state_slots, const int* __restrict__ positions,
                              float* __restrict__ qkv, float* __restrict__ beta, float* __restrict__ decay, int tokens,
                              int heads, int kv_heads, int key_dim, int value_dim, int decay_width, int taps) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x;
  const int first = blockIdx.x * RUN, last = min(first + RUN, tokens);
  const int keys = 2 * kv_heads, values = heads * value_dim;
  const int value_units = (values + 127) / 128, decay_units = (decay_width + 127) / 128;
  const int channels = keys * key_dim + values;
  int unit = blockIdx.y * kRunWarps + threadIdx.y;
  if (unit >= keys + value_units) {
    unit -= keys + value_units;
    if (unit < decay_units) {                                    // decays
      const int per_head = decay_width / heads;
      float rate[4], bias[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = unit * 128 + lane + 32 * e;
        rate[e] = j < decay_width ? -expf(a_log[j / per_head]) : 0.0f;
        bias[e] = j < decay_width ? dt_bias[j] : 0.0f;
      }
      const int my_position = positions[min(first + lane, last - 1)];
      constexpr int AHEAD = RUN < 4 ? RUN : 4;                   // tokens whose inputs are asked for together
#pragma unroll
      for (int i = 0; i < RUN; i += AHEAD) {
        float raw[AHEAD][4];
#pragma unroll
        for (int a = 0; a < AHEAD; ++a)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int j = unit * 128 + lane + 32 * e;
            raw[a][e] = first + i + a < last && j < decay_width ? to_float(decay_raw[(size_t)(first + i + a) * ld_decay + j]) : 0.0f;
          }
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) {
          const int t = first + i + a;
          if (__shfl_sync(0xffffffffu, my_position, i + a) < 0 || t >= last) continue;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int j = unit * 128 + lane + 32 * e;
            if (j < decay_width) decay[(size_t)t * decay_width + j] = expf(rate[e] * softplus(raw[a][e] + bias[e]));
          }
        }
      }
    } else if (unit == decay_units) {                            // the writes' factors
      for (int t = first; t < last; ++t) {
        if (positions[t] < 0) continue;
        for (int h = lane; h < heads; h += 32) beta[(size_t)t * heads + h] = sigmoid(to_float(beta_raw[(size_t)t * ld_beta + h]));
      }
    }
    return;
  }
  const bool key_head = unit < keys;
  const int base = key_head ? unit * key_dim : keys * key_dim + (unit - keys) * 128;
  const int count = key_head ? key_dim : min(128, values - (unit - keys) * 128);
  const bool active = lane * 4 < count;
  const int c = base + (active ? lane * 4 : 0);
  // the run's inputs, and which request each token belongs to
  using Raw = typename Quad<T>::Raw;
  Raw inputs[RUN];
#pragma unroll
  for (int i = 0; i < RUN; ++i)
    if (first + i < last) inputs[i] = *reinterpret_cast<const Raw*>(x + (size_t)(first + i) * ldx + c);
  const int mine = min(first + lane, last - 1);
  const int my_row = row_of_token[mine];
  const int my_start = query_starts[my_row], my_end = query_starts[my_row + 1], my_position = positions[mine];
  float taps_of[4][kRunTaps];                                    // [channel][tap], right-aligned: the last is the token's own
  if (taps == kRunTaps && (uintptr_t)w % (kRunTaps * sizeof(T)) == 0) {      // a channel's taps in one load (2,274 tokens, below: 75 to 70 us)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 own = quad_of(w + (size_t)(c + i) * kRunTaps);
      taps_of[i][0] = own.x; taps_of[i][1] = own.y; taps_of[i][2] = own.z; taps_of[i][3] = own.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < kRunTaps; ++j) {
        const int tap = j - (kRunTaps - taps);
        taps_of[i][j] = tap >= 0 ? to_float(w[(size_t)(c + i) * taps + tap]) : 0.0f;
      }
  }
  const float q_scale = rsqrtf((float)key_dim);
  float4 before[kRunTaps - 1] = {};                              // the inputs before the token, right-aligned
  int row = -1;
#pragma unroll
  for (int i = 0; i < RUN; ++i) {
    const int t = first + i;
    if (t >= last) break;
    const int here = __shfl_sync(0xffffffffu, my_row, i), start = __shfl_sync(0xffffffffu, my_start, i);
    const int end = __shfl_sync(0xffffffffu, my_end, i), position = __shfl_sync(0xffffffffu, my_position, i);
    if (position < 0) { row = -1; continue; }                    // padding
    if (here != row) {                                           // the run's first token of a request
      row = here;
      const float* old = tail + (size_t)state_slots[row] * (taps - 1) * channels;
#pragma unroll
      for (int j = 0; j < kRunTaps - 1; ++j) {
        const int tap = j - (kRunTaps - taps);                   // of the tail's taps - 1 inputs
        if (tap < 0) continue;
        const int src = t - start - (taps - 1) + tap;
        before[j] = src >= 0 ? quad_of(x + (size_t)(start + src) * ldx + c) : quad_of(old + (size_t)(taps - 1 + src) * channels + c);
      }
    }
    const float4 now = quad_of(reinterpret_cast<const T*>(&inputs[i]));
    float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < kRunTaps; ++j) {
      if (j < kRunTaps - taps) continue;
      const float4 in = j < kRunTaps - 1 ? before[j < kRunTaps - 1 ? j : 0] : now;
      y.x = fmaf(taps_of[0][j], in.x, y.x); y.y = fmaf(taps_of[1][j], in.y, y.y);
      y.z = fmaf(taps_of[2][j], in.z, y.z); y.w = fmaf(taps_of[3][j], in.w, y.w);
    }
    if (end - start == 1 && active) {                            // a request that brings one token: its tail moves on
      float* old = tail + (size_t)state_slots[row] * (taps - 1) * channels;
#pragma unroll
      for (int j = 0; j < kRunTaps - 1; ++j) {
        const int tap = j - (kRunTaps - taps);
        if (tap >= 0) *reinterpret_cast<float4*>(old + (size_t)tap * channels + c) = j + 1 < kRunTaps - 1 ? before[j + 1 < kRunTaps - 1 ? j + 1 : 0] : now;
      }
    }
    before[0] = before[1]; before[1] = before[2]; before[2] = now;
    y = make_float4(silu(y.x), silu(y.y), silu(y.z), silu(y.w));
    if (key_head) {                                              // a unit vector, the query's scaled
      const float square = active ? fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, y.w * y.w))) : 0.0f;
      const float factor = rsqrtf(warp_sum(square) + 1e-6f) * (unit < kv_heads ? q_scale : 1.0f);
      y.x *= factor; y.y *= factor; y.z *= factor; y.w *= factor;
    }
    if (active) *reinterpret_cast<float4*>(qkv + (size_t)t * channels + c) = y;
  }
}

constexpr int kScanWarps = 4;           // that walk
constexpr int kFetchWarps = 4;          // that copy what the others will need
constexpr int kScanThreads = (kScanWarps + kFetchWarps) * 32;
constexpr int kScanChunk = 16;          // tokens whose inputs one stage of shared memory holds
constexpr int kScanStages = 3;
constexpr int kScanLanes = 16, kScanColumns = 2;   // lanes that share a column of the state, columns a lane holds

// The recurrence.  LANES = 16 lanes share C = 2 columns of S (C value channels of one head): lane l holds the key channels
// 4 (m LANES + l) .. + 3 for m < PER / 4 in registers, so a warp works on 32 / LANES * C columns at once, the two dot
// products per token are log2(LANES) shuffle steps, and the state of a column (stored [head][value channel][key
// channel]) is read and written in 16-byte pieces that lie side by side across the lanes.  The inputs of a token are
// the same for every column of its head: the CTA (all its warps work on columns of one head) has kFetchWarps more that copy
// them for 16 tokens at a time into shared memory with cp.async, three stages.  blockDim (32, kScanWarps + kFetchWarps), grid
// (rows, heads, ceil(value_dim / (kScanWarps * 32 / LANES * C))).
//
// What bounds it: the chain from one token's state to the next (a decay, a dot product of PER channels, the sum over the
// lanes, the write's factor and a multiply-add) on the one walking warp a scheduler has, which can hide little of it.  So what can be kept away from that warp is: the copies and their addresses belong to the
// fetching warps, a token's inputs are in registers before the token before it ends, the read-out is summed over the
// lanes beside the next token's S^T k, a lane has C columns that share a token's inputs, and the arithmetic goes two
// numbers an instruction.  Every number is formed by the same operations in the same order
// whatever the step's shape, so a request's 32-bit results do not depend on how it was cut.
// Sixteen lanes with two columns each read a token's inputs half as often as eight lanes with one: a prompt of 2,048 tokens at
// 16 / 32 heads of 128 x 128 takes 375 / 520 us with a decay per channel (eight lanes: 476 / 707, thirty-two with four columns:
// 413 / 570; before the fetching warps: 630 / 870) and 345 / 465 with one per head.  One choice for every shape of step, so
// that a request's 32-bit results do not depend on how it was cut.
//   qkv    [tokens, 2 G D + H V] 32-bit: unit q | unit k | v (delta_rule_prepare)
//   beta   [tokens, H]; decay [tokens, H D] (PER_CHANNEL) or [tokens, H]
//   state  [slots, H, V, D] 32-bit;  out [tokens, H V] 32-bit: o before the head norm
template <int PER, bool PER_CHANNEL>
__global__ void __launch_bounds__(kScanThreads, 2)
delta_rule_scan_kernel(const float* __restrict__ qkv, const float* __restrict__ beta, const float* __restrict__ decay,
                       float* __restrict__ state, const int* __restrict__ query_starts,
                       const int* __restrict__ state_slots, const int* __restrict__ positions,
                       float* __restrict__ out, int heads, int kv_heads, int key_dim, int value_dim) {
  static_assert(PER % 4 == 0, "a lane holds whole 16-byte pieces");
  constexpr int LANES = kScanLanes, C = kScanColumns;
  extern __shared__ __align__(16) float staged[];              // [kScanStages][kScanChunk tokens][row]
  grid_dependency_wait();
  grid_launch_dependents();
  constexpr int COLUMNS = 32 / LANES * C;                       // per warp
  constexpr int BLOCK_COLUMNS = COLUMNS * kScanWarps;
  constexpr int PADDED = LANES * PER;                           // key channels with padding
  constexpr int DECAYS = PER_CHANNEL ? PADDED : 4;
  constexpr int VALUES = 2 * PADDED + DECAYS + 4;               // where a row's values begin
  constexpr int ROW = VALUES + BLOCK_COLUMNS;                   // q | k | decay | beta | v of this CTA's columns
  constexpr int STAGE = kScanChunk * ROW;
  const int lane = threadIdx.x;
  const int row = blockIdx.x, head = blockIdx.y;
  const int first_column = blockIdx.z * BLOCK_COLUMNS;
  const int start = query_starts[row], end = query_starts[row + 1];
  if (end <= start || positions[start] < 0) return;             // the whole CTA: an empty or padding row
  const int width = 2 * kv_heads * key_dim + heads * value_dim;
  // 16-byte accesses: every piece lies wholly inside or outside the head, and every row starts on a 16-byte boundary
  const bool wide = (key_dim % 4 == 0) && (width % 4 == 0);
  // padding channels (key_dim < PADDED) are read as q = k = 0: zero them once in all stages
  if (key_dim < PADDED) {
    for (int index = threadIdx.y * 32 + lane; index < kScanStages * STAGE; index += kScanThreads) staged[index] = 0.0f;
    __syncthreads();
  }
  const int chunks = (end - start + kScanChunk - 1) / kScanChunk;

  if (threadIdx.y >= kScanWarps) {                              // the fetching warps: tokens w, w + kFetchWarps, ... of a chunk
    const int kv_head = head / (heads / kv_heads), mine = threadIdx.y - kScanWarps;
    const int g_width = PER_CHANNEL ? heads * key_dim : heads;
    const bool wide_values = wide && value_dim % 4 == 0;
    const int step = wide ? 4 : 1, value_step = wide_values ? 4 : 1;
    const size_t key_at = (size_t)kv_heads * key_dim;
    const float* q0 = qkv + (size_t)kv_head * key_dim;
    const float* v0 = qkv + 2 * key_at + (size_t)head * value_dim + first_column;
    const float* b0 = beta + head;
    const float* g0 = decay + (size_t)head * (PER_CHANNEL ? key_dim : 1);
    const bool my_value = lane * value_step < BLOCK_COLUMNS && first_column + lane * value_step < value_dim;
    auto fetch = [&](int chunk) {
      const int from = start + chunk * kScanChunk;
#pragma unroll
      for (int tt = 0; tt < kScanChunk / kFetchWarps; ++tt) {
        const int t = mine + tt * kFetchWarps;
        const size_t token = from + t;
        if (from + t >= end) break;
        float* to = staged + (chunk % kScanStages) * STAGE + t * ROW;
        const float* q = q0 + token * width;
        const float* g = g0 + token * g_width;
        if (wide) {
          for (int i = lane * 4; i < key_dim; i += 128) {
            copy_async(to + i, q + i, true);
            copy_async(to + PADDED + i, q + key_at + i, true);
            if (PER_CHANNEL) copy_async(to + 2 * PADDED + i, g + i, true);
          }
        } else {
          for (int i = lane * step; i < key_dim; i += 32 * step) {
            copy_async(to + i, q + i, false);
            copy_async(to + PADDED + i, q + key_at + i, false);
            if (PER_CHANNEL) copy_async(to + 2 * PADDED + i, g + i, false);
          }
        }
        if (my_value) copy_async(to + VALUES + lane * value_step, v0 + token * width + lane * value_step, wide_values);
        // one copy of 4 bytes by two lanes: the write's factor, and (with a decay a head) the decay
        if (lane >= (PER_CHANNEL ? 31 : 30))
          copy_async(to + 2 * PADDED + (lane == 31 ? DECAYS : 0), lane == 31 ? b0 + token * heads : g, false);
      }
      copy_commit();
    };
    fetch(0);
    if (chunks > 1) fetch(1); else copy_commit();
    copy_wait<1>();
    __syncthreads();                                             // the first chunk is there
    for (int chunk = 0; chunk < chunks; ++chunk) {               // (into the stage of the chunk that was walked last)
      if (chunk + 2 < chunks) fetch(chunk + 2); else copy_commit();
      copy_wait<1>();
      __syncthreads();                                           // this chunk has been walked, and the next one is there
    }
    copy_wait<0>();
    return;
  }

  const int l = lane % LANES;
  const int local_column = threadIdx.y * COLUMNS + lane / LANES * C;
  const int column = first_column + local_column;                // idle lanes (beyond value_dim) still take part in the shuffles
  float* column_state = state + (((size_t)state_slots[row] * heads + head) * value_dim + column) * key_dim;
  Pair s[C][PER / 2];
#pragma unroll
  for (int c = 0; c < C; ++c)
    load_column<LANES, PER>(s[c], column_state + (size_t)c * key_dim, l, key_dim, column + c < value_dim, wide);

  struct Inputs {
    Pair q[PER / 2], k[PER / 2], g[PER_CHANNEL ? PER / 2 : 1];
    float beta, value[C];
  };
  auto load = [&](Inputs& in, const float* from) {
#pragma unroll
    for (int m = 0; m < PER; m += 4) {
      const int i = (m / 4 * LANES + l) * 4;
      const ulonglong2 key = *reinterpret_cast<const ulonglong2*>(from + PADDED + i);
      in.k[m / 2] = key.x; in.k[m / 2 + 1] = key.y;
      if (PER_CHANNEL) {
        const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(from + 2 * PADDED + i);
        in.g[m / 2] = g.x; in.g[m / 2 + 1] = g.y;
      }
      const ulonglong2 query = *reinterpret_cast<const ulonglong2*>(from + i);
      in.q[m / 2] = query.x; in.q[m / 2 + 1] = query.y;
    }
    if (!PER_CHANNEL) in.g[0] = pair_from(from[2 * PADDED], from[2 * PADDED]);
    in.beta = from[2 * PADDED + DECAYS];
#pragma unroll
    for (int c = 0; c < C; ++c) in.value[c] = from[VALUES + local_column + c];
  };
  float pending[C];                                              // the last token's read-outs, not yet summed over the lanes
#pragma unroll
  for (int c = 0; c < C; ++c) pending[c] = 0.0f;
  const int my_column = lane_sum<C>(l);                          // of the C columns, the one whose read-out this lane writes
  const bool writer = l < C && column + my_column < value_dim;
  const size_t out_step = (size_t)heads * value_dim;
  float* out_at = out + ((size_t)start * heads + head) * value_dim + column + my_column;
  bool has_pending = false;
  auto walk = [&](const Inputs& in) {
    float total[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      Pair seen[2] = {0, 0};
#pragma unroll
      for (int m = 0; m < PER / 2; ++m) {
        s[c][m] = pair_mul(s[c][m], in.g[PER_CHANNEL ? m : 0]);
        seen[m & 1] = pair_fma(s[c][m], in.k[m], seen[m & 1]);
      }
      total[c] = pair_total(seen);
    }
#pragma unroll
    for (int step = 1; step < LANES; step <<= 1)
#pragma unroll
      for (int c = 0; c < C; ++c) total[c] += __shfl_xor_sync(0xffffffffu, total[c], step);
    const float read_out = sum_lanes<LANES, C>(pending, l);
    if (has_pending) {
      if (writer) *out_at = read_out;
      out_at += out_step;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float update = in.beta * (in.value[c] - total[c]);
      const Pair both = pair_from(update, update);
      Pair read[2] = {0, 0};
#pragma unroll
      for (int m = 0; m < PER / 2; ++m) {
        s[c][m] = pair_fma(in.k[m], both, s[c][m]);
        read[m & 1] = pair_fma(s[c][m], in.q[m], read[m & 1]);
      }
      pending[c] = pair_total(read);
    }
    has_pending = true;
  };
  __syncthreads();                                               // the first chunk is there
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int count = min(kScanChunk, end - start - chunk * kScanChunk);
    const float* in = staged + (chunk % kScanStages) * STAGE;
    Inputs even, odd;
    load(even, in);
    int t = 0;
    for (; t + 2 <= count; t += 2, in += 2 * ROW) {
      load(odd, in + ROW);
      walk(even);
      if (t + 2 < count) load(even, in + 2 * ROW);
      walk(odd);
    }
    if (t < count) walk(even);
    __syncthreads();                                             // this chunk has been walked, and the next one is there
  }
  const float read_out = sum_lanes<LANES, C>(pending, l);        // the last token's
  if (writer) *out_at = read_out;
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (column + c < value_dim) store_column<LANES, PER>(s[c], column_state + (size_t)c * key_dim, l, key_dim, wide);
}

// A step of single tokens: the same operations on every number in the same order as delta_rule_scan_kernel (sixteen lanes a
// column; C columns a lane, whose number changes no result), but a token's inputs go from global memory to registers and
// nothing is staged: a step reads and writes the state once and has no next token to fetch for.  WIDE (16-byte accesses, as
// `wide` above) is known to the compiler, so that all loads are on their way before the first number is used: with a branch for
// it between them one row of 16 heads of 128 took 3.4 us.
// What bounds it: the bytes of the state.  64 rows of 32 heads of 128 x 128 61 us with a decay per channel (the walk's kernel 108), 49 with
// one a head (105), 268 MB either way; eight rows of 16 heads 4.9 us (7.6), two rows 3.6 (3.3).
// blockDim (32, kScanWarps), grid (rows, heads, ceil(value_dim / (kScanWarps * 2 C))).
template <int PER, int C, bool PER_CHANNEL, bool WIDE>
__global__ void __launch_bounds__(kScanWarps * 32)
delta_rule_step_kernel(const float* __restrict__ qkv, const float* __restrict__ beta, const float* __restrict__ decay,
                       float* __restrict__ state, const int* __restrict__ query_starts, const int* __restrict__ state_slots,
                       const int* __restrict__ positions, float* __restrict__ out, int heads, int kv_heads, int key_dim,
                       int value_dim) {
  constexpr int LANES = 16, COLUMNS = 32 / LANES * C;            // of a warp
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x, l = lane % LANES;
  const int row = blockIdx.x, head = blockIdx.y;
  const int start = query_starts[row], end = query_starts[row + 1], slot = state_slots[row];
  if (end <= start || positions[start] < 0) return;             // the whole CTA: an empty or padding row
  const int column = blockIdx.z * (COLUMNS * kScanWarps) + threadIdx.y * COLUMNS + lane / LANES * C;
  const int width = 2 * kv_heads * key_dim + heads * value_dim, kv_head = head / (heads / kv_heads);
  float* column_state = state + (((size_t)slot * heads + head) * value_dim + column) * key_dim;
  Pair s[C][PER / 2];
#pragma unroll
  for (int c = 0; c < C; ++c)
    load_column<LANES, PER>(s[c], column_state + (size_t)c * key_dim, l, key_dim, column + c < value_dim, WIDE);
  const int my_column = lane_sum<C>(l);                          // of the C columns, the one whose read-out this lane writes
  for (int at = start; at < end; ++at) {                         // (one token, but for steps whose other rows are empty)
    const float* from = qkv + (size_t)at * width + (size_t)kv_head * key_dim;
    const float* value_of = qkv + (size_t)at * width + (size_t)2 * kv_heads * key_dim + (size_t)head * value_dim;
    const float* g_of = decay + ((size_t)at * heads + head) * (PER_CHANNEL ? key_dim : 1);
    Pair q[PER / 2], k[PER / 2], g[PER_CHANNEL ? PER / 2 : 1];
    load_column<LANES, PER>(k, from + (size_t)kv_heads * key_dim, l, key_dim, true, WIDE);
    if constexpr (PER_CHANNEL) load_column<LANES, PER>(g, g_of, l, key_dim, true, WIDE);
    else g[0] = pair_from(*g_of, *g_of);
    load_column<LANES, PER>(q, from, l, key_dim, true, WIDE);
    const float factor = beta[(size_t)at * heads + head];
    float value[C], total[C], parts[C];
#pragma unroll
    for (int c = 0; c < C; ++c) value[c] = column + c < value_dim ? value_of[column + c] : 0.0f;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      Pair seen[2] = {0, 0};
#pragma unroll
      for (int m = 0; m < PER / 2; ++m) {
        s[c][m] = pair_mul(s[c][m], g[PER_CHANNEL ? m : 0]);
        seen[m & 1] = pair_fma(s[c][m], k[m], seen[m & 1]);
      }
      total[c] = pair_total(seen);
    }
#pragma unroll
    for (int step = 1; step < LANES; step <<= 1)
#pragma unroll
      for (int c = 0; c < C; ++c) total[c] += __shfl_xor_sync(0xffffffffu, total[c], step);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float update = factor * (value[c] - total[c]);
      const Pair both = pair_from(update, update);
      Pair read[2] = {0, 0};
#pragma unroll
      for (int m = 0; m < PER / 2; ++m) {
        s[c][m] = pair_fma(k[m], both, s[c][m]);
        read[m & 1] = pair_fma(s[c][m], q[m], read[m & 1]);
      }
      parts[c] = pair_total(read);
    }
    const float read_out = sum_lanes<LANES, C>(parts, l);
    if (l < C && column + my_column < value_dim) out[((size_t)at * heads + head) * value_dim + column + my_column] = read_out;
  }
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (column + c < value_dim) store_column<LANES, PER>(s[c], column_state + (size_t)c * key_dim, l, key_dim, WIDE);
}

// The recurrence four tokens at a time, for prompts whose results may be grouped by where the step begins (the bfloat16 engine;
// the 32-bit engine's results must not depend on the cut and run the kernel above).  With S the state before a group,
// G_t the product of the decays up to token t of it, G_ts the product of those behind token s up to t:
//     P_t = S^T (G_t k_t),  R_t = S^T (G_t q_t)                            eight dot products that need only S
//     u_t = beta_t (v_t - P_t - sum_{s<t} (k_t . G_ts k_s) u_s)            four short sums
//     o_t = R_t + sum_{s<=t} (q_t . G_ts k_s) u_s;   S <- G_4 S + sum_t (G_4t k_t) u_t^T
// Every factor is a product of decays, at most one: nothing is divided, nothing can overflow.  The vectors and the scalars
// do not depend on the column: delta_rule_group forms them once for a head, one warp a (group, head).
//   grouped [group, head, 13 PADDED + 28]: G_t k_t (4), G_t q_t (4), G_4t k_t (4), G_4 | the k products [1][0], [2][0..1],
//   [3][0..2] and two zeros | beta (4) | the q products [4][4], zero above the diagonal.  A request's groups begin at
//   start / 4 + its number; tokens a last group lacks have no key, no query, no decay (1) and no write.
constexpr int kGroup = 4, kGroupScalars = 28;
__host__ __device__ constexpr int group_floats(int padded) { return 13 * padded + kGroupScalars; }

template <int PADDED, bool PER_CHANNEL>
__global__ void __launch_bounds__(128)
delta_rule_group_kernel(const float* __restrict__ qkv, const float* __restrict__ beta, const float* __restrict__ decay,
                        const int* __restrict__ query_starts, const int* __restrict__ positions, float* __restrict__ grouped,
                        int rows, int heads, int kv_heads, int key_dim, int value_dim) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x, group = blockIdx.x, head = blockIdx.y * 4 + threadIdx.y;
  if (head >= heads) return;
  int start = -1, end = 0, begin = 0;
  for (int base = 0; base < rows && start < 0; base += 32) {     // whose group it is
    const int r = base + lane;
    const int a = r < rows ? query_starts[r] : 0, b = r < rows ? query_starts[r + 1] : 0, first = a / kGroup + r;
    const unsigned found = __ballot_sync(0xffffffffu, r < rows && group >= first && group < first + (b - a + kGroup - 1) / kGroup);
    if (found == 0) continue;
    const int source = __ffs(found) - 1;
    start = __shfl_sync(0xffffffffu, a, source);
    end = __shfl_sync(0xffffffffu, b, source);
    begin = start + (group - __shfl_sync(0xffffffffu, first, source)) * kGroup;
  }
  if (start < 0 || positions[start] < 0) return;
  const int kv_head = head / (heads / kv_heads);
  const int width = 2 * kv_heads * key_dim + heads * value_dim;
  const int g_width = PER_CHANNEL ? heads * key_dim : heads;
  const bool wide = key_dim % 4 == 0 && width % 4 == 0;
  auto read = [&](const float* from, int i) {                    // channels i .. i + 3 of a head, zeros beyond it
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (wide) {
      if (i < key_dim) v = *reinterpret_cast<const float4*>(from + i);
    } else {
      if (i < key_dim) v.x = from[i];
      if (i + 1 < key_dim) v.y = from[i + 1];
      if (i + 2 < key_dim) v.z = from[i + 2];
      if (i + 3 < key_dim) v.w = from[i + 3];
    }
    return v;
  };
  auto times = [](float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); };
  auto dot = [](float4 a, float4 b, float sum) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, sum)))); };
  float* to = grouped + ((size_t)group * heads + head) * group_floats(PADDED);
  float sums[16];                                                // k products (6), q products (10)
#pragma unroll
  for (int i = 0; i < 16; ++i) sums[i] = 0.0f;
#pragma unroll
  for (int piece = 0; piece < (PADDED + 127) / 128; ++piece) {
    const int i = piece * 128 + lane * 4;
    if (i >= PADDED) continue;                                   // (no shuffles inside)
    float4 k[kGroup], q[kGroup], g[kGroup];
#pragma unroll
    for (int t = 0; t < kGroup; ++t) {
      k[t] = q[t] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      g[t] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
      if (begin + t >= end) continue;
      const float* row = qkv + (size_t)(begin + t) * width + (size_t)kv_head * key_dim;
      q[t] = read(row, i);
      k[t] = read(row + (size_t)kv_heads * key_dim, i);
      const float* d = decay + (size_t)(begin + t) * g_width + (size_t)head * (PER_CHANNEL ? key_dim : 1);
      if (PER_CHANNEL) {
        if (g_width % 4 == 0 && key_dim % 4 == 0) g[t] = i < key_dim ? *reinterpret_cast<const float4*>(d + i) : g[t];
        else g[t] = read(d, i);
      } else {
        g[t] = make_float4(d[0], d[0], d[0], d[0]);
      }
    }
    float4 so_far = g[0];
#pragma unroll
    for (int t = 0; t < kGroup; ++t) {
      if (t > 0) so_far = times(so_far, g[t]);
      *reinterpret_cast<float4*>(to + t * PADDED + i) = times(k[t], so_far);
      *reinterpret_cast<float4*>(to + (kGroup + t) * PADDED + i) = times(q[t], so_far);
    }
    *reinterpret_cast<float4*>(to + 3 * kGroup * PADDED + i) = so_far;
#pragma unroll
    for (int s = 0; s < kGroup; ++s) {
      float4 reach = k[s];                                       // key s as token t sees it
      sums[6 + s * (s + 1) / 2 + s] = dot(q[s], reach, sums[6 + s * (s + 1) / 2 + s]);
#pragma unroll
      for (int t = s + 1; t < kGroup; ++t) {
        reach = times(reach, g[t]);
        sums[t * (t - 1) / 2 + s] = dot(k[t], reach, sums[t * (t - 1) / 2 + s]);
        sums[6 + t * (t + 1) / 2 + s] = dot(q[t], reach, sums[6 + t * (t + 1) / 2 + s]);
      }
      *reinterpret_cast<float4*>(to + (2 * kGroup + s) * PADDED + i) = reach;
    }
  }
  const float total = sum_lanes<32, 16>(sums, lane);
  float* scalars = to + 13 * PADDED;
  if (lane < 16) {
    const int number = lane_sum<16>(lane);
    if (number < 6) {
      scalars[number] = total;
    } else {
      int t = 0;
      while ((t + 1) * (t + 2) / 2 <= number - 6) ++t;
      scalars[12 + t * 4 + (number - 6 - t * (t + 1) / 2)] = total;
    }
  } else if (lane < 24) {                                        // what is never reached
    const int above[8] = {6, 7, 13, 14, 15, 18, 19, 23};
    scalars[above[lane - 16]] = 0.0f;
  } else if (lane < 28) {
    const int t = begin + lane - 24;
    scalars[8 + lane - 24] = t < end ? beta[(size_t)t * heads + head] : 0.0f;
  }
}

// The walk over groups: lanes, columns, roles and stages as in delta_rule_scan_kernel, LANES = 16.  A group costs its chain one
// sum over the lanes (4 C sums together, each in a lane of its own), one exchange and the four short sums, where four
// tokens one after the other cost four of each.
// What bounds it: one walking warp a scheduler, which issues in 0.38 (C = 2) and 0.49 (C = 4) of the cycles and otherwise waits
// on shared memory, shuffles and the latency of the operation before; shared memory's data path is 0.60 and 0.49 busy: a lane
// reads PER numbers of thirteen vectors a group whatever the columns it has, so C columns a lane cost 52 / C cycles a column.
// 2,048 tokens with the group kernel, decay per channel / head: 16 heads 268 / 266 us (a token at a time 377 / 345), 32 heads
// 392 / 388 (521 / 466); 1,400 and 874 tokens, 16 heads 267 / 264 (360 / 321), 32 heads 448 / 442 (598 / 537).
template <int PER, int C>
__global__ void __launch_bounds__(kScanThreads, 2)
delta_rule_grouped_scan_kernel(const float* __restrict__ grouped, const float* __restrict__ qkv, float* __restrict__ state,
                               const int* __restrict__ query_starts, const int* __restrict__ state_slots,
                               const int* __restrict__ positions, float* __restrict__ out, int heads, int kv_heads,
                               int key_dim, int value_dim) {
  constexpr int LANES = 16, PADDED = LANES * PER, SUMS = kGroup * C;
  constexpr int COLUMNS = 32 / LANES * C, BLOCK_COLUMNS = COLUMNS * kScanWarps;
  constexpr int GROUPED = group_floats(PADDED), ROW = GROUPED + kGroup * BLOCK_COLUMNS, CHUNK = kFetchWarps;   // groups of a stage
  constexpr int STAGE = CHUNK * ROW;
  constexpr int STAGES = 3;
  extern __shared__ __align__(16) float staged[];                // [STAGES][CHUNK groups][row]
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x;
  const int row = blockIdx.x, head = blockIdx.y;
  const int first_column = blockIdx.z * BLOCK_COLUMNS;
  const int start = query_starts[row], end = query_starts[row + 1];
  if (end <= start || positions[start] < 0) return;             // the whole CTA: an empty or padding row
  const int width = 2 * kv_heads * key_dim + heads * value_dim;
  const int groups = (end - start + kGroup - 1) / kGroup, first_group = start / kGroup + row;
  const int chunks = (groups + CHUNK - 1) / CHUNK;

  if (threadIdx.y >= kScanWarps) {                              // the fetching warps: a group of the stage each
    const int mine = threadIdx.y - kScanWarps;
    const float* v0 = qkv + (size_t)2 * kv_heads * key_dim + (size_t)head * value_dim + first_column;
    const bool wide = width % 4 == 0 && key_dim % 4 == 0 && value_dim % 4 == 0;
    auto fetch = [&](int chunk) {
      const int group = chunk * CHUNK + mine;
      if (group < groups) {
        float* to = staged + (chunk % STAGES) * STAGE + mine * ROW;
        const float* from = grouped + ((size_t)(first_group + group) * heads + head) * GROUPED;
#pragma unroll
        for (int i = 0; i < GROUPED; i += 128)
          if (GROUPED - i >= 128 || i + lane * 4 < GROUPED) copy_async(to + i + lane * 4, from + i + lane * 4, true);
        float* values = to + GROUPED;
        const int token = start + group * kGroup;
        if (wide) {
          constexpr int PIECES = BLOCK_COLUMNS / 4;              // 4 or 8: the lanes take all of them once
          static_assert(kGroup * PIECES <= 32, "a lane copies at most one piece of the values");
          const int t = lane / PIECES, c = lane % PIECES * 4;
          if (t < kGroup) {
            if (token + t < end && first_column + c < value_dim)
              copy_async(values + t * BLOCK_COLUMNS + c, v0 + (size_t)(token + t) * width + c, true);
            else
              *reinterpret_cast<float4*>(values + t * BLOCK_COLUMNS + c) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          }
        } else {
          for (int index = lane; index < kGroup * BLOCK_COLUMNS; index += 32) {
            const int t = index / BLOCK_COLUMNS, c = index % BLOCK_COLUMNS;
            if (token + t < end && first_column + c < value_dim) copy_async(values + index, v0 + (size_t)(token + t) * width + c, false);
            else values[index] = 0.0f;
          }
        }
      }
      copy_commit();
    };
    fetch(0);
    if (chunks > 1) fetch(1); else copy_commit();
    copy_wait<1>();
    __syncthreads();                                             // the first stage is there
    for (int chunk = 0; chunk < chunks; ++chunk) {               // (into the stage that was walked last)
      if (chunk + 2 < chunks) fetch(chunk + 2); else copy_commit();
      copy_wait<1>();
      __syncthreads();                                           // this stage has been walked, and the next one is there
    }
    copy_wait<0>();
    return;
  }

  const int l = lane % LANES, base_lane = lane & 16;
  const int local_column = threadIdx.y * COLUMNS + lane / LANES * C;
  const int column = first_column + local_column;                // idle lanes (beyond value_dim) still take part in the shuffles
  const bool wide = key_dim % 4 == 0;
  float* column_state = state + (((size_t)state_slots[row] * heads + head) * value_dim + column) * key_dim;
  Pair s[C][PER / 2];
#pragma unroll
  for (int c = 0; c < C; ++c)
    load_column<LANES, PER>(s[c], column_state + (size_t)c * key_dim, l, key_dim, column + c < value_dim, wide);
  auto pairs_at = [&](const float* vector, Pair (&to)[PER / 2]) {
#pragma unroll
    for (int m = 0; m < PER; m += 4) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(vector + (m / 4 * LANES + l) * 4);
      to[m / 2] = a.x;
      to[m / 2 + 1] = a.y;
    }
  };
  // sums of S^T (G_t k_t), and likewise of S^T (G_t q_t): token t = number / C, column number % C
  const int number = lane_sum<SUMS>(l);
  const int my_token = number / C, my_column = number % C;
  const bool writes = l < SUMS && column + my_column < value_dim;
  const size_t out_step = (size_t)heads * value_dim;
  float* out_of = out + ((size_t)start * heads + head) * value_dim + column + my_column;
  __syncthreads();                                               // the first stage is there
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int count = min(CHUNK, groups - chunk * CHUNK);
    const float* in = staged + (chunk % STAGES) * STAGE;
#pragma unroll 1
    for (int g = 0; g < count; ++g, in += ROW) {
      const float* scalars = in + 13 * PADDED;
      float seen_parts[SUMS], read_parts[SUMS];
#pragma unroll
      for (int t = 0; t < kGroup; ++t) {
        Pair key[PER / 2], query[PER / 2];
        pairs_at(in + t * PADDED, key);
        pairs_at(in + (kGroup + t) * PADDED, query);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          Pair seen[2] = {0, 0}, read[2] = {0, 0};
#pragma unroll
          for (int m = 0; m < PER / 2; ++m) {
            seen[m & 1] = pair_fma(s[c][m], key[m], seen[m & 1]);
            read[m & 1] = pair_fma(s[c][m], query[m], read[m & 1]);
          }
          seen_parts[t * C + c] = pair_total(seen);
          read_parts[t * C + c] = pair_total(read);
        }
      }
      const float4 k_low = *reinterpret_cast<const float4*>(scalars), k_high = *reinterpret_cast<const float4*>(scalars + 4);
      const float4 b = *reinterpret_cast<const float4*>(scalars + 8);
      const float4 reach = *reinterpret_cast<const float4*>(scalars + 12 + (my_token & 3) * 4);
      float v[kGroup][C];
#pragma unroll
      for (int t = 0; t < kGroup; ++t)
#pragma unroll
        for (int c = 0; c < C; ++c) v[t][c] = in[GROUPED + t * BLOCK_COLUMNS + local_column + c];
      const float seen_sum = sum_lanes<LANES, SUMS>(seen_parts, l);
      const float read_sum = sum_lanes<LANES, SUMS>(read_parts, l);
      float u[C][kGroup];
#pragma unroll
      for (int t = 0; t < kGroup; ++t)
#pragma unroll
        for (int c = 0; c < C; ++c) v[t][c] -= __shfl_sync(0xffffffffu, seen_sum, base_lane | lane_with<SUMS>(t * C + c));
#pragma unroll
      for (int c = 0; c < C; ++c) {
        u[c][0] = b.x * v[0][c];
        u[c][1] = b.y * fmaf(-k_low.x, u[c][0], v[1][c]);
        u[c][2] = b.z * fmaf(-k_low.z, u[c][1], fmaf(-k_low.y, u[c][0], v[2][c]));
        u[c][3] = b.w * fmaf(-k_high.y, u[c][2], fmaf(-k_high.x, u[c][1], fmaf(-k_low.w, u[c][0], v[3][c])));
      }
      const int token = (chunk * CHUNK + g) * kGroup + my_token;
      if (writes && token < end - start) {
        float mine[kGroup];
#pragma unroll
        for (int t = 0; t < kGroup; ++t) {
          mine[t] = u[0][t];
#pragma unroll
          for (int c = 1; c < C; ++c) mine[t] = my_column == c ? u[c][t] : mine[t];
        }
        out_of[(size_t)token * out_step] =
            fmaf(reach.w, mine[3], fmaf(reach.z, mine[2], fmaf(reach.y, mine[1], fmaf(reach.x, mine[0], read_sum))));
      }
      Pair decay[PER / 2];
      pairs_at(in + 3 * kGroup * PADDED, decay);
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int m = 0; m < PER / 2; ++m) s[c][m] = pair_mul(s[c][m], decay[m]);
#pragma unroll
      for (int t = 0; t < kGroup; ++t) {
        Pair key[PER / 2];
        pairs_at(in + (2 * kGroup + t) * PADDED, key);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const Pair both = pair_from(u[c][t], u[c][t]);
#pragma unroll
          for (int m = 0; m < PER / 2; ++m) s[c][m] = pair_fma(key[m], both, s[c][m]);
        }
      }
    }
    __syncthreads();                                             // this stage has been walked, and the next one is there
  }
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (column + c < value_dim) store_column<LANES, PER>(s[c], column_state + (size_t)c * key_dim, l, key_dim, wide);
}

// One warp per (token, head): out = o / sqrt(mean(o^2) + eps) * weight * act(gate); the weight is [value_dim], the
// same for every head, or (weight_per_head) [heads, value_dim].
template <typename T, typename TG>
__global__ void gated_head_norm_kernel(const float* __restrict__ o, const TG* __restrict__ gate, long long ld_gate,
                                       const float* __restrict__ weight, T* __restrict__ out, int units,
                                       int heads, int value_dim, float eps, int sigmoid_gate, int weight_per_head) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int unit = blockIdx.x * blockDim.y + threadIdx.y;       // token * heads + head
  if (unit >= units) return;
  const int lane = threadIdx.x;
  const float* src = o + (size_t)unit * value_dim;
  float sum = 0.0f;
  for (int d = lane; d < value_dim; d += 32) sum = fmaf(src[d], src[d], sum);
  const float inverse = rsqrtf(warp_sum(sum) / (float)value_dim + eps);
  const TG* gate_row = gate + (size_t)(unit / heads) * ld_gate + (size_t)(unit % heads) * value_dim;
  const float* scale = weight + (weight_per_head ? (size_t)(unit % heads) * value_dim : 0);
  for (int d = lane; d < value_dim; d += 32) {
    const float z = to_float(gate_row[d]);
    const float act = sigmoid_gate ? sigmoid(z) : silu(z);
    out[(size_t)unit * value_dim + d] = from_float<T>(src[d] * inverse * scale[d] * act);
  }
}

// The same for heads of up to LANES * PIECES numbers, which LANES lanes hold in registers: the head is read once, and its gate and
// weight asked for with it (the kernel above reads the head twice and the rest behind the sum: 2,274 tokens of 16 heads of 128
// 13.1 us, here 11.2, of 64 heads of 64 40.8, here 20.8; two tokens of 16 heads of 128 3.0, here 2.0).  The sum is that of the
// kernel above, bit for bit: there lane L has the numbers L, L + 32, ..., and the lanes' sums are added 16, 8, 4, 2 and 1
// apart; with 16 or 8 lanes a lane has the numbers of two or four of those lanes, and the first steps are its own.
template <typename T, typename TG, int LANES, int PIECES>
__global__ void __launch_bounds__(128) gated_row_norm_kernel(const float* __restrict__ o, const TG* __restrict__ gate,
                                                             long long ld_gate, const float* __restrict__ weight,
                                                             T* __restrict__ out, int units, int heads, int value_dim, float eps,
                                                             int sigmoid_gate, int weight_per_head) {
  const int unit = blockIdx.x * (128 / LANES) + threadIdx.x / LANES;       // token * heads + head
  const int l = threadIdx.x % LANES, head = unit % heads;
  const int count = unit < units ? value_dim : 0;                          // (a warp's last heads may not be there)
  const float* scale = weight + (weight_per_head ? (size_t)head * value_dim : 0);
  const TG* gate_row = gate + (size_t)(unit / heads) * ld_gate + (size_t)head * value_dim;
  const float* src = o + (size_t)unit * value_dim;
  float w[PIECES], v[PIECES];
  TG z[PIECES];
#pragma unroll
  for (int e = 0; e < PIECES; ++e) w[e] = l + LANES * e < count ? scale[l + LANES * e] : 0.0f;
  grid_dependency_wait();
  grid_launch_dependents();
#pragma unroll
  for (int e = 0; e < PIECES; ++e) v[e] = l + LANES * e < count ? src[l + LANES * e] : 0.0f;
#pragma unroll
  for (int e = 0; e < PIECES; ++e) z[e] = l + LANES * e < count ? gate_row[l + LANES * e] : from_float<TG>(0.0f);
  constexpr int OWN = 32 / LANES;                                // of the 32 sums, those of l, l + LANES, ...
  float sums[OWN];
#pragma unroll
  for (int i = 0; i < OWN; ++i) sums[i] = 0.0f;
#pragma unroll
  for (int e = 0; e < PIECES; ++e) sums[e % OWN] = fmaf(v[e], v[e], sums[e % OWN]);
#pragma unroll
  for (int half = OWN / 2; half > 0; half >>= 1)
#pragma unroll
    for (int i = 0; i < half; ++i) sums[i] += sums[i + half];
  float sum = sums[0];
#pragma unroll
  for (int step = LANES / 2; step > 0; step >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, step);
  const float inverse = rsqrtf(sum / (float)value_dim + eps);
#pragma unroll
  for (int e = 0; e < PIECES; ++e) {
    const float gated = to_float(z[e]);
    const float act = sigmoid_gate ? sigmoid(gated) : silu(gated);
    if (l + LANES * e < count) out[(size_t)unit * value_dim + l + LANES * e] = from_float<T>(v[e] * inverse * w[e] * act);
  }
}

template <typename T, typename TG>
int launch_gated_norm(const float* o, const TG* gate, long long ld_gate, const float* weight, T* out, int units, int heads,
                      int value_dim, float eps, int sigmoid_gate, int weight_per_head, cudaStream_t stream) {
#define MIR_NORM(LANES, PIECES)                                                                                           \
  return mir_launch("gated_head_norm", gated_row_norm_kernel<T, TG, LANES, PIECES>,                                      \
                    dim3((units + 128 / LANES - 1) / (128 / LANES)), dim3(128), 0, stream, 0, o, gate, ld_gate, weight, out, units, \
                    heads, value_dim, eps, sigmoid_gate, weight_per_head)
  if (value_dim <= 32) MIR_NORM(8, 4);
  if (value_dim <= 64) MIR_NORM(16, 4);
  if (value_dim <= 128) MIR_NORM(32, 4);
  if (value_dim <= 256) MIR_NORM(32, 8);
  return mir_launch("gated_head_norm", gated_head_norm_kernel<T, TG>, dim3((units + 3) / 4), dim3(32, 4), 0, stream, 0, o, gate,
                    ld_gate, weight, out, units, heads, value_dim, eps, sigmoid_gate, weight_per_head);
#undef MIR_NORM
}

// The same for wide rows (a norm over all heads at once): one CTA per (token, head), its sum by a fixed tree.  A thread keeps
// its columns in registers, V at a time in PIECES places blockDim.x * V columns apart; the gate's loads are on their way
// while the sum is formed.
template <typename T, int V>
__device__ __forceinline__ void load_columns(float (&v)[V], const T* __restrict__ from) {
  if constexpr (V == 4 && sizeof(T) == 4) {
    const float4 a = *reinterpret_cast<const float4*>(from);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  } else if constexpr (V == 4) {
    const uint2 a = *reinterpret_cast<const uint2*>(from);
    const float2 low = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.x));
    const float2 high = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.y));
    v[0] = low.x; v[1] = low.y; v[2] = high.x; v[3] = high.y;
  } else {
    v[0] = to_float(from[0]);
  }
}
template <typename T, typename TG, int V, int PIECES>
__global__ void __launch_bounds__(512) gated_wide_norm_kernel(const float* __restrict__ o, const TG* __restrict__ gate,
                                                              long long ld_gate, const float* __restrict__ weight,
                                                              T* __restrict__ out, int heads, int value_dim, float eps,
                                                              int sigmoid_gate, int weight_per_head) {
  __shared__ float scratch[32];
  const int unit = blockIdx.x;                                  // token * heads + head
  const float* scale = weight + (weight_per_head ? (size_t)(unit % heads) * value_dim : 0);
  float w[PIECES][V], x[PIECES][V], g[PIECES][V];
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int d = (p * blockDim.x + threadIdx.x) * V;
    if (d < value_dim) load_columns(w[p], scale + d);           // (older than the kernel before this one)
  }
  grid_dependency_wait();
  grid_launch_dependents();
  const float* src = o + (size_t)unit * value_dim;
  const TG* gate_row = gate + (size_t)(unit / heads) * ld_gate + (size_t)(unit % heads) * value_dim;
  float sum = 0.0f;
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int d = (p * blockDim.x + threadIdx.x) * V;
    if (d >= value_dim) continue;
    load_columns(x[p], src + d);
    load_columns(g[p], gate_row + d);
  }
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    if ((p * blockDim.x + threadIdx.x) * V >= value_dim) continue;
#pragma unroll
    for (int v = 0; v < V; ++v) sum = fmaf(x[p][v], x[p][v], sum);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
  sum = warp_sum(sum);
  if (lane == 0) scratch[warp] = sum;
  __syncthreads();
  float total = 0.0f;
  for (int i = 0; i < warps; ++i) total += scratch[i];
  const float inverse = rsqrtf(total / (float)value_dim + eps);
  T* dst = out + (size_t)unit * value_dim;
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int d = (p * blockDim.x + threadIdx.x) * V;
    if (d >= value_dim) continue;
#pragma unroll
    for (int v = 0; v < V; ++v) x[p][v] *= inverse * w[p][v] * (sigmoid_gate ? sigmoid(g[p][v]) : silu(g[p][v]));
    if constexpr (V == 4 && sizeof(T) == 4) {
      *reinterpret_cast<float4*>(dst + d) = make_float4(x[p][0], x[p][1], x[p][2], x[p][3]);
    } else if constexpr (V == 4) {
      uint2 packed;
      *reinterpret_cast<__nv_bfloat162*>(&packed.x) = __floats2bfloat162_rn(x[p][0], x[p][1]);
      *reinterpret_cast<__nv_bfloat162*>(&packed.y) = __floats2bfloat162_rn(x[p][2], x[p][3]);
      *reinterpret_cast<uint2*>(dst + d) = packed;
    } else {
      dst[d] = from_float<T>(x[p][0]);
    }
  }
}

template <typename T, typename TG>
int launch_gated_wide_norm(const float* o, const TG* gate, long long ld_gate, const float* weight, T* out, int units,
                           int heads, int value_dim, float eps, int sigmoid_gate, int weight_per_head, cudaStream_t stream) {
  const bool aligned = value_dim % 4 == 0 && ld_gate % 4 == 0 && ((uintptr_t)o & 15) == 0 && ((uintptr_t)weight & 15) == 0 &&
                       ((uintptr_t)gate & (4 * sizeof(TG) - 1)) == 0 && ((uintptr_t)out & (4 * sizeof(T) - 1)) == 0;
#define MIR_WIDE_NORM(V, P)                                                                                               \
  return mir_launch("gated_head_norm", gated_wide_norm_kernel<T, TG, V, P>, dim3(units), dim3(threads), 0, stream, 0, o, \
                    gate, ld_gate, weight, out, heads, value_dim, eps, sigmoid_gate, weight_per_head)
  const int per_thread = aligned ? 4 : 1;
  const int places = (value_dim + per_thread - 1) / per_thread;
  const int threads = places >= 512 ? 512 : (places + 31) / 32 * 32;
  const int pieces = (places + threads - 1) / threads;
  if (per_thread == 4) {
    if (pieces <= 1) MIR_WIDE_NORM(4, 1);
    if (pieces <= 2) MIR_WIDE_NORM(4, 2);
    if (pieces <= 4) MIR_WIDE_NORM(4, 4);
    if (pieces <= 8) MIR_WIDE_NORM(4, 8);
  } else {
    if (pieces <= 2) MIR_WIDE_NORM(1, 2);
    if (pieces <= 8) MIR_WIDE_NORM(1, 8);
    if (pieces <= 32) MIR_WIDE_NORM(1, 32);
  }
#undef MIR_WIDE_NORM
  mir_set_error("gated_head_norm: rows of %d numbers are wider than the kernel takes", value_dim);
  return MIR_BAD_ARGUMENT;
}
constexpr int kWideNormColumns = 512, kWideNormLimit = 16384;   // rows of these widths take a CTA each

template <int PER, bool PER_CHANNEL>
int launch_scan_as(cudaStream_t stream, const float* qkv, const float* beta, const float* decay, float* state,
                   const int* query_starts, const int* state_slots, const int* positions, float* out, int rows,
                   int heads, int kv_heads, int key_dim, int value_dim) {
  constexpr int columns = kScanWarps * (32 / kScanLanes) * kScanColumns;
  constexpr int padded = kScanLanes * PER;
  constexpr int row = 2 * padded + (PER_CHANNEL ? padded : 4) + 4 + columns;
  constexpr size_t smem = (size_t)kScanStages * kScanChunk * row * sizeof(float);
  static bool raised = false;                                    // more than 48 KB of shared memory needs the opt-in
  if (smem > 48 * 1024 && !raised) {
    const cudaError_t err = cudaFuncSetAttribute(delta_rule_scan_kernel<PER, PER_CHANNEL>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) {
      mir_set_error("delta_rule_scan: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(err));
      return MIR_CUDA_ERROR;
    }
    raised = true;
  }
  return mir_launch_alone("delta_rule_scan", delta_rule_scan_kernel<PER, PER_CHANNEL>,
                    dim3(rows, heads, (value_dim + columns - 1) / columns), dim3(32, kScanWarps + kFetchWarps), smem, stream, 0, qkv,
                    beta, decay, state, query_starts, state_slots, positions, out, heads, kv_heads, key_dim, value_dim);
}

template <int PER, int C, bool PER_CHANNEL>
int launch_step_as(cudaStream_t stream, const float* qkv, const float* beta, const float* decay, float* state,
                   const int* query_starts, const int* state_slots, const int* positions, float* out, int rows, int heads,
                   int kv_heads, int key_dim, int value_dim) {
  constexpr int columns = kScanWarps * 2 * C;
  const bool wide = key_dim % 4 == 0 && (2 * kv_heads * key_dim + heads * value_dim) % 4 == 0;
  return mir_launch("delta_rule_step", wide ? delta_rule_step_kernel<PER, C, PER_CHANNEL, true>
                                            : delta_rule_step_kernel<PER, C, PER_CHANNEL, false>,
                    dim3(rows, heads, (value_dim + columns - 1) / columns), dim3(32, kScanWarps), 0, stream, 0, qkv, beta,
                    decay, state, query_starts, state_slots, positions, out, heads, kv_heads, key_dim, value_dim);
}

template <bool PER_CHANNEL>
int launch_step(cudaStream_t stream, const float* qkv, const float* beta, const float* decay, float* state,
                const int* query_starts, const int* state_slots, const int* positions, float* out, int rows, int heads,
                int kv_heads, int key_dim, int value_dim) {
#define MIR_STEP(P, C)                                                                                               \
  return launch_step_as<P, C, PER_CHANNEL>(stream, qkv, beta, decay, state, query_starts, state_slots, positions, out, rows, \
                                           heads, kv_heads, key_dim, value_dim)
  // Four columns a lane share a token's inputs; two make twice as many CTAs of a few rows.
  const bool many = (long long)rows * heads * ((value_dim + 31) / 32) >= 2LL * mir_sm_count();
  if (key_dim <= 64) { if (many) MIR_STEP(4, 4); MIR_STEP(4, 2); }
  if (key_dim <= 128) { if (many) MIR_STEP(8, 4); MIR_STEP(8, 2); }
  if (key_dim <= 192) MIR_STEP(12, 2);
  MIR_STEP(16, 2);
#undef MIR_STEP
}

template <bool PER_CHANNEL>
int launch_scan(cudaStream_t stream, const float* qkv, const float* beta, const float* decay, float* state,
                const int* query_starts, const int* state_slots, const int* positions, float* out, int rows, int heads,
                int kv_heads, int key_dim, int value_dim, bool single_tokens) {
  if (key_dim > 32 * kMaxPerLane) {
    mir_set_error("delta_rule_scan: key_dim %d is larger than %d", key_dim, 32 * kMaxPerLane);
    return MIR_BAD_ARGUMENT;
  }
  if (single_tokens)
    return launch_step<PER_CHANNEL>(stream, qkv, beta, decay, state, query_starts, state_slots, positions, out, rows, heads,
                                    kv_heads, key_dim, value_dim);
#define MIR_SCAN(P)                                                                                                  \
  return launch_scan_as<P, PER_CHANNEL>(stream, qkv, beta, decay, state, query_starts, state_slots, positions, out, rows, \
                                        heads, kv_heads, key_dim, value_dim)
  if (key_dim <= 64) MIR_SCAN(4);
  if (key_dim <= 128) MIR_SCAN(8);
  if (key_dim <= 192) MIR_SCAN(12);
  MIR_SCAN(16);
#undef MIR_SCAN
}

template <int PER, int C>
int launch_grouped_walk(cudaStream_t stream, const float* grouped, const float* qkv, float* state, const int* query_starts,
                        const int* state_slots, const int* positions, float* out, int rows, int heads, int kv_heads, int key_dim,
                        int value_dim) {
  constexpr int columns = kScanWarps * 2 * C;
  constexpr int smem = 3 * kFetchWarps * (group_floats(16 * PER) + kGroup * columns) * (int)sizeof(float);
  const cudaError_t err = cudaFuncSetAttribute(delta_rule_grouped_scan_kernel<PER, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) {
    mir_set_error("delta_rule_scan: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(err));
    return MIR_CUDA_ERROR;
  }
  return mir_launch_alone("delta_rule_scan", delta_rule_grouped_scan_kernel<PER, C>,
                    dim3(rows, heads, (value_dim + columns - 1) / columns), dim3(32, kScanWarps + kFetchWarps), smem, stream, 0,
                    grouped, qkv, state, query_starts, state_slots, positions, out, heads, kv_heads, key_dim, value_dim);
}

template <int PER, bool PER_CHANNEL>
int launch_grouped_as(cudaStream_t stream, const float* qkv, const float* beta, const float* decay, float* state,
                      const int* query_starts, const int* state_slots, const int* positions, float* out, float* grouped,
                      int tokens, int rows, int heads, int kv_heads, int key_dim, int value_dim) {
  constexpr int padded = 16 * PER;
  int status = mir_launch("delta_rule_group", delta_rule_group_kernel<padded, PER_CHANNEL>,
                          dim3(tokens / kGroup + rows, (heads + 3) / 4), dim3(32, 4), 0, stream, 0, qkv, beta, decay,
                          query_starts, positions, grouped, rows, heads, kv_heads, key_dim, value_dim);
  if (status != MIR_OK) return status;
  // Two columns a lane while their CTAs get an SM each, else four, half as many CTAs with twice the columns for a group's reads.
  // 1,000 tokens, heads of 128, two / four columns: one request of 16 heads (128 CTAs of two columns) 134 / 187 us, of 20
  // heads (160 CTAs) 211 / 188, of 24 216 / 192, of 32 220 / 196; two requests of 32 heads 426 / 323.
  const long long ctas = (long long)rows * heads * ((value_dim + kScanWarps * 4 - 1) / (kScanWarps * 4));
  if (ctas > mir_sm_count())
    return launch_grouped_walk<PER, 4>(stream, grouped, qkv, state, query_starts, state_slots, positions, out, rows, heads, kv_heads,
                                       key_dim, value_dim);
  return launch_grouped_walk<PER, 2>(stream, grouped, qkv, state, query_starts, state_slots, positions, out, rows, heads, kv_heads,
                                     key_dim, value_dim);
}

template <bool PER_CHANNEL>
int launch_grouped(cudaStream_t stream, const float* qkv, const float* beta, const float* decay, float* state,
                   const int* query_starts, const int* state_slots, const int* positions, float* out, float* grouped,
                   int tokens, int rows, int heads, int kv_heads, int key_dim, int value_dim) {
#define MIR_GROUPED(P)                                                                                                    \
  return launch_grouped_as<P, PER_CHANNEL>(stream, qkv, beta, decay, state, query_starts, state_slots, positions, out,   \
                                           grouped, tokens, rows, heads, kv_heads, key_dim, value_dim)
  if (key_dim <= 64) MIR_GROUPED(4);
  MIR_GROUPED(8);
#undef MIR_GROUPED
}
constexpr int kGroupedKeys = 128;                                // the widest key head that is walked in groups

}  // namespace

// bf16: the type of x, w and beta_raw (and of decay_raw unless decay_f32).  decay_width: heads, or heads * key_dim for
// one decay per key channel.  Writes qkv [tokens, channels], beta [tokens, heads], decay [tokens, decay_width] (32-bit)
// and moves the convolution's tail [slots, taps - 1, channels] on.
MIR_EXPORT int mir_delta_rule_prepare(int bf16, int decay_f32, const void* x, long long ldx, const void* w, float* tail,
                                      const void* beta_raw, long long ld_beta, const void* decay_raw, long long ld_decay,
                                      const float* dt_bias, const float* a_log, const int* row_of_token,
                                      const int* query_starts, const int* state_slots, const int* positions, float* qkv,
                                      float* beta, float* decay, int tokens, int rows, int heads, int kv_heads,
                                      int key_dim, int value_dim, int decay_width, int taps, cudaStream_t stream) {
  if (tokens == 0 || rows == 0) return MIR_OK;
  if (tokens < 0 || rows < 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || key_dim <= 0 ||
      key_dim > 32 * kMaxPerLane || value_dim <= 0 || taps < 1 || taps > kMaxTaps ||
      (decay_width != heads && decay_width != heads * key_dim)) {
    mir_set_error("delta_rule_prepare: bad sizes (heads %d, kv heads %d, key_dim %d up to %d, value_dim %d, taps %d up "
                  "to %d, decay width %d)", heads, kv_heads, key_dim, 32 * kMaxPerLane, value_dim, taps, kMaxTaps,
                  decay_width);
    return MIR_BAD_ARGUMENT;
  }
  const int channels = 2 * kv_heads * key_dim + heads * value_dim;
  // one CTA per token where the step has many; with few tokens each token's work is shared out over several CTAs
  const int most = (2 * kv_heads + 7) / 8 > (channels + 255) / 256 ? (2 * kv_heads + 7) / 8 : (channels + 255) / 256;
  int parts = (2 * mir_sm_count() + tokens - 1) / tokens;
  parts = parts < 1 ? 1 : (parts > most ? most : parts);
  int status;
  const size_t element = bf16 ? 2 : 4;
  const bool paired = key_dim % 2 == 0 && (heads * value_dim) % 2 == 0 && ldx % 2 == 0 &&
                      (uintptr_t)x % (2 * element) == 0 && (uintptr_t)qkv % 8 == 0 && (uintptr_t)tail % 8 == 0;
  const int values = heads * value_dim;
  const bool runs = taps <= kRunTaps && key_dim <= 128 && key_dim % 4 == 0 && values % 4 == 0 && ldx % 4 == 0 &&
                    (uintptr_t)x % (4 * element) == 0 && ((uintptr_t)qkv | (uintptr_t)tail) % 16 == 0;
  const int units = 2 * kv_heads + (values + 127) / 128 + (decay_width + 127) / 128 + 1;
  // eight tokens a warp (sixteen: 59 us where eight take 38) once that still makes several warps for every SM's schedulers
  // - but single tokens have no neighbour to share inputs with, and eight of them behind one another in a warp wait for eight
  // tails (200 rows of 32 heads of 64, decays per channel: 23 us)
  const bool long_runs = tokens != rows && (long long)tokens * units >= 8LL * 16 * mir_sm_count();
#define MIR_PREPARE_RUN(T, TD, RUN)                                                                                    \
  status = mir_launch("delta_rule_prepare", delta_rule_prepare_run_kernel<T, TD, RUN>,                                 \
                      dim3((tokens + RUN - 1) / RUN, (units + kRunWarps - 1) / kRunWarps), dim3(32, kRunWarps), 0,     \
                      stream, 0, (const T*)x, ldx, (const T*)w, tail, (const T*)beta_raw, ld_beta,                     \
                      (const TD*)decay_raw, ld_decay, dt_bias, a_log, row_of_token, query_starts, state_slots,         \
                      positions, qkv, beta, decay, tokens, heads, kv_heads, key_dim, value_dim, decay_width, taps)
#define MIR_PREPARE_AS(T, TD, P)                                                                                       \
  status = mir_launch("delta_rule_prepare", delta_rule_prepare_kernel<T, TD, P>, dim3(tokens, parts), dim3(256), 0,    \
                      stream, 0, (const T*)x, ldx, (const T*)w, tail, (const T*)beta_raw, ld_beta,       \
                      (const TD*)decay_raw, ld_decay, dt_bias, a_log, row_of_token, query_starts, state_slots,         \
                      positions, qkv, beta, decay, heads, kv_heads, key_dim, value_dim, decay_width, taps)
#define MIR_PREPARE(T, TD)                                                                                             \
  do {                                                                                                                 \
    if (runs && long_runs) MIR_PREPARE_RUN(T, TD, 8);                                                                  \
    else if (runs) MIR_PREPARE_RUN(T, TD, 1);                                                                          \
    else if (paired) MIR_PREPARE_AS(T, TD, true);                                                                      \
    else MIR_PREPARE_AS(T, TD, false);                                                                                 \
  } while (0)
  if (bf16 && decay_f32) MIR_PREPARE(__nv_bfloat16, float);
  else if (bf16) MIR_PREPARE(__nv_bfloat16, __nv_bfloat16);
  else MIR_PREPARE(float, float);
#undef MIR_PREPARE
#undef MIR_PREPARE_AS
#undef MIR_PREPARE_RUN
  // rows of one token have moved their tails on themselves; a step of single tokens needs nothing more
  if (status != MIR_OK || taps == 1 || tokens == rows) return status;
  const int threads = channels >= 256 ? 256 : ((channels + 31) / 32) * 32;
  const dim3 tail_grid(rows, (channels + threads - 1) / threads);
  if (bf16)
    return mir_launch("short_conv_tail", short_conv_tail_kernel<__nv_bfloat16>, tail_grid, dim3(threads), 0, stream, 0,
                      (const __nv_bfloat16*)x, ldx, tail, query_starts, state_slots, positions, channels, taps, 1);
  return mir_launch("short_conv_tail", short_conv_tail_kernel<float>, tail_grid, dim3(threads), 0, stream, 0,
                    (const float*)x, ldx, tail, query_starts, state_slots, positions, channels, taps, 1);
}

// qkv, beta, decay as delta_rule_prepare leaves them; per_channel: decay is [tokens, heads * key_dim].  grouped: null, or
// 32-bit scratch (16-byte aligned) of (tokens / 4 + rows) * heads * (13 padded + 28) numbers, padded = the key width rounded
// up to 64 or 128: a step that brings more than single tokens then walks four tokens at a time (results then depend, in the
// last places, on where a request's portions begin); not used for key heads wider than 128.
MIR_EXPORT int mir_delta_rule_scan(int per_channel, const float* qkv, const float* beta, const float* decay, float* state,
                                   const int* query_starts, const int* state_slots, const int* positions, float* out,
                                   float* grouped, int tokens, int rows, int heads, int kv_heads, int key_dim, int value_dim,
                                   cudaStream_t stream) {
  if (rows == 0) return MIR_OK;
  if (rows < 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || key_dim <= 0 || value_dim <= 0) {
    mir_set_error("delta_rule_scan: bad sizes (rows %d, heads %d, kv heads %d, key_dim %d, value_dim %d)", rows, heads,
                  kv_heads, key_dim, value_dim);
    return MIR_BAD_ARGUMENT;
  }
  if (grouped != nullptr && tokens != rows && key_dim <= kGroupedKeys && ((uintptr_t)grouped & 15) == 0 && heads <= 4 * 65535) {
    if (per_channel)
      return launch_grouped<true>(stream, qkv, beta, decay, state, query_starts, state_slots, positions, out, grouped, tokens,
                                  rows, heads, kv_heads, key_dim, value_dim);
    return launch_grouped<false>(stream, qkv, beta, decay, state, query_starts, state_slots, positions, out, grouped, tokens,
                                 rows, heads, kv_heads, key_dim, value_dim);
  }
  if (per_channel)
    return launch_scan<true>(stream, qkv, beta, decay, state, query_starts, state_slots, positions, out, rows, heads,
                             kv_heads, key_dim, value_dim, tokens == rows);
  return launch_scan<false>(stream, qkv, beta, decay, state, query_starts, state_slots, positions, out, rows, heads,
                            kv_heads, key_dim, value_dim, tokens == rows);
}

// o [tokens, heads, value_dim] 32-bit; gate element (t, h, d) at gate[t * ld_gate + h * value_dim + d], in the
// activations' type or (gate_f32) in 32-bit; out [tokens, heads * value_dim] contiguous in the activations' type.
MIR_EXPORT int mir_gated_head_norm(int bf16, int gate_f32, const float* o, const void* gate, long long ld_gate,
                                   const float* weight, void* out, int tokens, int heads, int value_dim, float eps,
                                   int sigmoid_gate, int weight_per_head, cudaStream_t stream) {
  if (tokens == 0) return MIR_OK;
  if (tokens < 0 || heads <= 0 || value_dim <= 0) { mir_set_error("gated_head_norm: bad sizes"); return MIR_BAD_ARGUMENT; }
  const int units = tokens * heads;
  if (value_dim >= kWideNormColumns && value_dim <= kWideNormLimit) {
    if (bf16 && gate_f32)
      return launch_gated_wide_norm(o, (const float*)gate, ld_gate, weight, (__nv_bfloat16*)out, units, heads, value_dim, eps,
                                    sigmoid_gate, weight_per_head, stream);
    if (bf16)
      return launch_gated_wide_norm(o, (const __nv_bfloat16*)gate, ld_gate, weight, (__nv_bfloat16*)out, units, heads,
                                    value_dim, eps, sigmoid_gate, weight_per_head, stream);
    return launch_gated_wide_norm(o, (const float*)gate, ld_gate, weight, (float*)out, units, heads, value_dim, eps,
                                  sigmoid_gate, weight_per_head, stream);
  }
  if (bf16 && gate_f32)
    return launch_gated_norm(o, (const float*)gate, ld_gate, weight, (__nv_bfloat16*)out, units, heads, value_dim, eps,
                             sigmoid_gate, weight_per_head, stream);
  if (bf16)
    return launch_gated_norm(o, (const __nv_bfloat16*)gate, ld_gate, weight, (__nv_bfloat16*)out, units, heads, value_dim, eps,
                             sigmoid_gate, weight_per_head, stream);
  return launch_gated_norm(o, (const float*)gate, ld_gate, weight, (float*)out, units, heads, value_dim, eps, sigmoid_gate,
                           weight_per_head, stream);
}
