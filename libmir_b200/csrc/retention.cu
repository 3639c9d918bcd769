// The recurrence of the retention mixer: linear attention with one fixed decay per head and no softmax.
//
//   per head, S [key channel, value channel] (stored per value channel, a column contiguous):
//     S_t = d S_t-1 + k_t v_t^T;   o_t = S_t^T q_t = d (S_t-1^T q_t) + (q_t . k_t) v_t
//   q and k are the projections' results rotated by the token's position (half-split pairs i, i + r/2 of the first r
//   channels; angle = position * inv_freq[i], a 32-bit product), k also times key_scale, both in 32-bit while a chunk
//   of tokens is staged in shared memory: nothing rotated is ever rounded to the storage type.
//   With `activated` the recurrence's inputs are silu of the projections' results (of q and k before the rotation, and of
//   v), also in 32-bit while they are staged.
// The decay, the rotation, the state and every sum are 32-bit; T is the storage type of the projections' results.
// One lane count and one order of sums for every shape of step: a request's 32-bit results do not depend on how it was
// cut into steps.  A row of a captured decode batch whose position is negative is padding: nothing is read or written.
#include "common.cuh"
#include "scan_pairs.cuh"

using namespace mir;

namespace {

constexpr int kWarps = 4;
constexpr int kFetchWarps = 4;          // of the walk over prepared rows: they copy what the others will need

// A token's q and k of one head, staged by one warp.  Lane `lane` owns the channels i = lane + 32 e.  A channel of the
// first half of the rotated ones is rotated together with its partner i + half by the lane that owns it (one sine and
// cosine for the pair, for q and k alike); the partner's owner has nothing to do there.  `load_token` only issues the
// loads, in the storage type; `stage_token` rotates, scales the key, and writes q at row[i], k at row[PADDED + i] and
// q . k at row[2 PADDED] (32-bit, to shared or global memory).  Every product and sum is spelled out, so that the
// kernels that share this code leave the same bits.
template <typename T, int PER_LANE>
struct TokenInputs {
  static constexpr int PAIRED = (PER_LANE + 1) / 2;              // 32 e < half <= PADDED / 2 for these e alone
  T q[PER_LANE], k[PER_LANE], partner_q[PAIRED], partner_k[PAIRED];
  float position;
};

// What enters the recurrence of a projection's element: the element, or its silu.
__device__ __forceinline__ float entering(float z, int activated) {
  return activated ? z / (1.0f + expf(-z)) : z;
}

template <typename T, int PER_LANE>
__device__ __forceinline__ void load_token(TokenInputs<T, PER_LANE>& in, const T* __restrict__ q,
                                           const T* __restrict__ k, size_t source, bool live, float position, int lane,
                                           int dim, int half, int rotary_dim) {
  in.position = live ? position : 0.0f;
#pragma unroll
  for (int e = 0; e < PER_LANE; ++e) {
    const int i = lane + 32 * e;
    const bool mine = live && i < dim && !(i >= half && i < rotary_dim);
    in.q[e] = mine ? q[source + i] : T(0.0f);
    in.k[e] = mine ? k[source + i] : T(0.0f);
    if (e < TokenInputs<T, PER_LANE>::PAIRED) {
      const bool paired = live && i < half;
      in.partner_q[e] = paired ? q[source + i + half] : T(0.0f);
      in.partner_k[e] = paired ? k[source + i + half] : T(0.0f);
    }
  }
}

template <typename T, int PER_LANE>
__device__ __forceinline__ void stage_token(const TokenInputs<T, PER_LANE>& in, const float* frequency, float key_scale,
                                            int lane, int half, int rotary_dim, int activated, float* row) {
  constexpr int PADDED = 32 * PER_LANE;
  float sum = 0.0f;
#pragma unroll
  for (int e = 0; e < PER_LANE; ++e) {
    const int i = lane + 32 * e;
    if (32 * e >= half && 32 * e + 32 <= rotary_dim) continue;   // a warp of partners: their owners write them
    const float qi = entering(to_float(in.q[e]), activated), ki = entering(to_float(in.k[e]), activated);
    if (e < TokenInputs<T, PER_LANE>::PAIRED && i < half) {
      // the first of a pair becomes u cos - v sin, the second v cos + u sin
      const float qp = entering(to_float(in.partner_q[e]), activated), kp = entering(to_float(in.partner_k[e]), activated);
      float sine, cosine;
      sincosf(__fmul_rn(in.position, frequency[e]), &sine, &cosine);
      const float q_first = fmaf(qi, cosine, -__fmul_rn(qp, sine)), q_second = fmaf(qp, cosine, __fmul_rn(qi, sine));
      const float k_first = __fmul_rn(fmaf(ki, cosine, -__fmul_rn(kp, sine)), key_scale);
      const float k_second = __fmul_rn(fmaf(kp, cosine, __fmul_rn(ki, sine)), key_scale);
      sum = fmaf(q_first, k_first, sum);
      sum = fmaf(q_second, k_second, sum);
      row[i] = q_first; row[PADDED + i] = k_first;
      row[i + half] = q_second; row[PADDED + i + half] = k_second;
    } else if (!(i >= half && i < rotary_dim)) {                 // not rotated (or beyond dim: zeros)
      const float scaled = __fmul_rn(ki, key_scale);
      sum = fmaf(qi, scaled, sum);
      row[i] = qi; row[PADDED + i] = scaled;
    }
  }
  sum = warp_sum(sum);
  if (lane == 0) row[2 * PADDED] = sum;
}

// blockDim (32, kWarps), grid (rows, heads, ceil(value_dim / (kWarps * 32 / kLanes))).  kLanes lanes share one column of
// the state (a function of the head's width alone: 16 from 33 key channels on, so that a single prompt fills the GPU
// with short chains); lane l of a column holds the key channels 4 (m kLanes + l) .. + 3, m < PER / 4.  The inputs of
// CHUNK tokens at a time are staged in shared memory (every column of a head reads the same q and k): a warp stages
// whole tokens, rotating as it goes, and leaves the token's q . k beside them.  What the next chunk needs is fetched
// into registers before the walk over the current chunk starts.  SHORT: a step of single tokens stages one token a warp.
template <typename T, int PER, int kLanes, bool SHORT>
__global__ void __launch_bounds__(kWarps * 32)
retention_scan_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, long long ld,
                      const float* __restrict__ inv_freq, int rotary_dim, const float* __restrict__ decays,
                      float key_scale, float* __restrict__ state, const int* __restrict__ query_starts,
                      const int* __restrict__ state_slots, const int* __restrict__ positions, float* __restrict__ out,
                      int heads, int dim, int value_dim, int activated) {
  constexpr int COLUMNS = 32 / kLanes;
  constexpr int BLOCK_COLUMNS = COLUMNS * kWarps;
  constexpr int PADDED = kLanes * PER;
  constexpr int ROW = 2 * PADDED + 4 + BLOCK_COLUMNS;             // q | k | q . k | v of this CTA's columns
  constexpr int CHUNK = SHORT ? kWarps : (PADDED <= 64 ? 32 : (PADDED <= 128 ? 16 : 8));
  __shared__ __align__(16) float staged[CHUNK * ROW];
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x, warp = threadIdx.y;
  const int thread = warp * 32 + lane;
  const int l = lane % kLanes;
  const int row = blockIdx.x, head = blockIdx.y;
  const int first_column = blockIdx.z * BLOCK_COLUMNS;
  const int local_column = warp * COLUMNS + lane / kLanes;
  const int column = first_column + local_column;
  const int start = query_starts[row], end = query_starts[row + 1];
  if (end <= start || positions[start] < 0) return;              // the whole CTA: an empty or padding row
  const bool active = column < value_dim;
  const bool wide = dim % 4 == 0;
  const float decay = decays[head];
  const int half = rotary_dim / 2;
  float* column_state = state + (((size_t)state_slots[row] * heads + head) * value_dim + (active ? column : 0)) * dim;

  float s[PER];
#pragma unroll
  for (int m = 0; m < PER; m += 4) {
    const int i = (m / 4 * kLanes + l) * 4;
    if (wide) {
      const float4 piece = (active && i < dim) ? *reinterpret_cast<const float4*>(column_state + i)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
      s[m] = piece.x; s[m + 1] = piece.y; s[m + 2] = piece.z; s[m + 3] = piece.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) s[m + e] = (active && i + e < dim) ? column_state[i + e] : 0.0f;
    }
  }
  const size_t key_at = (size_t)head * dim, value_at = (size_t)head * value_dim;
  constexpr int TOKENS_PER_WARP = CHUNK / kWarps;
  constexpr int PER_LANE = PADDED / 32;
  constexpr int VALUES_PER_THREAD = (CHUNK * BLOCK_COLUMNS + kWarps * 32 - 1) / (kWarps * 32);
  // `fetch` only issues the loads: nothing waits for them before `commit`, which runs after the walk over the chunk
  // before.
  using Inputs = TokenInputs<T, PER_LANE>;
  Inputs next[TOKENS_PER_WARP];
  T next_v[VALUES_PER_THREAD];
  float frequency[Inputs::PAIRED];                               // of the pairs this lane rotates
#pragma unroll
  for (int e = 0; e < Inputs::PAIRED; ++e) frequency[e] = lane + 32 * e < half ? inv_freq[lane + 32 * e] : 0.0f;
  auto fetch = [&](int from) {
    const int count = min(CHUNK, end - from);
#pragma unroll
    for (int tt = 0; tt < TOKENS_PER_WARP; ++tt) {
      const int t = warp + tt * kWarps;
      const bool live = t < count;
      load_token(next[tt], q, k, (size_t)(from + (live ? t : 0)) * ld + key_at, live,
                 live ? (float)positions[from + t] : 0.0f, lane, dim, half, rotary_dim);
    }
#pragma unroll
    for (int j = 0; j < VALUES_PER_THREAD; ++j) {
      const int index = thread + j * kWarps * 32;
      const int t = index / BLOCK_COLUMNS, c = index - t * BLOCK_COLUMNS;
      next_v[j] = (t < count && first_column + c < value_dim)
                      ? v[(size_t)(from + t) * ld + value_at + first_column + c] : T(0.0f);
    }
  };
  auto commit = [&](int from) {
    const int count = min(CHUNK, end - from);
#pragma unroll
    for (int tt = 0; tt < TOKENS_PER_WARP; ++tt) {
      const int t = warp + tt * kWarps;
      if (t >= count) continue;                                  // (the same for the whole warp)
      stage_token(next[tt], frequency, key_scale, lane, half, rotary_dim, activated, staged + t * ROW);
    }
#pragma unroll
    for (int j = 0; j < VALUES_PER_THREAD; ++j) {
      const int index = thread + j * kWarps * 32;
      const int t = index / BLOCK_COLUMNS, c = index - t * BLOCK_COLUMNS;
      if (t < CHUNK) staged[t * ROW + 2 * PADDED + 4 + c] = entering(to_float(next_v[j]), activated);
    }
  };
  fetch(start);
  const size_t out_width = (size_t)heads * value_dim;
  for (int from = start; from < end; from += CHUNK) {
    const int count = min(CHUNK, end - from);
    __syncthreads();                                             // the chunk before has been read
    commit(from);
    __syncthreads();
    if (from + CHUNK < end) fetch(from + CHUNK);
#pragma unroll 4
    for (int t = 0; t < count; ++t) {
      const float* in = staged + t * ROW;
      const float value = in[2 * PADDED + 4 + local_column];
      float read[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int m = 0; m < PER; m += 4) {
        const int i = (m / 4 * kLanes + l) * 4;
        const float4 query = *reinterpret_cast<const float4*>(in + i);
        const float4 key = *reinterpret_cast<const float4*>(in + PADDED + i);
        read[0] = fmaf(s[m], query.x, read[0]);
        read[1] = fmaf(s[m + 1], query.y, read[1]);
        read[2] = fmaf(s[m + 2], query.z, read[2]);
        read[3] = fmaf(s[m + 3], query.w, read[3]);
        s[m] = fmaf(s[m], decay, key.x * value);
        s[m + 1] = fmaf(s[m + 1], decay, key.y * value);
        s[m + 2] = fmaf(s[m + 2], decay, key.z * value);
        s[m + 3] = fmaf(s[m + 3], decay, key.w * value);
      }
      float total = (read[0] + read[1]) + (read[2] + read[3]);
#pragma unroll
      for (int step = 1; step < kLanes; step <<= 1) total += __shfl_xor_sync(0xffffffffu, total, step);
      if (l == 0 && active)
        out[(size_t)(from + t) * out_width + value_at + column] = fmaf(in[2 * PADDED], value, decay * total);
    }
  }
  if (!active) return;
#pragma unroll
  for (int m = 0; m < PER; m += 4) {
    const int i = (m / 4 * kLanes + l) * 4;
    if (wide) {
      if (i < dim) *reinterpret_cast<float4*>(column_state + i) = make_float4(s[m], s[m + 1], s[m + 2], s[m + 3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (i + e < dim) column_state[i + e] = s[m + e];
    }
  }
}

// The staging alone, for steps that bring portions of prompts: one warp per (token, head) writes what `stage_token`
// makes into prepared[token, head, 2 PADDED + 4] (32-bit), so that the walk below has nothing but copies between its
// chunks and no CTA of a head repeats another's rotation.  blockDim (32, kWarps), grid ceil(tokens * heads / kWarps).
template <typename T, int PER_LANE>
__global__ void __launch_bounds__(kWarps * 32)
retention_prepare_kernel(const T* __restrict__ q, const T* __restrict__ k, long long ld,
                         const float* __restrict__ inv_freq, int rotary_dim, float key_scale,
                         const int* __restrict__ positions, float* __restrict__ prepared, int tokens, int heads, int dim,
                         int activated) {
  constexpr int PADDED = 32 * PER_LANE;
  using Inputs = TokenInputs<T, PER_LANE>;
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x;
  const long long unit = (long long)blockIdx.x * kWarps + threadIdx.y;
  if (unit >= (long long)tokens * heads) return;
  const int token = (int)(unit / heads), head = (int)(unit - (long long)token * heads);
  const int position = positions[token];
  if (position < 0) return;                                      // padding
  const int half = rotary_dim / 2;
  float frequency[Inputs::PAIRED];
#pragma unroll
  for (int e = 0; e < Inputs::PAIRED; ++e) frequency[e] = lane + 32 * e < half ? inv_freq[lane + 32 * e] : 0.0f;
  Inputs in;
  load_token(in, q, k, (size_t)token * ld + (size_t)head * dim, true, (float)position, lane, dim, half, rotary_dim);
  stage_token(in, frequency, key_scale, lane, half, rotary_dim, activated, prepared + (size_t)unit * (2 * PADDED + 4));
}

// The walk over prepared rows: the results of retention_scan_kernel, bit for bit (the same lanes, the same order of sums).
// kWarps warps walk, C columns a lane; kFetchWarps more copy the next chunks' q, k, q . k and v into shared memory (three
// stages).  Several tokens' inputs are in registers at a time, their read-outs are summed over the lanes together, and the
// arithmetic goes two numbers an instruction.
// blockDim (32, kWarps + kFetchWarps), grid (rows, heads, ceil(value_dim / (kWarps * 32 / kLanes * C))).
// What bounds it: one walking warp a scheduler, which issues in 0.36 (C = 2) and 0.46 (C = 4) of the cycles and otherwise waits on
// the latency of the operation before and on shared memory, whose data path is 0.46 and 0.41 busy.  One column a lane spends
// four reads of shared memory on 24 operations of the state; with C columns those reads are shared.
template <typename T, int PER, int kLanes, int C>
__global__ void __launch_bounds__((kWarps + kFetchWarps) * 32, 2)
retention_scan_prepared_kernel(const float* __restrict__ prepared, const T* __restrict__ v, long long ld,
                               const float* __restrict__ decays, float* __restrict__ state,
                               const int* __restrict__ query_starts, const int* __restrict__ state_slots,
                               const int* __restrict__ positions, float* __restrict__ out, int heads, int dim,
                               int value_dim, int activated) {
  constexpr int BLOCK_COLUMNS = 32 / kLanes * kWarps * C;
  constexpr int PADDED = kLanes * PER;
  constexpr int PREPARED = 2 * PADDED + 4;                        // q | k | q . k
  constexpr int ROW = PREPARED + BLOCK_COLUMNS;                   // and v of this CTA's columns
  constexpr int CHUNK = PADDED <= 128 ? 16 : 8, STAGES = 3, STAGE = CHUNK * ROW;
  extern __shared__ __align__(16) float staged[];                 // [STAGES][CHUNK][ROW]
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x;
  const int row = blockIdx.x, head = blockIdx.y;
  const int first_column = blockIdx.z * BLOCK_COLUMNS;
  const int start = query_starts[row], end = query_starts[row + 1];
  if (end <= start || positions[start] < 0) return;
  const size_t value_at = (size_t)head * value_dim;
  const int chunks = (end - start + CHUNK - 1) / CHUNK;

  if (threadIdx.y >= kWarps) {                                    // the fetching warps: tokens w, w + kFetchWarps, ... of a chunk
    constexpr int TOKENS = CHUNK / kFetchWarps, VALUES = (BLOCK_COLUMNS + 31) / 32;
    const int mine = threadIdx.y - kWarps;
    T next_v[TOKENS][VALUES];
    auto fetch = [&](int chunk) {                                 // issues the copies; v passes through registers
      const int from = start + chunk * CHUNK;
#pragma unroll
      for (int tt = 0; tt < TOKENS; ++tt) {
        const int t = mine + tt * kFetchWarps;
        const size_t token = from + t;
        const bool there = from + t < end;
        float* to = staged + (chunk % STAGES) * STAGE + t * ROW;
        const float* source = prepared + (token * heads + head) * PREPARED;
#pragma unroll
        for (int i = 0; i < PREPARED; i += 128)
          if (there && i + lane * 4 < PREPARED) copy_async(to + i + lane * 4, source + i + lane * 4, true);
#pragma unroll
        for (int e = 0; e < VALUES; ++e) {
          const int c = e * 32 + lane;
          next_v[tt][e] = there && c < BLOCK_COLUMNS && first_column + c < value_dim ? v[token * ld + value_at + first_column + c] : T(0.0f);
        }
      }
      copy_commit();
    };
    auto commit_values = [&](int chunk) {
      float* to = staged + (chunk % STAGES) * STAGE + mine * ROW + PREPARED + lane;
#pragma unroll
      for (int tt = 0; tt < TOKENS; ++tt)
#pragma unroll
        for (int e = 0; e < VALUES; ++e)
          if (e * 32 + lane < BLOCK_COLUMNS) to[tt * kFetchWarps * ROW + e * 32] = entering(to_float(next_v[tt][e]), activated);
    };
    fetch(0);
    commit_values(0);
    if (chunks > 1) fetch(1); else copy_commit();
    copy_wait<1>();
    __syncthreads();                                              // the first chunk is there
    for (int chunk = 0; chunk < chunks; ++chunk) {                // (into the stage of the chunk that was walked last)
      if (chunk + 1 < chunks) commit_values(chunk + 1);
      if (chunk + 2 < chunks) fetch(chunk + 2); else copy_commit();
      copy_wait<1>();
      __syncthreads();                                            // this chunk has been walked, and the next one is there
    }
    copy_wait<0>();
    return;
  }

  const int l = lane % kLanes;
  const int local_column = (threadIdx.y * (32 / kLanes) + lane / kLanes) * C;
  const int column = first_column + local_column;
  const bool wide = dim % 4 == 0;
  const float decay = decays[head];
  const Pair both_decays = pair_from(decay, decay);
  float* column_state = state + (((size_t)state_slots[row] * heads + head) * value_dim + column) * dim;
  Pair s[C][PER / 2];
#pragma unroll
  for (int c = 0; c < C; ++c)
    load_column<kLanes, PER>(s[c], column_state + (size_t)c * dim, l, dim, column + c < value_dim, wide);
  struct Inputs {
    Pair q[PER / 2], k[PER / 2];
    float value[C];
  };
  auto load = [&](Inputs& in, const float* from) {
#pragma unroll
    for (int m = 0; m < PER; m += 4) {
      const int i = (m / 4 * kLanes + l) * 4;
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(from + i);
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(from + PADDED + i);
      in.q[m / 2] = a.x; in.q[m / 2 + 1] = a.y;
      in.k[m / 2] = b.x; in.k[m / 2 + 1] = b.y;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) in.value[c] = from[PREPARED + local_column + c];
  };
  auto walk = [&](const Inputs& in, float* parts) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const Pair values = pair_from(in.value[c], in.value[c]);
      Pair read[2] = {0, 0};
#pragma unroll
      for (int m = 0; m < PER / 2; ++m) {
        read[m & 1] = pair_fma(s[c][m], in.q[m], read[m & 1]);
        s[c][m] = pair_fma(s[c][m], both_decays, pair_mul(in.k[m], values));
      }
      parts[c] = pair_total(read);
    }
  };
  // A run of GROUP tokens: their inputs, their walk, then the sums of all their columns at once, each of which ends in a lane of
  // its own that writes it.
  constexpr int GROUP = kLanes / C < 4 ? kLanes / C : 4, SUMS = GROUP * C;
  const size_t out_width = (size_t)heads * value_dim;
  float* const out_of = out + (size_t)start * out_width + value_at + column;
  auto finish = [&](float total, int number, const float* from, int token) {
    const int t = number / C, c = number % C;
    if (column + c < value_dim)
      out_of[(size_t)(token + t) * out_width + c] =
          fmaf(from[t * ROW + 2 * PADDED], from[t * ROW + PREPARED + local_column + c], decay * total);
  };
  __syncthreads();                                                // the first chunk is there
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int count = min(CHUNK, end - start - chunk * CHUNK);
    const float* in = staged + (chunk % STAGES) * STAGE;
    int t = 0;
#pragma unroll 1
    for (; t + GROUP <= count; t += GROUP, in += GROUP * ROW) {
      Inputs inputs[GROUP];
#pragma unroll
      for (int g = 0; g < GROUP; ++g) load(inputs[g], in + g * ROW);
      float parts[SUMS];
#pragma unroll
      for (int g = 0; g < GROUP; ++g) walk(inputs[g], parts + g * C);
      const float total = sum_lanes<kLanes, SUMS>(parts, l);
      if (l < SUMS) finish(total, lane_sum<SUMS>(l), in, chunk * CHUNK + t);
    }
#pragma unroll 1
    for (; t < count; ++t, in += ROW) {
      Inputs inputs;
      load(inputs, in);
      float parts[C];
      walk(inputs, parts);
      const float total = sum_lanes<kLanes, C>(parts, l);
      if (l < C) finish(total, lane_sum<C>(l), in, chunk * CHUNK + t);
    }
    __syncthreads();                                              // this chunk has been walked, and the next one is there
  }
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (column + c < value_dim) store_column<kLanes, PER>(s[c], column_state + (size_t)c * dim, l, dim, wide);
}

template <typename T, int PER, int kLanes, int C>
int launch_walk(cudaStream_t stream, const float* prepared, const void* v, long long ld, const float* decays, float* state,
                const int* query_starts, const int* state_slots, const int* positions, float* out, int rows, int heads,
                int dim, int value_dim, int activated) {
  constexpr int columns = kWarps * (32 / kLanes) * C;
  constexpr int smem = 3 * (kLanes * PER <= 128 ? 16 : 8) * (2 * kLanes * PER + 4 + columns) * (int)sizeof(float);
  const cudaError_t err = cudaFuncSetAttribute(retention_scan_prepared_kernel<T, PER, kLanes, C>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) {
    mir_set_error("retention_scan: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(err));
    return MIR_CUDA_ERROR;
  }
  return mir_launch_alone("retention_scan", retention_scan_prepared_kernel<T, PER, kLanes, C>,
                    dim3(rows, heads, (value_dim + columns - 1) / columns), dim3(32, kWarps + kFetchWarps), smem, stream, 0,
                    prepared, (const T*)v, ld, decays, state, query_starts, state_slots, positions, out, heads, dim,
                    value_dim, activated);
}

template <typename T, int PER, int kLanes>
int launch_prepared(cudaStream_t stream, const void* q, const void* k, const void* v, long long ld, const float* inv_freq,
                    int rotary_dim, const float* decays, float key_scale, float* state, const int* query_starts,
                    const int* state_slots, const int* positions, float* out, float* prepared, int tokens, int rows,
                    int heads, int dim, int value_dim, int activated) {
  const long long units = (long long)tokens * heads;
  int status = mir_launch("retention_prepare", retention_prepare_kernel<T, kLanes * PER / 32>,
                          dim3((unsigned)((units + kWarps - 1) / kWarps)), dim3(32, kWarps), 0, stream, 0, (const T*)q,
                          (const T*)k, ld, inv_freq, rotary_dim, key_scale, positions, prepared, tokens, heads, dim,
                          activated);
  if (status != MIR_OK) return status;
#define MIR_WALK(C)                                                                                                    \
  return launch_walk<T, PER, kLanes, C>(stream, prepared, v, ld, decays, state, query_starts, state_slots, positions, \
                                        out, rows, heads, dim, value_dim, activated)
  // More columns a lane share a token's reads of shared memory; fewer fill the GPU with the heads of few requests: two until their
  // CTAs have to share an SM (1,000 tokens, heads of 128, two / four columns: 16 heads, 128 CTAs, 113 / 133 us; 20 heads, 160
  // CTAs, 152 / 136; heads of 64: 36 heads, 144 CTAs, 91 / 105, 40 heads, 160 CTAs, 116 / 106).
  const int narrow = kWarps * (32 / kLanes) * 2;                  // columns of a CTA with two a lane
  if constexpr (PER <= 8)
    if ((long long)rows * heads * ((value_dim + narrow - 1) / narrow) > mir_sm_count()) MIR_WALK(4);
  MIR_WALK(2);
#undef MIR_WALK
}

template <typename T, int PER, int kLanes, bool SHORT>
int launch_scan(cudaStream_t stream, const void* q, const void* k, const void* v, long long ld, const float* inv_freq,
                int rotary_dim, const float* decays, float key_scale, float* state, const int* query_starts,
                const int* state_slots, const int* positions, float* out, int rows, int heads, int dim, int value_dim,
                int activated) {
  constexpr int columns = kWarps * (32 / kLanes);
  return mir_launch("retention_scan", retention_scan_kernel<T, PER, kLanes, SHORT>,
                    dim3(rows, heads, (value_dim + columns - 1) / columns), dim3(32, kWarps), 0, stream, 0, (const T*)q,
                    (const T*)k, (const T*)v, ld, inv_freq, rotary_dim, decays, key_scale, state, query_starts,
                    state_slots, positions, out, heads, dim, value_dim, activated);
}

template <typename T>
int launch_scan_for(cudaStream_t stream, const void* q, const void* k, const void* v, long long ld,
                    const float* inv_freq, int rotary_dim, const float* decays, float key_scale, float* state,
                    const int* query_starts, const int* state_slots, const int* positions, float* out, int rows,
                    int heads, int dim, int value_dim, bool single_tokens, float* prepared, int tokens, int activated) {
#define MIR_RETENTION(P, L)                                                                                         \
  if (prepared && !single_tokens)                                                                                   \
    return launch_prepared<T, P, L>(stream, q, k, v, ld, inv_freq, rotary_dim, decays, key_scale, state,           \
                                    query_starts, state_slots, positions, out, prepared, tokens, rows, heads, dim,  \
                                    value_dim, activated);                                                          \
  if (single_tokens)                                                                                                \
    return launch_scan<T, P, L, true>(stream, q, k, v, ld, inv_freq, rotary_dim, decays, key_scale, state,         \
                                      query_starts, state_slots, positions, out, rows, heads, dim, value_dim, activated); \
  return launch_scan<T, P, L, false>(stream, q, k, v, ld, inv_freq, rotary_dim, decays, key_scale, state,          \
                                     query_starts, state_slots, positions, out, rows, heads, dim, value_dim, activated);
  if (dim <= 32) { MIR_RETENTION(4, 8) }
  if (dim <= 64) { MIR_RETENTION(4, 16) }
  if (dim <= 128) { MIR_RETENTION(8, 16) }
  if (dim <= 192) { MIR_RETENTION(12, 16) }
  if (dim <= 256) { MIR_RETENTION(16, 16) }
#undef MIR_RETENTION
  mir_set_error("retention_scan: heads of %d key channels are wider than 256", dim);
  return MIR_BAD_ARGUMENT;
}

}  // namespace

// q, k [tokens, heads * dim] and v [tokens, heads * value_dim] with one row stride ld in the activations' type (views
// of one packed projection); inv_freq [rotary_dim / 2] 32-bit (may be null with rotary_dim 0); decays [heads] 32-bit;
// state [slots, heads, value_dim, dim] 32-bit; out [tokens, heads * value_dim] 32-bit: o before the head norm.
// prepared: null, or 32-bit scratch of tokens * heads * (2 * padded + 4) numbers, padded = the key width rounded up to
// 32, 64, 128, 192 or 256: a step that brings more than single tokens then rotates in a kernel of its own first.
// activated: silu on q, k and v as they enter.
MIR_EXPORT int mir_retention_scan(int bf16, const void* q, const void* k, const void* v, long long ld,
                                  const float* inv_freq, int rotary_dim, const float* decays, float key_scale,
                                  float* state, const int* query_starts, const int* state_slots, const int* positions,
                                  float* out, float* prepared, int tokens, int rows, int heads, int dim, int value_dim,
                                  int activated, cudaStream_t stream) {
  if (tokens == 0 || rows == 0) return MIR_OK;
  if (tokens < 0 || rows < 0 || heads <= 0 || dim <= 0 || value_dim <= 0 || heads > 65535 || rotary_dim < 0 ||
      rotary_dim > dim || (rotary_dim & 1) || (rotary_dim > 0 && inv_freq == nullptr)) {
    mir_set_error("retention_scan: bad sizes (tokens %d, rows %d, heads %d, dim %d, value_dim %d, rotary_dim %d)",
                  tokens, rows, heads, dim, value_dim, rotary_dim);
    return MIR_BAD_ARGUMENT;
  }
  const bool single_tokens = tokens == rows;                     // a step of decoded tokens: every row brings one
  if (bf16)
    return launch_scan_for<__nv_bfloat16>(stream, q, k, v, ld, inv_freq, rotary_dim, decays, key_scale, state,
                                          query_starts, state_slots, positions, out, rows, heads, dim, value_dim,
                                          single_tokens, prepared, tokens, activated);
  return launch_scan_for<float>(stream, q, k, v, ld, inv_freq, rotary_dim, decays, key_scale, state, query_starts,
                                state_slots, positions, out, rows, heads, dim, value_dim, single_tokens, prepared, tokens,
                                activated);
}
