// Kernels of the wkv mixer: time mixing with a matrix state per head, a decay per head and key channel, and a bonus for
// the current token.
//
//   wkv_mix    the five inputs of the projections: mix_s[t] = h[t] + (h[t - 1] - h[t]) * mu_s, with h[t - 1] of a
//              portion's first token taken from the request's state (zeros at its start); a request that brings one
//              token moves its state on in the same kernel, the others in wkv_tail
//   wkv_scan   per head, with S [key channel, value channel] (stored per value channel, a column contiguous):
//                o_t = S^T r_t + (sum_i r_i u_i k_i) v_t;   S <- diag(w_t) S + k_t v_t^T;   w_t = exp(-exp(z_t + w0))
//              (wkv_step for a step of single tokens, with the same operations in the same order)
// The decays, the state and every sum are 32-bit; T is the storage type of the projections' results.
#include "common.cuh"
#include "scan_pairs.cuh"

using namespace mir;

namespace {

constexpr int kMixes = 5;

template <typename T>
__global__ void wkv_mix_kernel(const T* __restrict__ h, long long ld, float* __restrict__ tail,
                               const float* __restrict__ mu, const int* __restrict__ row_of_token,
                               const int* __restrict__ query_starts, const int* __restrict__ state_slots,
                               const int* __restrict__ positions, T* __restrict__ out, int tokens, int width) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int token = blockIdx.x;
  if (positions[token] < 0) return;                              // a padding row of a captured batch
  const int row = row_of_token[token];
  const int start = query_starts[row], end = query_starts[row + 1];
  const T* mine = h + (size_t)token * ld;
  const T* before = token > start ? h + (size_t)(token - 1) * ld : nullptr;
  float* kept = tail + (size_t)state_slots[row] * width;
  const bool alone = end - start == 1;
  // the CTAs of a token (gridDim.y of them, more where a step has few tokens) share its columns out
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < width; c += gridDim.y * blockDim.x) {
    const float x = to_float(mine[c]);
    const float previous = before != nullptr ? to_float(before[c]) : kept[c];
    const float step = previous - x;
#pragma unroll
    for (int s = 0; s < kMixes; ++s)
      out[((size_t)s * tokens + token) * width + c] = from_float<T>(fmaf(step, mu[(size_t)s * width + c], x));
    if (alone) kept[c] = x;
  }
}

// The state's last input of every request that brought more than one token.
template <typename T>
__global__ void wkv_tail_kernel(const T* __restrict__ h, long long ld, float* __restrict__ tail,
                                const int* __restrict__ query_starts, const int* __restrict__ state_slots,
                                const int* __restrict__ positions, int width) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x;
  const int start = query_starts[row], end = query_starts[row + 1];
  if (end - start < 2 || positions[start] < 0) return;
  const T* last = h + (size_t)(end - 1) * ld;
  float* kept = tail + (size_t)state_slots[row] * width;
  for (int c = threadIdx.x; c < width; c += blockDim.x) kept[c] = to_float(last[c]);
}

constexpr int kScanWarps = 4;                                   // that walk
constexpr int kLanes = 8;                                       // lanes that share one column of the state

// What the walk needs of a run of CHUNK tokens of one head, staged in shared memory by kScanWarps warps, warp w the tokens
// w, w + kScanWarps, ...: r, k and the decay exp(-exp(z + w0)) of every channel, the token's bonus term sum_i r_i u_i k_i (the
// same for every column of the head), and v of this CTA's columns.  `fetch` only issues the loads; nothing waits for them
// before `commit`.
template <typename T, int PADDED, int CHUNK, int BLOCK_COLUMNS>
struct Stager {
  static constexpr int ROW = 3 * PADDED + 4 + BLOCK_COLUMNS;     // r | k | decay | bonus term | v of this CTA's columns
  static constexpr int TOKENS_PER_WARP = CHUNK / kScanWarps;
  static constexpr int PER_LANE = PADDED / 32;
  static constexpr int VALUES_PER_THREAD = (CHUNK * BLOCK_COLUMNS + kScanWarps * 32 - 1) / (kScanWarps * 32);
  T next_r[TOKENS_PER_WARP][PER_LANE], next_k[TOKENS_PER_WARP][PER_LANE], next_v[VALUES_PER_THREAD];
  float next_w[TOKENS_PER_WARP][PER_LANE];

  __device__ __forceinline__ void fetch(const T* __restrict__ r, const T* __restrict__ k, const T* __restrict__ v, long long ld,
                                        const float* __restrict__ decay_raw, int from, int count, int warp, int lane,
                                        size_t head_at, int width, int dim, int first_column) {
#pragma unroll
    for (int tt = 0; tt < TOKENS_PER_WARP; ++tt) {
      const int t = warp + tt * kScanWarps;
#pragma unroll
      for (int e = 0; e < PER_LANE; ++e) {
        const int i = lane + 32 * e;
        next_r[tt][e] = T(0.0f); next_k[tt][e] = T(0.0f); next_w[tt][e] = 0.0f;
        if (t < count && i < dim) {
          const size_t source = (size_t)(from + t) * ld + head_at + i;
          next_r[tt][e] = r[source];
          next_k[tt][e] = k[source];
          next_w[tt][e] = decay_raw[(size_t)(from + t) * width + head_at + i];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < VALUES_PER_THREAD; ++j) {
      const int index = warp * 32 + lane + j * kScanWarps * 32;
      const int t = index / BLOCK_COLUMNS, c = index - t * BLOCK_COLUMNS;
      next_v[j] = (t < count && first_column + c < dim) ? v[(size_t)(from + t) * ld + head_at + first_column + c] : T(0.0f);
      // (t may lie beyond the chunk where the chunk has fewer values than there are threads: commit skips those)
    }
  }
  __device__ __forceinline__ void commit(float* staged, const float* __restrict__ decay_bias, const float* __restrict__ bonus,
                                         int count, int warp, int lane, size_t head_at, int dim) const {
#pragma unroll
    for (int tt = 0; tt < TOKENS_PER_WARP; ++tt) {
      const int t = warp + tt * kScanWarps;
      if (t >= count) continue;                                  // (the same for the whole warp)
      float* at = staged + t * ROW;
      float sum = 0.0f;
#pragma unroll
      for (int e = 0; e < PER_LANE; ++e) {
        const int i = lane + 32 * e;
        float ww = 0.0f;
        const float rr = to_float(next_r[tt][e]), kk = to_float(next_k[tt][e]);
        if (i < dim) {
          ww = expf(-expf(next_w[tt][e] + decay_bias[head_at + i]));
          sum = fmaf(rr * bonus[head_at + i], kk, sum);
        }
        at[i] = rr; at[PADDED + i] = kk; at[2 * PADDED + i] = ww;
      }
      sum = warp_sum(sum);
      if (lane == 0) at[3 * PADDED] = sum;
    }
#pragma unroll
    for (int j = 0; j < VALUES_PER_THREAD; ++j) {
      const int index = warp * 32 + lane + j * kScanWarps * 32;
      const int t = index / BLOCK_COLUMNS, c = index - t * BLOCK_COLUMNS;
      if (t < CHUNK) staged[t * ROW + 3 * PADDED + 4 + c] = to_float(next_v[j]);
    }
  }
};

// One token through C columns of the state (lane l of a column holds the key channels 4 (m kLanes + l) .. + 3, m < PER / 4):
// the read-out's parts, and the state after the token.  One lane count and one order of sums for every shape of step.
template <int PER, int C>
struct Token {
  Pair r[PER / 2], k[PER / 2], w[PER / 2];
  float value[C];
  __device__ __forceinline__ void load(const float* from, int l, int local_column) {
    constexpr int PADDED = kLanes * PER;
#pragma unroll
    for (int m = 0; m < PER; m += 4) {
      const int i = (m / 4 * kLanes + l) * 4;
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(from + i);
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(from + PADDED + i);
      const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(from + 2 * PADDED + i);
      r[m / 2] = a.x; r[m / 2 + 1] = a.y;
      k[m / 2] = b.x; k[m / 2 + 1] = b.y;
      w[m / 2] = c.x; w[m / 2 + 1] = c.y;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) value[c] = from[3 * PADDED + 4 + local_column + c];
  }
  __device__ __forceinline__ void walk(Pair (&s)[C][PER / 2], float* parts) const {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const Pair both = pair_from(value[c], value[c]);
      Pair read[2] = {0, 0};
#pragma unroll
      for (int m = 0; m < PER / 2; ++m) {
        read[m & 1] = pair_fma(s[c][m], r[m], read[m & 1]);
        s[c][m] = pair_fma(s[c][m], w[m], pair_mul(k[m], both));
      }
      parts[c] = pair_total(read);
    }
  }
};

// A step of single tokens.  blockDim (32, kScanWarps), grid (rows, heads, ceil(dim / (kScanWarps * 4))): few registers, so that
// all its CTAs are resident at once.
template <typename T, int PER>
__global__ void __launch_bounds__(kScanWarps * 32)
wkv_step_kernel(const T* __restrict__ r, const T* __restrict__ k, const T* __restrict__ v, long long ld,
                const float* __restrict__ decay_raw, const float* __restrict__ decay_bias, const float* __restrict__ bonus,
                float* __restrict__ state, const int* __restrict__ query_starts, const int* __restrict__ state_slots,
                const int* __restrict__ positions, float* __restrict__ out, int heads, int dim) {
  constexpr int BLOCK_COLUMNS = 32 / kLanes * kScanWarps;
  using Stage = Stager<T, kLanes * PER, kScanWarps, BLOCK_COLUMNS>;
  __shared__ __align__(16) float staged[kScanWarps * Stage::ROW];
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x, warp = threadIdx.y, l = lane % kLanes;
  const int row = blockIdx.x, head = blockIdx.y;
  const int first_column = blockIdx.z * BLOCK_COLUMNS;
  const int local_column = warp * (32 / kLanes) + lane / kLanes;
  const int column = first_column + local_column;
  const int start = query_starts[row], end = query_starts[row + 1];
  if (end <= start || positions[start] < 0) return;             // the whole CTA: an empty or padding row
  const bool active = column < dim;
  const int width = heads * dim;
  const size_t head_at = (size_t)head * dim;
  float* column_state = state + (((size_t)state_slots[row] * heads + head) * dim + (active ? column : 0)) * dim;
  Pair s[1][PER / 2];
  load_column<kLanes, PER>(s[0], column_state, l, dim, active, dim % 4 == 0);
  for (int at = start; at < end; ++at) {
    Stage stage;
    stage.fetch(r, k, v, ld, decay_raw, at, 1, warp, lane, head_at, width, dim, first_column);
    if (at > start) __syncthreads();                             // the token before has been read
    stage.commit(staged, decay_bias, bonus, 1, warp, lane, head_at, dim);
    __syncthreads();
    Token<PER, 1> token;
    token.load(staged, l, local_column);
    float parts[1];
    token.walk(s, parts);
    const float total = sum_lanes<kLanes, 1>(parts, l);
    if (l == 0 && active) out[(size_t)at * width + head_at + column] = fmaf(staged[3 * kLanes * PER], token.value[0], total);
  }
  if (active) store_column<kLanes, PER>(s[0], column_state, l, dim, dim % 4 == 0);
}

// What the walk over a portion needs of a token and head, one warp for each: prepared[token, head, 4 PADDED + 4] (32-bit) is
// r | k | decay | v | the bonus term.
template <typename T, int PER_LANE>
__global__ void __launch_bounds__(kScanWarps * 32)
wkv_prepare_kernel(const T* __restrict__ r, const T* __restrict__ k, const T* __restrict__ v, long long ld,
                   const float* __restrict__ decay_raw, const float* __restrict__ decay_bias, const float* __restrict__ bonus,
                   const int* __restrict__ positions, float* __restrict__ prepared, int tokens, int heads, int dim) {
  constexpr int PADDED = 32 * PER_LANE;
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x;
  const long long unit = (long long)blockIdx.x * kScanWarps + threadIdx.y;
  if (unit >= (long long)tokens * heads) return;
  const int token = (int)(unit / heads), head = (int)(unit - (long long)token * heads);
  if (positions[token] < 0) return;                              // padding
  const size_t at = (size_t)token * ld + (size_t)head * dim, of_head = (size_t)head * dim;
  float* row = prepared + (size_t)unit * (4 * PADDED + 4);
  float sum = 0.0f;
#pragma unroll
  for (int e = 0; e < PER_LANE; ++e) {
    const int i = lane + 32 * e;
    float rr = 0.0f, kk = 0.0f, ww = 0.0f, vv = 0.0f;
    if (i < dim) {
      rr = to_float(r[at + i]);
      kk = to_float(k[at + i]);
      vv = to_float(v[at + i]);
      ww = expf(-expf(decay_raw[(size_t)token * heads * dim + of_head + i] + decay_bias[of_head + i]));
      sum = fmaf(rr * bonus[of_head + i], kk, sum);
    }
    row[i] = rr; row[PADDED + i] = kk; row[2 * PADDED + i] = ww; row[3 * PADDED + i] = vv;
  }
  sum = warp_sum(sum);
  if (lane == 0) row[4 * PADDED] = sum;
}

// Portions of prompts: the walk over prepared rows.  kScanWarps warps walk over a request's tokens, C columns a lane;
// kFetchWarps more copy the next chunks' rows into shared memory (three stages), so that the walk has nothing but reads of shared memory and the
// state's arithmetic, two numbers an instruction; several tokens' inputs are in registers at a time and their read-outs
// are summed over the lanes together.
// blockDim (32, kScanWarps + kFetchWarps), grid (rows, heads, ceil(dim / (kScanWarps * 4 C))).
// What bounds it: one walking warp a scheduler, which issues in 0.24 (C = 1) and 0.32 (C = 2) of the cycles and otherwise waits on
// shared memory and on the latency of the operation before; shared memory's data path is 0.57 busy.  C is chosen by the
// launcher.  A prompt of 2,048 tokens with 32 / 64 heads of 64 x 64, the preparation included: 224 / 257 us (640 / 693 when
// the walking warps also formed the decays).
constexpr int kFetchWarps = 4, kChunk = 16, kStages = 3;
template <int PER, int C>
__global__ void __launch_bounds__((kScanWarps + kFetchWarps) * 32, 2)
wkv_scan_kernel(const float* __restrict__ prepared, float* __restrict__ state, const int* __restrict__ query_starts,
                const int* __restrict__ state_slots, const int* __restrict__ positions, float* __restrict__ out, int heads,
                int dim) {
  constexpr int BLOCK_COLUMNS = 32 / kLanes * kScanWarps * C;
  constexpr int PADDED = kLanes * PER;
  constexpr int PREPARED = 4 * PADDED + 4;
  constexpr int ROW = 3 * PADDED + 4 + BLOCK_COLUMNS;            // r | k | decay | bonus term | v of this CTA's columns
  constexpr int STAGE = kChunk * ROW;
  extern __shared__ __align__(16) float staged[];                // [kStages][kChunk][ROW]
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x;
  const int row = blockIdx.x, head = blockIdx.y;
  const int first_column = blockIdx.z * BLOCK_COLUMNS;
  const int start = query_starts[row], end = query_starts[row + 1];
  if (end <= start || positions[start] < 0) return;             // the whole CTA: an empty or padding row
  const int width = heads * dim;
  const size_t head_at = (size_t)head * dim;
  const int chunks = (end - start + kChunk - 1) / kChunk;

  if (threadIdx.y >= kScanWarps) {                              // the fetching warps: tokens w, w + kFetchWarps, ... of a chunk
    const int mine = threadIdx.y - kScanWarps;
    auto fetch = [&](int chunk) {
      const int from = start + chunk * kChunk;
#pragma unroll
      for (int tt = 0; tt < kChunk / kFetchWarps; ++tt) {
        const int t = mine + tt * kFetchWarps;
        if (from + t >= end) break;
        float* to = staged + (chunk % kStages) * STAGE + t * ROW;
        const float* source = prepared + ((size_t)(from + t) * heads + head) * PREPARED;
#pragma unroll
        for (int i = 0; i < 3 * PADDED; i += 128)
          if (3 * PADDED - i >= 128 || i + lane * 4 < 3 * PADDED) copy_async(to + i + lane * 4, source + i + lane * 4, true);
        // the bonus term's piece and the values (a CTA's last columns may lie beyond the padded head: they are not used)
        const int c = lane * 4;
        if (c < BLOCK_COLUMNS + 4) {
          const bool term = c == BLOCK_COLUMNS;
          const int column = min(first_column + c, PADDED - 4);
          copy_async(to + 3 * PADDED + (term ? 0 : 4 + c), source + (term ? 4 * PADDED : 3 * PADDED + column), true);
        }
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

  const int l = lane % kLanes;
  const int local_column = (threadIdx.y * (32 / kLanes) + lane / kLanes) * C;
  const int column = first_column + local_column;
  const bool wide = dim % 4 == 0;
  float* column_state = state + (((size_t)state_slots[row] * heads + head) * dim + column) * dim;
  Pair s[C][PER / 2];
#pragma unroll
  for (int c = 0; c < C; ++c) load_column<kLanes, PER>(s[c], column_state + (size_t)c * dim, l, dim, column + c < dim, wide);
  // A run of GROUP tokens: their inputs, their walk, then the sums of all their columns at once, each of which ends in a lane of
  // its own that writes it.
  constexpr int GROUP = PER > 16 ? 1 : (kLanes / C < 4 ? kLanes / C : 4), SUMS = GROUP * C;
  float* const out_of = out + (size_t)start * width + head_at + column;
  auto finish = [&](float total, int number, const float* from, int token) {
    const int t = number / C, c = number % C;
    if (column + c < dim)
      out_of[(size_t)(token + t) * width + c] =
          fmaf(from[t * ROW + 3 * kLanes * PER], from[t * ROW + 3 * kLanes * PER + 4 + local_column + c], total);
  };
  __syncthreads();                                               // the first chunk is there
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int count = min(kChunk, end - start - chunk * kChunk);
    const float* in = staged + (chunk % kStages) * STAGE;
    int t = 0;
#pragma unroll 1
    for (; t + GROUP <= count; t += GROUP, in += GROUP * ROW) {
      Token<PER, C> tokens[GROUP];
#pragma unroll
      for (int g = 0; g < GROUP; ++g) tokens[g].load(in + g * ROW, l, local_column);
      float parts[SUMS];
#pragma unroll
      for (int g = 0; g < GROUP; ++g) tokens[g].walk(s, parts + g * C);
      const float total = sum_lanes<kLanes, SUMS>(parts, l);
      if (l < SUMS) finish(total, lane_sum<SUMS>(l), in, chunk * kChunk + t);
    }
#pragma unroll 1
    for (; t < count; ++t, in += ROW) {
      Token<PER, C> token;
      token.load(in, l, local_column);
      float parts[C];
      token.walk(s, parts);
      const float total = sum_lanes<kLanes, C>(parts, l);
      if (l < C) finish(total, lane_sum<C>(l), in, chunk * kChunk + t);
    }
    __syncthreads();                                             // this chunk has been walked, and the next one is there
  }
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (column + c < dim) store_column<kLanes, PER>(s[c], column_state + (size_t)c * dim, l, dim, wide);
}

template <int PER, int C>
int launch_walk(cudaStream_t stream, const float* prepared, float* state, const int* query_starts, const int* state_slots,
                const int* positions, float* out, int rows, int heads, int dim) {
  constexpr int columns = kScanWarps * (32 / kLanes) * C;
  constexpr int smem = kStages * kChunk * (3 * kLanes * PER + 4 + columns) * (int)sizeof(float);
  const cudaError_t err = cudaFuncSetAttribute(wkv_scan_kernel<PER, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) {
    mir_set_error("wkv_scan: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(err));
    return MIR_CUDA_ERROR;
  }
  return mir_launch_alone("wkv_scan", wkv_scan_kernel<PER, C>, dim3(rows, heads, (dim + columns - 1) / columns),
                    dim3(32, kScanWarps + kFetchWarps), smem, stream, 0, prepared, state, query_starts, state_slots, positions,
                    out, heads, dim);
}

template <typename T, int PER>
int launch_scan_for(cudaStream_t stream, const void* r, const void* k, const void* v, long long ld,
                    const float* decay_raw, const float* decay_bias, const float* bonus, float* state,
                    const int* query_starts, const int* state_slots, const int* positions, float* out, float* prepared,
                    int tokens, int rows, int heads, int dim, bool single_tokens) {
  if (single_tokens) {
    constexpr int columns = kScanWarps * (32 / kLanes);
    return mir_launch("wkv_scan", wkv_step_kernel<T, PER>, dim3(rows, heads, (dim + columns - 1) / columns),
                      dim3(32, kScanWarps), 0, stream, 0, (const T*)r, (const T*)k, (const T*)v, ld, decay_raw, decay_bias,
                      bonus, state, query_starts, state_slots, positions, out, heads, dim);
  }
  const long long units = (long long)tokens * heads;
  const int status = mir_launch("wkv_prepare", wkv_prepare_kernel<T, kLanes * PER / 32>,
                                dim3((unsigned)((units + kScanWarps - 1) / kScanWarps)), dim3(32, kScanWarps), 0, stream, 0,
                                (const T*)r, (const T*)k, (const T*)v, ld, decay_raw, decay_bias, bonus, positions, prepared,
                                tokens, heads, dim);
  if (status != MIR_OK) return status;
#define MIR_WKV(C)                                                                                                       \
  return launch_walk<PER, C>(stream, prepared, state, query_starts, state_slots, positions, out, rows, heads, dim)
  // More columns a lane share a token's reads of shared memory; fewer fill the GPU with the heads of few requests: one, two or four
  // as the CTAs of one column are up to an SM's worth, up to two, or more (1,000 tokens, heads of 64, one / two / four: 144
  // CTAs 115 / 119 / 159 us, 160 170 / 122 / 160, 288 185 / 136 / 175, 320 328 / 190 / 178).
  if constexpr (PER <= 8) {
    const long long units = (long long)rows * heads * ((dim + 15) / 16);     // CTAs with one column a lane
    if (units > 2LL * mir_sm_count()) MIR_WKV(4);
    if (units > mir_sm_count()) MIR_WKV(2);
  }
  MIR_WKV(1);
#undef MIR_WKV
}

template <typename T>
int launch_scan_width(cudaStream_t stream, const void* r, const void* k, const void* v, long long ld,
                      const float* decay_raw, const float* decay_bias, const float* bonus, float* state,
                      const int* query_starts, const int* state_slots, const int* positions, float* out, float* prepared,
                      int tokens, int rows, int heads, int dim, bool single_tokens) {
#define MIR_WKV(P)                                                                                                    \
  return launch_scan_for<T, P>(stream, r, k, v, ld, decay_raw, decay_bias, bonus, state, query_starts, state_slots,  \
                               positions, out, prepared, tokens, rows, heads, dim, single_tokens)
  if (dim <= 32) MIR_WKV(4);
  if (dim <= 64) MIR_WKV(8);
  if (dim <= 96) MIR_WKV(12);
  if (dim <= 128) MIR_WKV(16);
  if (dim <= 192) MIR_WKV(24);
  if (dim <= 256) MIR_WKV(32);
#undef MIR_WKV
  mir_set_error("wkv_scan: heads of %d channels are wider than 256", dim);
  return MIR_BAD_ARGUMENT;
}

}  // namespace

// h [tokens, width] with row stride ld; tail [slots, width] 32-bit; mu [5, width] 32-bit; out [5, tokens, width].
MIR_EXPORT int mir_wkv_mix(int bf16, const void* h, long long ld, float* tail, const float* mu, const int* row_of_token,
                           const int* query_starts, const int* state_slots, const int* positions, void* out, int tokens,
                           int rows, int width, int single_tokens_only, cudaStream_t stream) {
  if (tokens == 0) return MIR_OK;
  if (tokens < 0 || rows <= 0 || width <= 0) {
    mir_set_error("wkv_mix: bad sizes (tokens %d, rows %d, width %d)", tokens, rows, width);
    return MIR_BAD_ARGUMENT;
  }
  const int threads = width >= 1024 ? 256 : 128;
  // three tokens of 2,048 columns: 9.1 us with one CTA each, a column's loads behind the other's
  const int most = (width + threads - 1) / threads, wanted = (4 * mir_sm_count() + tokens - 1) / tokens;
  const int parts = wanted < 1 ? 1 : (wanted > most ? most : wanted);
  int status;
  if (bf16)
    status = mir_launch("wkv_mix", wkv_mix_kernel<__nv_bfloat16>, dim3(tokens, parts), dim3(threads), 0, stream, 0,
                        (const __nv_bfloat16*)h, ld, tail, mu, row_of_token, query_starts, state_slots, positions,
                        (__nv_bfloat16*)out, tokens, width);
  else
    status = mir_launch("wkv_mix", wkv_mix_kernel<float>, dim3(tokens, parts), dim3(threads), 0, stream, 0, (const float*)h, ld,
                        tail, mu, row_of_token, query_starts, state_slots, positions, (float*)out, tokens, width);
  if (status != MIR_OK || single_tokens_only) return status;
  if (bf16)
    return mir_launch("wkv_tail", wkv_tail_kernel<__nv_bfloat16>, dim3(rows), dim3(threads), 0, stream, 0,
                      (const __nv_bfloat16*)h, ld, tail, query_starts, state_slots, positions, width);
  return mir_launch("wkv_tail", wkv_tail_kernel<float>, dim3(rows), dim3(threads), 0, stream, 0, (const float*)h, ld, tail,
                    query_starts, state_slots, positions, width);
}

// r, k, v [tokens, heads * dim] with row stride ld in the activations' type; decay_raw [tokens, heads * dim] 32-bit
// (the low-rank pair's result), decay_bias and bonus [heads * dim] 32-bit; state [slots, heads, dim (value channel),
// dim (key channel)] 32-bit; out [tokens, heads * dim] 32-bit: o before the head norm.  prepared: 32-bit scratch of tokens *
// heads * (4 padded + 4) numbers, padded = the heads' width rounded up to 32, 64, 96, 128, 192 or 256; not used by a step
// of single tokens (and may be null there).
MIR_EXPORT int mir_wkv_scan(int bf16, const void* r, const void* k, const void* v, long long ld, const float* decay_raw,
                            const float* decay_bias, const float* bonus, float* state, const int* query_starts,
                            const int* state_slots, const int* positions, float* out, float* prepared, int tokens, int rows,
                            int heads, int dim, cudaStream_t stream) {
  if (tokens == 0 || rows == 0) return MIR_OK;
  if (tokens < 0 || rows < 0 || heads <= 0 || dim <= 0 || heads > 65535 || (tokens != rows && prepared == nullptr)) {
    mir_set_error("wkv_scan: bad sizes (tokens %d, rows %d, heads %d, dim %d)", tokens, rows, heads, dim);
    return MIR_BAD_ARGUMENT;
  }
  const bool single_tokens = tokens == rows;                     // a step of decoded tokens: every row brings one
  if (bf16)
    return launch_scan_width<__nv_bfloat16>(stream, r, k, v, ld, decay_raw, decay_bias, bonus, state, query_starts,
                                            state_slots, positions, out, prepared, tokens, rows, heads, dim, single_tokens);
  return launch_scan_width<float>(stream, r, k, v, ld, decay_raw, decay_bias, bonus, state, query_starts, state_slots,
                                  positions, out, prepared, tokens, rows, heads, dim, single_tokens);
}
