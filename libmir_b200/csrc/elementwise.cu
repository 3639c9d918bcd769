// Embedding gather, RMSNorm, SiLU-gate and bias kernels.  The residual stream is 32-bit in both
// engine dtypes; T is the storage type of weights and activations (float or bf16).
//
// What each replaces in libmir: embedding_bf16.cu:3-19, rms_norm_bf16.cu:3-36,
// elementwise_bf16.cu:42-70 (packed gate|up), select_row_bf16.cu (row gather, folded into the norm).
#include <cuda_fp16.h>
#include "common.cuh"

using namespace mir;

// out[r, :] = float(table[ids[r], :]) * scale.  An id outside [0, vocab) gives a row of zeros;
// the host rejects such ids before the launch.
template <typename T>
__global__ void embed_kernel(const T* __restrict__ table, const int* __restrict__ ids, float* __restrict__ out,
                             int hidden, int vocab, float scale) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x;
  const int id = ids[row];
  const bool ok = id >= 0 && id < vocab;
  const T* src = table + (size_t)(ok ? id : 0) * hidden;
  float* dst = out + (size_t)row * hidden;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) dst[c] = ok ? to_float(src[c]) * scale : 0.0f;
}

// The same, 16 bytes of the table a thread (hidden a multiple of 8, rows on 16-byte boundaries): one load a thread for bfloat16
// rows of up to 4,096 (2 rows of 4,096: 8.5 us column by column).
template <typename T>
__global__ void __launch_bounds__(512) embed_wide_kernel(const T* __restrict__ table, const int* __restrict__ ids,
                                                         float* __restrict__ out, int hidden, int vocab, float scale) {
  constexpr int V = 16 / sizeof(T);
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x;
  const int id = ids[row];
  const bool ok = id >= 0 && id < vocab;
  const T* src = table + (size_t)(ok ? id : 0) * hidden;
  float* dst = out + (size_t)row * hidden;
  for (int c = threadIdx.x * V; c < hidden; c += blockDim.x * V) {
    float v[V];
    if constexpr (V == 8) load8(src + c, v);
    else *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src + c);
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = ok ? v[i] * scale : 0.0f;
#pragma unroll
    for (int i = 0; i < V; i += 4) reinterpret_cast<float4*>(dst + c)[i / 4] = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
  }
}

// out[r, :] = float(table[ids[r], :]) * scale + float(pairs[bucket(r), :]): a second table indexed by a hash of the
// token and the token before it in its request, bucket = (previous * mul_previous + id * mul_current) mod buckets;
// a request's first token (previous < 0) takes row `buckets`, the table's last.
template <typename T>
__global__ void embed_pairs_kernel(const T* __restrict__ table, const T* __restrict__ pairs, const int* __restrict__ ids,
                                   const int* __restrict__ previous, float* __restrict__ out, int hidden, int vocab,
                                   int buckets, long long mul_previous, long long mul_current, float scale) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x;
  const int id = ids[row];
  const int before = previous[row];
  const bool ok = id >= 0 && id < vocab;
  const long long bucket = before < 0 ? (long long)buckets
                                      : (((long long)before * mul_previous + (long long)id * mul_current) % buckets + buckets) % buckets;
  const T* src = table + (size_t)(ok ? id : 0) * hidden;
  const T* pair = pairs + (size_t)bucket * hidden;
  float* dst = out + (size_t)row * hidden;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x)
    dst[c] = ok ? to_float(src[c]) * scale + to_float(pair[c]) : 0.0f;
}

// x <- 0.5 x (1 + tanh(sqrt(2 / pi) (x + 0.044715 x^3))), in place.
template <typename T>
__global__ void gelu_tanh_kernel(T* __restrict__ x, size_t total) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total) return;
  const float z = to_float(x[index]);
  const float inner = 0.7978845608028654f * fmaf(0.044715f * z * z, z, z);
  x[index] = from_float<T>(0.5f * z * (1.0f + tanhf(inner)));
}

// Kernels that keep a row in registers: four columns a thread in a few places.  The threads follow from the row's
// width alone, so that a row's result does not depend on how many rows there are.
constexpr int kRowThreads = 512;
inline int row_pieces(int quads) { return (quads + kRowThreads - 1) / kRowThreads; }
inline int row_threads(int quads) {
  const int pieces = row_pieces(quads), each = (quads + pieces - 1) / pieces;
  return (each + 31) / 32 * 32;
}
__device__ __forceinline__ void store_rounded(__nv_bfloat16* row, int quad, float4 v) {
  uint2 packed;
  *reinterpret_cast<__nv_bfloat162*>(&packed.x) = __floats2bfloat162_rn(v.x, v.y);
  *reinterpret_cast<__nv_bfloat162*>(&packed.y) = __floats2bfloat162_rn(v.z, v.w);
  reinterpret_cast<uint2*>(row)[quad] = packed;
}
__device__ __forceinline__ void store_rounded(float* row, int quad, float4 v) { reinterpret_cast<float4*>(row)[quad] = v; }

// residual[r, :] += scale * sum over branches b of branch_b[r, :] * rsqrt(mean(branch_b[r, :]^2) + eps) * weight_b:
// several branch outputs (32-bit rows), each normalised over the model width with a weight of its own, added to the
// residual stream in one pass.  Fixed reduction tree per branch.
struct NormedBranches {
  const float* rows[4];
  const float* weight[4];
  int count;
};
// `rounded` (may be null): the updated residual's rows once more, rounded to bfloat16, for the product that reads them next.
__global__ void add_normed_branches_kernel(NormedBranches branches, float* __restrict__ residual,
                                           __nv_bfloat16* __restrict__ rounded, int hidden, float eps, float scale) {
  __shared__ float scratch[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x;
  float inverse[4];
  for (int b = 0; b < branches.count; ++b) {
    const float* src = branches.rows[b] + (size_t)row * hidden;
    float sum = 0.0f;
    for (int c = threadIdx.x; c < hidden; c += blockDim.x) sum = fmaf(src[c], src[c], sum);
    sum = block_sum(sum, scratch);
    inverse[b] = rsqrtf(sum / (float)hidden + eps);
  }
  float* dst = residual + (size_t)row * hidden;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    float total = 0.0f;
    for (int b = 0; b < branches.count; ++b)
      total += branches.rows[b][(size_t)row * hidden + c] * inverse[b] * branches.weight[b][c];
    const float updated = dst[c] + scale * total;
    dst[c] = updated;
    if (rounded) rounded[(size_t)row * hidden + c] = __float2bfloat16(updated);
  }
}

// The same with 16-byte accesses (hidden a multiple of 4, every pointer 16-byte aligned), for rows wider than the registers of a
// CTA take; the second pass finds the rows in L1 (2,000 rows of 12,288, one branch: 66 us, column by column 170).
__global__ void add_normed_branches_vec4_kernel(NormedBranches branches, float* __restrict__ residual,
                                                __nv_bfloat16* __restrict__ rounded, int hidden, float eps, float scale) {
  __shared__ float scratch[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t base = (size_t)blockIdx.x * hidden;
  const int quads = hidden >> 2;
  float inverse[4];
  for (int b = 0; b < branches.count; ++b) {
    const float4* src = reinterpret_cast<const float4*>(branches.rows[b] + base);
    float sum = 0.0f;
    for (int c = threadIdx.x; c < quads; c += blockDim.x) {
      const float4 v = src[c];
      sum = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, sum))));
    }
    sum = block_sum(sum, scratch);
    inverse[b] = rsqrtf(sum / (float)hidden + eps);
  }
  for (int c = threadIdx.x; c < quads; c += blockDim.x) {
    float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int b = 0; b < branches.count; ++b) {
      const float4 v = reinterpret_cast<const float4*>(branches.rows[b] + base)[c];
      const float4 w = __ldg(reinterpret_cast<const float4*>(branches.weight[b]) + c);
      total.x += v.x * inverse[b] * w.x; total.y += v.y * inverse[b] * w.y;
      total.z += v.z * inverse[b] * w.z; total.w += v.w * inverse[b] * w.w;
    }
    float4 r = reinterpret_cast<float4*>(residual + base)[c];
    r.x += scale * total.x; r.y += scale * total.y; r.z += scale * total.z; r.w += scale * total.w;
    reinterpret_cast<float4*>(residual + base)[c] = r;
    if (rounded) store_rounded(rounded + base, c, r);
  }
}

// The same with the row of every branch in registers, read once, four columns a thread in PIECES places; the residual and the
// weights are asked for with them, and all branches are summed behind one barrier.  Few rows are bound by these latencies (2 rows of
// 4,096: 8.7 us when the row was read twice and the weights behind the sum), many by their bytes.
template <int BRANCHES, int PIECES, bool EARLY>
__global__ void __launch_bounds__(256) add_normed_branches_row_kernel(
    NormedBranches branches, float* __restrict__ residual, __nv_bfloat16* __restrict__ rounded, int hidden, float eps, float scale) {
  __shared__ float scratch[BRANCHES][32];
  const int quads = hidden >> 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  float4 w[BRANCHES][PIECES], v[BRANCHES][PIECES], old[PIECES];
#pragma unroll
  for (int b = 0; b < BRANCHES; ++b)
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int c = p * blockDim.x + threadIdx.x;
      if (EARLY && c < quads) w[b][p] = __ldg(reinterpret_cast<const float4*>(branches.weight[b]) + c);
    }
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t base = (size_t)blockIdx.x * hidden;
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int c = p * blockDim.x + threadIdx.x;
#pragma unroll
    for (int b = 0; b < BRANCHES; ++b)
      v[b][p] = c < quads ? reinterpret_cast<const float4*>(branches.rows[b] + base)[c] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (c < quads) old[p] = reinterpret_cast<const float4*>(residual + base)[c];
  }
  float inverse[BRANCHES];
#pragma unroll
  for (int b = 0; b < BRANCHES; ++b) {
    float sum = 0.0f;
#pragma unroll
    for (int p = 0; p < PIECES; ++p)
      sum = fmaf(v[b][p].x, v[b][p].x, fmaf(v[b][p].y, v[b][p].y, fmaf(v[b][p].z, v[b][p].z, fmaf(v[b][p].w, v[b][p].w, sum))));
    sum = warp_sum(sum);
    if (lane == 0) scratch[b][warp] = sum;
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < BRANCHES; ++b) inverse[b] = rsqrtf(warp_sum(lane < warps ? scratch[b][lane] : 0.0f) / (float)hidden + eps);
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int c = p * blockDim.x + threadIdx.x;
    if (c >= quads) continue;
    float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int b = 0; b < BRANCHES; ++b) {
      if (!EARLY) w[b][p] = __ldg(reinterpret_cast<const float4*>(branches.weight[b]) + c);
      total.x += v[b][p].x * inverse[b] * w[b][p].x; total.y += v[b][p].y * inverse[b] * w[b][p].y;
      total.z += v[b][p].z * inverse[b] * w[b][p].z; total.w += v[b][p].w * inverse[b] * w[b][p].w;
    }
    float4 r = old[p];
    r.x += scale * total.x; r.y += scale * total.y; r.z += scale * total.z; r.w += scale * total.w;
    reinterpret_cast<float4*>(residual + base)[c] = r;
    if (rounded) store_rounded(rounded + base, c, r);
  }
}

// residual[r, :] = u * rsqrt(mean(u^2) + eps) * weight with u = alpha * residual[r, :] + sum over branches b of
// scale_b * branch_b[r, :]: what stands behind a sublayer whose norm comes after the sum.  One CTA per row, which stays
// in registers between the sum and the norm (V columns a thread and access, PIECES of them blockDim.x * V columns apart).
// `rounded` (may be null): the new rows once more, rounded to bfloat16, for the product that reads them next.
struct ScaledBranches {
  const float* rows[4];
  float scale[4];
  int count;
};
template <int V, int PIECES>
__global__ void __launch_bounds__(512) norm_scaled_sum_kernel(ScaledBranches branches, float* __restrict__ residual,
                                                              const float* __restrict__ weight,
                                                              __nv_bfloat16* __restrict__ rounded, int hidden, float alpha,
                                                              float eps) {
  __shared__ float scratch[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
  const size_t base = (size_t)blockIdx.x * hidden;
  auto load = [](float (&v)[V], const float* from) {
    if constexpr (V == 4) {
      const float4 a = *reinterpret_cast<const float4*>(from);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
      v[0] = *from;
    }
  };
  // one piece a thread (few rows' shortest chain): the weight, older than the kernel before this one, is asked for ahead;
  // more pieces: the registers serve the rows in flight, and the weight comes behind the sum
  constexpr bool kEarly = PIECES == 1;
  float early[V];
  if (kEarly && threadIdx.x * V < hidden) load(early, weight + threadIdx.x * V);
  grid_dependency_wait();
  grid_launch_dependents();
  float u[PIECES][V];
  float sum = 0.0f;
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int c = (p * blockDim.x + threadIdx.x) * V;
#pragma unroll
    for (int v = 0; v < V; ++v) u[p][v] = 0.0f;
    if (c >= hidden) continue;
    load(u[p], residual + base + c);
#pragma unroll
    for (int v = 0; v < V; ++v) u[p][v] *= alpha;
    for (int b = 0; b < branches.count; ++b) {
      float piece[V];
      load(piece, branches.rows[b] + base + c);
#pragma unroll
      for (int v = 0; v < V; ++v) u[p][v] = fmaf(branches.scale[b], piece[v], u[p][v]);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) sum = fmaf(u[p][v], u[p][v], sum);
  }
  sum = warp_sum(sum);
  if (lane == 0) scratch[warp] = sum;
  __syncthreads();
  float total = 0.0f;
  for (int i = 0; i < warps; ++i) total += scratch[i];
  const float inverse = rsqrtf(total / (float)hidden + eps);
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int c = (p * blockDim.x + threadIdx.x) * V;
    if (c >= hidden) continue;
    float w[V];
    if (kEarly) {
#pragma unroll
      for (int v = 0; v < V; ++v) w[v] = early[v];
    } else {
      load(w, weight + c);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) u[p][v] *= inverse * w[v];
    if constexpr (V == 4) {
      *reinterpret_cast<float4*>(residual + base + c) = make_float4(u[p][0], u[p][1], u[p][2], u[p][3]);
      if (rounded) {
        uint2 packed;
        *reinterpret_cast<__nv_bfloat162*>(&packed.x) = __floats2bfloat162_rn(u[p][0], u[p][1]);
        *reinterpret_cast<__nv_bfloat162*>(&packed.y) = __floats2bfloat162_rn(u[p][2], u[p][3]);
        *reinterpret_cast<uint2*>(rounded + base + c) = packed;
      }
    } else {
      residual[base + c] = u[p][0];
      if (rounded) rounded[base + c] = __float2bfloat16(u[p][0]);
    }
  }
}

// out[i] (+)= sum over branches b of scale_b * branch_b[i].
__global__ void scaled_sum_kernel(ScaledBranches branches, float* __restrict__ out, size_t total, int accumulate) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total) return;
  float sum = accumulate ? out[index] : 0.0f;
  for (int b = 0; b < branches.count; ++b) sum = fmaf(branches.scale[b], branches.rows[b][index], sum);
  out[index] = sum;
}

// gelu_tanh on eight bfloat16 values per thread (16-byte accesses).
__global__ void gelu_tanh_bf16x8_kernel(__nv_bfloat16* __restrict__ x, size_t total8) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total8) return;
  float z[8];
  load8(x + index * 8, z);
  uint4 packed;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = z[2 * i], b = z[2 * i + 1];
    h[i] = __floats2bfloat162_rn(0.5f * a * (1.0f + tanhf(0.7978845608028654f * fmaf(0.044715f * a * a, a, a))),
                                 0.5f * b * (1.0f + tanhf(0.7978845608028654f * fmaf(0.044715f * b * b, b, b))));
  }
  *reinterpret_cast<uint4*>(x + index * 8) = packed;
}

// y[r, :] = x[src(r), :] * rsqrt(mean(x^2) + eps) * w, src(r) = rows ? rows[r] : r.
// Sum of squares and scaling in 32-bit with a fixed reduction tree.
template <typename Tout>
__global__ void rms_norm_kernel(const float* __restrict__ x, const float* __restrict__ weight,
                                Tout* __restrict__ out, const int* __restrict__ rows, int hidden, float eps) {
  __shared__ float scratch[32];
  grid_dependency_wait();
  grid_launch_dependents();

  const int row = blockIdx.x;
  const float* src = x + (size_t)(rows ? rows[row] : row) * hidden;
  float sum = 0.0f;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    const float v = src[c];
    sum = fmaf(v, v, sum);
  }
  sum = block_sum(sum, scratch);
  const float inverse = rsqrtf(sum / (float)hidden + eps);
  Tout* dst = out + (size_t)row * hidden;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) dst[c] = from_float<Tout>(src[c] * inverse * weight[c]);
}

// The same with 16-byte loads (hidden a multiple of 4), for rows wider than the registers of a CTA take: the second pass finds
// the row in L1 (2,000 rows of 20,480: 54 us, column by column 119).
template <typename Tout>
__global__ void rms_norm_vec4_kernel(const float* __restrict__ x, const float* __restrict__ weight,
                                     Tout* __restrict__ out, const int* __restrict__ rows, int hidden, float eps) {
  __shared__ float scratch[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x;
  const float4* src = reinterpret_cast<const float4*>(x + (size_t)(rows ? rows[row] : row) * hidden);
  const float4* w4 = reinterpret_cast<const float4*>(weight);
  const int quads = hidden >> 2;
  float sum = 0.0f;
  for (int c = threadIdx.x; c < quads; c += blockDim.x) {
    const float4 v = src[c];
    sum = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, sum))));
  }
  sum = block_sum(sum, scratch);
  const float inverse = rsqrtf(sum / (float)hidden + eps);
  for (int c = threadIdx.x; c < quads; c += blockDim.x) {
    const float4 v = src[c], w = __ldg(w4 + c);
    store_rounded(out + (size_t)row * hidden, c,
                  make_float4(v.x * inverse * w.x, v.y * inverse * w.y, v.z * inverse * w.z, v.w * inverse * w.w));
  }
}

// The same with the row in registers, read once, and the weights (EARLY) asked for with it; with PAIR a second norm of the same
// rows, out_b = x * s * weight_b with the same s.
template <typename Tout, bool PAIR, int PIECES, int THREADS, bool EARLY = true>
__global__ void __launch_bounds__(THREADS) rms_norm_row_kernel(const float* __restrict__ x, const float* __restrict__ weight,
                                                               const float* __restrict__ weight_b, Tout* __restrict__ out,
                                                               Tout* __restrict__ out_b, const int* __restrict__ rows,
                                                               int hidden, float eps) {
  __shared__ float scratch[32];
  const int quads = hidden >> 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  float4 w[PIECES], second[PAIR ? PIECES : 1], v[PIECES];
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int c = p * blockDim.x + threadIdx.x;
    if (!EARLY || c >= quads) continue;
    w[p] = __ldg(reinterpret_cast<const float4*>(weight) + c);
    if (PAIR) second[p] = __ldg(reinterpret_cast<const float4*>(weight_b) + c);
  }
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x;
  const float4* src = reinterpret_cast<const float4*>(x + (size_t)(rows ? rows[row] : row) * hidden);
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int c = p * blockDim.x + threadIdx.x;
    v[p] = c < quads ? src[c] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  float sum = 0.0f;
#pragma unroll
  for (int p = 0; p < PIECES; ++p) sum = fmaf(v[p].x, v[p].x, fmaf(v[p].y, v[p].y, fmaf(v[p].z, v[p].z, fmaf(v[p].w, v[p].w, sum))));
  sum = warp_sum(sum);
  if (lane == 0) scratch[warp] = sum;
  __syncthreads();
  const float inverse = rsqrtf(warp_sum(lane < warps ? scratch[lane] : 0.0f) / (float)hidden + eps);
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int c = p * blockDim.x + threadIdx.x;
    if (c >= quads) continue;
    if (!EARLY) w[p] = __ldg(reinterpret_cast<const float4*>(weight) + c);
    const float4 n = make_float4(v[p].x * inverse, v[p].y * inverse, v[p].z * inverse, v[p].w * inverse);
    store_rounded(out + (size_t)row * hidden, c, make_float4(n.x * w[p].x, n.y * w[p].y, n.z * w[p].z, n.w * w[p].w));
    if (PAIR)
      store_rounded(out_b + (size_t)row * hidden, c,
                    make_float4(n.x * second[p].x, n.y * second[p].y, n.z * second[p].z, n.w * second[p].w));
  }
}
// 256 threads a row (128 below 1,024 columns): more are no faster (2,000 rows of 8,192 15 us, with 512 threads 18; two rows the
// same), and the order of the sum is one for rows in registers and rows that are read twice.  The weights are asked for with a
// row of up to 5,120, and with a wider one where no SM has a second row (two rows of 8,192: 2.5 us, 3.1 behind the sum; 2,000 rows
// 17 and 15).
template <typename Tout>
int launch_rms_norm(const float* x, const float* weight, Tout* out, const int* rows, int n_rows, int hidden, float eps,
                    cudaStream_t stream) {
  const int threads = hidden >= 1024 ? 256 : 128, pieces = ((hidden >> 2) + threads - 1) / threads;
#define MIR_RMS(P)                                                                                                        \
  return mir_launch("rms_norm", P <= 5 || n_rows <= mir_sm_count() ? rms_norm_row_kernel<Tout, false, P, 256, true> \
                                                                   : rms_norm_row_kernel<Tout, false, P, 256, P <= 5>, dim3(n_rows), dim3(threads), 0, stream, 0, x,  \
                    weight, nullptr, out, nullptr, rows, hidden, eps)
  if (pieces == 1) MIR_RMS(1);
  if (pieces == 2) MIR_RMS(2);
  if (pieces == 3) MIR_RMS(3);
  if (pieces == 4) MIR_RMS(4);
  if (pieces == 5) MIR_RMS(5);
  if (pieces <= 8) MIR_RMS(8);
  if (pieces <= 16) MIR_RMS(16);
#undef MIR_RMS
  return mir_launch("rms_norm", rms_norm_vec4_kernel<Tout>, dim3(n_rows), dim3(threads), 0, stream, 0, x, weight, out, rows,
                    hidden, eps);
}
constexpr int kPairLimit = 8 * 4 * kRowThreads;                  // the widest row that the register form of the pair takes
template <typename Tout>
int launch_rms_norm_pair(const float* x, const float* weight, const float* weight_b, Tout* out, Tout* out_b, int n_rows,
                         int hidden, float eps, cudaStream_t stream) {
  const int quads = hidden >> 2, pieces = row_pieces(quads);
#define MIR_RMS(P)                                                                                                        \
  return mir_launch("rms_norm_pair", rms_norm_row_kernel<Tout, true, P, kRowThreads>, dim3(n_rows), dim3(row_threads(quads)), \
                    0, stream, 0, x, weight, weight_b, out, out_b, nullptr, hidden, eps)
  if (pieces == 1) MIR_RMS(1);
  if (pieces == 2) MIR_RMS(2);
  if (pieces <= 4) MIR_RMS(4);
  MIR_RMS(8);
#undef MIR_RMS
}

// out[r, c] = silu(gu[r, c]) * gu[r, inter + c]; gu rows are [gate | up].
template <typename T>
__global__ void silu_mul_kernel(const T* __restrict__ gu, T* __restrict__ out, int inter, size_t total) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total) return;
  const size_t row = index / inter;
  const int col = (int)(index - row * inter);
  const float g = to_float(gu[row * 2 * inter + col]);
  const float u = to_float(gu[row * 2 * inter + inter + col]);
  out[index] = from_float<T>(g / (1.0f + expf(-g)) * u);
}

// The same, 8 columns per thread with 16-byte loads and stores (inter a multiple of 8, bf16).
__global__ void silu_mul_bf16x8_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                                       int inter, size_t total8) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total8) return;
  const int per_row = inter / 8;
  const size_t row = index / per_row;
  const int col = (int)(index - row * per_row) * 8;
  float g[8], u[8];
  load8(gu + row * 2 * inter + col, g);
  load8(gu + row * 2 * inter + inter + col, u);
  uint4 packed;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    h[i] = __floats2bfloat162_rn(g[2 * i] / (1.0f + expf(-g[2 * i])) * u[2 * i],
                                 g[2 * i + 1] / (1.0f + expf(-g[2 * i + 1])) * u[2 * i + 1]);
  *reinterpret_cast<uint4*>(out + row * inter + col) = packed;
}

// x[r, c] += bias[c]  (32-bit residual; used when a projection that accumulates into the residual has a bias).
template <typename T>
__global__ void add_bias_kernel(float* __restrict__ x, const T* __restrict__ bias, int cols, size_t total) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total) return;
  x[index] += to_float(bias[index % cols]);
}

// dst[i] = T(src[i]) for the load-time casts (dense_cast.cu:4-18) and for copying logits rows.
template <typename Tin, typename Tout>
__global__ void cast_kernel(const Tin* __restrict__ src, Tout* __restrict__ dst, size_t total) {
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index < total) dst[index] = from_float<Tout>(to_float(src[index]));
}

// A thread for each of `total` elements.
template <typename... KernelArgs, typename... Args>
int launch_each(const char* what, void (*kernel)(KernelArgs...), size_t total, cudaStream_t stream, Args... args) {
  if (total == 0) return MIR_OK;
  return mir_launch(what, kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, 0, args...);
}

// The same for what writes weights: not released early, since the kernels that stream weights ask for them before they wait.
#define LAUNCH_1D(kernel, total, ...)                                                      \
  do {                                                                                     \
    const size_t n_ = (total);                                                             \
    if (n_ == 0) return MIR_OK;                                                            \
    kernel<<<(unsigned)((n_ + 255) / 256), 256, 0, stream>>>(__VA_ARGS__);                 \
  } while (0)

MIR_EXPORT int mir_embed(int bf16, const void* table, const int* ids, float* out, int rows, int hidden, int vocab,
                         float scale, cudaStream_t stream) {
  if (rows == 0) return MIR_OK;
  if (rows < 0 || hidden <= 0 || vocab <= 0) { mir_set_error("embed: bad sizes"); return MIR_BAD_ARGUMENT; }
  if (hidden % 8 == 0 && (((uintptr_t)table | (uintptr_t)out) & 15) == 0) {
    const int threads = row_threads(bf16 ? hidden / 8 : hidden / 4);
    if (bf16)
      return mir_launch("embed", embed_wide_kernel<__nv_bfloat16>, dim3(rows), dim3(threads), 0, stream, 0,
                        (const __nv_bfloat16*)table, ids, out, hidden, vocab, scale);
    return mir_launch("embed", embed_wide_kernel<float>, dim3(rows), dim3(threads), 0, stream, 0, (const float*)table, ids, out,
                      hidden, vocab, scale);
  }
  if (bf16)
    return mir_launch("embed", embed_kernel<__nv_bfloat16>, dim3(rows), dim3(256), 0, stream, 0,
                      (const __nv_bfloat16*)table, ids, out, hidden, vocab, scale);
  return mir_launch("embed", embed_kernel<float>, dim3(rows), dim3(256), 0, stream, 0, (const float*)table, ids, out,
                    hidden, vocab, scale);
}

MIR_EXPORT int mir_embed_pairs(int bf16, const void* table, const void* pairs, const int* ids, const int* previous,
                               float* out, int rows, int hidden, int vocab, int buckets, long long mul_previous,
                               long long mul_current, float scale, cudaStream_t stream) {
  if (rows == 0) return MIR_OK;
  if (rows < 0 || hidden <= 0 || vocab <= 0 || buckets <= 0) { mir_set_error("embed_pairs: bad sizes"); return MIR_BAD_ARGUMENT; }
  if (bf16)
    return mir_launch("embed_pairs", embed_pairs_kernel<__nv_bfloat16>, dim3(rows), dim3(256), 0, stream, 0,
                      (const __nv_bfloat16*)table, (const __nv_bfloat16*)pairs, ids, previous, out, hidden, vocab,
                      buckets, mul_previous, mul_current, scale);
  return mir_launch("embed_pairs", embed_pairs_kernel<float>, dim3(rows), dim3(256), 0, stream, 0, (const float*)table,
                    (const float*)pairs, ids, previous, out, hidden, vocab, buckets, mul_previous, mul_current, scale);
}

// x <- act(x) in place: kind 1 the exact GELU 0.5 x (1 + erf(x / sqrt 2)), kind 2 tanh, kind 3 the square of relu;
// computed in 32-bit.
template <typename T>
__global__ void activation_kernel(T* __restrict__ x, size_t total, int kind) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total) return;
  const float z = to_float(x[index]);
  const float positive = fmaxf(z, 0.0f);
  x[index] = from_float<T>(kind == 1 ? 0.5f * z * (1.0f + erff(z * 0.70710678118654752f))
                                     : (kind == 2 ? tanhf(z) : positive * positive));
}

// x <- cap * tanh(x / cap) on 32-bit logits.
__global__ void softcap_kernel(float* __restrict__ x, size_t total, float cap) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index < total) x[index] = cap * tanhf(x[index] / cap);
}

// residual[r, :] += rows[r, :] (if given) + vector (if given): what a pass of a looped run of layers starts with.
__global__ void add_rows_kernel(float* __restrict__ residual, const float* __restrict__ rows,
                                const float* __restrict__ vector, int hidden, size_t total) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total) return;
  float v = residual[index];
  if (rows != nullptr) v += rows[index];
  if (vector != nullptr) v += vector[index % hidden];
  residual[index] = v;
}

// Two norms of the same rows: out_a = x * s * weight_a, out_b = x * s * weight_b with one s = rsqrt(mean(x^2) + eps).
template <typename Tout>
__global__ void rms_norm_pair_kernel(const float* __restrict__ x, const float* __restrict__ weight_a,
                                     const float* __restrict__ weight_b, Tout* __restrict__ out_a,
                                     Tout* __restrict__ out_b, int hidden, float eps) {
  __shared__ float scratch[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x;
  const float* src = x + (size_t)row * hidden;
  float sum = 0.0f;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    const float v = src[c];
    sum = fmaf(v, v, sum);
  }
  sum = block_sum(sum, scratch);
  const float inverse = rsqrtf(sum / (float)hidden + eps);
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    const float v = src[c] * inverse;
    out_a[(size_t)row * hidden + c] = from_float<Tout>(v * weight_a[c]);
    out_b[(size_t)row * hidden + c] = from_float<Tout>(v * weight_b[c]);
  }
}

MIR_EXPORT int mir_gelu_tanh(int bf16, void* x, size_t total, cudaStream_t stream) {
  if (bf16 && total % 8 == 0 && ((uintptr_t)x & 15) == 0) return launch_each("gelu_tanh", gelu_tanh_bf16x8_kernel, total / 8, stream, x, total / 8);
  if (bf16) return launch_each("gelu_tanh", gelu_tanh_kernel<__nv_bfloat16>, total, stream, x, total);
  return launch_each("gelu_tanh", gelu_tanh_kernel<float>, total, stream, x, total);
}

// rows_b, weight_b: `count` (1 to 4) pointers each, to 32-bit [rows, hidden] and [hidden].  rounded: null, or bfloat16
// [rows, hidden] that receives the updated residual.
MIR_EXPORT int mir_add_normed_branches(const float* const* branch_rows, const float* const* branch_weights, int count,
                                       float* residual, void* rounded, int rows, int hidden, float eps, float scale,
                                       cudaStream_t stream) {
  if (rows == 0) return MIR_OK;
  if (rows < 0 || hidden <= 0 || count < 1 || count > 4) { mir_set_error("add_normed_branches: bad sizes"); return MIR_BAD_ARGUMENT; }
  NormedBranches branches = {};
  branches.count = count;
  for (int b = 0; b < count; ++b) { branches.rows[b] = branch_rows[b]; branches.weight[b] = branch_weights[b]; }
  bool aligned = (hidden & 3) == 0 && ((uintptr_t)residual & 15) == 0 && ((uintptr_t)rounded & 7) == 0;
  for (int b = 0; b < count; ++b)
    aligned = aligned && ((uintptr_t)branch_rows[b] & 15) == 0 && ((uintptr_t)branch_weights[b] & 15) == 0;
  // 256 threads a row (128 below 4,096 columns), so that two CTAs and more share an SM and three or four branches do not spill
  // (2,000 rows of 2,048, four branches, with 512 threads: 65 us); the order of the sums is the same in both forms.  The
  // weights are asked for with the rows while both take 100 registers at most, and 224 where no SM has a second row (two rows
  // of 8,192, two branches: 3.4 us, 4.5 behind the sums; 2,000 rows 53 and 46).
  const int threads_of_row = hidden >= 4096 ? 256 : 128, pieces = ((hidden >> 2) + threads_of_row - 1) / threads_of_row;
#define MIR_NORMED(B, P)                                                                                             \
  return mir_launch("add_normed_branches", rows <= mir_sm_count() ? add_normed_branches_row_kernel<B, P, (2 * B + 1) * P * 4 <= 224> \
                                                                  : add_normed_branches_row_kernel<B, P, (2 * B + 1) * P * 4 <= 100>, \
                    dim3(rows), dim3(threads_of_row), 0, stream, 0, branches, residual, (__nv_bfloat16*)rounded, hidden, eps, scale)
  if (aligned && count == 1) {
    if (pieces == 1) MIR_NORMED(1, 1);
    if (pieces == 2) MIR_NORMED(1, 2);
    if (pieces <= 4) MIR_NORMED(1, 4);
    if (pieces <= 5) MIR_NORMED(1, 5);
    if (pieces <= 8) MIR_NORMED(1, 8);
    if (pieces <= 16) MIR_NORMED(1, 16);
  }
  if (aligned && count == 2) {
    if (pieces <= 2) MIR_NORMED(2, 2);
    if (pieces <= 4) MIR_NORMED(2, 4);
    if (pieces <= 5) MIR_NORMED(2, 5);
    if (pieces <= 8) MIR_NORMED(2, 8);
  }
  if (aligned && count == 3 && pieces <= 5) MIR_NORMED(3, 5);
  if (aligned && count == 3 && pieces <= 8) MIR_NORMED(3, 8);
  if (aligned && count == 4 && pieces <= 5) MIR_NORMED(4, 5);
  if (aligned && count == 4 && pieces <= 8) MIR_NORMED(4, 8);
  if (aligned)
    return mir_launch("add_normed_branches", add_normed_branches_vec4_kernel, dim3(rows), dim3(threads_of_row), 0, stream, 0,
                      branches, residual, (__nv_bfloat16*)rounded, hidden, eps, scale);
#undef MIR_NORMED
  const int threads = hidden >= 2048 ? 512 : 256;
  return mir_launch("add_normed_branches", add_normed_branches_kernel, dim3(rows), dim3(threads), 0, stream, 0, branches,
                    residual, (__nv_bfloat16*)rounded, hidden, eps, scale);
}

// branch_rows: `count` (1 to 4) pointers to 32-bit [rows, hidden]; scales: as many numbers; the rest as
// norm_scaled_sum_kernel says.
MIR_EXPORT int mir_norm_scaled_sum(const float* const* branch_rows, const float* scales, int count, float* residual,
                                   const float* weight, void* rounded, int rows, int hidden, float alpha, float eps,
                                   cudaStream_t stream) {
  if (rows == 0) return MIR_OK;
  if (rows < 0 || hidden <= 0 || count < 1 || count > 4) { mir_set_error("norm_scaled_sum: bad sizes"); return MIR_BAD_ARGUMENT; }
  ScaledBranches branches = {};
  branches.count = count;
  bool aligned = (hidden & 3) == 0 && ((uintptr_t)residual & 15) == 0 && ((uintptr_t)weight & 15) == 0 &&
                 ((uintptr_t)rounded & 7) == 0;
  for (int b = 0; b < count; ++b) {
    branches.rows[b] = branch_rows[b];
    branches.scale[b] = scales[b];
    aligned = aligned && ((uintptr_t)branch_rows[b] & 15) == 0;
  }
#define MIR_NORM_SUM(V, P)                                                                                              \
  return mir_launch("norm_scaled_sum", norm_scaled_sum_kernel<V, P>, dim3(rows), dim3(threads), 0, stream, 0, branches, \
                    residual, weight, (__nv_bfloat16*)rounded, hidden, alpha, eps)
  const int per_thread = aligned ? 4 : 1;
  const int places = (hidden + per_thread - 1) / per_thread;
  // (a prompt's rows: two pieces a thread, twice the loads in flight; a few rows: the shortest chain)
  const int wanted = rows >= 256 ? (places + 1) / 2 : places;
  const int threads = wanted >= 512 ? 512 : (wanted + 31) / 32 * 32;
  const int pieces = (places + threads - 1) / threads;
  if (per_thread == 4) {
    if (pieces <= 1) MIR_NORM_SUM(4, 1);
    if (pieces <= 2) MIR_NORM_SUM(4, 2);
    if (pieces <= 4) MIR_NORM_SUM(4, 4);
    if (pieces <= 8) MIR_NORM_SUM(4, 8);
  } else {
    if (pieces <= 2) MIR_NORM_SUM(1, 2);
    if (pieces <= 8) MIR_NORM_SUM(1, 8);
    if (pieces <= 32) MIR_NORM_SUM(1, 32);
  }
#undef MIR_NORM_SUM
  mir_set_error("norm_scaled_sum: rows of %d numbers are wider than the kernel takes", hidden);
  return MIR_BAD_ARGUMENT;
}

MIR_EXPORT int mir_scaled_sum(const float* const* branch_rows, const float* scales, int count, float* out, size_t total,
                              int accumulate, cudaStream_t stream) {
  if (count < 1 || count > 4) { mir_set_error("scaled_sum: one to four branches"); return MIR_BAD_ARGUMENT; }
  ScaledBranches branches = {};
  branches.count = count;
  for (int b = 0; b < count; ++b) { branches.rows[b] = branch_rows[b]; branches.scale[b] = scales[b]; }
  return launch_each("scaled_sum", scaled_sum_kernel, total, stream, branches, out, total, accumulate);
}

MIR_EXPORT int mir_rms_norm(int bf16, const float* x, const float* weight, void* out, const int* rows, int n_rows,
                            int hidden, float eps, cudaStream_t stream) {
  if (n_rows == 0) return MIR_OK;
  if (n_rows < 0 || hidden <= 0) { mir_set_error("rms_norm: bad sizes"); return MIR_BAD_ARGUMENT; }
  if ((hidden & 3) == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)weight & 15) == 0 && ((uintptr_t)out & 15) == 0) {
    if (bf16) return launch_rms_norm(x, weight, (__nv_bfloat16*)out, rows, n_rows, hidden, eps, stream);
    return launch_rms_norm(x, weight, (float*)out, rows, n_rows, hidden, eps, stream);
  }
  const int threads = hidden >= 2048 ? 512 : 256;
  if (bf16)
    return mir_launch("rms_norm", rms_norm_kernel<__nv_bfloat16>, dim3(n_rows), dim3(threads), 0, stream, 0, x, weight,
                      (__nv_bfloat16*)out, rows, hidden, eps);
  return mir_launch("rms_norm", rms_norm_kernel<float>, dim3(n_rows), dim3(threads), 0, stream, 0, x, weight,
                    (float*)out, rows, hidden, eps);
}

MIR_EXPORT int mir_activation(int kind, int bf16, void* x, size_t total, cudaStream_t stream) {
  if (kind < 1 || kind > 3) { mir_set_error("activation: unknown kind %d", kind); return MIR_BAD_ARGUMENT; }
  const char* name = kind == 1 ? "gelu_erf" : (kind == 2 ? "tanh" : "relu_squared");
  return bf16 ? launch_each(name, activation_kernel<__nv_bfloat16>, total, stream, x, total, kind)
              : launch_each(name, activation_kernel<float>, total, stream, x, total, kind);
}

MIR_EXPORT int mir_softcap(float* x, size_t total, float cap, cudaStream_t stream) {
  if (!(cap > 0.0f)) { mir_set_error("softcap: the cap must be greater than zero"); return MIR_BAD_ARGUMENT; }
  return launch_each("softcap", softcap_kernel, total, stream, x, total, cap);
}

MIR_EXPORT int mir_add_rows(float* residual, const float* rows, const float* vector, int n_rows, int hidden,
                            cudaStream_t stream) {
  if (n_rows < 0 || hidden <= 0) { mir_set_error("add_rows: bad sizes"); return MIR_BAD_ARGUMENT; }
  const size_t total = (size_t)n_rows * hidden;
  return launch_each("add_rows", add_rows_kernel, total, stream, residual, rows, vector, hidden, total);
}

MIR_EXPORT int mir_rms_norm_pair(int bf16, const float* x, const float* weight_a, const float* weight_b, void* out_a,
                                 void* out_b, int n_rows, int hidden, float eps, cudaStream_t stream) {
  if (n_rows == 0) return MIR_OK;
  if (n_rows < 0 || hidden <= 0) { mir_set_error("rms_norm_pair: bad sizes"); return MIR_BAD_ARGUMENT; }
  if ((hidden & 3) == 0 && (((uintptr_t)x | (uintptr_t)weight_a | (uintptr_t)weight_b | (uintptr_t)out_a | (uintptr_t)out_b) & 15) == 0 &&
      hidden <= kPairLimit) {
    if (bf16)
      return launch_rms_norm_pair(x, weight_a, weight_b, (__nv_bfloat16*)out_a, (__nv_bfloat16*)out_b, n_rows, hidden, eps, stream);
    return launch_rms_norm_pair(x, weight_a, weight_b, (float*)out_a, (float*)out_b, n_rows, hidden, eps, stream);
  }
  const int threads = hidden >= 2048 ? 512 : 256;
  if (bf16)
    return mir_launch("rms_norm_pair", rms_norm_pair_kernel<__nv_bfloat16>, dim3(n_rows), dim3(threads), 0, stream, 0, x,
                      weight_a, weight_b, (__nv_bfloat16*)out_a, (__nv_bfloat16*)out_b, hidden, eps);
  return mir_launch("rms_norm_pair", rms_norm_pair_kernel<float>, dim3(n_rows), dim3(threads), 0, stream, 0, x, weight_a,
                    weight_b, (float*)out_a, (float*)out_b, hidden, eps);
}

MIR_EXPORT int mir_silu_mul(int bf16, const void* gu, void* out, int rows, int inter, cudaStream_t stream) {
  if (rows < 0 || inter <= 0) { mir_set_error("silu_mul: bad sizes"); return MIR_BAD_ARGUMENT; }
  const size_t total = (size_t)rows * inter;
  if (bf16 && inter % 8 == 0 && ((uintptr_t)gu & 15) == 0 && ((uintptr_t)out & 15) == 0)
    return launch_each("silu_mul", silu_mul_bf16x8_kernel, total / 8, stream, gu, out, inter, total / 8);
  if (bf16) return launch_each("silu_mul", silu_mul_kernel<__nv_bfloat16>, total, stream, gu, out, inter, total);
  return launch_each("silu_mul", silu_mul_kernel<float>, total, stream, gu, out, inter, total);
}

MIR_EXPORT int mir_add_bias(int bf16, float* x, const void* bias, int rows, int cols, cudaStream_t stream) {
  if (rows < 0 || cols <= 0) { mir_set_error("add_bias: bad sizes"); return MIR_BAD_ARGUMENT; }
  const size_t total = (size_t)rows * cols;
  return bf16 ? launch_each("add_bias", add_bias_kernel<__nv_bfloat16>, total, stream, x, bias, cols, total)
              : launch_each("add_bias", add_bias_kernel<float>, total, stream, x, bias, cols, total);
}

// kind: 0 f32->bf16, 1 bf16->f32, 2 f16->bf16, 3 f16->f32 (what a checkpoint may store, to what the engine keeps).
MIR_EXPORT int mir_cast(int kind, const void* src, void* dst, size_t total, cudaStream_t stream) {
  if (kind == 0) LAUNCH_1D(cast_kernel, total, (const float*)src, (__nv_bfloat16*)dst, total);
  else if (kind == 1) LAUNCH_1D(cast_kernel, total, (const __nv_bfloat16*)src, (float*)dst, total);
  else if (kind == 2) LAUNCH_1D(cast_kernel, total, (const __half*)src, (__nv_bfloat16*)dst, total);
  else if (kind == 3) LAUNCH_1D(cast_kernel, total, (const __half*)src, (float*)dst, total);
  else { mir_set_error("cast: unknown kind %d", kind); return MIR_BAD_ARGUMENT; }
  return mir_check_launch("cast");
}

// Random weights on the device: element i of a tensor is a normal deviate (Box-Muller on two uniforms from the
// SplitMix64 of seed + 2 i and seed + 2 i + 1) times `deviation`: the same for a seed whatever the launch shape.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
template <typename T>
__global__ void random_normal_kernel(T* __restrict__ out, size_t total, unsigned long long seed, float deviation) {
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total) return;
  const unsigned long long a = splitmix64(seed + 2ull * index), b = splitmix64(seed + 2ull * index + 1ull);
  const float u = ((float)(a >> 40) + 0.5f) * (1.0f / 16777216.0f);      // (0, 1)
  const float v = (float)(b >> 40) * (1.0f / 16777216.0f);               // [0, 1)
  out[index] = from_float<T>(deviation * sqrtf(-2.0f * logf(u)) * cospif(2.0f * v));
}

MIR_EXPORT int mir_random_normal(int bf16, void* out, size_t total, unsigned long long seed, float deviation,
                                 cudaStream_t stream) {
  if (bf16) LAUNCH_1D(random_normal_kernel, total, (__nv_bfloat16*)out, total, seed, deviation);
  else LAUNCH_1D(random_normal_kernel, total, (float*)out, total, seed, deviation);
  return mir_check_launch("random_normal");
}

// The fixed-size states of newly admitted requests: zero.  regions[2 n], [2 n + 1]: where the n-th state tensor starts and the
// bytes one request's record takes in it.  One launch for all tensors and up to kSlotsAtOnce requests, whose slots travel in the
// launch: 24 tensors filled one by one cost a prompt 24 launches and a copy before its first kernel.
constexpr int kSlotsAtOnce = 64, kZeroPiece = 64 * 1024;
struct ZeroSlots { int slot[kSlotsAtOnce]; };

__global__ void __launch_bounds__(256) zero_slots_kernel(const long long* __restrict__ regions, ZeroSlots slots) {
  grid_dependency_wait();
  grid_launch_dependents();
  char* base = reinterpret_cast<char*>(regions[2 * blockIdx.y]);
  const long long bytes = regions[2 * blockIdx.y + 1];
  char* record = base + (long long)slots.slot[blockIdx.z] * bytes;
  const long long first = (long long)blockIdx.x * kZeroPiece, last = min(bytes, first + kZeroPiece);
  if (((reinterpret_cast<uintptr_t>(record) | (uintptr_t)bytes) & 15) == 0) {
    for (long long i = first + threadIdx.x * 16; i < last; i += 256 * 16) *reinterpret_cast<uint4*>(record + i) = make_uint4(0, 0, 0, 0);
  } else {
    for (long long i = first + threadIdx.x; i < last; i += 256) record[i] = 0;
  }
}

// ---- decode batches that run as a captured graph -------------------------------------------------
// Before the layers: where each row's new key/value goes, from its position and block table.  A row
// with a negative position is padding (the batch is smaller than the captured size): no cache write.
__global__ void decode_prepare_kernel(const int* __restrict__ positions, const int* __restrict__ block_table,
                                      int table_width, int page_size, int* __restrict__ slot_mapping,
                                      int* __restrict__ context_lens, int rows) {
  grid_dependency_wait();                         // (no early release: what follows reads these numbers before it waits)
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  const int position = positions[row];
  int slot = -1;
  if (position >= 0) {
    const int block = position / page_size;
    const int page = block < table_width ? block_table[(size_t)row * table_width + block] : -1;
    if (page >= 0) slot = page * page_size + position % page_size;
  }
  slot_mapping[row] = slot;
  context_lens[row] = position >= 0 ? position + 1 : 0;
}

// After sampling: the sampled token is the next step's input, positions move on by one, and the token is
// appended to a log so that several steps can run without the host reading each one.
__global__ void decode_advance_kernel(const int* __restrict__ sampled, int* __restrict__ tokens,
                                      int* __restrict__ positions, int* __restrict__ token_log, int log_steps,
                                      int* __restrict__ step_counter, int rows, int* __restrict__ previous) {
  grid_dependency_wait();                         // (no early release: the next step reads the positions before it waits)
  const int step = *step_counter;
  __syncthreads();
  for (int row = threadIdx.x; row < rows; row += blockDim.x) {
    const int token = sampled[row];
    if (previous) previous[row] = tokens[row];      // the token before the next one, for models that look at pairs
    tokens[row] = token;
    if (positions[row] >= 0) positions[row] += 1;
    if (step < log_steps) token_log[(size_t)step * rows + row] = token;
  }
  if (threadIdx.x == 0) *step_counter = step + 1;
}

// regions [states][2] on the device as above, largest: the most bytes a record takes; slots on the host.
MIR_EXPORT int mir_zero_slots(const long long* regions, int states, long long largest, const int* slots, int count,
                              cudaStream_t stream) {
  if (states < 0 || states > 65535 || largest < 0 || count < 0) {
    mir_set_error("zero_slots: bad sizes (states %d, largest %lld, count %d)", states, largest, count);
    return MIR_BAD_ARGUMENT;
  }
  if (states == 0 || largest == 0) return MIR_OK;
  for (int done = 0; done < count; done += kSlotsAtOnce) {
    const int now = min(kSlotsAtOnce, count - done);
    ZeroSlots these = {};
    for (int i = 0; i < now; ++i) these.slot[i] = slots[done + i];
    const int status = mir_launch("zero_slots", zero_slots_kernel, dim3((unsigned)((largest + kZeroPiece - 1) / kZeroPiece), states, now),
                                  dim3(256), 0, stream, 0, regions, these);
    if (status != MIR_OK) return status;
  }
  return MIR_OK;
}

MIR_EXPORT int mir_decode_prepare(const int* positions, const int* block_table, int table_width, int page_size,
                                  int* slot_mapping, int* context_lens, int rows, cudaStream_t stream) {
  if (rows <= 0) return MIR_OK;
  return mir_launch("decode_prepare", decode_prepare_kernel, dim3((rows + 127) / 128), dim3(128), 0, stream, 0,
                    positions, block_table, table_width, page_size, slot_mapping, context_lens, rows);
}

MIR_EXPORT int mir_decode_advance(const int* sampled, int* tokens, int* positions, int* token_log, int log_steps,
                                  int* step_counter, int rows, int* previous, cudaStream_t stream) {
  if (rows <= 0) return MIR_OK;
  return mir_launch("decode_advance", decode_advance_kernel, dim3(1), dim3(256), 0, stream, 0, sampled, tokens,
                    positions, token_log, log_steps, step_counter, rows, previous);
}
