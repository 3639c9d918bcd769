// C[M, N] = beta * C + A[M, K] . W[N, K]^T (+ bias[N]) in true 32-bit: plain FMA on CUDA cores, no
// tensor cores and no TF32.  This is the matrix product of the float32 engine.
//
// Each output element is one chain of fmaf over k = 0 .. K-1 in ascending order, so its value does
// not depend on M, on the kernel and tile it falls in or on what else is in the batch.  libmir has no 32-bit
// model path on CUDA (its ProjectionFormat has no F32 member, cuda/src/backend/linear/mod.rs:80-88);
// this kernel exists to show faults that bf16 rounding hides.
//
// Two kernels, both fed by rings of cp.async stages whose rows keep their k order in shared memory, padded by four
// floats so that eight neighbouring rows read as 16-byte pieces meet all banks once:
//   gemm_f32_rows   up to 16 rows of A: bound by reading W once.  A CTA takes 16 rows of W and all of A; a thread owns one
//                   output and walks down k, so the least a product can take is K dependent multiply-adds (four cycles
//                   each, 4.2 us for 2,048), which several CTAs on an SM, each with a ring of four
//                   stages of 128 k that two warps of its own fill, hide behind the reads (3 rows, the products of
//                   a layer of 2,048 with 5,504 inside: 27.6 us on average; all warps filling the ring: 29.5).
//   gemm_f32_tile   more rows: bound by issue slots, 0.76 of them taken by 3.4 warps a scheduler (the multiply-adds' pipe 0.58
//                   busy, shared memory's data path 0.61).  A thread owns TM x TN outputs whose rows and columns lie
//                   (tile / threads) apart, and reads four k of each with one load.
#include "common.cuh"

namespace {

__device__ __forceinline__ void copy_async(float* to, const float* from, int bytes) {     // the rest of 16 bytes is zero
  const unsigned at = (unsigned)__cvta_generic_to_shared(to);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_async_one(float* to, const float* from, bool there) {
  const unsigned at = (unsigned)__cvta_generic_to_shared(to);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at), "l"(from), "r"(there ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// ROWS rows of K-major data from row `row0` and column k0 on into [ROWS][DEPTH + 4]; what lies outside is zero.  WIDE: rows
// start on 16-byte boundaries and k is a multiple of four.
template <int ROWS, int DEPTH, int THREADS, bool WIDE>
__device__ __forceinline__ void load_tile(float* tile, const float* __restrict__ from, int ld, int row0, int rows, int k0, int k,
                                          int thread) {
  if (WIDE) {
    constexpr int PIECES = DEPTH / 4;
    for (int index = thread; index < ROWS * PIECES; index += THREADS) {
      const int r = index / PIECES, kk = (index % PIECES) * 4;
      const bool there = row0 + r < rows && k0 + kk < k;
      copy_async(tile + r * (DEPTH + 4) + kk, there ? from + (size_t)(row0 + r) * ld + k0 + kk : from, there ? 16 : 0);
    }
  } else {
    for (int index = thread; index < ROWS * DEPTH; index += THREADS) {
      const int r = index / DEPTH, kk = index % DEPTH;
      const bool there = row0 + r < rows && k0 + kk < k;
      copy_async_one(tile + r * (DEPTH + 4) + kk, there ? from + (size_t)(row0 + r) * ld + k0 + kk : from, there);
    }
  }
}

__device__ __forceinline__ void finish(float* c, int ldc, const float* bias, float beta, int row, int column, float value) {
  if (bias) value += bias[column];
  float* dst = c + (size_t)row * ldc + column;
  *dst = beta != 0.0f ? fmaf(beta, *dst, value) : value;
}

template <int BM, int BN, int TM, int TN, int DEPTH, int STAGES, bool WIDE>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 3)
gemm_f32_tile_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, const float* __restrict__ bias,
                     float* __restrict__ c, int ldc, int m, int n, int k, float beta) {
  constexpr int ACROSS = BN / TN, DOWN = BM / TM, THREADS = ACROSS * DOWN, ROW = DEPTH + 4;
  extern __shared__ __align__(16) float shared[];
  const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
  const int tx = threadIdx.x % ACROSS, ty = threadIdx.x / ACROSS;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
  const int steps = (k + DEPTH - 1) / DEPTH;
  mir::grid_dependency_wait();
  mir::grid_launch_dependents();
  auto fetch = [&](int step) {
    float* stage = shared + (step % STAGES) * (BM + BN) * ROW;
    load_tile<BM, DEPTH, THREADS, WIDE>(stage, a, lda, row0, m, step * DEPTH, k, threadIdx.x);
    load_tile<BN, DEPTH, THREADS, WIDE>(stage + BM * ROW, w, ldw, col0, n, step * DEPTH, k, threadIdx.x);
  };
#pragma unroll
  for (int step = 0; step < STAGES - 1; ++step) {
    if (step < steps) fetch(step);
    copy_commit();
  }
  for (int step = 0; step < steps; ++step) {
    copy_wait<STAGES - 2>();
    __syncthreads();                               // this stage is there for everybody, and the one before has been read
    if (step + STAGES - 1 < steps) fetch(step + STAGES - 1);
    copy_commit();
    const float* at = shared + (step % STAGES) * (BM + BN) * ROW + ty * ROW;
    const float* wt = shared + (step % STAGES) * (BM + BN) * ROW + (BM + tx) * ROW;
    float4 av[2][TM], wv[2][TN];                   // the next four k are read while these four are multiplied
    auto read = [&](int buffer, int kk) {
#pragma unroll
      for (int i = 0; i < TM; ++i) av[buffer][i] = *reinterpret_cast<const float4*>(at + i * DOWN * ROW + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j) wv[buffer][j] = *reinterpret_cast<const float4*>(wt + j * ACROSS * ROW + kk);
    };
    read(0, 0);
#pragma unroll
    for (int kk = 0; kk < DEPTH; kk += 4) {
      const int buffer = kk / 4 & 1;
      if (kk + 4 < DEPTH) read(buffer ^ 1, kk + 4);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          acc[i][j] = fmaf(av[buffer][i].x, wv[buffer][j].x, acc[i][j]);
          acc[i][j] = fmaf(av[buffer][i].y, wv[buffer][j].y, acc[i][j]);
          acc[i][j] = fmaf(av[buffer][i].z, wv[buffer][j].z, acc[i][j]);
          acc[i][j] = fmaf(av[buffer][i].w, wv[buffer][j].w, acc[i][j]);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int row = row0 + ty + i * DOWN;
    if (row >= m) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int column = col0 + tx + j * ACROSS;
      if (column < n) finish(c, ldc, bias, beta, row, column, acc[i][j]);
    }
  }
}

constexpr int kRowsColumns = 16, kRowsDepth = 128, kRowsStages = 4, kRowsThreads = 128, kRowsLoaders = 64, kRun = 4;

// MT: rows of A rounded up to a power of two (1 to 16).  With MT = 16 a thread owns two outputs.
template <int MT, bool WIDE>
__global__ void __launch_bounds__(kRowsThreads + kRowsLoaders, 3)
gemm_f32_rows_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, const float* __restrict__ bias,
                     float* __restrict__ c, int ldc, int m, int n, int k, float beta) {
  constexpr int ROW = kRowsDepth + 4, STAGE = (kRowsColumns + MT) * ROW;
  constexpr int EACH = MT * kRowsColumns > kRowsThreads ? MT * kRowsColumns / kRowsThreads : 1;
  constexpr int DOWN = MT / EACH;
  extern __shared__ __align__(16) float shared[];
  const int col0 = blockIdx.x * kRowsColumns;
  const int tx = threadIdx.x % kRowsColumns, ty = threadIdx.x / kRowsColumns;
  const bool owner = ty < DOWN;
  float acc[EACH];
#pragma unroll
  for (int e = 0; e < EACH; ++e) acc[e] = 0.0f;
  const int steps = (k + kRowsDepth - 1) / kRowsDepth;
  mir::grid_launch_dependents();
  if (threadIdx.x >= kRowsThreads) {               // two warps fetch: the others' chain of multiply-adds is not interrupted
    const int thread = threadIdx.x - kRowsThreads;
    auto fetch_weights = [&](int step) {
      if (step < steps)
        load_tile<kRowsColumns, kRowsDepth, kRowsLoaders, WIDE>(shared + (step % kRowsStages) * STAGE, w, ldw, col0, n,
                                                                step * kRowsDepth, k, thread);
    };
    auto fetch_rows = [&](int step) {
      if (step < steps)
        load_tile<MT, kRowsDepth, kRowsLoaders, WIDE>(shared + (step % kRowsStages) * STAGE + kRowsColumns * ROW, a, lda, 0, m,
                                                      step * kRowsDepth, k, thread);
    };
    auto fetch = [&](int step) {
      fetch_weights(step);
      fetch_rows(step);
      copy_commit();
    };
    // the weights belong to no kernel: the ring's are on their way before the kernel in front is over
#pragma unroll
    for (int step = 0; step < kRowsStages - 1; ++step) fetch_weights(step);
    mir::grid_dependency_wait();
#pragma unroll
    for (int step = 0; step < kRowsStages - 1; ++step) {
      fetch_rows(step);
      copy_commit();
    }
    copy_wait<kRowsStages - 2>();
    __syncthreads();                               // the first stage is there
    for (int step = 0; step < steps; ++step) {     // (into the stage that was multiplied last)
      fetch(step + kRowsStages - 1);
      copy_wait<kRowsStages - 2>();
      __syncthreads();                             // this stage has been read, and the next one is there
    }
    copy_wait<0>();
    return;
  }
  __syncthreads();
  for (int step = 0; step < steps; ++step) {
    const float* wt = shared + (step % kRowsStages) * STAGE + tx * ROW;
    const float* at = shared + (step % kRowsStages) * STAGE + (kRowsColumns + ty) * ROW;
    // Runs of kRun pieces of four k, the next run's reads on their way while this one's chain of multiply-adds goes on.
    float4 wv[2][kRun], av[2][EACH][kRun];
    auto read = [&](int buffer, int kk) {
#pragma unroll
      for (int i = 0; i < kRun; ++i) {
        wv[buffer][i] = *reinterpret_cast<const float4*>(wt + kk + 4 * i);
#pragma unroll
        for (int e = 0; e < EACH; ++e) av[buffer][e][i] = *reinterpret_cast<const float4*>(at + e * DOWN * ROW + kk + 4 * i);
      }
    };
    auto multiply = [&](int buffer) {
#pragma unroll
      for (int i = 0; i < kRun; ++i)
#pragma unroll
        for (int e = 0; e < EACH; ++e) {
          acc[e] = fmaf(av[buffer][e][i].x, wv[buffer][i].x, acc[e]);
          acc[e] = fmaf(av[buffer][e][i].y, wv[buffer][i].y, acc[e]);
          acc[e] = fmaf(av[buffer][e][i].z, wv[buffer][i].z, acc[e]);
          acc[e] = fmaf(av[buffer][e][i].w, wv[buffer][i].w, acc[e]);
        }
    };
    if (owner) {
      read(0, 0);
#pragma unroll 1
      for (int kk = 0; kk < kRowsDepth; kk += 8 * kRun) {
        read(1, kk + 4 * kRun);
        multiply(0);
        if (kk + 8 * kRun < kRowsDepth) read(0, kk + 8 * kRun);
        multiply(1);
      }
    }
    __syncthreads();
  }
  mir::grid_dependency_wait();                     // (c may be what an earlier kernel left)
  if (!owner || col0 + tx >= n) return;
#pragma unroll
  for (int e = 0; e < EACH; ++e)
    if (ty + e * DOWN < m) finish(c, ldc, bias, beta, ty + e * DOWN, col0 + tx, acc[e]);
}

struct Product {
  const float* a; int lda;
  const float* w; int ldw;
  const float* bias;
  float* c; int ldc;
  int m, n, k;
  float beta;
  cudaStream_t stream;
};

// early: whether it may start beside the kernel in front.
template <typename Kernel>
int launch(bool early, Kernel kernel, dim3 grid, int threads, int smem, const Product& p) {
  const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) {
    mir_set_error("gemm_f32: %s", cudaGetErrorString(err));
    return MIR_CUDA_ERROR;
  }
  return mir_launch_with(early && mir_pdl_enabled(), "gemm_f32", kernel, grid, dim3(threads), smem, p.stream, 0, p.a, p.lda, p.w, p.ldw, p.bias, p.c, p.ldc, p.m, p.n,
                    p.k, p.beta);
}

template <int MT, bool WIDE>
int launch_rows(const Product& p) {
  constexpr int smem = kRowsStages * (kRowsColumns + MT) * (kRowsDepth + 4) * (int)sizeof(float);
  // Started early, a grid that does not fill the GPU lands on the SMs that are left first, several CTAs on one.  Within decode
  // steps of three rows, plainly / early (us): 128 CTAs, K 2,048 and 5,504 together, 18.8 / 23.4; 192, K 2,048, 12.0 / 15.2; 688
  // 34.6 / 28.1.  One such product behind the other: 128 CTAs, K 2,048 11.9 / 11.9, K 5,504 27.3 / 26.7; 192 13.0 / 14.2; 688 35 / 32.
  const int ctas = (p.n + kRowsColumns - 1) / kRowsColumns;
  return launch(ctas >= 3 * mir_sm_count(), gemm_f32_rows_kernel<MT, WIDE>, dim3(ctas), kRowsThreads + kRowsLoaders, smem, p);
}

template <int BM, int BN, int TM, int TN, bool WIDE>
int launch_tile(const Product& p) {
  constexpr int DEPTH = 32, STAGES = 3, smem = STAGES * (BM + BN) * (DEPTH + 4) * (int)sizeof(float);
  const dim3 grid((p.n + BN - 1) / BN, (p.m + BM - 1) / BM);
  if (grid.y > 65535) {
    mir_set_error("gemm_f32: %d rows exceed the grid limit", p.m);
    return MIR_BAD_ARGUMENT;
  }
  // (never early: 290 rows, tiles of two waves or less, 212 us plainly and 246 beside the kernel in front)
  return launch(false, gemm_f32_tile_kernel<BM, BN, TM, TN, DEPTH, STAGES, WIDE>, grid, (BM / TM) * (BN / TN), smem, p);
}

template <bool WIDE>
int choose(const Product& p) {
  if (p.m <= 1) return launch_rows<1, WIDE>(p);
  if (p.m <= 2) return launch_rows<2, WIDE>(p);
  if (p.m <= 4) return launch_rows<4, WIDE>(p);
  if (p.m <= 8) return launch_rows<8, WIDE>(p);
  if (p.m <= 16) return launch_rows<16, WIDE>(p);
  if (p.m <= 32) return launch_tile<32, 64, 4, 4, WIDE>(p);
  // The tile whose busiest SM has the least to do: multiply-adds of its tiles, a thread of the smaller tile reading more of
  // shared memory for each (by the weights below).  290 rows: N 11,008, K 2,048 by 64 x 64 364 us, the average of a layer's
  // products by 64 x 64 249 us and by 32 x 64 212 (each where it is taken); 2,048 rows, N 2,048, K 5,504: 1,107 us (41.7 TF).
  // Larger tiles are no better: 64 x 128 with 64 outputs a thread 373 us for what these two do in 230, 128 x 128 1,173 us
  // for the last product and the same to 1 % for N 11,008.
  const int sms = mir_sm_count();
  auto cost = [&](int rows, int columns, int weight) {
    const long long tiles = (long long)((p.m + rows - 1) / rows) * ((p.n + columns - 1) / columns);
    return (tiles + sms - 1) / sms * rows * columns * weight;
  };
  if (cost(64, 64, 5) <= cost(32, 64, 6)) return launch_tile<64, 64, 8, 4, WIDE>(p);
  return launch_tile<32, 64, 4, 4, WIDE>(p);
}

}  // namespace

MIR_EXPORT int mir_gemm_f32(const float* a, int lda, const float* w, int ldw, const float* bias, float* c, int ldc,
                            int m, int n, int k, float beta, cudaStream_t stream) {
  if (m == 0 || n == 0) return MIR_OK;
  if (m < 0 || n < 0 || k <= 0 || lda < k || ldw < k || ldc < n) {
    mir_set_error("gemm_f32: bad sizes m %d n %d k %d lda %d ldw %d ldc %d", m, n, k, lda, ldw, ldc);
    return MIR_BAD_ARGUMENT;
  }
  const Product p{a, lda, w, ldw, bias, c, ldc, m, n, k, beta, stream};
  const bool wide = k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)a | (uintptr_t)w) % 16 == 0;
  return wide ? choose<true>(p) : choose<false>(p);
}
