// bf16 matrix products for many rows on the 5th-generation tensor cores (tcgen05), written by hand:
//
//   out[M, N] = epilogue(x[M, K] . w[N, K]^T)          x, w row-major bf16 ("K-major" for both operands)
//
// One CTA per SM walks over tiles of the output: 128 tokens x `width` accumulator columns (for the SwiGLU
// epilogue width / 2 gate features and the width / 2 up features that belong to them); width is 256 unless
// the product has fewer columns.  Three roles:
//
//   producer   one thread.  Per 64-wide step of K it asks the TMA unit for the x box (128 rows x 64) and the
//              w box(es) with cp.async.bulk.tensor.2d into a ring of shared-memory stages laid out with the
//              128-byte swizzle that tcgen05.mma reads.  Out-of-range rows and k arrive as zeros, so M, N and K
//              need not be multiples of the tile.  An mbarrier per stage counts the bytes in.
//   issuer     one warp that stays converged, the products predicated on its elected lane (tcgen05.cuh says why).
//              When a stage is full it issues four tcgen05.mma (128 x width x 16 each, operands
//              straight from shared memory through matrix descriptors, accumulator in tensor memory) and then
//              tcgen05.commit, which arrives on the stage's "empty" barrier once the tensor cores have read the
//              stage, so the producer can refill it.  After a tile's last step a commit arrives on the
//              accumulator's "full" barrier.  Two accumulators alternate: the products of the next tile run
//              while the epilogue reads the last one.
//   epilogue   eight warps; warp i may read accumulator lanes 32 (i mod 4) .. + 31 (one token row per thread),
//              and the two warps of a quarter take alternate chunks of 32 columns.  They
//              wait for "full", read the accumulator with tcgen05.ld (32 columns at a time), hand the
//              accumulator back ("free" barrier) as soon as its last columns are in registers, apply the
//              epilogue and write the row to global memory.
//
// Epilogues:  STORE  out bf16 = acc (+ bias)
//             ACCUM  out float += acc (+ bias)            the residual stream
//             F32    out float = acc (+ bias)
//             SWIGLU out bf16 = silu(acc_gate) * acc_up   w holds [gate rows; up rows]; the [M, 2 I] intermediate
//                                                         of the two-kernel formulation is never written
// Tensor memory: all 512 columns (two accumulators of 128 lanes x 256 columns), allocated by one warp and freed
// by the same warp; the shared-memory ring leaves room for one CTA per SM only.
// Every wait is bounded in time; a role whose wait runs out raises g_tc_gemm_error and stops waiting, the CTA
// still frees its tensor memory and returns.
// libmir takes these products from a library (DenseMatmulPlan / CublasLtBf16Plan of the mircuda crate,
// cuda/src/backend/linear/mod.rs:141-194) and applies the gate in a second kernel
// (cuda/kernels/elementwise_bf16.cu:42-70).
#include <algorithm>
#include "tcgen05.cuh"

using namespace mir;
using namespace mir::tc;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int kTileM = 128;                 // tokens per CTA
constexpr int kStepK = 64;                  // k per stage: 128 bytes, one swizzle row
constexpr int kStages = 4;                  // shared-memory ring
constexpr int kStageStride = (kTileM + 256) * 128;   // 48 KB: 128 token rows and up to 256 weight rows of 128 bytes
constexpr int kEpilogueWarps = 8;          // two per quarter of the accumulator lanes; they share its columns
constexpr int kThreads = (2 + kEpilogueWarps) * 32;  // producer warp, issuer warp, epilogue warps
constexpr int kPlaces = 64;                 // tiles of a CTA whose places are looked up before the first of them
constexpr uint32_t kTmemColumns = 512;      // two accumulators of up to 256 columns
static_assert(kStages * kStageStride + 1024 + kLeastSharedBeside > kSharedOfSm, "no other kernel with tensor memory beside this one");
// GELU: STORE of gelu_tanh(acc), no bias; GELU_ERF: the same with the exact form 0.5 z (1 + erf(z / sqrt 2)); RELU2: the
// same with the square of relu
enum Epilogue : int { STORE = 0, ACCUM = 1, F32 = 2, SWIGLU = 3, GELU = 4, GELU_ERF = 5, RELU2 = 6 };

__device__ int g_tc_gemm_error = 0;

// The rows of a grouped product (routed experts): the rows are sorted by group, every group multiplies with its own
// weight rows, and which tiles of 128 rows there are is known on the device only.  tiles[2 i], tiles[2 i + 1]: group and
// first row of tile i (a tile ends with its group's rows, offsets[group + 1], the rest of its 128 rows is computed and
// dropped); tile_count[0] tiles in all; group g's weight rows start at row g * group_rows of the weight matrix; the
// result of sorted row r goes to row scatter[r] of out (to row r without scatter).  tiles == nullptr: a plain product.
struct GroupedRows {
  const int* tiles;
  const int* tile_count;
  const int* offsets;
  const int* scatter;
  int group_rows;
};

// Where a tile of the output lies: its tile of rows, its tile of columns.  Plain products: token tile fastest, so CTAs that
// run together share weight rows in L2.  Grouped ones: one group behind the other, a group's row tiles fastest, so that its
// weights are read once and its rows stay in L2 for all its column tiles (14,800 pairs of 64 experts, 2 x 1,024 columns, K
// 2,048: 131 us; with the row tiles of all groups fastest, which goes over all rows for every column tile, 172).  The weights'
// boxes brought into the L2 ten steps ahead: 155 us.
// A grouped tile's place takes four reads behind one another, which the producer would wait for at every tile: the threads of
// a CTA look its first kPlaces up side by side before the first tile.
struct Place { int m0, row_end, n0, w0; };                   // first row, end of the rows, first column, first row of the weights
__device__ __forceinline__ Place place_of(int tile, int token_tiles, int column_tiles, int out_width, int m, const GroupedRows& grouped) {
  if (grouped.tiles == nullptr) {
    const int n0 = tile / token_tiles * out_width;
    return Place{tile % token_tiles * kTileM, m, n0, n0};
  }
  const int inside = tile / column_tiles;                    // some row tile of the group: its tiles lie one behind the other
  const int group = grouped.tiles[2 * inside], begin = grouped.offsets[group];
  const int first = inside - (grouped.tiles[2 * inside + 1] - begin) / kTileM;
  const int end = grouped.offsets[group + 1], count = (end - begin + kTileM - 1) / kTileM, local = tile - first * column_tiles;
  const int n0 = local / count * out_width;
  return Place{begin + local % count * kTileM, end, n0, group * grouped.group_rows + n0};
}

// One CTA per SM walks over output tiles (their order: place_of).  A tile is 128 tokens x `width` accumulator columns (width a multiple of 16, at most 256; with the SwiGLU
// epilogue width / 2 gate columns followed by width / 2 up columns).  Two accumulators of 256 columns alternate,
// so the epilogue of one tile overlaps the products of the next.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map,
               const void* __restrict__ bias, void* __restrict__ out, int ldo, int m, int n, int k, int up_offset,
               int width, int token_tiles, int tiles, GroupedRows grouped, int column_tiles) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long barriers[2 * kStages + 4];   // full, empty, accumulator full[2], free[2]
  __shared__ uint32_t tmem_base_slot;
  __shared__ Place places[kPlaces];
  if (*reinterpret_cast<volatile int*>(&g_tc_gemm_error) != 0) {            // an earlier wait ran out: do not queue up more
    grid_dependency_wait();                                 // (what follows takes the kernels in front of this one for over)
    return;
  }
  // the swizzle pattern repeats every 1024 bytes; the stages start on such a boundary
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(&barriers[0]), empty0 = smem_u32(&barriers[kStages]);
  const uint32_t acc_full0 = smem_u32(&barriers[2 * kStages]), acc_free0 = smem_u32(&barriers[2 * kStages + 2]);
  const int steps = (k + kStepK - 1) / kStepK;
  const int out_width = MODE == SWIGLU ? width / 2 : width;  // output columns of a tile
  const uint32_t stage_bytes = (uint32_t)(kTileM + width) * 128u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * s) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + 8 * s) : "memory");
    }
    for (int b = 0; b < 2; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(acc_full0 + 8 * b) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(acc_free0 + 8 * b), "r"(kEpilogueWarps) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {                                          // this warp owns the tensor memory: all 512 columns
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"(kTmemColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_slot;
  grid_dependency_wait();                                   // x (and out for ACCUM) come from earlier kernels
  grid_launch_dependents();
  if (grouped.tiles != nullptr) {                           // the list of row tiles was written by an earlier kernel
    token_tiles = grouped.tile_count[0];
    tiles = token_tiles * column_tiles;
    const int tile = blockIdx.x + threadIdx.x * gridDim.x;
    if (threadIdx.x < kPlaces && tile < tiles) places[threadIdx.x] = place_of(tile, token_tiles, column_tiles, out_width, m, grouped);
    __syncthreads();
  }
  auto place_at = [&](int tile, int number) {                // of this CTA's number-th tile
    return grouped.tiles != nullptr && number < kPlaces ? places[number]
                                                        : place_of(tile, token_tiles, column_tiles, out_width, m, grouped);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      const uint64_t xm = reinterpret_cast<uint64_t>(&x_map), wm = reinterpret_cast<uint64_t>(&w_map);
      uint32_t count = 0;                                    // stages filled so far, over all tiles
      bool alive = true;
      int number = 0;
      for (int tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x, ++number) {
        const Place place = place_at(tile, number);
        const int m0 = place.m0, w0 = place.w0;
        for (int step = 0; step < steps; ++step, ++count) {
          const uint32_t stage = count % kStages, parity = (count / kStages) & 1u;
          if (!wait_barrier(empty0 + 8 * stage, parity ^ 1u)) { g_tc_gemm_error = 1; alive = false; break; }
          const uint32_t barrier = full0 + 8 * stage;
          const uint32_t dst = smem_u32(smem + (size_t)stage * kStageStride);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barrier), "r"(stage_bytes) : "memory");
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                  "r"(dst), "l"(xm), "r"(barrier), "r"(step * kStepK), "r"(m0)
              : "memory");
          // the weight map's box has out_width rows: one box, or a gate box and an up box behind it
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                  "r"(dst + kTileM * 128), "l"(wm), "r"(barrier), "r"(step * kStepK), "r"(w0)
              : "memory");
          if (MODE == SWIGLU)
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
                    "r"(dst + (kTileM + out_width) * 128), "l"(wm), "r"(barrier), "r"(step * kStepK), "r"(up_offset + w0)
                : "memory");
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ issuer: the whole warp stays converged, the
    // products are predicated on the elected lane (see tcgen05.cuh on issuing from a whole warp)
    {
      const uint32_t idesc = instruction_descriptor(kTileM, width);
      const uint32_t elected = elect_one();
      const uint32_t a_low0 = operand_low(smem_u32(smem)), b_low0 = operand_low(smem_u32(smem) + kTileM * 128);
      uint32_t stage = 0, parity = 0, local = 0;             // of the stages consumed so far; tiles of this CTA
      bool alive = true;
      for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++local) {
        const uint32_t buffer = local & 1u, use = (local >> 1) & 1u;
        // the epilogue must have read this accumulator's previous tile
        if (alive && !wait_barrier(acc_free0 + 8 * buffer, use ^ 1u)) { g_tc_gemm_error = 2; alive = false; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t accumulator = tmem_base + buffer * 256u;
        for (int step = 0; step < steps; ++step) {
          if (alive && !wait_barrier(full0 + 8 * stage, parity)) { g_tc_gemm_error = 2; alive = false; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_low = a_low0 + stage * (uint32_t)(kStageStride >> 4);
          const uint32_t b_low = b_low0 + stage * (uint32_t)(kStageStride >> 4);
          // 16 k = 32 bytes further along the swizzled rows: the start address moves by 32 bytes
          mma_bf16_ss_halves(accumulator, a_low, b_low, idesc, step > 0 ? 1u : 0u, elected);
#pragma unroll
          for (int kk = 1; kk < kStepK / 16; ++kk)
            mma_bf16_ss_halves<true>(accumulator, a_low + 2u * kk, b_low + 2u * kk, idesc, elected);
          mma_commit_elected(empty0 + 8 * stage, elected);   // the stage is free once these have read it
          if (++stage == (uint32_t)kStages) { stage = 0; parity ^= 1u; }
        }
        mma_commit_elected(acc_full0 + 8 * buffer, elected); // this tile's accumulator is complete
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: one token row per thread
    const int quarter = warp & 3;                            // the accumulator lanes this warp may read
    const int half = (warp - 2) >> 2;                        // which of every two 32-column chunks it takes
    uint32_t local = 0;
    bool alive = true;
    for (int tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x, ++local) {
      const uint32_t buffer = local & 1u, use = (local >> 1) & 1u;
      const Place place = place_at(tile, (int)local);
      const int n0 = place.n0, m0 = place.m0, row_end = place.row_end;
      const int source_row = m0 + quarter * 32 + lane;
      // where this thread's row of results goes: its own row, or the place the sorted row came from
      const int row = (grouped.tiles != nullptr && grouped.scatter != nullptr && source_row < row_end)
                          ? grouped.scatter[source_row] : source_row;
      if (!wait_barrier(acc_full0 + 8 * buffer, use)) { g_tc_gemm_error = 3; alive = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lane_base = tmem_base + buffer * 256u + ((uint32_t)(quarter * 32) << 16);
      bool released = false;
      auto release = [&]() {                                 // this warp has read all it needs of the accumulator
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_free0 + 8 * buffer) : "memory");
        released = true;
      };
#pragma unroll 1
      for (int c0 = half * 32; c0 < out_width; c0 += 64) {
        float v[32];
        tmem_load_32(lane_base + c0, v);
        if (MODE == SWIGLU) {
          float u[32];
          tmem_load_32(lane_base + out_width + c0, u);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __fdividef(v[i], 1.0f + __expf(-v[i])) * u[i];
        }
        if (MODE == GELU) {                                   // 0.5 z (1 + tanh(sqrt(2 / pi) (z + 0.044715 z^3)))
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            float t;
            asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.7978845608028654f * fmaf(0.044715f * v[i] * v[i], v[i], v[i])));
            v[i] = 0.5f * v[i] * (1.0f + t);
          }
        }
        if (MODE == GELU_ERF) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0.5f * v[i] * (1.0f + erff(v[i] * 0.70710678118654752f));
        }
        if (MODE == RELU2) {
#pragma unroll
          for (int i = 0; i < 32; ++i) { const float positive = fmaxf(v[i], 0.0f); v[i] = positive * positive; }
        }
        if (c0 + 64 >= out_width) release();                 // the last columns are in registers
        const int limit = min(n, n0 + out_width);            // columns of this tile that exist
        if (MODE == F32 && n0 + c0 + 32 <= limit && (ldo % 4) == 0 && bias == nullptr) {
          // 32-bit rows: through shared memory, so that a store writes four rows of 128 bytes instead of sixteen bytes of
          // each of 32 rows (19,800 sorted rows of 2,048 columns, K 1,024: 86 us, 106 the other way)
          float4* block = reinterpret_cast<float4*>(smem + (size_t)kStages * kStageStride) + (warp - 2) * 256;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            block[lane * 8 + (i ^ (lane & 7))] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          __syncwarp();
          const int place = source_row < row_end ? row : -1;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = i * 4 + (lane >> 3);
            const int to = __shfl_sync(0xffffffffu, place, r);
            if (to >= 0)
              reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + (size_t)to * ldo + n0 + c0)[lane & 7] =
                  block[r * 8 + ((lane & 7) ^ (r & 7))];
          }
          __syncwarp();                                      // (the block is written again for the next columns)
        } else if (source_row < row_end) {
          if (MODE == STORE || MODE == SWIGLU || MODE == GELU || MODE == GELU_ERF || MODE == RELU2) {
            bf16* dst = reinterpret_cast<bf16*>(out) + (size_t)row * ldo + n0 + c0;
            if (n0 + c0 + 32 <= limit && (ldo % 8) == 0) {
#pragma unroll
              for (int i = 0; i < 32; i += 8) {
                float b8[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                if (MODE == STORE && bias) {
#pragma unroll
                  for (int j = 0; j < 8; ++j) b8[j] = __bfloat162float(reinterpret_cast<const bf16*>(bias)[n0 + c0 + i + j]);
                }
                uint4 packed;
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
                for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[i + 2 * j] + b8[2 * j], v[i + 2 * j + 1] + b8[2 * j + 1]);
                *reinterpret_cast<uint4*>(dst + i) = packed;
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                if (n0 + c0 + i < limit) {
                  float value = v[i];
                  if (MODE == STORE && bias) value += __bfloat162float(reinterpret_cast<const bf16*>(bias)[n0 + c0 + i]);
                  dst[i] = __float2bfloat16_rn(value);
                }
              }
            }
          } else {
            float* dst = reinterpret_cast<float*>(out) + (size_t)row * ldo + n0 + c0;
            if (n0 + c0 + 32 <= limit && (ldo % 4) == 0 && bias == nullptr) {
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                float4 value = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                if (MODE == ACCUM) {
                  const float4 old = *reinterpret_cast<const float4*>(dst + i);
                  value.x += old.x; value.y += old.y; value.z += old.z; value.w += old.w;
                }
                *reinterpret_cast<float4*>(dst + i) = value;
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                if (n0 + c0 + i < limit) {
                  float value = v[i];
                  if (bias) value += reinterpret_cast<const float*>(bias)[n0 + c0 + i];
                  dst[i] = MODE == ACCUM ? dst[i] + value : value;
                }
              }
            }
          }
        }
      }
      if (!released) release();                              // a tile too narrow to give this warp any columns
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColumns) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------ host
int g_forced_width = 0;                                      // for measurements: 0 = choose

int sm_count() {
  static int count = 0;
  if (count == 0) {
    int device = 0;
    cudaGetDevice(&device);
    if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count <= 0) count = 148;
  }
  return count;
}

// Accumulator columns of a tile.  Measured on B200 (2,048 tokens, K 2,560 to 9,728): a step of K takes about
// 0.4 us whether the tile is 192, 224 or 256 columns wide (the ring of four stages is bound by the latency of
// its refills, not by the products), so the widest tile is the fastest even where a narrower one would fill the
// last round of tiles better.  `columns` is the number of accumulator columns over all tiles (2 n with the
// SwiGLU epilogue), `step` what the width must be a multiple of.
int choose_width(long long columns, int step) {
  if (g_forced_width >= step && g_forced_width <= 256 && g_forced_width % step == 0) return g_forced_width;
  const long long rounded = (columns + step - 1) / step * step;
  return (int)std::min<long long>(256, rounded);
}

template <int MODE>
int launch(const void* x, int ldx, const void* w, const void* bias, void* out, int ldo, int m, int n, int k,
           int up_offset, cudaStream_t stream) {
  const int token_tiles = (m + kTileM - 1) / kTileM;
  const int width = MODE == SWIGLU ? choose_width(2ll * n, 32) : choose_width(n, 16);
  const int out_width = MODE == SWIGLU ? width / 2 : width;
  CUtensorMap x_map, w_map;
  int status = tensor_map_for(x, m, k, ldx, kTileM, &x_map);
  if (status != MIR_OK) return status;
  status = tensor_map_for(w, MODE == SWIGLU ? up_offset + n : n, k, k, out_width, &w_map);
  if (status != MIR_OK) return status;
  const size_t smem = (size_t)kStages * kStageStride + 1024 + (MODE == F32 ? kEpilogueWarps * 4096 : 0);
  static bool configured = false;
  if (!configured) {
    const cudaError_t err = cudaFuncSetAttribute(tc_gemm_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) {
      mir_set_error("tc_gemm: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(err));
      return MIR_CUDA_ERROR;
    }
    configured = true;
  }
  const long long tiles = (long long)((n + out_width - 1) / out_width) * token_tiles;
  if (tiles > 0x7fffffffll) { mir_set_error("tc_gemm: too many tiles"); return MIR_BAD_ARGUMENT; }
  const dim3 grid((unsigned)std::min<long long>(tiles, sm_count()));
  return mir_launch("tc_gemm", tc_gemm_kernel<MODE>, grid, dim3(kThreads), smem, stream, 0, x_map, w_map, bias, out, ldo,
                    m, n, k, up_offset, width, token_tiles, (int)tiles, GroupedRows{nullptr, nullptr, nullptr, nullptr, 0}, 0);
}

// The grouped form: x [rows, k] sorted by group, w [weight_rows, k] with group g's n rows from row g * n on (and, for
// the SwiGLU epilogue, its up rows up_offset further), the row tiles from a list on the device (at most max_row_tiles).
template <int MODE>
int launch_grouped(const void* x, int ldx, int rows, const void* w, int weight_rows, void* out, int ldo, int n, int k,
                   int up_offset, const GroupedRows& grouped, int max_row_tiles, cudaStream_t stream) {
  const int width = MODE == SWIGLU ? choose_width(2ll * n, 32) : choose_width(n, 16);
  const int out_width = MODE == SWIGLU ? width / 2 : width;
  CUtensorMap x_map, w_map;
  int status = tensor_map_for(x, rows, k, ldx, kTileM, &x_map);
  if (status != MIR_OK) return status;
  status = tensor_map_for(w, weight_rows, k, k, out_width, &w_map);
  if (status != MIR_OK) return status;
  const size_t smem = (size_t)kStages * kStageStride + 1024 + (MODE == F32 ? kEpilogueWarps * 4096 : 0);
  static bool configured = false;
  if (!configured) {
    const cudaError_t err = cudaFuncSetAttribute(tc_gemm_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) {
      mir_set_error("tc_gemm: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(err));
      return MIR_CUDA_ERROR;
    }
    configured = true;
  }
  const int column_tiles = (n + out_width - 1) / out_width;
  const long long tiles = (long long)column_tiles * max_row_tiles;
  if (tiles > 0x7fffffffll) { mir_set_error("tc_gemm: too many tiles"); return MIR_BAD_ARGUMENT; }
  const dim3 grid((unsigned)std::min<long long>(std::max<long long>(tiles, 1), sm_count()));
  return mir_launch("tc_gemm_grouped", tc_gemm_kernel<MODE>, grid, dim3(kThreads), smem, stream, 0, x_map, w_map,
                    (const void*)nullptr, out, ldo, rows, n, k, up_offset, width, 0, 0, grouped, column_tiles);
}

}  // namespace

// 0 if no bounded wait of the tcgen05 product ever ran out; else which role gave up last (1 producer, 2 issuer,
// 3 epilogue).  Synchronises the device.
MIR_EXPORT int mir_gemm_tc_error() {
  int flag = 0;
  if (cudaMemcpyFromSymbol(&flag, g_tc_gemm_error, sizeof(int)) != cudaSuccess) return -1;
  return flag;
}

// The products of routed experts on rows sorted by expert.  mode 3 (SwiGLU): out bf16 [rows, n] = silu(x w_gate[g]^T) *
// (x w_up[g]^T) with w = [experts * n gate rows; experts * n up rows] (up_offset = experts * n); mode 2: out float
// [*, n] = x w[g]^T, the row of sorted row r written to out row scatter[r].  tiles / tile_count / offsets: the list of
// 128-row tiles, their number and the experts' row ranges, all on the device; max_row_tiles bounds the list.  k and ldx
// multiples of 8, x and w 16-byte aligned.
MIR_EXPORT int mir_gemm_tc_grouped_bf16(int mode, const void* x, int ldx, int rows, const void* w, int experts,
                                        void* out, int ldo, int n, int k, const int* tiles, const int* tile_count,
                                        const int* offsets, const int* scatter, int max_row_tiles, cudaStream_t stream) {
  if (rows == 0 || n == 0) return MIR_OK;
  if (rows < 0 || n < 0 || k <= 0 || (k % 8) || (ldx % 8) || ldx < k || ldo < n || ((uintptr_t)x & 15) ||
      ((uintptr_t)w & 15) || experts <= 0 || max_row_tiles <= 0 || tiles == nullptr || tile_count == nullptr ||
      offsets == nullptr) {
    mir_set_error("tc_gemm_grouped: k and the row stride must be multiples of 8 and the operands 16-byte aligned "
                  "(rows %d n %d k %d ldx %d ldo %d)", rows, n, k, ldx, ldo);
    return MIR_BAD_ARGUMENT;
  }
  const GroupedRows grouped{tiles, tile_count, offsets, scatter, n};
  if (mode == SWIGLU)
    return launch_grouped<SWIGLU>(x, ldx, rows, w, 2 * experts * n, out, ldo, n, k, experts * n, grouped, max_row_tiles, stream);
  if (mode == F32)
    return launch_grouped<F32>(x, ldx, rows, w, experts * n, out, ldo, n, k, 0, grouped, max_row_tiles, stream);
  mir_set_error("tc_gemm_grouped: mode %d is neither the SwiGLU nor the float epilogue", mode);
  return MIR_BAD_ARGUMENT;
}

// For measurements: fix the accumulator width of a tile (a multiple of 32, 32..256), or 0 to let the launcher
// choose.
MIR_EXPORT int mir_gemm_tc_set_width(int width) {
  if (width != 0 && (width < 32 || width > 256 || width % 32)) {
    mir_set_error("tc_gemm: the width must be 0 or a multiple of 32 up to 256");
    return MIR_BAD_ARGUMENT;
  }
  g_forced_width = width;
  return MIR_OK;
}

// mode: 0 store bf16, 1 accumulate into float, 2 float, 4 store bf16 of the tanh GELU, 5 of the exact GELU, 6 of the
// square of relu, 3 SwiGLU (w = [gate; up],
// up rows start at up_offset, n = number of output columns).  k and ldx must be multiples of 8, x and w 16-byte
// aligned; m, n, k need not be multiples of the tile sizes.
MIR_EXPORT int mir_gemm_tc_bf16(int mode, const void* x, int ldx, const void* w, const void* bias, void* out, int ldo,
                                int m, int n, int k, int up_offset, cudaStream_t stream) {
  if (m == 0 || n == 0) return MIR_OK;
  if (m < 0 || n < 0 || k <= 0 || (k % 8) || (ldx % 8) || ldx < k || ldo < n || ((uintptr_t)x & 15) ||
      ((uintptr_t)w & 15) || m > 65535 * kTileM) {
    mir_set_error("tc_gemm: k and the row stride must be multiples of 8 and the operands 16-byte aligned "
                  "(m %d n %d k %d ldx %d ldo %d)", m, n, k, ldx, ldo);
    return MIR_BAD_ARGUMENT;
  }
  switch (mode) {
    case STORE: return launch<STORE>(x, ldx, w, bias, out, ldo, m, n, k, 0, stream);
    case ACCUM: return launch<ACCUM>(x, ldx, w, bias, out, ldo, m, n, k, 0, stream);
    case F32: return launch<F32>(x, ldx, w, bias, out, ldo, m, n, k, 0, stream);
    case SWIGLU:
      if (bias) { mir_set_error("tc_gemm: the SwiGLU epilogue takes no bias"); return MIR_BAD_ARGUMENT; }
      return launch<SWIGLU>(x, ldx, w, nullptr, out, ldo, m, n, k, up_offset, stream);
    case GELU:
      if (bias) { mir_set_error("tc_gemm: the GELU epilogue takes no bias"); return MIR_BAD_ARGUMENT; }
      return launch<GELU>(x, ldx, w, nullptr, out, ldo, m, n, k, 0, stream);
    case GELU_ERF:
      if (bias) { mir_set_error("tc_gemm: the GELU epilogue takes no bias"); return MIR_BAD_ARGUMENT; }
      return launch<GELU_ERF>(x, ldx, w, nullptr, out, ldo, m, n, k, 0, stream);
    case RELU2:
      if (bias) { mir_set_error("tc_gemm: the squared-relu epilogue takes no bias"); return MIR_BAD_ARGUMENT; }
      return launch<RELU2>(x, ldx, w, nullptr, out, ldo, m, n, k, 0, stream);
  }
  mir_set_error("tc_gemm: unknown mode %d", mode);
  return MIR_BAD_ARGUMENT;
}
