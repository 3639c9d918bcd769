// Helpers of the recurrences' kernels: 32-bit arithmetic two numbers an instruction, 16-byte copies into shared memory, and
// the sum of several columns' parts over the lanes that share them.
#pragma once
#include "common.cuh"

namespace mir {

// Two 32-bit numbers side by side in one register pair: one instruction for two multiplications or multiply-adds, each
// rounded as its scalar form is.
typedef unsigned long long Pair;
__device__ __forceinline__ Pair pair_from(float x, float y) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 pair_split(Pair p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ Pair pair_mul(Pair a, Pair b) {
  Pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ Pair pair_fma(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// The sum of four partial sums kept as two pairs (elements 0, 1 and 2, 3 of every run of four).
__device__ __forceinline__ float pair_total(const Pair (&sums)[2]) {
  const float2 a = pair_split(sums[0]), b = pair_split(sums[1]);
  return (a.x + a.y) + (b.x + b.y);
}

// PER channels of a column of `count` 32-bit numbers, held by one of LANES lanes as 16-byte pieces side by side across the
// lanes: lane l has 4 (m LANES + l) .. + 3, m < PER / 4.  `wide`: count is a multiple of four and the column starts on a
// 16-byte boundary.
template <int LANES, int PER>
__device__ __forceinline__ void load_column(Pair (&s)[PER / 2], const float* column, int l, int count, bool live, bool wide) {
#pragma unroll
  for (int m = 0; m < PER; m += 4) {
    const int i = (m / 4 * LANES + l) * 4;
    float4 piece = make_float4(0.f, 0.f, 0.f, 0.f);
    if (wide) {
      if (live && i < count) piece = *reinterpret_cast<const float4*>(column + i);
    } else if (live) {
      if (i < count) piece.x = column[i];
      if (i + 1 < count) piece.y = column[i + 1];
      if (i + 2 < count) piece.z = column[i + 2];
      if (i + 3 < count) piece.w = column[i + 3];
    }
    s[m / 2] = pair_from(piece.x, piece.y);
    s[m / 2 + 1] = pair_from(piece.z, piece.w);
  }
}
template <int LANES, int PER>
__device__ __forceinline__ void store_column(const Pair (&s)[PER / 2], float* column, int l, int count, bool wide) {
#pragma unroll
  for (int m = 0; m < PER; m += 4) {
    const int i = (m / 4 * LANES + l) * 4;
    const float2 a = pair_split(s[m / 2]), b = pair_split(s[m / 2 + 1]);
    if (wide) {
      if (i < count) *reinterpret_cast<float4*>(column + i) = make_float4(a.x, a.y, b.x, b.y);
    } else {
      if (i < count) column[i] = a.x;
      if (i + 1 < count) column[i + 1] = a.y;
      if (i + 2 < count) column[i + 2] = b.x;
      if (i + 3 < count) column[i + 3] = b.y;
    }
  }
}

// parts[i]: this lane's part of sum i, i < N (a power of two up to LANES).  The parts of LANES lanes are added neighbours
// first, then pairs of pairs, and so on; while a lane has several sums each step hands half of them to the lane it adds
// with, so that N sums cost little more than one.  Returns the sum number lane_sum<N>(l).
template <int N> __device__ __forceinline__ int lane_sum(int l) {
  int index = 0;
#pragma unroll
  for (int bit = 1, half = N / 2; half > 0; bit <<= 1, half >>= 1) index += (l & bit) ? half : 0;
  return index;
}
// The lane that has sum `index`: lane_sum<N>(lane_with<N>(index)) == index.
template <int N> __host__ __device__ constexpr int lane_with(int index) {
  int lane = 0;
  for (int bit = 1, half = N / 2; half > 0; bit <<= 1, half >>= 1) lane += (index & half) ? bit : 0;
  return lane;
}
template <int LANES, int N, int STEP = 1>
__device__ __forceinline__ float sum_lanes(const float (&parts)[N], int l) {
  if constexpr (N == 1) {
    float sum = parts[0];
#pragma unroll
    for (int step = STEP; step < LANES; step <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, step);
    return sum;
  } else {
    const bool upper = (l & STEP) != 0;
    float half[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      const float given = __shfl_xor_sync(0xffffffffu, upper ? parts[i] : parts[i + N / 2], STEP);
      half[i] = (upper ? parts[i + N / 2] : parts[i]) + given;
    }
    return sum_lanes<LANES, N / 2, STEP * 2>(half, l);
  }
}

__device__ __forceinline__ void copy_async(float* to, const float* from, bool wide) {       // 16 or 4 bytes
  const unsigned target = (unsigned)__cvta_generic_to_shared(to);
  if (wide) asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(target), "l"(from) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(target), "l"(from) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

}  // namespace mir
