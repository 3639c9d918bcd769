// Kernels of a mixture of gated experts.  P = tokens * top pairs of (token, chosen expert); pair p = token * top + slot.
//
//   moe_route     per token, from the router's 32-bit logits (a product of the framework): sigmoid scores (or a softmax
//                 over all experts), choice among the experts of the best groups by score + correction (a group judged
//                 by the sum of its two largest choice scores, or by its largest), weights = chosen scores / their sum
//                 * scale; and the shared expert's gate.  The last experts of the router may be identity experts, which
//                 have no weights: the sort leaves their pairs out, and moe_combine adds weight * the token's own input
//   moe_sort      the pairs ordered by expert (a stable counting sort: a CTA per expert counts, one CTA scans, a CTA
//                 per expert places), each expert's range, and the list of tiles (8 or 128 pairs of one expert)
//                 that the grouped products walk over
//   moe_grouped   products on the sorted pairs with each pair's own expert's weights: hidden = silu(Wg x) * (Wu x)
//                 from the tokens' rows, and the down projection of the hidden rows into one 32-bit row per pair, as
//                 32-bit multiply-adds on tiles of 8 pairs (any type and size).  bfloat16 rows of 16-byte pieces run
//                 the tcgen05 product of csrc/gemm_tc.cu instead, on tiles of 128 pairs of this file's list, after
//                 moe_gather_rows has brought the tokens' rows into the pairs' order; steps of few tokens run the weight
//                 streaming product of csrc/gemm_tc_stream.cu behind moe_plan_few, which is the route, the sort and the
//                 gathering in one kernel
//   moe_combine   residual[t] += sum over slots of weight * the pair's row (+ gate * the shared expert's row)
// Everything the host needs to launch them is known before the step: no count is read back.
#include <cfloat>
#include "common.cuh"

using namespace mir;

namespace {

constexpr int kExpertTile = 8;        // pairs of one expert that a CTA of the grouped product takes
constexpr int kTensorTile = 128;      // rows of a tile of the tcgen05 grouped product (csrc/gemm_tc.cu)
constexpr int kMaxExperts = 1024;

__device__ __forceinline__ float sigmoid_of(float z) { return 1.0f / (1.0f + expf(-z)); }

// One warp per token, four tokens a CTA.  logits [tokens, >= experts (+ 1)] 32-bit: the router's logits and, behind
// them, the shared expert's gate logit (has_gate).  Shared memory per warp: score[E] | choice[E] | group score[groups] |
// the chosen scores[top] (RANKED).
// Among equal scores the expert (or group) with the lower index wins.
constexpr int kRouteWarps = 4;
// Whether a token's experts are ranked by counting, every expert against every other (a lane's own ones at a time), or searched
// for slot by slot.  The first takes experts / 32 rounds of `experts` comparisons, a slot of the second about as long as 32 of
// them: three tokens, 64 experts 4.1 us ranked and 2.8 / 3.4 / 5.3 / 6.3 searched for 1 / 2 / 6 / 8 slots, 32 experts 2.7 and 2.7 to
// 5.7.  More than 64 are never ranked: 2,000 tokens, 96 experts 9.7 us ranked and 5.2 to 7.9 searched, 256 experts 47 and 6.7 to 9.3.
__host__ __device__ constexpr bool route_by_rank(int experts, int top) {
  return experts <= 64 && (experts + 31) / 32 * experts <= 32 * top;
}

__device__ __forceinline__ void warp_best(float& value, int& index, bool want_max) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_xor_sync(0xffffffffu, value, o);
    const int other_index = __shfl_xor_sync(0xffffffffu, index, o);
    const bool better = want_max ? (other > value || (other == value && other_index < index))
                                 : (other < value || (other == value && other_index > index));
    if (other_index >= 0 && (index < 0 || better)) { value = other; index = other_index; }
  }
}

// One token's choice by one warp.  z: its logits; score, choice [experts], group_score [groups], chosen [top] (RANKED): shared
// memory of this warp.  ids_out, weights_out [top]: shared or global memory.
struct RouteRule {
  const float* correction;
  int experts, top, groups, keep;
  float scale;
  int softmax_scores, group_by_max;
};
template <bool RANKED>
__device__ __forceinline__ void route_token(const float* z, const RouteRule& rule, float* score, float* choice,
                                            float* group_score, float* chosen, int lane, int* ids_out, float* weights_out) {
  const int experts = rule.experts, top = rule.top, groups = rule.groups, keep = rule.keep;
  float softmax_top = 0.0f, softmax_inverse = 1.0f;
  if (rule.softmax_scores) {                                     // over all the router's experts, in 32-bit
    float high = -FLT_MAX;
    for (int e = lane; e < experts; e += 32) high = fmaxf(high, z[e]);
    softmax_top = warp_max(high);
    float sum = 0.0f;
    for (int e = lane; e < experts; e += 32) sum += expf(z[e] - softmax_top);
    softmax_inverse = 1.0f / warp_sum(sum);
  }
  for (int e = lane; e < experts; e += 32) {
    const float s = rule.softmax_scores ? expf(z[e] - softmax_top) * softmax_inverse : sigmoid_of(z[e]);
    score[e] = s;
    // (plain softmax scores are in the logits' order: the choice then looks at the logits, which do not underflow)
    choice[e] = rule.correction != nullptr ? s + rule.correction[e] : (rule.softmax_scores && keep >= groups ? z[e] : s);
  }
  __syncwarp();
  const int per_group = experts / groups;
  if (keep < groups) {
    // a group's score: the sum of its two largest choice scores (of its one score where a group is one expert)
    for (int g = lane; g < groups; g += 32) {
      float first = -FLT_MAX, second = -FLT_MAX;
#pragma unroll 8
      for (int e = g * per_group; e < (g + 1) * per_group; ++e) {
        const float c = choice[e];
        if (c > first) { second = first; first = c; }
        else if (c > second) second = c;
      }
      group_score[g] = (per_group > 1 && !rule.group_by_max) ? first + second : first;
    }
    __syncwarp();
    // experts of all but the `keep` best groups cannot be chosen: their choice scores count as minus infinity
    if (groups <= 32) {                                          // a group's rank: how many are better (or as good and before it)
      const float mine = lane < groups ? group_score[lane] : 0.0f;
      int rank = 0;
#pragma unroll 8
      for (int g = 0; g < groups; ++g) {
        const float other = group_score[g];
        rank += other > mine || (other == mine && g < lane);
      }
      const unsigned dropped = __ballot_sync(0xffffffffu, lane < groups && rank >= keep);
      for (int e = lane; e < experts; e += 32)
        if (dropped >> (e / per_group) & 1) choice[e] = -FLT_MAX;
      __syncwarp();
    } else
    for (int round = 0; round < groups - keep; ++round) {
      float low = FLT_MAX;
      int worst = -1;
      for (int g = lane; g < groups; g += 32) {
        const float v = group_score[g];
        if (v != FLT_MAX && (worst < 0 || v <= low)) { low = v; worst = g; }     // (among equals the later group goes)
      }
      warp_best(low, worst, false);
      if (worst < 0) break;
      if (lane == 0) group_score[worst] = FLT_MAX;                // marked as dropped
      for (int e = worst * per_group + lane; e < (worst + 1) * per_group; e += 32) choice[e] = -FLT_MAX;
      __syncwarp();
    }
  }
  float total = 0.0f;
  if constexpr (RANKED) {
    // An expert's rank among those that can be chosen is its slot: every lane counts for its own experts at once, instead
    // of one search over the warp for each slot (three tokens, 64 experts in 8 groups, 6 chosen: 9.2 us by searches).
    // route_by_rank: at most 64 experts, two a lane.
    const int e0 = lane, e1 = lane + 32;
    const float mine0 = e0 < experts ? choice[e0] : -FLT_MAX, mine1 = e1 < experts ? choice[e1] : -FLT_MAX;
    const bool can0 = mine0 > -FLT_MAX, can1 = mine1 > -FLT_MAX;
    int rank0 = 0, rank1 = 0;
#pragma unroll 16
    for (int other = 0; other < experts; ++other) {
      const float theirs = choice[other];
      rank0 += theirs > mine0 || (theirs == mine0 && other < e0);
      rank1 += theirs > mine1 || (theirs == mine1 && other < e1);
    }
    if (can0 && rank0 < top) { ids_out[rank0] = e0; chosen[rank0] = score[e0]; }
    if (can1 && rank1 < top) { ids_out[rank1] = e1; chosen[rank1] = score[e1]; }
    const int choosable = __popc(__ballot_sync(0xffffffffu, can0)) + __popc(__ballot_sync(0xffffffffu, can1));
    for (int slot = choosable + lane; slot < top; slot += 32) {  // (fewer choosable experts than top: not a valid model)
      ids_out[slot] = 0;
      chosen[slot] = score[0];
    }
    __syncwarp();
#pragma unroll 8
    for (int slot = 0; slot < top; ++slot) total += chosen[slot];
    const float factor = rule.scale / (total + 1e-20f);
    for (int slot = lane; slot < top; slot += 32) weights_out[slot] = chosen[slot] * factor;
  } else {
    for (int slot = 0; slot < top; ++slot) {
      float high = -FLT_MAX;
      int best = -1;
      for (int e = lane; e < experts; e += 32) {
        const float c = choice[e];
        if (c > high) { high = c; best = e; }
      }
      if (best >= 0 && high == -FLT_MAX) best = -1;
      warp_best(high, best, true);
      if (best < 0) best = 0;                                      // (fewer choosable experts than top: not a valid model)
      if (lane == 0) {
        choice[best] = -FLT_MAX;
        ids_out[slot] = best;
        weights_out[slot] = score[best];
      }
      total += score[best];
      __syncwarp();
    }
    const float factor = rule.scale / (total + 1e-20f);
    for (int slot = lane; slot < top; slot += 32) weights_out[slot] *= factor;
  }
}

template <bool RANKED>
__global__ void moe_route_kernel(const float* __restrict__ logits, long long ld, int has_gate, int* __restrict__ ids,
                                 float* __restrict__ weights, float* __restrict__ shared_gate, int tokens, RouteRule rule) {
  extern __shared__ float route_shared[];
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x, warp = threadIdx.y;
  const int token = blockIdx.x * kRouteWarps + warp;
  if (token >= tokens) return;
  const int experts = rule.experts;
  float* score = route_shared + (size_t)warp * (2 * experts + rule.groups + (RANKED ? rule.top : 0));
  const float* z = logits + (size_t)token * ld;
  if (has_gate && lane == 0) shared_gate[token] = sigmoid_of(z[experts]);
  route_token<RANKED>(z, rule, score, score + experts, score + 2 * experts, score + 2 * experts + rule.groups, lane,
                      ids + (size_t)token * rule.top, weights + (size_t)token * rule.top);
}

// The pairs ordered by expert, in three small kernels.  order[i] = the i-th pair when the pairs are sorted by expert
// (pairs of one expert stay in their own order); offsets[e] .. offsets[e + 1] is expert e's range in it; tiles[2 n],
// tiles[2 n + 1] = expert and first sorted pair of the n-th tile of tile_pairs pairs, tile_count[0] = how many there are.

// All of the sort in one CTA, for the pairs of decoded tokens (up to kFewPairs): three launches' work in one
// (18 pairs of 64 experts 3.0 us, the three 5.5; 256 pairs 4.8 and 5.3).  A pair's place is counted over the pairs before it,
// which is why more go to the kernels below (384 pairs 5.9 us and 6.3; 510 pairs 7.1 and 6.3).
constexpr int kFewPairs = 416;
__global__ void __launch_bounds__(kMaxExperts)
moe_sort_few_kernel(const int* __restrict__ ids, int pairs, int experts, int tile_pairs, int* __restrict__ order,
                    int* __restrict__ offsets, int* __restrict__ tiles, int* __restrict__ tile_count) {
  __shared__ int id_s[kFewPairs], count_s[kMaxExperts], base_s[kMaxExperts], pair_sums[32], tile_sums[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5;       // a thread: one expert, and one pair
  count_s[e] = 0;
  const int id = e < pairs ? ids[e] : -1;
  if (e < pairs) id_s[e] = id;
  __syncthreads();
  const bool sorted = id >= 0 && id < experts;                   // (identity experts have ids beyond: they are left out)
  if (sorted) atomicAdd(&count_s[id], 1);
  __syncthreads();
  const int mine = e < experts ? count_s[e] : 0;
  const int my_tiles = (mine + tile_pairs - 1) / tile_pairs;
  int pair_scan = mine, tile_scan = my_tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, pair_scan, o), t = __shfl_up_sync(0xffffffffu, tile_scan, o);
    if (lane >= o) { pair_scan += a; tile_scan += t; }
  }
  if (lane == 31) { pair_sums[warp] = pair_scan; tile_sums[warp] = tile_scan; }
  __syncthreads();
  int pair_base = pair_scan - mine, tile_base = tile_scan - my_tiles;
  for (int w = 0; w < warp; ++w) { pair_base += pair_sums[w]; tile_base += tile_sums[w]; }
  base_s[e] = pair_base;
  if (e < experts) {
    offsets[e] = pair_base;
    for (int t = 0; t < my_tiles; ++t) {
      tiles[2 * (tile_base + t)] = e;
      tiles[2 * (tile_base + t) + 1] = pair_base + t * tile_pairs;
    }
  }
  if (e == experts - 1) {
    offsets[experts] = pair_base + mine;
    tile_count[0] = tile_base + my_tiles;
  }
  __syncthreads();
  if (!sorted) return;
  int before = 0;                                                // pairs of the same expert ahead of this one
#pragma unroll 8
  for (int p = 0; p < e; ++p) before += id_s[p] == id;
  order[base_s[id] + before] = e;
}

// Everything between the router's logits and the grouped products for a step of few tokens, in one kernel: a warp routes a
// token, the pairs are ordered as moe_sort_few_kernel orders them, and the tokens' rows are brought into that order.  Every
// CTA routes for itself (it takes the time of one token's chain of dependent steps, whoever does it).  The first one leaves
// the results and the lists; the others hold 16 bytes of one token a thread, asked for beside the logits, and store them at
// the places of the token's pairs.  A place is counted over all pairs, which needs no barrier but the one behind the routing.
// It goes over its instructions twice: first, while the kernel in front still runs, on logits of zero, leaving nothing.  A
// decoded token's weights have pushed this code out of the caches by the time a layer comes here, and a chain of
// instruction fetches from memory takes longer than the routing.  Three tokens, 64 experts in 8 groups, 6 chosen, rows of
// 2,048, inside a captured decode step: route, sort and gathering took 6.3 + 3.2 + 2.5 us one behind the other, this kernel
// 8.1 without the first pass and 5.4 with it.
// Shared memory: ids [pairs, a multiple of four, the rest INT_MAX] | weights, later the places [pairs] | zeros [experts] |
// the warps' scratch of route_token.
constexpr int kPlanThreads = 512;
template <bool RANKED>
__global__ void __launch_bounds__(kPlanThreads)
moe_plan_few_kernel(const float* logits, long long ld, int has_gate, int* __restrict__ ids,
                    float* __restrict__ weights, float* __restrict__ shared_gate, int tokens, RouteRule rule, int real_experts,
                    int tile_pairs, int* __restrict__ order, int* __restrict__ offsets, int* __restrict__ tiles,
                    int* __restrict__ tile_count, const uint4* h, long long ld_pieces, uint4* __restrict__ sorted_rows,
                    int pieces) {
  // (logits and h carry no __restrict__: as invariant loads the compiler moves them in front of both passes, and so in front
  // of the wait)
  extern __shared__ __align__(16) float plan_shared[];
  __shared__ int tile_sums[kPlanThreads / 32];
  const int thread = threadIdx.x, lane = thread & 31, warp = thread >> 5;
  const int top = rule.top, pairs = tokens * top, quads = (pairs + 3) / 4;
  const int scratch = 2 * rule.experts + rule.groups + (RANKED ? top : 0);
  int* id_s = reinterpret_cast<int*>(plan_shared);
  float* weight_s = plan_shared + 4 * quads;
  float* zeros = weight_s + pairs;
  float* scratch_s = zeros + rule.experts;
  if (thread < 4) id_s[4 * quads - 1 - thread] = 0x7fffffff;
  for (int e = thread; e < rule.experts; e += kPlanThreads) zeros[e] = 0.0f;
  const long long copied = (long long)((int)blockIdx.x - 1) * kPlanThreads + thread;   // of the tokens' pieces
  const int token = copied >= 0 && copied < (long long)tokens * pieces ? (int)(copied / pieces) : -1;
  const int piece = (int)(copied - (long long)token * pieces);
  __syncthreads();
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const bool real = pass == 1;
    if (real) {
      grid_dependency_wait();
      grid_launch_dependents();
    }
    uint4 held = make_uint4(0, 0, 0, 0);
    if (real && token >= 0) held = h[(size_t)token * ld_pieces + piece];
#pragma unroll 1
    for (int t = warp; t < tokens; t += kPlanThreads / 32) {
      const float* z = real ? logits + (size_t)t * ld : zeros;
      float* score = scratch_s + (size_t)t * scratch;
      if (real && has_gate && lane == 0 && blockIdx.x == 0) shared_gate[t] = sigmoid_of(z[rule.experts]);
      route_token<RANKED>(z, rule, score, score + rule.experts, score + 2 * rule.experts, score + 2 * rule.experts + rule.groups,
                          lane, id_s + t * top, weight_s + t * top);
    }
    __syncthreads();
    // the place of pair p: the pairs of experts before its own, and those of its own ahead of it; -1 for an identity
    // expert, whose pairs are left out
    auto place_of = [&](int p) {
      const int id = id_s[p];
      int place = 0;
#pragma unroll 4
      for (int q = 0; q < quads; ++q) {
        const int4 ids4 = reinterpret_cast<const int4*>(id_s)[q];
        place += ids4.x < id || (ids4.x == id && 4 * q < p);
        place += ids4.y < id || (ids4.y == id && 4 * q + 1 < p);
        place += ids4.z < id || (ids4.z == id && 4 * q + 2 < p);
        place += ids4.w < id || (ids4.w == id && 4 * q + 3 < p);
      }
      return id < real_experts ? place : -1;
    };
    if (blockIdx.x > 0) {
      int* place_s = reinterpret_cast<int*>(weight_s);
      for (int p = thread; p < pairs; p += kPlanThreads) place_s[p] = place_of(p);
      __syncthreads();
      if (token >= 0)
        for (int slot = 0; slot < top; ++slot) {
          const int place = place_s[token * top + slot];
          if (real && place >= 0) sorted_rows[(size_t)place * pieces + piece] = held;
        }
    } else {
      for (int p = thread; p < pairs; p += kPlanThreads) {
        const int place = place_of(p);
        if (real) {
          ids[p] = id_s[p];
          weights[p] = weight_s[p];
          if (place >= 0) order[place] = p;
        }
      }
      int tiles_before = 0;                                      // tiles of the experts of earlier rounds
#pragma unroll 1
      for (int first = 0; first < real_experts; first += kPlanThreads) {
        const int e = first + thread;
        int before = 0, mine = 0;                                // pairs of the experts before e, and of e
#pragma unroll 4
        for (int q = 0; q < quads; ++q) {
          const int4 ids4 = reinterpret_cast<const int4*>(id_s)[q];
          before += (ids4.x < e) + (ids4.y < e) + (ids4.z < e) + (ids4.w < e);
          mine += (ids4.x == e) + (ids4.y == e) + (ids4.z == e) + (ids4.w == e);
        }
        const int my_tiles = e < real_experts ? (mine + tile_pairs - 1) / tile_pairs : 0;
        int scan = my_tiles;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, scan, o);
          if (lane >= o) scan += t;
        }
        if (lane == 31) tile_sums[warp] = scan;
        __syncthreads();
        int base = tiles_before + scan - my_tiles;
#pragma unroll 4
        for (int w = 0; w < kPlanThreads / 32; ++w) {
          if (w < warp) base += tile_sums[w];
          tiles_before += tile_sums[w];
        }
        if (real && e < real_experts) {
          offsets[e] = before;
          for (int t = 0; t < my_tiles; ++t) {
            tiles[2 * (base + t)] = e;
            tiles[2 * (base + t) + 1] = before + t * tile_pairs;
          }
          if (e == real_experts - 1) {
            offsets[real_experts] = before + mine;
            tile_count[0] = base + my_tiles;
          }
        }
        __syncthreads();                                         // (tile_sums is written again in the next round)
      }
    }
    __syncthreads();                                             // (the ids are written again in the next pass)
  }
}

// One CTA per expert: how many pairs chose it.  (A prompt's 15,000 pairs are a few trips over the L2 for 1,024 threads.)
template <int THREADS>
__global__ void __launch_bounds__(THREADS) moe_count_kernel(const int* __restrict__ ids, int pairs, int* __restrict__ counts) {
  __shared__ float scratch[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const int expert = blockIdx.x;
  int n = 0;
#pragma unroll 4
  for (int p = threadIdx.x; p < pairs; p += THREADS) n += ids[p] == expert;
  const float total = block_sum((float)n, scratch);              // (exact: fewer than 2^24 pairs)
  if (threadIdx.x == 0) counts[expert] = (int)(total + 0.5f);
}

// One CTA: the experts' ranges and first tiles (an exclusive scan over at most kMaxExperts counts).
__global__ void moe_offsets_kernel(const int* __restrict__ counts, int experts, int tile_pairs, int* __restrict__ offsets,
                                   int* __restrict__ first_tile, int* __restrict__ tile_count) {
  __shared__ int pair_sums[32], tile_sums[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;    // 1024 threads: one expert each
  const int e = threadIdx.x;
  const int mine = e < experts ? counts[e] : 0;
  const int my_tiles = (mine + tile_pairs - 1) / tile_pairs;
  int pair_scan = mine, tile_scan = my_tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, pair_scan, o), t = __shfl_up_sync(0xffffffffu, tile_scan, o);
    if (lane >= o) { pair_scan += a; tile_scan += t; }
  }
  if (lane == 31) { pair_sums[warp] = pair_scan; tile_sums[warp] = tile_scan; }
  __syncthreads();
  if (warp == 0) {
    int a = pair_sums[lane], t = tile_sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) { a += x; t += y; }
    }
    pair_sums[lane] = a;
    tile_sums[lane] = t;
  }
  __syncthreads();
  const int pair_base = (warp ? pair_sums[warp - 1] : 0) + pair_scan - mine;
  const int tile_base = (warp ? tile_sums[warp - 1] : 0) + tile_scan - my_tiles;
  if (e < experts) {
    offsets[e] = pair_base;
    first_tile[e] = tile_base;
  }
  if (e == experts - 1) {
    offsets[experts] = pair_base + mine;
    tile_count[0] = tile_base + my_tiles;
  }
}

// One CTA per expert: its pairs into their places, in their own order, and its tiles.  A warp counts a run of the pairs, and
// behind one barrier places them (15,000 pairs, 64 experts: 19.5 us when every 256 pairs met at two barriers).
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
moe_place_kernel(const int* __restrict__ ids, int pairs, int tile_pairs, const int* __restrict__ offsets,
                 const int* __restrict__ first_tile, int* __restrict__ order, int* __restrict__ tiles) {
  constexpr int WARPS = THREADS / 32;
  __shared__ int warp_counts[WARPS];
  grid_dependency_wait();
  grid_launch_dependents();
  const int expert = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int begin = offsets[expert], total = offsets[expert + 1] - begin;
  const int n = (total + tile_pairs - 1) / tile_pairs;
  for (int t = threadIdx.x; t < n; t += THREADS) {
    tiles[2 * (first_tile[expert] + t)] = expert;
    tiles[2 * (first_tile[expert] + t) + 1] = begin + t * tile_pairs;
  }
  const int run = ((pairs + WARPS - 1) / WARPS + 31) / 32 * 32;  // pairs of a warp
  const int first = warp * run, last = min(first + run, pairs);
  int mine = 0;
#pragma unroll 4
  for (int p = first + lane; p < last; p += 32) mine += ids[p] == expert;
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0) warp_counts[warp] = mine;
  __syncthreads();
  int at = begin;
  for (int w = 0; w < warp; ++w) at += warp_counts[w];
  if (mine == 0) return;
#pragma unroll 4
  for (int base = first; base < last; base += 32) {
    const int p = base + lane;
    const bool here = p < last && ids[p] == expert;
    const unsigned ballot = __ballot_sync(0xffffffffu, here);
    if (here) order[at + __popc(ballot & ((1u << lane) - 1u))] = p;
    at += __popc(ballot);
  }
}

__device__ __forceinline__ void load4(const float* p, float (&out)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&out)[4]) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
  const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
  out[0] = a.x; out[1] = a.y; out[2] = b.x; out[3] = b.y;
}

constexpr int kGroupedWarps = 8;
constexpr int kGroupedPerWarp = 4;                               // outputs a warp computes for the tile's pairs
constexpr int kGroupedChunk = 512;                               // inputs staged at a time

// blockDim (32, kGroupedWarps); grid (tile slots, ceil(N / 32)).  The rows of a tile's pairs are staged in shared
// memory 512 inputs at a time; a warp walks over a weight row with its lanes side by side (4 inputs a lane) and keeps
// one sum per pair.  Every output is the same chain of partial sums and the same tree over the lanes whatever the
// batch holds.  x row of sorted pair i: gather == null ? i : gather[i] / gather_div; out row: scatter == null ? i :
// scatter[i].  GATED: out = silu(w_a x) * (w_b x), else out = w_a x.
template <typename T, typename TO, bool GATED>
__global__ void __launch_bounds__(kGroupedWarps * 32)
moe_grouped_kernel(const T* __restrict__ x, long long ldx, const int* __restrict__ gather, int gather_div,
                   const T* __restrict__ w_a, const T* __restrict__ w_b, TO* __restrict__ out, long long ldo,
                   const int* __restrict__ scatter, const int* __restrict__ tiles, const int* __restrict__ tile_count,
                   const int* __restrict__ offsets, int K, int N) {
  __shared__ __align__(16) float rows[kExpertTile][kGroupedChunk];
  __shared__ int source[kExpertTile];
  grid_dependency_wait();
  grid_launch_dependents();
  if ((int)blockIdx.x >= tile_count[0]) return;
  const int lane = threadIdx.x, warp = threadIdx.y, thread = warp * 32 + lane;
  const int expert = tiles[2 * blockIdx.x], start = tiles[2 * blockIdx.x + 1];
  const int count = min(kExpertTile, offsets[expert + 1] - start);
  if (thread < kExpertTile)
    source[thread] = thread < count ? (gather != nullptr ? gather[start + thread] / gather_div : start + thread) : -1;
  const int first_output = blockIdx.y * (kGroupedWarps * kGroupedPerWarp) + warp * kGroupedPerWarp;
  float acc_a[kGroupedPerWarp][kExpertTile], acc_b[GATED ? kGroupedPerWarp : 1][kExpertTile];
#pragma unroll
  for (int j = 0; j < kGroupedPerWarp; ++j)
#pragma unroll
    for (int r = 0; r < kExpertTile; ++r) {
      acc_a[j][r] = 0.0f;
      if (GATED) acc_b[j][r] = 0.0f;
    }
  const bool wide = K % 4 == 0;
  for (int from = 0; from < K; from += kGroupedChunk) {
    const int here = min(kGroupedChunk, K - from);
    __syncthreads();
    for (int index = thread; index < kExpertTile * here; index += kGroupedWarps * 32) {
      const int r = index / here, i = index - r * here;
      rows[r][i] = source[r] >= 0 ? to_float(x[(size_t)source[r] * ldx + from + i]) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kGroupedPerWarp; ++j) {
      const int o = first_output + j;
      if (o >= N) break;
      const T* row_a = w_a + ((size_t)expert * N + o) * K + from;
      const T* row_b = GATED ? w_b + ((size_t)expert * N + o) * K + from : nullptr;
      if (wide) {
        for (int i = lane * 4; i < here; i += 128) {
          float a[4], b[4];
          load4(row_a + i, a);
          if (GATED) load4(row_b + i, b);
#pragma unroll
          for (int r = 0; r < kExpertTile; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(&rows[r][i]);
            acc_a[j][r] = fmaf(a[3], v.w, fmaf(a[2], v.z, fmaf(a[1], v.y, fmaf(a[0], v.x, acc_a[j][r]))));
            if (GATED) acc_b[j][r] = fmaf(b[3], v.w, fmaf(b[2], v.z, fmaf(b[1], v.y, fmaf(b[0], v.x, acc_b[j][r]))));
          }
        }
      } else {
        for (int i = lane; i < here; i += 32) {
          const float a = to_float(row_a[i]);
          const float b = GATED ? to_float(row_b[i]) : 0.0f;
#pragma unroll
          for (int r = 0; r < kExpertTile; ++r) {
            acc_a[j][r] = fmaf(a, rows[r][i], acc_a[j][r]);
            if (GATED) acc_b[j][r] = fmaf(b, rows[r][i], acc_b[j][r]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kGroupedPerWarp; ++j) {
    const int o = first_output + j;
#pragma unroll
    for (int r = 0; r < kExpertTile; ++r) {
      const float a = warp_sum(acc_a[j][r]);
      const float b = GATED ? warp_sum(acc_b[j][r]) : 0.0f;
      if (lane == r && r < count && o < N) {
        const int to = scatter != nullptr ? scatter[start + r] : start + r;
        const float value = GATED ? a / (1.0f + expf(-a)) * b : a;
        out[(size_t)to * ldo + o] = from_float<TO>(value);
      }
    }
  }
}

// One CTA per token: residual[t] += sum_s weights[t, s] * pair_rows[t * top + s] (+ shared_gate[t] * shared_rows[t], or
// + shared_rows[t] without a gate), slots in their own order.  A slot whose expert is an identity expert (ids[pair] >=
// real_experts) has no row: it adds weight * the token's own input (identity_rows, in the activations' type).
// overwrite: the sum replaces residual[t] instead of being added to it.
// A thread takes V neighbouring columns of one token (V = 4 where rows and pointers allow 16-byte accesses), a CTA a
// run of columns (blockIdx.y): few tokens still fill the GPU.  A column's sum runs over the slots in ascending order,
// then the shared expert, whatever V is.
template <typename T, int V>
__global__ void moe_combine_kernel(float* __restrict__ residual, const float* __restrict__ pair_rows,
                                   const float* __restrict__ weights, const float* __restrict__ shared_rows,
                                   const float* __restrict__ shared_gate, int width, int top, int overwrite,
                                   const int* __restrict__ ids, int real_experts, const T* __restrict__ identity_rows,
                                   long long identity_stride) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int token = blockIdx.x;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * V;
  if (c >= width) return;
  float total[V];
#pragma unroll
  for (int v = 0; v < V; ++v) total[v] = 0.0f;
  const size_t at = (size_t)token * width + c;
  // What does not depend on the slots, and the rows of kAhead slots, are asked for before the first sum: one trip to memory
  // for them instead of one for every slot (three tokens, six slots, rows of 2,048: 4.2 us, now 2.4).
  alignas(16) float old[V], shared[V];
#pragma unroll
  for (int v = 0; v < V; ++v) old[v] = overwrite ? 0.0f : residual[at + v];
#pragma unroll
  for (int v = 0; v < V; ++v) shared[v] = shared_rows != nullptr ? shared_rows[at + v] : 0.0f;
  const float gate = shared_rows != nullptr && shared_gate != nullptr ? shared_gate[token] : 1.0f;
  constexpr int kAhead = 4;
  for (int s0 = 0; s0 < top; s0 += kAhead) {
    alignas(16) float row[kAhead][V];
    float weight[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (s0 + j >= top) break;
      const size_t pair = (size_t)token * top + s0 + j;
      weight[j] = __ldg(weights + pair);
      if (ids != nullptr && __ldg(ids + pair) >= real_experts) {
        const T* src = identity_rows + (size_t)token * identity_stride + c;
#pragma unroll
        for (int v = 0; v < V; ++v) row[j][v] = to_float(src[v]);
      } else if (V == 4) {
        *reinterpret_cast<float4*>(row[j]) = *reinterpret_cast<const float4*>(pair_rows + pair * width + c);
      } else {
        row[j][0] = pair_rows[pair * width + c];
      }
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (s0 + j >= top) break;
#pragma unroll
      for (int v = 0; v < V; ++v) total[v] = fmaf(weight[j], row[j][v], total[v]);
    }
  }
  if (shared_rows != nullptr) {
#pragma unroll
    for (int v = 0; v < V; ++v) total[v] = fmaf(gate, shared[v], total[v]);
  }
#pragma unroll
  for (int v = 0; v < V; ++v) residual[at + v] = overwrite ? total[v] : old[v] + total[v];
}

template <typename T, typename TO, bool GATED>
int launch_grouped(cudaStream_t stream, const void* x, long long ldx, const int* gather, int gather_div, const void* w_a,
                   const void* w_b, void* out, long long ldo, const int* scatter, const int* tiles, const int* tile_count,
                   const int* offsets, int pairs, int experts, int K, int N) {
  const int slots = pairs / kExpertTile + experts;               // no more tiles than this, whatever the routing
  const dim3 grid(slots, (N + kGroupedWarps * kGroupedPerWarp - 1) / (kGroupedWarps * kGroupedPerWarp));
  return mir_launch(GATED ? "moe_grouped_gate_up" : "moe_grouped_down", moe_grouped_kernel<T, TO, GATED>, grid,
                    dim3(32, kGroupedWarps), 0, stream, 0, (const T*)x, ldx, gather, gather_div, (const T*)w_a,
                    (const T*)w_b, (TO*)out, ldo, scatter, tiles, tile_count, offsets, K, N);
}

}  // namespace

// logits [tokens, >= experts + has_gate] 32-bit with row stride ld: the router's logits (and the shared expert's gate
// logit behind them); correction [experts] (or null) 32-bit; ids, weights [tokens, top]; shared_gate [tokens].
MIR_EXPORT int mir_moe_route(const float* logits, long long ld, const float* correction, int has_gate, int* ids,
                             float* weights, float* shared_gate, int tokens, int experts, int top, int groups, int keep,
                             float scale, int softmax_scores, int group_by_max, cudaStream_t stream) {
  if (tokens == 0) return MIR_OK;
  if (tokens < 0 || experts <= 0 || experts > kMaxExperts || top <= 0 || top > experts || groups <= 0 ||
      experts % groups || keep <= 0 || keep > groups || (long long)keep * (experts / groups) < top ||
      (has_gate && shared_gate == nullptr)) {
    mir_set_error("moe_route: bad sizes (tokens %d, experts %d, top %d, groups %d of which %d are kept)", tokens, experts,
                  top, groups, keep);
    return MIR_BAD_ARGUMENT;
  }
  const bool ranked = route_by_rank(experts, top);
  const size_t smem = (size_t)kRouteWarps * (2 * experts + groups + (ranked ? top : 0)) * sizeof(float);
  return mir_launch("moe_route", ranked ? moe_route_kernel<true> : moe_route_kernel<false>,
                    dim3((tokens + kRouteWarps - 1) / kRouteWarps), dim3(32, kRouteWarps), smem, stream, 0, logits, ld,
                    has_gate, ids, weights, shared_gate, tokens,
                    RouteRule{correction, experts, top, groups, keep, scale, softmax_scores, group_by_max});
}

// Whether mir_moe_plan_few takes a step of these sizes: places are counted over all pairs, and its shared memory needs no
// opt-in.
static size_t plan_few_shared(int tokens, int experts, int top, int groups) {
  const size_t scratch = 2 * (size_t)experts + groups + (route_by_rank(experts, top) ? top : 0);
  return (tokens * scratch + 2 * (size_t)tokens * top + 3 + experts) * sizeof(float);
}
MIR_EXPORT int mir_moe_plan_few_takes(int tokens, int experts, int real_experts, int top, int groups) {
  return tokens > 0 && tokens <= 128 && real_experts > 0 && (long long)tokens * top <= kFewPairs && experts <= kMaxExperts &&
         plan_few_shared(tokens, experts, top, groups) <= 47 * 1024;
}

// mir_moe_route, mir_moe_sort (tiles of tile_pairs pairs) and mir_moe_gather_rows in one kernel, for the sizes that
// mir_moe_plan_few_takes says; the arguments are theirs.  `experts` counts the router's experts, `real_experts` those that
// have weights; h [tokens, width] bfloat16, sorted_rows [tokens * top, width].
MIR_EXPORT int mir_moe_plan_few(const float* logits, long long ld, const float* correction, int has_gate, int* ids,
                                float* weights, float* shared_gate, int tokens, int experts, int real_experts, int top,
                                int groups, int keep, float scale, int softmax_scores, int group_by_max, int tile_pairs,
                                int* order, int* offsets, int* tiles, int* tile_count, const void* h, long long ld_h,
                                void* sorted_rows, int width, cudaStream_t stream) {
  if (tokens == 0) return MIR_OK;
  if (tokens < 0 || experts <= 0 || experts > kMaxExperts || real_experts <= 0 || real_experts > experts || top <= 0 ||
      top > experts || groups <= 0 || experts % groups || keep <= 0 || keep > groups ||
      (long long)keep * (experts / groups) < top || (has_gate && shared_gate == nullptr) || tile_pairs <= 0 || width <= 0 ||
      width % 8 || ld_h % 8 || ((uintptr_t)h & 15) || ((uintptr_t)sorted_rows & 15) ||
      !mir_moe_plan_few_takes(tokens, experts, real_experts, top, groups)) {
    mir_set_error("moe_plan_few: bad sizes (tokens %d, experts %d of which %d have weights, top %d, groups %d of which %d are "
                  "kept, tiles of %d pairs, rows of %d with stride %lld)", tokens, experts, real_experts, top, groups, keep,
                  tile_pairs, width, ld_h);
    return MIR_BAD_ARGUMENT;
  }
  const bool ranked = route_by_rank(experts, top);
  const int pieces = width / 8;
  const long long copies = ((long long)tokens * pieces + kPlanThreads - 1) / kPlanThreads;
  return mir_launch_with(mir_pdl_for_streaming(), "moe_plan_few", ranked ? moe_plan_few_kernel<true> : moe_plan_few_kernel<false>,
                         dim3((unsigned)(1 + copies)), dim3(kPlanThreads), plan_few_shared(tokens, experts, top, groups), stream, 0,
                         logits, ld, has_gate, ids, weights, shared_gate, tokens,
                         RouteRule{correction, experts, top, groups, keep, scale, softmax_scores, group_by_max}, real_experts,
                         tile_pairs, order, offsets, tiles, tile_count, (const uint4*)h, ld_h / 8, (uint4*)sorted_rows, pieces);
}

// How many tiles of tile_pairs pairs there can be at most for `pairs` pairs over `experts` experts (`tiles` holds two
// ints for each).
MIR_EXPORT int mir_moe_tile_slots(int pairs, int experts, int tile_pairs) { return pairs / tile_pairs + experts; }

// tile_pairs: 8 for the 32-bit grouped products of this file, 128 for the tcgen05 product (csrc/gemm_tc.cu).
// counts, first_tile: scratch of `experts` ints each.
MIR_EXPORT int mir_moe_sort(const int* ids, int pairs, int experts, int tile_pairs, int* order, int* offsets, int* tiles,
                            int* tile_count, int* counts, int* first_tile, cudaStream_t stream) {
  if (pairs == 0) return MIR_OK;
  if (pairs < 0 || experts <= 0 || experts > kMaxExperts ||
      (tile_pairs != kExpertTile && tile_pairs != kTensorTile)) {
    mir_set_error("moe_sort: bad sizes (pairs %d, experts %d, tiles of %d)", pairs, experts, tile_pairs);
    return MIR_BAD_ARGUMENT;
  }
  if (pairs <= kFewPairs)
    return mir_launch("moe_sort_few", moe_sort_few_kernel, dim3(1), dim3(kMaxExperts), 0, stream, 0, ids, pairs, experts,
                      tile_pairs, order, offsets, tiles, tile_count);
  // 1,024 threads an expert, but 256 where more CTAs of that size than an SM each holds have few pairs to go over: 768 pairs of
  // 300 experts 6.8 us (1,024 threads: 7.9), 1,536 of 300 7.8 (8.7), 4,096 of 300 10.0 (9.1); 768 of 200 6.8 (7.0), 1,536 of
  // 200 the same, 4,096 of 200 10.0 (7.8); 768 of 64 6.5 (6.3).
  const int sms = mir_sm_count();
  const bool many = experts <= sms || pairs >= (experts <= 2 * sms ? 1024 : 4096);
  int status = mir_launch("moe_count", many ? moe_count_kernel<1024> : moe_count_kernel<256>, dim3(experts), dim3(many ? 1024 : 256), 0, stream, 0, ids, pairs, counts);
  if (status != MIR_OK) return status;
  status = mir_launch("moe_offsets", moe_offsets_kernel, dim3(1), dim3(kMaxExperts), 0, stream, 0, counts, experts,
                      tile_pairs, offsets, first_tile, tile_count);
  if (status != MIR_OK) return status;
  return mir_launch("moe_place", many ? moe_place_kernel<1024> : moe_place_kernel<256>, dim3(experts), dim3(many ? 1024 : 256), 0, stream, 0, ids, pairs, tile_pairs,
                    offsets, first_tile, order, tiles);
}

// hidden[i] = silu(w_gate[e] x) * (w_up[e] x) for the i-th sorted pair, x the row of its token (order[i] / top) of h.
// w_gate, w_up [experts, inter, width]; hidden [pairs, inter] in the activations' type.
MIR_EXPORT int mir_moe_gate_up(int bf16, const void* h, long long ld, const int* order, int top, const void* w_gate,
                               const void* w_up, void* hidden, const int* tiles, const int* tile_count,
                               const int* offsets, int pairs, int experts, int width, int inter, int tile_pairs,
                               cudaStream_t stream) {
  if (pairs == 0) return MIR_OK;
  if (tile_pairs != kExpertTile) { mir_set_error("moe_gate_up: this kernel works on tiles of %d pairs", kExpertTile); return MIR_BAD_ARGUMENT; }
  if (bf16)
    return launch_grouped<__nv_bfloat16, __nv_bfloat16, true>(stream, h, ld, order, top, w_gate, w_up, hidden, inter,
                                                              nullptr, tiles, tile_count, offsets, pairs, experts, width,
                                                              inter);
  return launch_grouped<float, float, true>(stream, h, ld, order, top, w_gate, w_up, hidden, inter, nullptr, tiles,
                                            tile_count, offsets, pairs, experts, width, inter);
}

// pair_rows[order[i]] = w_down[e] hidden[i]: one 32-bit row [width] per pair, at the pair's own index.
MIR_EXPORT int mir_moe_down(int bf16, const void* hidden, const int* order, const void* w_down, float* pair_rows,
                            const int* tiles, const int* tile_count, const int* offsets, int pairs, int experts,
                            int width, int inter, int tile_pairs, cudaStream_t stream) {
  if (pairs == 0) return MIR_OK;
  if (tile_pairs != kExpertTile) { mir_set_error("moe_down: this kernel works on tiles of %d pairs", kExpertTile); return MIR_BAD_ARGUMENT; }
  if (bf16)
    return launch_grouped<__nv_bfloat16, float, false>(stream, hidden, inter, nullptr, 1, w_down, nullptr, pair_rows,
                                                       width, order, tiles, tile_count, offsets, pairs, experts, inter,
                                                       width);
  return launch_grouped<float, float, false>(stream, hidden, inter, nullptr, 1, w_down, nullptr, pair_rows, width, order,
                                             tiles, tile_count, offsets, pairs, experts, inter, width);
}

// sorted[i, :] = h[order[i] / top, :]: the tokens' rows in the order of the sorted pairs (16-byte pieces).
__global__ void moe_gather_rows_kernel(const uint4* __restrict__ h, long long ld_pieces, const int* __restrict__ order, int top,
                                       uint4* __restrict__ sorted, int pieces, size_t total,
                                       const int* __restrict__ sorted_count) {
  grid_dependency_wait();
  grid_launch_dependents();
  const size_t index = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= total) return;
  const size_t row = index / pieces;
  if (sorted_count != nullptr && row >= (size_t)sorted_count[0]) return;     // (pairs of identity experts are in no order)
  const int piece = (int)(index - row * pieces);
  sorted[index] = h[(size_t)(order[row] / top) * ld_pieces + piece];
}

// h [tokens, width] bfloat16 (row stride ld, both multiples of 8); sorted [pairs, width].  sorted_count (or null): one
// number on the device, how many of the pairs the order holds (the pairs of identity experts are left out of it).
MIR_EXPORT int mir_moe_gather_rows(const void* h, long long ld, const int* order, int top, void* sorted, int pairs,
                                   int width, const int* sorted_count, cudaStream_t stream) {
  if (pairs == 0) return MIR_OK;
  if (pairs < 0 || width <= 0 || width % 8 || ld % 8 || top <= 0) {
    mir_set_error("moe_gather_rows: rows of 16-byte pieces are needed (width %d, stride %lld)", width, ld);
    return MIR_BAD_ARGUMENT;
  }
  const int pieces = width / 8;
  const size_t total = (size_t)pairs * pieces;
  return mir_launch("moe_gather_rows", moe_gather_rows_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, 0,
                    (const uint4*)h, ld / 8, order, top, (uint4*)sorted, pieces, total, sorted_count);
}

MIR_EXPORT int mir_moe_combine(float* residual, const float* pair_rows, const float* weights, const float* shared_rows,
                               const float* shared_gate, int tokens, int width, int top, int overwrite, const int* ids,
                               int real_experts, int bf16, const void* identity_rows, long long identity_stride,
                               cudaStream_t stream) {
  if (tokens == 0) return MIR_OK;
  if (ids != nullptr && identity_rows == nullptr) {
    mir_set_error("moe_combine: identity experts need the tokens' input rows");
    return MIR_BAD_ARGUMENT;
  }
  const bool wide = width % 4 == 0 && ((uintptr_t)pair_rows & 15) == 0;
  const int per_thread = wide ? 4 : 1;
  const int threads = width >= 1024 * per_thread ? 256 : 128;
  const dim3 grid(tokens, (width + threads * per_thread - 1) / (threads * per_thread));
#define MIR_COMBINE(T, V)                                                                                             \
  return mir_launch("moe_combine", moe_combine_kernel<T, V>, grid, dim3(threads), 0, stream, 0, residual, pair_rows,   \
                    weights, shared_rows, shared_gate, width, top, overwrite, ids, real_experts, (const T*)identity_rows, \
                    identity_stride)
  if (bf16) {
    if (wide) MIR_COMBINE(__nv_bfloat16, 4);
    MIR_COMBINE(__nv_bfloat16, 1);
  }
  if (wide) MIR_COMBINE(float, 4);
  MIR_COMBINE(float, 1);
#undef MIR_COMBINE
}
