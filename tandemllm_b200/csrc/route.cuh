// The router's choice for one row, run by one full warp: scores (the sigmoid of each logit, or the softmax over all
// experts' logits), the top-k of score + bias (the bias for the choice only), weights = chosen scores, divided by
// (their sum + floor) when normalised, times scale.
// Ties go to the lower expert id; a NaN score is chosen only when nothing else is left.
// (engine/models/lfm2_moe/ref.py:185-197, engine/models/lfm2_moe/kernels.py:265-287 of the reference; the softmax
// scoring is what its other routed families use, engine/models/flashnext/ref.py:479-487)
// The third scoring function takes the bias as part of the logit: the k largest logits + bias are chosen, and their weights are
// the softmax over the chosen ones only (computed from the row's largest logit, which is always chosen).
//
// The launchers' `normalize` argument carries the router's choices: bit 0 = divide the chosen weights by their sum,
// bits 1..3 = the scoring function (TL_SCORE_SIGMOID 0, TL_SCORE_SOFTMAX 1, TL_SCORE_CHOSEN 2), bits 4..9 = the number of expert groups
// (0: the choice is free) and bits 10..15 = how many of them are kept.
//
// Group-limited choice: the experts form `groups` equal groups of neighbours; a group's score is the sum of its two
// largest choice scores (score + bias); only the experts of the `keep` best groups (ties to the lower group) can be
// chosen: the others' choice scores count as minus infinity.
#pragma once

#include "common.cuh"

namespace tl {

#define TL_SCORE_SIGMOID 0
#define TL_SCORE_SOFTMAX 1
#define TL_SCORE_CHOSEN 2
#define TL_SCORE_LAST 2
#define TL_ROUTE_SCORING(flags) (((flags) >> 1) & 7)
#define TL_ROUTE_GROUPS(flags) (((flags) >> 4) & 63)
#define TL_ROUTE_KEEP(flags) (((flags) >> 10) & 63)
#define TL_ROUTE_MAX_GROUPS 32

constexpr int MAX_EXPERTS = 1024;
constexpr int MAX_TOP_K = 32;

// A number as a whole number in the same order (minus infinity the smallest but above 0; both zeros alike; not for NaN), and back.
__device__ __forceinline__ uint32_t route_key(float f) {
  const uint32_t u = __float_as_uint(f == 0.f ? 0.f : f);
  return u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float route_value(uint32_t key) {
  return __uint_as_float(key ^ ((key >> 31) ? 0x80000000u : 0xffffffffu));
}

// `lg`: the row's E <= 32 PER logits (global or shared memory). Lanes 0..k-1 write ids[lane] and wts[lane], in the
// order of the choice (best first). PER: experts a lane holds.
template <int PER>
__device__ __forceinline__ void warp_route_sized(const float* lg, const float* __restrict__ bias, int E, int k,
                                                 int normalize, float floor_, float scale, int* ids, float* wts) {
  const int lane = threadIdx.x & 31;
  const int scoring = TL_ROUTE_SCORING(normalize);
  const int n_groups = TL_ROUTE_GROUPS(normalize), keep_groups = TL_ROUTE_KEEP(normalize);
  normalize &= 1;
  if (scoring == TL_SCORE_CHOSEN) {
    normalize = 1;
    floor_ = 0.f;
  }
  float score[PER], choice[PER];
  float top = -INFINITY, denom = 1.f;
  if (scoring == TL_SCORE_SOFTMAX) {        // the row's largest logit and the sum of exponentials, over the whole warp
#pragma unroll
    for (int t = 0; t < PER; ++t)
      if (lane + 32 * t < E) top = fmaxf(top, lg[lane + 32 * t]);
    top = warp_max(top);
    float part = 0.f;
#pragma unroll
    for (int t = 0; t < PER; ++t)
      if (lane + 32 * t < E) part += expf(lg[lane + 32 * t] - top);
    denom = warp_sum(part);
  }
  if (scoring == TL_SCORE_CHOSEN) {
#pragma unroll
    for (int t = 0; t < PER; ++t) {
      const int e = lane + 32 * t;
      if (e < E) top = fmaxf(top, bias ? lg[e] + bias[e] : lg[e]);
    }
    top = warp_max(top);
  }
#pragma unroll
  for (int t = 0; t < PER; ++t) {
    const int e = lane + 32 * t;
    if (e < E) {
      if (scoring == TL_SCORE_CHOSEN) {
        choice[t] = bias ? lg[e] + bias[e] : lg[e];
        score[t] = expf(choice[t] - top);
      } else {
        const float s = scoring == TL_SCORE_SOFTMAX ? expf(lg[e] - top) / denom : 1.f / (1.f + expf(-lg[e]));
        score[t] = s;
        choice[t] = bias ? s + bias[e] : s;
      }
      if (!(choice[t] == choice[t])) choice[t] = -INFINITY;
    } else {
      score[t] = 0.f;
      choice[t] = -INFINITY;
    }
  }
  // From here on a choice score is a whole number in the same order (route_key; 0: taken), so that the warp's largest is one
  // instruction. The loops over groups and over the chosen stay loops: one warp runs this once a row, with its instructions cold, and
  // unrolled it waited for those (64 experts, top-6 of 4 of 8 groups: the norm kernel 11.0 us with unrolled shuffles, 7.9 us so; 32
  // experts, top-4: 6.6 and 6.1 us).
  uint32_t key[PER];
#pragma unroll
  for (int t = 0; t < PER; ++t) key[t] = lane + 32 * t < E ? route_key(choice[t]) : 0u;
  if (n_groups > 1 && keep_groups < n_groups) {
    // lane g ends up with group g's score (at most 32 groups); every lane learns which groups are kept
    // (whether an expert is of a group is asked of its distance to the group's first: a group number kept for each of a lane's 32 experts
    // of a wide router spilled, the norm kernel with 512 experts 159 -> 174 us at 300 rows)
    const int per = E / n_groups;
    float mine = -INFINITY;
#pragma unroll 1
    for (int g = 0; g < n_groups; ++g) {
      uint32_t a = 0u, b = 0u;                      // the two largest keys of group g in this lane
#pragma unroll
      for (int t = 0; t < PER; ++t) {
        const uint32_t c = (unsigned)(lane + 32 * t - g * per) < (unsigned)per ? key[t] : 0u;
        b = max(b, min(a, c));
        a = max(a, c);
      }
      const uint32_t first = __reduce_max_sync(0xffffffffu, a);
      const int holder = __ffs(__ballot_sync(0xffffffffu, a == first)) - 1;
      const uint32_t second = __reduce_max_sync(0xffffffffu, lane == holder ? b : a);
      const float fa = route_value(first), fb = second ? route_value(second) : -INFINITY;
      if (lane == g) mine = fb == -INFINITY ? fa : fa + fb;
    }
    int rank = 0;
#pragma unroll 1
    for (int g = 0; g < n_groups; ++g) {
      const float other = __shfl_sync(0xffffffffu, mine, g);
      rank += (other > mine) || (other == mine && g < lane);
    }
    const unsigned kept = __ballot_sync(0xffffffffu, lane < n_groups && rank < keep_groups);
#pragma unroll
    for (int t = 0; t < PER; ++t)
      if (key[t] && !((kept >> ((lane + 32 * t) / per)) & 1u)) key[t] = route_key(-INFINITY);
  }
  float sum = 0.f, my_w = 0.f;
  int my_id = 0;
#pragma unroll 1
  for (int j = 0; j < k; ++j) {
    uint32_t best = 0u;
#pragma unroll
    for (int t = 0; t < PER; ++t) best = max(best, key[t]);
    const uint32_t top_key = __reduce_max_sync(0xffffffffu, best);
    uint32_t e = 0xffffffffu;                       // this lane's lowest expert with that key
#pragma unroll
    for (int t = PER - 1; t >= 0; --t)
      if (key[t] == top_key) e = lane + 32 * t;
    const int best_e = (int)__reduce_min_sync(0xffffffffu, e);
    float won = 0.f;
#pragma unroll
    for (int t = 0; t < PER; ++t)
      if (lane + 32 * t == best_e) {                // the owner retires the winner
        won = score[t];
        key[t] = 0u;
      }
    won = __shfl_sync(0xffffffffu, won, best_e & 31);
    sum += won;
    if (lane == j) {
      my_id = best_e;
      my_w = won;
    }
  }
  if (lane < k) {
    float w = my_w;
    if (normalize) w = w / (sum + floor_);
    ids[lane] = my_id;
    wts[lane] = w * scale;
  }
}

__device__ __forceinline__ void warp_route(const float* lg, const float* __restrict__ bias, int E, int k, int normalize,
                                           float floor_, float scale, int* ids, float* wts) {
  if (E <= 32) warp_route_sized<1>(lg, bias, E, k, normalize, floor_, scale, ids, wts);
  else if (E <= 64) warp_route_sized<2>(lg, bias, E, k, normalize, floor_, scale, ids, wts);
  else if (E <= 128) warp_route_sized<4>(lg, bias, E, k, normalize, floor_, scale, ids, wts);
  else warp_route_sized<MAX_EXPERTS / 32>(lg, bias, E, k, normalize, floor_, scale, ids, wts);
}

}  // namespace tl
