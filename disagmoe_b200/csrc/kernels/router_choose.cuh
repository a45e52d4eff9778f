// The choice of experts from a row's logits, by one warp.
#pragma once
#include "sm100.cuh"

namespace dmoe {

constexpr int kMaxExperts = 256, kMaxTop = 32;

// lg [E]: logits, overwritten; score [E], group [groups]: scratch of a sigmoid router. See DmoeRouter.
__device__ __forceinline__ void choose_experts(float* lg, float* score, float* group, int E, int K, int renorm, int sigmoid, int groups,
                                               int keep, const float* correction, float wscale, int lane, int* ids, float* wts,
                                               int* counts) {
  const auto warp_sum = [](float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  float mx = -INFINITY, den = 0.f;
  if (sigmoid) {
    for (int e = lane; e < E; e += 32) {
      score[e] = 1.f / (1.f + expf(-lg[e]));
      lg[e] = score[e] + (correction != nullptr ? correction[e] : 0.f);
    }
    __syncwarp();
    if (keep < groups) {
      const int per = E / groups;
      float* sum = group;
      for (int g = lane; g < groups; g += 32) {
        float first = -INFINITY, second = -INFINITY;
        for (int e = g * per; e < (g + 1) * per; ++e) {
          const float c = lg[e];
          if (c > first) { second = first; first = c; }
          else if (c > second) second = c;
        }
        sum[g] = per > 1 ? first + second : first;
      }
      __syncwarp();
      for (int g = lane; g < groups; g += 32) {
        int ahead = 0;
        for (int q = 0; q < groups; ++q) ahead += sum[q] > sum[g] || (sum[q] == sum[g] && q < g);
        if (ahead >= keep)
          for (int e = g * per; e < (g + 1) * per; ++e) lg[e] = -INFINITY;
      }
      __syncwarp();
    }
  } else {
    for (int e = lane; e < E; e += 32) mx = fmaxf(mx, lg[e]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    for (int e = lane; e < E; e += 32) den += expf(lg[e] - mx);
    den = warp_sum(den);
  }
  int my_id = -1;           // lane k keeps the k-th choice
  float my_w = 0.f, total = 0.f;
  for (int k = 0; k < K; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32)
      if (lg[e] > best) { best = lg[e]; bi = e; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    float s = sigmoid ? (bi < E ? score[bi] : 0.f) : expf(best - mx) / den;
    if (bi >= E) {        // no finite logit left: the lowest expert not chosen yet, so that the ids stay valid
      for (bi = 0; __any_sync(0xffffffffu, my_id == bi);) ++bi;
      s = 0.f;
    }
    if (lane == k) { my_id = bi; my_w = s; }
    total += s;
    __syncwarp();
    if (lane == 0) lg[bi] = -INFINITY;
    __syncwarp();
  }
  if (lane < K) {
    ids[lane] = my_id;
    wts[lane] = (renorm && total > 0.f ? my_w / total : my_w) * wscale;
    if (counts != nullptr) atomicAdd(&counts[my_id], 1);
  }
}

}  // namespace dmoe
