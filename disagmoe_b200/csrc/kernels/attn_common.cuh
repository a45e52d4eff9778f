// Options of the attention kernels and the scalar pieces of their softmax.
#pragma once
#include "dmoe_kernels.h"
#include "sm100.cuh"

namespace dmoe {

// Options of the EXT instantiations of the paged attention kernels (plain ones compile without them):
//   window > 0: a query at position p sees only keys in (p - window, p];
//   chunk > 0: it sees only keys of its own chunk of `chunk` positions, counted from position 0;
//   cap_log2 > 0: score <- cap * tanh(score / cap) before the softmax (cap_log2 = cap * log2 e, cap_in = 2 scale log2 e / cap);
//   sink != NULL: exp(sink[head]) enters the softmax denominator (no key, no value);
//   temp_every > 0: scores are multiplied by the query temperature 1 + temp_coef ln(floor((p + 1) / temp_every) + 1);
//   gate != NULL: head outputs are multiplied by sigmoid(gate[row, head]) (row stride ld_gate);
//   gq: query heads per kv head where the instantiation leaves it open (GQ = 0).
// The EXT kernels also keep the softmax weights at fp32 accuracy in the P V product: P = hi + lo, both bf16, two MMAs.
struct AttnExt {
  int window, chunk;
  float cap_in, cap_log2;
  const float* sink;
  int gq;
  const void* gate;
  long long ld_gate;
  float temp_coef;
  int temp_every;
};
__device__ __forceinline__ float query_temperature(const AttnExt& x, int p) {
  return x.temp_every > 0 ? 1.f + x.temp_coef * logf(static_cast<float>((p + 1) / x.temp_every + 1)) : 1.f;
}
template <typename T>
__device__ __forceinline__ float head_gate(const AttnExt& x, long long row, int head) {
  return x.gate != nullptr ? 1.f / (1.f + expf(-static_cast<float>(static_cast<const T*>(x.gate)[row * x.ld_gate + head]))) : 1.f;
}
constexpr float kLog2e = 1.4426950408889634f;
// first key that a query at position p sees
__device__ __forceinline__ int first_key(int p, int window, int chunk) {
  int lo = window > 0 ? max(0, p - window + 1) : 0;
  if (chunk > 0) lo = max(lo, p / chunk * chunk);
  return lo;
}
// raw q.k -> score in base-2 units. tanh(x) = 1 - 2 / (exp(2x) + 1), good to ~1e-7 absolute.
template <bool EXT>
__device__ __forceinline__ float attn_score(float raw, float scale_log2, const AttnExt& x) {
  if (EXT && x.cap_log2 > 0.f) return x.cap_log2 * (1.f - __fdividef(2.f, exp2f(raw * x.cap_in) + 1.f));
  return raw * scale_log2;
}

// 1 / denominator of a row with running maximum m (base 2) and sum l, the sink included; 0 for a row that saw nothing.
__device__ __forceinline__ float sink_inverse(float m, float l, float sink) {
  const float sk = sink * kLog2e, M = fmaxf(m, sk), f = exp2f(m - M);
  return f / (l * f + exp2f(sk - M));
}

// Options of a launch as the kernels take them (softcap <= 0: none; window, chunk <= 0: every key).
inline AttnExt make_ext(float scale, int window, int chunk, float softcap, const float* sink, int gq, const DmoeAttnExtra* extra) {
  AttnExt x;
  x.gate = extra != nullptr ? extra->gate : nullptr;
  x.ld_gate = extra != nullptr ? extra->ld_gate : 0;
  x.temp_coef = extra != nullptr ? extra->temp_coef : 0.f;
  x.temp_every = extra != nullptr ? extra->temp_every : 0;
  x.sink = sink;
  x.gq = gq;
  x.window = window > 0 ? window : 0;
  x.chunk = chunk > 0 ? chunk : 0;
  x.cap_in = softcap > 0.f ? 2.f * scale * 1.4426950408889634f / softcap : 0.f;
  x.cap_log2 = softcap > 0.f ? softcap * 1.4426950408889634f : 0.f;
  return x;
}

}  // namespace dmoe
