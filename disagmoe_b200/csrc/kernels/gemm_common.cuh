// What the GEMM kernels share: tile constants, gate activations and the tensor maps of their operands.
#pragma once

#include "dmoe_kernels.h"
#include "sm100.cuh"

namespace dmoe {

constexpr int kBM = 128;       // rows of the M operand that one CTA stages and accumulates
constexpr int kBK = 64;        // K elements per stage: 64 bf16 = 128 bytes = one swizzle span
constexpr int kUmmaK = 16;     // K per tcgen05.mma for 16-bit inputs
constexpr int kMaxGroups = 1024;

enum { EPI_PLAIN = 0, EPI_SWIGLU = 1, EPI_COMBINE = 2 };

// n / (1 + e) for e >= 0, rounded to nearest where the quotient is of normal size (3 of 2^30 random ones were a unit off the
// operator's); signed zeros, infinities and NaN as the division has them. The quotient by an approximate reciprocal is corrected
// by its remainder, which a fused multiply-add gives exactly (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990); both sides are scaled so that the reciprocal stays normal. Straight code: the operator's slow
// path, which zero rows of a ragged tile take, and its branch keep the chains of an epilogue thread from overlapping. Measured on B200, SwiGLU of 2500 x 5632 x 2048: 119 us with the operator, 88 us here;
// one row of 5632 x 2048: 50 us with the operator, 27 us here.
__device__ __forceinline__ float over_1p(float n, float e) {
  constexpr float kScale = 0.0625f;
  const float ds = fmaf(e, kScale, kScale), ns = n * kScale;      // rounded as 1 + e is
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(ds));
  const float q = ns * r, c = fmaf(fmaf(-ds, q, ns), r, q);
  return fabsf(c) > 0.f ? c : q;
}

// silu(g) = g sigmoid(g); the tanh form of gelu is g sigmoid(2 sqrt(2 / pi) (g + 0.044715 g^3))
template <int ACT>
__device__ __forceinline__ float gate_act(float g) {
  const float z = ACT == 0 ? g : 1.5957691216057308f * (g + 0.044715f * g * g * g);
  return over_1p(g, __expf(-z));
}

// g <- act(g) * u for N values; clamped (act 3): min(g, limit) sigmoid(1.702 min(g, limit)) (clamp(u, -limit, limit) + 1).
// The activation is chosen outside the loops, so that the N chains of special-function instructions overlap.
template <int N>
__device__ __forceinline__ void gated(float (&g)[N], const float (&u)[N], int act, float limit) {
  if (act == 0) {
#pragma unroll
    for (int j = 0; j < N; ++j) g[j] = gate_act<0>(g[j]) * u[j];
  } else if (act == 1) {
#pragma unroll
    for (int j = 0; j < N; ++j) g[j] = gate_act<1>(g[j]) * u[j];
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float m = fminf(g[j], limit);
      g[j] = __fdividef(m, 1.f + __expf(-1.702f * m)) * (fminf(fmaxf(u[j], -limit), limit) + 1.f);
    }
  }
}

// tanh(x) = 1 - 2 / (exp(2x) + 1), good to about 1e-7 absolute
__device__ __forceinline__ float out_tanh(float x) { return 1.f - __fdividef(2.f, __expf(fminf(2.f * x, 40.f)) + 1.f); }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
    }
  }
  return fn;
}

// Tensor map over a row-major [rows, K] bf16 matrix with a [box_rows, 64] box and the 128-byte swizzle.
inline int make_map_2d(CUtensorMap* map, const void* ptr, long long rows, long long K, long long ld_elems,
                       int box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return -1;
  cuuint64_t gdim[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
  cuuint64_t gstride[1] = {static_cast<cuuint64_t>(ld_elems) * 2};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(kBK), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}


// gemm_wide.cu: the same product with the tokens as the M operand (see there). Checks have been made by dmoe_gemm.
int gemm_wide(const DmoeGemm* d, cudaStream_t stream);
// gemm_split.cu: dense launches of one wave, K cut over a cluster. Checks as above, but for the token tile.
int gemm_split(const DmoeGemm* d, cudaStream_t stream);

}  // namespace dmoe
