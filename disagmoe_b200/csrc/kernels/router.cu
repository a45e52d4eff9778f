// Router over normalised bf16 rows: logits on the tensor cores, then the choice of experts.
//
// One CTA has 16 rows; eighths of the width x halves of the experts go to its 16 warps, so that a router weight is read once
// per 16 rows (straight from L2 as 16-byte pieces in the order the mma fragments want: the order of k inside a step does not
// matter as long as both operands share it) and no row passes through shared memory. At decode batches a handful of CTAs runs
// and the time is the latency of the weight reads: the loop is unrolled by four steps of the width, and one CTA per SM leaves
// 128 registers per thread for their loads (37 rows x 60 experts of 2048: 16.4 us with two CTAs per SM, 14.3 with one).
//
// The logits choose experts, so they are as exact as fp32 multiply-adds. The tensor core truncates what it adds to an
// accumulator; chained over the width that made the errors three to eight times as large (4096 wide: 4.8e-7 of the logits'
// root mean square, against 9.4e-8 for the CUDA cores). Every mma therefore starts from zero, and its 16 products are added in
// rounded fp32: first over four steps of the width, then over those; the eight slices are added in fp64. Errors against fp64,
// root mean square, CUDA cores -> here: 4096 wide 9.4e-8 -> 7.1e-8, 2048 wide 7.9e-8 -> 6.5e-8, 256 wide 5.6e-8 -> 4.4e-8.
//
// Afterwards every warp chooses for one row. The kernels that norm the rows (moe.cu: route_kernel, layer_ops.cu: sum_norm_kernel)
// have a router of their own on the CUDA cores, bound by its fp32 multiply-adds and shared-memory reads; ops/functional.py:
// separate_router says where each is used.
#include "dmoe_kernels.h"
#include "mma_sync.cuh"
#include "router_choose.cuh"

namespace dmoe {

constexpr int kRtRows = 16, kRtSlices = 8, kRtThreads = 512;

// NT: groups of 8 experts per pass and warp
template <int NT>
__global__ void __launch_bounds__(kRtThreads, 1)
router_kernel(const __nv_bfloat16* __restrict__ h, long long ld_h, int T, int H, const DmoeRouter r, const float* __restrict__ bias,
              float* __restrict__ logits_out) {
  extern __shared__ float s_part[];                        // [slices][rows][E8]
  __shared__ float s_lg[kRtRows][kMaxExperts], s_score[kRtRows][kMaxExperts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
  const int E = r.E, E8 = (E + 7) / 8 * 8;
  const long long row0 = static_cast<long long>(blockIdx.x) * kRtRows;
  const int slice = warp % kRtSlices, per = H / kRtSlices, k0 = slice * per + tq * 8;
  const __nv_bfloat16* W = static_cast<const __nv_bfloat16*>(r.weight);
  const bool v0 = row0 + g < T, v1 = row0 + g + 8 < T;
  const __nv_bfloat16* x0 = h + (v0 ? row0 + g : 0) * ld_h + k0;
  const __nv_bfloat16* x1 = h + (v1 ? row0 + g + 8 : 0) * ld_h + k0;
  for (int e0 = warp / kRtSlices * 8 * NT; e0 < E; e0 += 16 * NT) {
    float acc[NT][4] = {}, run[NT][4] = {};
    const __nv_bfloat16* w[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) w[n] = W + static_cast<long long>(min(e0 + n * 8 + g, E - 1)) * H + k0;
#pragma unroll 4
    for (int k = 0; k < per; k += 32) {
      uint4 a0 = __ldg(reinterpret_cast<const uint4*>(x0 + k)), a1 = __ldg(reinterpret_cast<const uint4*>(x1 + k)), b[NT];
      if (!v0) a0 = make_uint4(0, 0, 0, 0);
      if (!v1) a1 = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int n = 0; n < NT; ++n) b[n] = __ldg(reinterpret_cast<const uint4*>(w[n] + k));
      const uint32_t lo[4] = {a0.x, a1.x, a0.y, a1.y}, hi[4] = {a0.z, a1.z, a0.w, a1.w};
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        float t[4] = {}, u[4] = {};
        mma_bf16_16816(t, lo, b[n].x, b[n].y);
        mma_bf16_16816(u, hi, b[n].z, b[n].w);
#pragma unroll
        for (int i = 0; i < 4; ++i) run[n][i] += t[i] + u[i];
        if (k % 128 == 96) {
#pragma unroll
          for (int i = 0; i < 4; ++i) { acc[n][i] += run[n][i]; run[n][i] = 0.f; }
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int e = e0 + n * 8 + 2 * tq;
      if (e >= E8) continue;
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[n][i] += run[n][i];
      float* p = s_part + (slice * kRtRows + g) * E8 + e;
      *reinterpret_cast<float2*>(p) = make_float2(acc[n][0], acc[n][1]);
      *reinterpret_cast<float2*>(p + 8 * E8) = make_float2(acc[n][2], acc[n][3]);
    }
  }
  __syncthreads();
  const int j = warp;
  const long long t = row0 + j;
  if (t >= T) return;
  for (int e = lane; e < E; e += 32) {
    double sum = 0.;
#pragma unroll
    for (int p = 0; p < kRtSlices; ++p) sum += s_part[(p * kRtRows + j) * E8 + e];
    float z = static_cast<float>(sum);
    if (bias != nullptr) z += bias[e];
    if (logits_out != nullptr) logits_out[t * E + e] = z;
    s_lg[j][e] = z;
  }
  __syncwarp();
  // the partial logits of this row are read: their first slice holds the sums of the groups
  choose_experts(s_lg[j], s_score[j], s_part + j * E8, E, r.K, r.renorm, r.sigmoid, r.groups, r.keep, r.correction, r.wscale, lane,
                 r.ids + t * r.K, r.wts + t * r.K, r.counts);
}

template <int NT>
static int launch_router(const void* h, long long ld_h, int T, int H, const DmoeRouter& r, const float* bias, float* logits,
                         cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(kRtSlices) * kRtRows * ((r.E + 7) / 8 * 8) * sizeof(float);
  static PerDeviceOnce configured;
  const int rc = configured.run([] {
    return static_cast<int>(cudaFuncSetAttribute(router_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 kRtSlices * kRtRows * kMaxExperts * 4));
  });
  if (rc != 0) return rc;
  router_kernel<NT><<<(T + kRtRows - 1) / kRtRows, kRtThreads, smem, stream>>>(static_cast<const __nv_bfloat16*>(h), ld_h, T, H, r, bias,
                                                                              logits);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace dmoe

using namespace dmoe;

extern "C" int dmoe_router(const void* h, long long ld_h, int T, int H, const DmoeRouter* r, const float* logit_bias, float* logits,
                           void* stream_) {
  const auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (H < 256 || H % 256 != 0 || ld_h % 8 != 0 || !al16(h) || !al16(r->weight) || r->weight == nullptr || r->E < 1 || r->E > kMaxExperts ||
      r->K < 1 || r->K > kMaxTop || r->K > r->E || r->ids == nullptr || r->wts == nullptr ||
      (r->sigmoid && (r->groups < 1 || r->E % r->groups != 0 || r->keep < 1)))
    return -10;
  if (T == 0) return 0;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (r->E <= 8) return launch_router<1>(h, ld_h, T, H, *r, logit_bias, logits, stream);
  if (r->E <= 32) return launch_router<2>(h, ld_h, T, H, *r, logit_bias, logits, stream);
  return launch_router<4>(h, ld_h, T, H, *r, logit_bias, logits, stream);
}
