// Causal attention of prompt rows over the paged cache on tcgen05: S = Q K^T and O += P V with accumulators in TMEM.
//
// One CTA owns one tile of up to 128 query rows (consecutive tokens x the query heads of one kv head). K and V pages go straight
// from the cache to swizzled shared memory by TMA, 128 keys at a time (one box of 64 head dimensions per page and half), and are
// worked through 64 keys at a time: S lands in TMEM; four warps, one row per thread, apply options and the online softmax and put P
// back into TMEM over S, from where it is the A operand of P V. Two score buffers of 64 columns: the scores of the next 64 keys are
// there when a thread is done with these, and Q K^T and P V run under the softmax. The output accumulator stays in TMEM. Warp 0
// loads, warp 1 issues the MMAs. Two CTAs share an SM (96 KB of shared memory, 256 TMEM columns each). Weights as the A operand in
// TMEM, and rescaling the output only when a row's maximum grew by more than 2^8 (the sums use the same stale maximum, so nothing is
// lost), are published ideas of attention on this chip (T. Dao et al., FlashAttention-4, 2025).
//
// With options the softmax weights keep fp32 accuracy: P = hi + lo, both bf16, two products. EXACT, without options: weights are
// rounded to bf16 once, relative to the maximum after every 64 keys, as in the mma.sync kernel of attention.cu, which has the same
// blocks: both round the same weights the same way. (Other roundings make decoders with few large experts choose other experts for
// nearly tied rows.) The output is then rescaled whenever a maximum grows.
//
// LATENT: the same for prompt runs of latent attention over expanded keys and values (latent_attention.cu has the layout): a
// tile is 128 tokens of one head, a key is 128 numbers of its expanded row and the 64 rotated ones of its cache row, and the
// keys of a sequence are consecutive rows, so that a box holds 128 of them. With 128 KB of shared memory one CTA fits an SM.
//
// Measured on B200 (1965 MHz) against the mma.sync kernel of attention.cu (64 rows per CTA, every warp re-reading all of K and V from
// shared memory), and this one with one score buffer of 128 keys between: 4096 tokens of 16 heads, window 1024, soft cap 366 -> 131 -> 96
// us; 3000 tokens, sinks 219 -> 64 -> 48 us; latent, 4096 tokens of 16 heads 208 -> 157 us; without options, 4096 tokens of 32 heads in
// three prompts 390 -> 111 us. Bound by the issue slots of its softmax. The mma.sync kernel stays for other head sizes, page sizes that
// do not divide 128 keys, unaligned rows and prompts of few keys.
#include <string.h>

#include "attn_common.cuh"
#include "gemm_common.cuh"
#include "mma_sync.cuh"

namespace dmoe {

constexpr int kFaRows = 128, kFaKeys = 128, kFaDim = 128;
constexpr int kFaSub = 64;                          // keys per step
constexpr int kFaThreads = 192;
constexpr int kFaHalf = 128 * 128;                  // bytes of 128 rows x 64 bf16
constexpr int kFaTile = 2 * kFaHalf;                // one of Q, K, V
constexpr int kFaRot = 64;                          // rotated part of a latent key
constexpr int fa_smem(bool lat) { return 3 * kFaTile + (lat ? 2 * kFaHalf : 0) + 1024 /*alignment*/ + 128; }
enum { FA_PAGED = 0, FA_LATENT = 1 };
constexpr float kFaSlack = 8.f;                     // growth of a row's maximum (base 2) that is left in P

__device__ __forceinline__ void fa_load(uint32_t dst, const CUtensorMap* m, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// LATENT: tmK is the map of the expanded keys and values, tmV that of the cache rows, base the row of position 0 per tile
template <int KIND, bool EXACT>
__global__ void __launch_bounds__(kFaThreads, KIND == FA_LATENT ? 1 : 2)
prefill_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                  const __nv_bfloat16* __restrict__ q, long long ld_q, const int* __restrict__ block_tables, int max_blocks,
                  const int4* __restrict__ tiles, int n_tiles, int n_kv, int block_size, float scale_log2, __nv_bfloat16* __restrict__ out,
                  long long ld_out, AttnExt ext, const int* __restrict__ base, int rankp, int* status) {
  constexpr bool LAT = KIND == FA_LATENT;
  constexpr int kQd = kFaDim + (LAT ? kFaRot : 0);                 // numbers of a query / key
  constexpr int kQk = kFaTile + (LAT ? kFaHalf : 0);               // bytes of Q, K
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * kQk + kFaTile);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
  int* abort_word = reinterpret_cast<int*>(tmem_slot + 1);
  const uint32_t sq = smem_u32(smem), sk = sq + kQk, sv = sk + kQk;
  // K / V landed, K / V consumed, output accumulated; scores ready and weights ready in each of two buffers; output complete. A thread
  // that waits for the output of a step knows that the step before is complete, so that the parity says which step is meant; the end
  // has a barrier of its own, because warps come to it one or two steps late
  const uint32_t k_full = smem_u32(bars), v_full = k_full + 8, k_empty = k_full + 16, v_empty = k_full + 24, o_full = k_full + 32,
                 s_full = k_full + 40, p_full = k_full + 56, o_done = k_full + 72;

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  // tiles of a prompt are in order of position: the longest run first
  const int4 tile = tiles[n_tiles - 1 - blockIdx.x / n_kv];
  const int hkv = blockIdx.x % n_kv, gq = ext.gq;
  const int row0 = tile.x, ntok = min(tile.y, kFaRows / gq), pos0 = tile.w;
  const int* bt = LAT ? nullptr : block_tables + static_cast<long long>(tile.z) * max_blocks;
  const int kmax = pos0 + ntok;
  // first key block: from the first key that anyone sees, at the start of a page
  const int first = first_key(pos0, ext.window, ext.chunk), kbase = LAT ? first : first / kFaKeys * kFaKeys;
  const int nkb = (kmax - kbase + kFaKeys - 1) / kFaKeys;
  // uniform for the compiler; steps of 64 keys that anyone sees
  const int blocks = __shfl_sync(0xffffffffu, nkb, 0), first_block = __shfl_sync(0xffffffffu, kbase, 0);
  const int steps = __shfl_sync(0xffffffffu, (kmax - kbase + kFaSub - 1) / kFaSub, 0);

  if (threadIdx.x == 0) {
    *abort_word = 0;
    for (int i = 0; i < 10; ++i) mbar_init(k_full + 8 * i, i == 7 || i == 8 ? 4 : 1);      // weights: one arrival per softmax warp
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 256);
    tmem_relinquish();
  }
  // query row of a softmax thread: its lane of the TMEM quarter that its warp may access
  const int r = warp >= 2 ? (warp & 3) * 32 + lane : -1;
  const int tok = r >= 0 ? r / gq : 0, head = hkv * gq + (r >= 0 ? r % gq : 0);
  const bool live = r >= 0 && tok < ntok;
  if (warp >= 2) {
    // the row's head vector into the two halves of the K-major, 128-byte swizzled Q tile
    const uint4* src = reinterpret_cast<const uint4*>(q + static_cast<long long>(row0 + (live ? tok : 0)) * ld_q + head * kQd);
#pragma unroll
    for (int c = 0; c < kQd / 8; ++c) {
      const uint4 x = live ? __ldg(src + c) : make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(smem + (c >> 3) * kFaHalf + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = x;
    }
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // scores / weights [2 x 64 columns], output [128 columns]
  const uint32_t t_s = __shfl_sync(0xffffffffu, *tmem_slot, 0), t_o = t_s + 2 * kFaSub;

  if (warp == 0) {
    // ------------------------------------------------------------ loads
    if (LAT) {
      // one box of 128 keys per 64 numbers
      const int at = __shfl_sync(0xffffffffu, base[n_tiles - 1 - blockIdx.x / n_kv], 0) + first_block, col = hkv * (2 * kFaDim);
      for (int j = 0; j < blocks; ++j) {
        const int row = at + j * kFaKeys;
        if (!mbar_wait_warp(k_empty, (j & 1) ^ 1, abort_word)) break;
        if (elect_one()) {
          mbar_expect_tx(k_full, kQk);
          fa_load(sk, &tmK, col, row, k_full);
          fa_load(sk + kFaHalf, &tmK, col + 64, row, k_full);
          fa_load(sk + 2 * kFaHalf, &tmV, rankp, row, k_full);
        }
        __syncwarp();
        if (!mbar_wait_warp(v_empty, (j & 1) ^ 1, abort_word)) break;
        if (elect_one()) {
          mbar_expect_tx(v_full, kFaTile);
          fa_load(sv, &tmK, col + kFaDim, row, v_full);
          fa_load(sv + kFaHalf, &tmK, col + kFaDim + 64, row, v_full);
        }
        __syncwarp();
      }
    } else {
      // lane = (page of the block, half of the head)
      const int pages = kFaKeys / block_size;
      const int page = lane >> 1, half = lane & 1;
      for (int j = 0; j < nkb; ++j) {
        const int key0 = kbase + j * kFaKeys;
        const int there = min(pages, (kmax - key0 + block_size - 1) / block_size);      // pages that hold visible keys
        const bool mine = page < there;
        const int slot = mine ? bt[key0 / block_size + page] * block_size : 0;
        const uint32_t at = half * kFaHalf + page * block_size * 128;
        bool ok = true;
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          const uint32_t full = kv ? v_full : k_full;
          ok = ok && mbar_wait_warp(kv ? v_empty : k_empty, (j & 1) ^ 1, abort_word);
          if (!ok) break;
          if (lane == 0) mbar_expect_tx(full, there * block_size * 256);
          __syncwarp();
          if (mine) tma_load_3d((kv ? sv : sk) + at, kv ? &tmV : &tmK, half * 64, hkv, slot, full);
        }
        if (!ok) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMAs (the warp converged, an elected lane issues)
    constexpr uint32_t id_qk = umma_idesc_bf16(kFaRows, kFaSub);
    constexpr uint32_t id_pv = umma_idesc_bf16(kFaRows, kFaDim) | (1u << 16);      // V is MN-major
    const auto scores = [&](int t) {      // step t; its buffer is free
      if ((t & 1) == 0 && !mbar_wait_warp(k_full, (t >> 1) & 1, abort_word)) return false;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t k0 = sk + (t & 1) * kFaSub * 128;
#pragma unroll
        for (int k = 0; k < kQd / kUmmaK; ++k) {
          const uint32_t off = (k >> 2) * kFaHalf + (k & 3) * 32;
          umma_f16(t_s + (t & 1) * kFaSub, umma_desc_sw128(sq + off), umma_desc_sw128(k0 + off), id_qk, k > 0 ? 1u : 0u);
        }
        umma_commit(s_full + 8 * (t & 1));
        if ((t & 1) != 0 || t == steps - 1) umma_commit(k_empty);
      }
      __syncwarp();
      return true;
    };
    bool ok = scores(0) && (steps < 2 || scores(1));
    for (int t = 0; ok && t < steps; ++t) {
      ok = mbar_wait_warp(p_full + 8 * (t & 1), (t >> 1) & 1, abort_word);
      if (ok && (t & 1) == 0) ok = mbar_wait_warp(v_full, (t >> 1) & 1, abort_word);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t p0 = t_s + (t & 1) * kFaSub, v0 = sv + (t & 1) * kFaSub * 128;
#pragma unroll
        for (int part = 0; part < (EXACT ? 1 : 2); ++part)
#pragma unroll
          for (int k = 0; k < kFaSub / kUmmaK; ++k)
            umma_f16_ta(t_o, p0 + part * (kFaSub / 2) + k * (kUmmaK / 2), umma_desc_sw128_mn(v0 + k * kUmmaK * 128, kFaHalf), id_pv,
                        (t > 0 || part > 0 || k > 0) ? 1u : 0u);
        umma_commit(o_full);
        if (t == steps - 1) umma_commit(o_done);
        if ((t & 1) != 0 || t == steps - 1) umma_commit(v_empty);
      }
      __syncwarp();
      // the next scores of this buffer overwrite the weights that this product reads from tensor memory. The order of two products is
      // only given for the same accumulator, so it has to be complete
      if (t + 2 < steps) ok = mbar_wait_warp(o_full, t & 1, abort_word) && scores(t + 2);
    }
  } else {
    // ------------------------------------------------------------ softmax: one query row per thread
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int qpos = pos0 + tok;
    const float temp = EXACT ? 1.f : query_temperature(ext, qpos);
    const int lo = EXACT ? 0 : first_key(qpos, ext.window, ext.chunk);
    // steps that need no mask: all keys visible to the first and the last token of the tile
    const int lo_last = EXACT ? 0 : first_key(kmax - 1, ext.window, ext.chunk);
    const float scale = scale_log2 * temp;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int t = 0; t < steps; ++t) {
      const int key0 = kbase + t * kFaSub;
      const uint32_t buf = t_s + lanes + (t & 1) * kFaSub;
      if (!mbar_wait(s_full + 8 * (t & 1), (t >> 1) & 1, abort_word)) { ok = false; break; }
      tc_fence_after();
      uint32_t s[2][32];
      tmem_ld32(buf, s[0]);
      tmem_ld32(buf + 32, s[1]);
      tmem_ld_wait();
      const bool masked = key0 + kFaSub - 1 > pos0 || key0 < lo_last;
      float mx = -INFINITY, mul = 1.f;      // scores are s times mul: the factor goes into the exponent's subtraction where it can
      if (!EXACT && ext.cap_log2 > 0.f) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 32; ++e) s[i][e] = __float_as_uint(attn_score<true>(__uint_as_float(s[i][e]) * temp, scale_log2, ext));
      } else if (scale > 0.f) {
        mul = scale;
      } else {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 32; ++e) s[i][e] = __float_as_uint(__uint_as_float(s[i][e]) * scale);
      }
      if (masked) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int key = key0 + i * 32 + e;
            if (key > qpos || key < lo) s[i][e] = __float_as_uint(-INFINITY);
          }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float a = __uint_as_float(s[i][0]), b = __uint_as_float(s[i][1]);
#pragma unroll
        for (int e = 2; e < 32; e += 2) {
          a = fmaxf(a, __uint_as_float(s[i][e]));
          b = fmaxf(b, __uint_as_float(s[i][e + 1]));
        }
        mx = fmaxf(mx, fmaxf(a, b));
      }
      mx *= mul;
      const bool grow = EXACT ? mx > m : mx > m + kFaSlack;      // true for the first finite maximum: m is -inf before it
      if (__any_sync(0xffffffffu, grow)) {
        const float to = grow ? mx : m;
        if (t > 0) {
          ok = mbar_wait_warp(o_full, (t - 1) & 1, abort_word);
          if (!ok) break;
          tc_fence_after();
          const float f = grow ? exp2f(m - to) : 1.f;      // -inf - finite: 0, and what it scales is 0
          l *= f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t o[2][16];
            tmem_ld16(t_o + lanes + i * 32, o[0]);
            tmem_ld16(t_o + lanes + i * 32 + 16, o[1]);
            tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
              for (int e = 0; e < 16; ++e) o[h][e] = __float_as_uint(__uint_as_float(o[h][e]) * f);
              tmem_st16(t_o + lanes + i * 32 + h * 16, o[h]);
            }
          }
        }
        m = to;
      }
      const float sub = m == -INFINITY ? 0.f : m;      // a row with nothing visible yet: weights 0, not NaN
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t hi[16], rest[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          // exp2f and not the instruction alone, which makes 0 of weights below 2^-126
          const float p0 = exp2f(fmaf(__uint_as_float(s[i][2 * e]), mul, -sub)), p1 = exp2f(fmaf(__uint_as_float(s[i][2 * e + 1]), mul, -sub));
          sum[e & 3] += p0 + p1;
          if (EXACT) hi[e] = pack_bf16(p0, p1);
          else split2(p0, p1, hi[e], rest[e]);
        }
        tmem_st16(buf + i * 16, hi);
        if (!EXACT) tmem_st16(buf + kFaSub / 2 + i * 16, rest);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      if (key0 + kFaSub > kmax) {
        // keys past the last one: their weights are 0, but 0 times whatever the page holds there need not be
        if (!mbar_wait(v_full, (t >> 1) & 1, abort_word)) ok = false;
        const int key = (threadIdx.x - 64) & (kFaSub - 1), half = (threadIdx.x - 64) / kFaSub;
        if (key0 + key >= kmax) {
          uint8_t* row = smem + 2 * kQk + half * kFaHalf + ((t & 1) * kFaSub + key) * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(row + (c << 4)) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + 8 * (t & 1));
      if (!ok) break;
    }
    if (ok && mbar_wait(o_done, 0, abort_word)) {
      tc_fence_after();
      float inv = l > 0.f ? 1.f / l : 0.f;
      if (!EXACT && ext.sink != nullptr) inv = sink_inverse(m, l, ext.sink[head]);
      if (!EXACT && ext.gate != nullptr && live) inv *= head_gate<__nv_bfloat16>(ext, row0 + tok, head);
      __nv_bfloat16* y = out + static_cast<long long>(row0 + tok) * ld_out + head * kFaDim;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t o[32];
        tmem_ld32(t_o + lanes + i * 32, o);
        tmem_ld_wait();
        if (live) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 pk;
            uint32_t* pp = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              pp[e] = pack_bf16(__uint_as_float(o[c * 8 + 2 * e]) * inv, __uint_as_float(o[c * 8 + 2 * e + 1]) * inv);
            *reinterpret_cast<uint4*>(y + i * 32 + c * 8) = pk;
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_word) {
    if (threadIdx.x == 0 && status != nullptr) atomicCAS(status, kStatusOk, kStatusBarrierTimeout);
    // give copies that may still be in flight time to land before shared memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(*tmem_slot, 256);
  }
}

// The cache [blocks * block_size, n_kv, 128] as boxes of one page x one head x 64 dimensions.
static int page_map(CUtensorMap* map, const void* cache, long long slots, int n_kv, int block_size) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return -20;
  cuuint64_t dim[3] = {static_cast<cuuint64_t>(kFaDim), static_cast<cuuint64_t>(n_kv), static_cast<cuuint64_t>(slots)};
  cuuint64_t stride[2] = {kFaDim * 2, static_cast<cuuint64_t>(n_kv) * kFaDim * 2};
  cuuint32_t box[3] = {64, 1, static_cast<cuuint32_t>(block_size)};
  cuuint32_t step[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(cache), dim, stride, box, step,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -21;
}

template <int KIND, bool EXACT>
static int launch_tc(const CUtensorMap& tmK, const CUtensorMap& tmV, const void* q, long long ld_q, const int* bt, int max_blocks,
                     const void* tiles, int n_tiles, int block_size, int n_kv, float scale, void* out, long long ld_out, AttnExt ext,
                     const int* base, int rankp, int* status, cudaStream_t stream) {
  constexpr int smem = fa_smem(KIND == FA_LATENT);
  static PerDeviceOnce configured;
  const int crc = configured.run([] {
    return static_cast<int>(cudaFuncSetAttribute(prefill_tc_kernel<KIND, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  });
  if (crc != 0) return crc;
  prefill_tc_kernel<KIND, EXACT><<<n_kv * n_tiles, kFaThreads, smem, stream>>>(
      tmK, tmV, static_cast<const __nv_bfloat16*>(q), ld_q, bt, max_blocks, static_cast<const int4*>(tiles), n_tiles, n_kv,
      block_size, scale * kLog2e, static_cast<__nv_bfloat16*>(out), ld_out, ext, base, rankp, status);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace dmoe

using namespace dmoe;

extern "C" int dmoe_prefill_attention_tc(const void* q, long long ld_q, const void* kcache, const void* vcache, int n_blocks,
                                         const int* block_tables, int max_blocks, const void* tiles, int n_tiles, int block_size,
                                         int n_q, int n_kv, float scale, int window, int chunk, float softcap,
                                         const float* sink, void* out, long long ld_out, const DmoeAttnExtra* extra, int exact,
                                         int* status, void* stream_) {
  if (n_tiles == 0) return 0;
  if (n_kv < 1 || n_q % n_kv != 0 || n_q / n_kv > kFaRows || n_tiles < 0 || static_cast<long long>(n_tiles) * n_kv > 0x7fffffff ||
      tiles == nullptr || n_blocks < 1 || block_size < 8 || kFaKeys % block_size != 0)
    return -10;
  if (exact && (window > 0 || chunk > 0 || softcap > 0.f || sink != nullptr || extra != nullptr)) return -10;
  CUtensorMap tmK, tmV;
  const long long slots = static_cast<long long>(n_blocks) * block_size;
  int rc = page_map(&tmK, kcache, slots, n_kv, block_size);
  if (rc == 0) rc = page_map(&tmV, vcache, slots, n_kv, block_size);
  if (rc != 0) return rc;
  const AttnExt ext = make_ext(scale, window, chunk, softcap, sink, n_q / n_kv, extra);
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const auto launch = exact ? launch_tc<FA_PAGED, true> : launch_tc<FA_PAGED, false>;
  return launch(tmK, tmV, q, ld_q, block_tables, max_blocks, tiles, n_tiles, block_size, n_kv, scale, out, ld_out, ext, nullptr, 0, status,
                stream);
}

extern "C" int dmoe_latent_prefill_tc(const void* q, long long ld_q, const void* kv, long long ld_kv, const void* lat, long long ld_lat,
                                      long long n_keys, const void* tiles, const int* base, int n_tiles, int heads, int rankp,
                                      float scale, int window, const float* sink, const void* gate, long long ld_gate, void* out,
                                      long long ld_out, int* status, void* stream) {
  if (n_tiles == 0) return 0;
  if (heads < 1 || n_tiles < 0 || n_keys < 1 || static_cast<long long>(n_tiles) * heads > 0x7fffffff || rankp % 8 != 0) return -10;
  CUtensorMap tmKV, tmL;
  if (make_map_2d(&tmKV, kv, n_keys, static_cast<long long>(heads) * 2 * kFaDim, ld_kv, kFaKeys) != 0 ||
      make_map_2d(&tmL, lat, n_keys, rankp + kFaRot, ld_lat, kFaKeys) != 0)
    return -20;
  const DmoeAttnExtra extra = {gate, ld_gate, 0.f, 0};
  const AttnExt ext = make_ext(scale, window, 0, 0.f, sink, 1, &extra);
  return launch_tc<FA_LATENT, false>(tmKV, tmL, q, ld_q, nullptr, 0, tiles, n_tiles, kFaKeys, heads, scale, out, ld_out, ext, base, rankp, status,
                              static_cast<cudaStream_t>(stream));
}
