// Grouped / dense bf16 GEMM for prompt-sized batches: the product of gemm.cu with the TOKENS as the M operand.
//
// gemm.cu keeps the weights in the M rows so that a handful of tokens never pads to 128 rows. From a few hundred tokens on
// that layout is bound by what its rounds stage: a 128 x 256 tile of one CTA takes 48 KB per 512 tensor cycles, and every
// output chunk has to be transposed through shared memory. Here a cluster of two CTAs computes a tile of 256 tokens x 256
// weight rows with tcgen05.mma.cta_group::2: each CTA stages its own 128 token rows and HALF of the weight rows (32 KB per
// 512 tensor cycles). A stage holds two K blocks, three stages fit: a round of the issuing warp takes about 400 cycles, and
// was what bounded a K block when every block had a round of its own (SwiGLU of K up to 512 takes 1 to 5 % longer so: 2952 x 2816 x 256
// 20.0 -> 20.7 us; 3000 x 5632 x 1024 59 -> 51, 1024 x 5632 x 2048 42.1 -> 38.6). A TMEM lane is a token, so an epilogue thread owns
// consecutive features of one output row: no transposition, no barrier between the epilogue warps. For SwiGLU the even CTA
// stages 128 gate rows and the odd one the matching 128 up rows; gate and up of a feature then sit 128 TMEM columns apart
// in the same lane.
//
// A tile of up to 128 tokens (the last one of a group) takes 64 token rows per CTA and the product of 128 rows, half the tensor
// time and 24 instead of 32 KB per K block: the tokens of a CTA then lie in lanes 0 .. 63 with the accumulator columns of the even
// CTA's weight rows and in lanes 64 .. 127 with those of the odd one's; for SwiGLU each CTA stages 64 gate and the matching 64 up rows.
// Full product -> this (with the turn of WideTurn), us: 64 experts of 1408 x 2048, SwiGLU, 104 rows each 150 -> 126, 281: 264 -> 236,
// their down-projections 77 -> 66 and 137 -> 125; 8 experts of 14336 x 4096, 281 rows 626 -> 562 and 346 -> 318. Results equal
// bit for bit. Tiles of 256 weight rows only: dense launches of narrower ones have too few tails to shorten a wave.
//
// Warp roles (192 threads per CTA): warp 0 TMA producer (its own CTA's operands), warp 1 TMEM owner and, in the even CTA,
// MMA issuer for both, warps 2..5 epilogue of the CTA's 128 accumulator lanes. Two accumulators of 256 columns fill TMEM:
// the epilogue of a tile runs under the next one's main loop. Dense launches may take tiles of fewer weight rows (any multiple of
// 32), so that their count fills whole waves of pairs. Persistent: a pair runs a tile of every wave (WideTurn); tiles are
// numbered group after group with the token tile fastest, so that concurrent pairs share a weight tile in L2.
//
// Measured on B200 against gemm.cu, see ops/gemm.py: want_wide, which holds the rule that chooses between the two.
#include <string.h>

#include "gemm_common.cuh"

namespace dmoe {

constexpr int kWThreads = 192;
constexpr int kWTokens = 2 * kBM;                        // tokens per tile
constexpr int kWCols = 256;                              // accumulator columns = weight rows per tile, at most
constexpr int kWSub = 2;                                 // K blocks per stage
constexpr int kWMaxStages = 4;
constexpr int kWSmemMax = 227 * 1024;                    // three stages of 256 columns, or four of 160 where there are no groups
constexpr int kWPutBytes = 32 * 64;                      // 32 rows x 32 output columns on their way to global memory
constexpr int kWPutRoom = 4 * 2 * kWPutBytes;            // two of them per epilogue warp
constexpr int kWOperandBytes = kBM * kBK * 2;            // 128 rows x 64 bf16: one CTA's tokens
constexpr int kWBarBytes = 256;
// shared memory of a launch: stages, output on its way, barriers, first row and tile of every group
constexpr int wide_smem(int stages, int stage_bytes, int groups) {
  return 1024 /*alignment slack*/ + stages * stage_bytes + kWPutRoom + kWBarBytes + (2 * groups + 1) * 4;
}

struct WideArgs {
  int cols, stages;      // weight rows per tile: a multiple of 32 up to kWCols
  const int* offs;
  int G, T, F, K, w_rows, w_blocked;
  void* Y;
  long long ldy;
  int y_f32;
  const __nv_bfloat16* R;
  long long ldr;
  const int4* recs;
  void* const* bases;
  int unit_weights;
  int act;
  float act_limit;
  int act_cols;
  const float2* rope_table;
  const int* positions;
  const long long* slots;
  __nv_bfloat16* kcache;
  __nv_bfloat16* vcache;
  int n_q, n_kv, hd, rope_max_pos;
  int* status;
  int put;      // rows of Y by TMA
  int tails;    // tiles of up to 128 tokens as such
};

__device__ __forceinline__ uint4 pack8(const float* x) {
  uint4 pk;
  __nv_bfloat162* pp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
  for (int i = 0; i < 4; ++i) pp[i] = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
  return pk;
}

// 32 consecutive values of one row; ``n`` of them exist (a multiple of 8)
__device__ __forceinline__ void store32(__nv_bfloat16* y, const float (&x)[32], int n) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (8 * i < n) *reinterpret_cast<uint4*>(y + 8 * i) = pack8(x + 8 * i);
}

// Tiles of a pair: one of every wave of `pairs` tiles, each time the one before. Groups often have the same count of token tiles with
// a tail as the last; always at the same place of a wave, every second pair would have all the tails (8 experts of 14336 x 4096, 281
// rows each, SwiGLU: 646 us, 562 with the turn).
struct WideTurn {
  int base, slot, pairs;
  __device__ __forceinline__ WideTurn(int pair, int n) : base(0), slot(pair), pairs(n) {}
  __device__ __forceinline__ int tile() const { return base + slot; }
  __device__ __forceinline__ void next() {
    base += pairs;
    slot = slot == 0 ? pairs - 1 : slot - 1;
  }
};

// Tile of this pair: cursor over the groups, whose tiles start at tile0[g].
struct WideTile {
  int g, n, row0, ntok;
  __device__ __forceinline__ bool locate(int tile, const int* start, const int* tile0, int G, int NT, int T) {
    while (g < G && tile >= tile0[g + 1]) ++g;
    if (g >= G) return false;
    const int r = tile - tile0[g], mt = (tile0[g + 1] - tile0[g]) / NT;
    const int m = r % mt;
    n = r / mt;
    row0 = start[g] + m * kWTokens;
    const int end = g + 1 < G ? start[g + 1] : T;
    ntok = min(kWTokens, end - row0);
    return true;
  }
};

template <int EPI>
__global__ void __launch_bounds__(kWThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY,
                 const __grid_constant__ CUtensorMap tmW64, const __grid_constant__ CUtensorMap tmX64, const WideArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int prank = __shfl_sync(0xffffffffu, static_cast<int>(cluster_ctarank()), 0);
  const bool leader = prank == 0;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int feat = EPI == EPI_SWIGLU ? a.cols / 2 : a.cols;           // output features per tile
  const int half = a.cols / 2, w_bytes = half * kBK * 2;              // weight rows that a CTA stages
  const int sub_bytes = kWOperandBytes + w_bytes, stage_bytes = kWSub * sub_bytes;      // tokens, then weights of one K block
  uint8_t* put_rows = smem + a.stages * stage_bytes;      // of the epilogue warps
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(put_rows + kWPutRoom);
  uint64_t* empty_bar = full_bar + kWMaxStages;
  uint64_t* tfull_bar = empty_bar + kWMaxStages;      // [2]
  uint64_t* tempty_bar = tfull_bar + 2;            // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  int* abort_word = reinterpret_cast<int*>(tmem_slot + 1);
  int* s_start = reinterpret_cast<int*>(put_rows + kWPutRoom + kWBarBytes);      // [G] first row
  int* s_tile0 = s_start + a.G;                                                     // [G + 1] first tile

  const int NT = (a.F + feat - 1) / feat;
  const int kblocks = (a.K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    *abort_word = 0;
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&tfull_bar[b]), 1);
      mbar_init(smem_u32(&tempty_bar[b]), 8);      // one arrival per epilogue warp of both CTAs
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), 2 * kWCols);
    tmem_relinquish_pair();
  }
  pdl_trigger();
  if (warp == 0) {
    if (lane == 0) { tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX); }
    pdl_wait();
    if (a.offs == nullptr) {
      if (lane == 0) {
        s_start[0] = 0;
        s_tile0[0] = 0;
        s_tile0[1] = (a.T + kWTokens - 1) / kWTokens * NT;
      }
    } else {
      int base = 0;
      for (int g0 = 0; g0 < a.G; g0 += 32) {
        const int g = g0 + lane;
        int t = 0;
        if (g < a.G) {
          const int o0 = a.offs[g], o1 = a.offs[g + 1];
          s_start[g] = o0;
          t = o1 > o0 ? (o1 - o0 + kWTokens - 1) / kWTokens * NT : 0;
        }
        int sum = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int x = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += x;
        }
        if (g < a.G) s_tile0[g] = base + sum - t;
        base += __shfl_sync(0xffffffffu, sum, 31);
      }
      if (lane == 0) s_tile0[a.G] = base;
    }
  }
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // both CTAs' barriers are initialised before either is signalled from outside
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  WideTile u;
  u.g = 0;
  // the rows of a group end where the next one starts; the last one ends at T, or where offs says
  const int t_end = a.offs != nullptr ? a.offs[a.G] : a.T;

  const int steps = (kblocks + kWSub - 1) / kWSub;
  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    const uint64_t pol_first = l2_policy_evict_first(), pol_last = l2_policy_evict_last();
    // the bytes of both CTAs are counted on the even CTA's barriers, which its producer arms
    const uint32_t full0 = __shfl_sync(0xffffffffu, mapa_rank(smem_u32(full_bar), 0), 0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (WideTurn w(pair, pairs); ok && u.locate(w.tile(), s_start, s_tile0, a.G, NT, t_end); w.next()) {
      const bool both = __shfl_sync(0xffffffffu, u.ntok, 0) > kBM;             // the odd CTA has token rows of its own
      const bool tail = a.tails && !both;
      const bool mine = leader || both;
      // a weight tile that one token tile reads streams through L2, one that several read stays
      const bool once = __shfl_sync(0xffffffffu, s_tile0[u.g + 1] - s_tile0[u.g], 0) == NT;
      const int xrow = __shfl_sync(0xffffffffu, u.row0, 0) + prank * kBM;
      const int wrow = __shfl_sync(0xffffffffu, u.g * a.w_rows + u.n * feat, 0) + prank * (EPI == EPI_SWIGLU ? tail ? 64 : a.F : half);
      for (int i = 0; i < steps; ++i) {
        ok = mbar_wait_warp(smem_u32(&empty_bar[stage]), phase ^ 1, abort_word);
        if (!ok) break;
        const uint32_t fb = full0 + 8 * stage, st = smem_u32(smem) + stage * stage_bytes;
        const int kb = i * kWSub, n = min(kWSub, kblocks - kb);
        if (elect_one()) {
          // a tail has two halves of one operand's token rows
          if (leader) mbar_expect_tx(smem_u32(&full_bar[stage]), n * ((both ? 2 : 1) * kWOperandBytes + 2 * w_bytes));
#pragma unroll
          for (int j = 0; j < kWSub; ++j) {
            if (j < n) {
              const uint32_t sx = st + j * sub_bytes;
              const int x = a.w_blocked ? 0 : (kb + j) * kBK, y = a.w_blocked ? (wrow / kBM * kblocks + kb + j) * kBM : wrow;
              const uint64_t pol = once ? pol_first : pol_last;
              if (EPI == EPI_SWIGLU && tail) {      // 64 gate rows and the matching 64 up rows
                const int up = wrow + a.F;
                tma_load_2d_pair(sx + kWOperandBytes, &tmW64, x, a.w_blocked ? y + wrow % kBM : wrow, fb, pol);
                tma_load_2d_pair(sx + kWOperandBytes + w_bytes / 2, &tmW64, x,
                                 a.w_blocked ? (up / kBM * kblocks + kb + j) * kBM + up % kBM : up, fb, pol);
              } else {
                tma_load_2d_pair(sx + kWOperandBytes, &tmW, x, y, fb, pol);
              }
              if (tail) tma_load_2d_pair(sx, &tmX64, (kb + j) * kBK, xrow - prank * 64, fb, pol_last);
              else if (mine) tma_load_2d_pair(sx, &tmX, (kb + j) * kBK, xrow, fb, pol_last);
            }
          }
        }
        __syncwarp();
        if (++stage == a.stages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the even CTA's)
    if (leader) {
      const uint32_t idesc_full = umma_idesc_bf16(2 * kBM, a.cols), idesc_tail = umma_idesc_bf16(kBM, a.cols);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (WideTurn w(pair, pairs); ok && u.locate(w.tile(), s_start, s_tile0, a.G, NT, t_end); w.next(), ++it) {
        const int buf = it & 1;
        const uint32_t idesc = a.tails && __shfl_sync(0xffffffffu, u.ntok, 0) <= kBM ? idesc_tail : idesc_full;
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(smem_u32(&tempty_bar[buf]), ((it >> 1) & 1) ^ 1, abort_word, DMOE_WAIT_CYCLES));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d0 = tmem_base + buf * kWCols;
        for (int i = 0; i < steps; ++i) {
          ok = mbar_wait_warp(smem_u32(&full_bar[stage]), phase, abort_word);
          if (!ok) break;
          tc_fence_after();
          const uint32_t st = smem_u32(smem) + stage * stage_bytes;
          const int n = min(kWSub, kblocks - i * kWSub);
          if (elect_one()) {
#pragma unroll
            for (int j = 0; j < kWSub; ++j) {
              if (j < n) {
                const uint64_t da = umma_desc_sw128(st + j * sub_bytes), db = umma_desc_sw128(st + j * sub_bytes + kWOperandBytes);
#pragma unroll
                for (int k = 0; k < kBK / kUmmaK; ++k)
                  umma_f16_pair(d0, da + 2 * k, db + 2 * k, idesc, (i > 0 || j > 0 || k > 0) ? 1u : 0u);
              }
            }
            umma_commit_both(smem_u32(&empty_bar[stage]));
          }
          __syncwarp();
          if (++stage == a.stages) { stage = 0; phase ^= 1; }
        }
        if (ok && elect_one()) umma_commit_both(smem_u32(&tfull_bar[buf]));
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5): lane = token
    const int q = warp & 3;
    int it = 0, put_buf = 0;
    const uint32_t put_smem = smem_u32(put_rows) + q * 2 * kWPutBytes;
    // 32 columns from x of the warp's 32 rows from y. A lane has a row, so plain stores are 16 bytes of 32 rows, four times; through
    // 64-byte swizzled shared memory (no bank is met twice) the copy engine writes rows of 64 bytes while the next columns are read
    // from TMEM. Plain stores -> this, us: 2500 x 7184 x 2048 54.7 -> 52.6, 3000 x 4096 x 512 20.4 -> 19.5, 576 x 6144 x 2048 20.0 ->
    // 18.8, 2500 x 2048 x 1024 15.4 -> 14.3; median of 42 sizes 2 %; SwiGLU 2952 x 2816 x
    // 256 21.3 -> 20.7, 4096 x 14336 x 1024 169 -> 161
    const auto put = [&](const float (&o)[32], int x, int y) {
      if (lane == 0) bulk_wait_read<1>();
      __syncwarp();
      const uint32_t base = put_smem + put_buf * kWPutBytes;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint4 v = pack8(o + 8 * i);
        const uint32_t at = base + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmY, base, x, y);
        bulk_commit();
      }
      put_buf ^= 1;
    };
    for (WideTurn turn(pair, pairs); u.locate(turn.tile(), s_start, s_tile0, a.G, NT, t_end); turn.next(), ++it) {
      const int buf = it & 1;
      if (!mbar_wait(smem_u32(&tfull_bar[buf]), (it >> 1) & 1, abort_word)) break;
      tc_fence_after();
      const uint32_t t0 = tmem_base + buf * kWCols + (static_cast<uint32_t>(q * 32) << 16);
      // A tail's accumulator has the tokens of the CTA in lanes 0 .. 63 with the columns of the even CTA's weights, and again in
      // lanes 64 .. 127 with those of the odd one's
      const bool tail = a.tails && u.ntok <= kBM;
      const int first = tail ? prank * 64 + (q & 1) * 32 : prank * kBM + q * 32;      // first token of this warp inside the tile
      const int width = tail ? feat / 2 : feat;                                       // columns of this warp
      const bool ok_row = first + lane < u.ntok;
      const long long t = u.row0 + first + lane;
      const int f0 = u.n * feat + (tail ? (q >> 1) * width : 0);
      const uint32_t back = mapa_rank(smem_u32(&tempty_bar[buf]), 0);
      // after a warp's last read of the accumulator
      const auto hand_back = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(back);
      };
      if (first >= u.ntok || f0 >= a.F) {
        hand_back();
        continue;
      }
      // rows past the last one are past the end of Y, but for groups, whose rows are followed by those of the next
      const bool whole = a.put != 0 && (a.offs == nullptr || first + 32 <= u.ntok);
      if (EPI == EPI_SWIGLU) {
        const int cols = min(width, a.F - f0), chunks = (cols + 31) / 32;
        const float s = a.recs != nullptr && ok_row ? __int_as_float(__ldg(&a.recs[t].z)) : 1.f;
        __nv_bfloat16* y = static_cast<__nv_bfloat16*>(a.Y) + t * a.ldy + f0;
#pragma unroll 1
        for (int c = 0; c < chunks; ++c) {
          uint32_t g[32], up[32];
          tmem_ld32(t0 + c * 32, g);
          tmem_ld32(t0 + width + c * 32, up);
          tmem_ld_wait();
          if (c == chunks - 1) hand_back();
          float o[32], x[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) { o[j] = __uint_as_float(g[j]) * s; x[j] = __uint_as_float(up[j]) * s; }
          gated(o, x, a.act, a.act_limit);
          if (whole && (c * 32 + 32 <= cols || f0 + cols == a.F)) put(o, f0 + c * 32, u.row0 + first);
          else if (ok_row) store32(y + c * 32, o, cols - c * 32);
        }
      } else if (EPI == EPI_PLAIN && a.rope_table != nullptr) {
        // QKV: rotation partners are hd / 2 columns apart in the same lane. The accumulator is rounded to bf16 before the
        // rotation, as the unfused path stores and re-reads it. A tile holds whole heads (gemm_wide checks its columns).
        const int half = a.hd >> 1, hc = half >> 5;              // 32-column chunks per half head
        const int heads = min(a.cols, a.F - f0) / a.hd;
        int pos = ok_row ? __ldg(a.positions + t) : 0;
        pos = pos < 0 ? 0 : (pos >= a.rope_max_pos ? a.rope_max_pos - 1 : pos);
        const long long slot = ok_row && a.slots != nullptr ? __ldg(a.slots + t) : -1;
#pragma unroll 1
        for (int h = 0; h < heads; ++h) {
          const int head = f0 / a.hd + h;
          const bool rot = head < a.n_q + a.n_kv;
          __nv_bfloat16* dst;
          bool put = ok_row;
          if (head < a.n_q) {
            dst = static_cast<__nv_bfloat16*>(a.Y) + t * a.ldy + static_cast<long long>(head) * a.hd;
          } else {
            const int kvh = head - a.n_q;
            put = put && slot >= 0;
            dst = (kvh < a.n_kv ? a.kcache : a.vcache) + (slot * a.n_kv + (kvh < a.n_kv ? kvh : kvh - a.n_kv)) * a.hd;
          }
#pragma unroll 1
          for (int c = 0; c < hc; ++c) {
            uint32_t lo[32], hi[32];
            tmem_ld32(t0 + h * a.hd + c * 32, lo);
            tmem_ld32(t0 + h * a.hd + half + c * 32, hi);
            tmem_ld_wait();
            if (h == heads - 1 && c == hc - 1) hand_back();
            float x[32], z[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) { x[j] = __uint_as_float(lo[j]); z[j] = __uint_as_float(hi[j]); }
            if (rot) {
              const float4* cs = reinterpret_cast<const float4*>(a.rope_table + static_cast<long long>(pos) * half + c * 32);
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const float4 v = __ldg(cs + j);      // (cos, sin) of two consecutive rotation pairs
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const float p = __bfloat162float(__float2bfloat16(x[2 * j + e])), r = __bfloat162float(__float2bfloat16(z[2 * j + e]));
                  const float co = e ? v.z : v.x, si = e ? v.w : v.y;
                  x[2 * j + e] = p * co - r * si;
                  z[2 * j + e] = r * co + p * si;
                }
              }
            }
            if (put) {
              store32(dst + c * 32, x, 32);
              store32(dst + half + c * 32, z, 32);
            }
          }
        }
      } else {
        const int cols = min(width, a.F - f0), chunks = (cols + 31) / 32;
        int4 rec = make_int4(0, -1, 0, 0);
        __nv_bfloat16* y = nullptr;
        float w = 1.f;
        if (EPI == EPI_COMBINE) {
          if (ok_row) rec = __ldg(&a.recs[t]);
          if (rec.y >= 0) y = static_cast<__nv_bfloat16*>(a.bases[rec.x]) + static_cast<long long>(rec.y) * a.ldy + f0;
          if (!a.unit_weights) w = __int_as_float(rec.z);
        } else if (ok_row && !a.y_f32) {
          y = static_cast<__nv_bfloat16*>(a.Y) + t * a.ldy + f0;
        }
        float* yf = EPI == EPI_PLAIN && ok_row && a.y_f32 ? static_cast<float*>(a.Y) + t * a.ldy + f0 : nullptr;
        const __nv_bfloat16* res = EPI == EPI_PLAIN && a.R != nullptr && ok_row ? a.R + t * a.ldr + f0 : nullptr;
#pragma unroll 1
        for (int c = 0; c < chunks; ++c) {
          const int left = cols - c * 32;
          uint32_t v[32];
          tmem_ld32(t0 + c * 32, v);
          uint4 rr[4];
          if (EPI == EPI_PLAIN && res != nullptr) {
#pragma unroll
            for (int i = 0; i < 4; ++i) rr[i] = 8 * i < left ? *reinterpret_cast<const uint4*>(res + c * 32 + 8 * i) : make_uint4(0, 0, 0, 0);
          }
          tmem_ld_wait();
          if (c == chunks - 1) hand_back();
          float o[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __uint_as_float(v[j]);
          if (EPI == EPI_COMBINE) {
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] *= w;
          } else {
            if (a.act == 2) {
#pragma unroll
              for (int j = 0; j < 32; ++j) o[j] = out_tanh(o[j]);
            }
            const int silu = a.act == 4 ? a.act_cols - f0 - c * 32 : 0;      // columns of this chunk that take it
            if (silu >= 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j) o[j] = gate_act<0>(o[j]);
            } else if (silu > 0) {
#pragma unroll
              for (int j = 0; j < 32; ++j) o[j] = j < silu ? gate_act<0>(o[j]) : o[j];
            }
            if (res != nullptr) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162* rp = reinterpret_cast<const __nv_bfloat162*>(&rr[i]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 rf = __bfloat1622float2(rp[e]);
                  o[8 * i + 2 * e] += rf.x;
                  o[8 * i + 2 * e + 1] += rf.y;
                }
              }
            }
            if (yf != nullptr) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                if (4 * i < left) *reinterpret_cast<float4*>(yf + c * 32 + 4 * i) = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
            }
          }
          if (EPI == EPI_PLAIN && whole && !a.y_f32) put(o, f0 + c * 32, u.row0 + first);      // 256 columns, or those up to the end of Y
          else if (y != nullptr) store32(y + c * 32, o, left);
        }
      }
    }
  }

  if (warp >= 2 && lane == 0) bulk_wait_read<0>();
  // ---------------------------------------------------------------- tear-down
  tc_fence_before();
  __syncthreads();
  if (*abort_word) {
    if (threadIdx.x == 0 && a.status != nullptr) atomicCAS(a.status, kStatusOk, kStatusBarrierTimeout);
    // give copies that may still be in flight time to land before shared memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();      // neither CTA leaves (or frees TMEM) while the other may still signal or use it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * kWCols);
  }
}

template <int EPI>
static int launch_wide(const CUtensorMap& tmW, const CUtensorMap& tmX, const CUtensorMap& tmY, const CUtensorMap& tmW64,
                       const CUtensorMap& tmX64, const WideArgs& a, int smem, int max_tiles, cudaStream_t stream) {
  static PerDeviceOnce configured;
  const int crc = configured.run([] {
    return static_cast<int>(cudaFuncSetAttribute(gemm_wide_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWSmemMax));
  });
  if (crc != 0) return crc;
  int pairs = device_num_sms() / 2;
  if (max_tiles < pairs) pairs = max_tiles;
  if (pairs < 1) pairs = 1;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(kWThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_wide_kernel<EPI>, tmW, tmX, tmY, tmW64, tmX64, a));
}

// Y [rows, F] as boxes of 32 rows x 32 columns with the 64-byte swizzle
static int make_put_map(CUtensorMap* map, void* y, long long rows, long long F, long long ld) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return -1;
  cuuint64_t dim[2] = {static_cast<cuuint64_t>(F), static_cast<cuuint64_t>(rows)};
  cuuint64_t stride[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {32, 32}, step[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, y, dim, stride, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
             CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -2;
}

int gemm_wide(const DmoeGemm* d, cudaStream_t stream) {
  WideArgs a;
  memset(&a, 0, sizeof(a));
  a.cols = d->wide > 1 ? d->wide : kWCols;
  if (a.cols < 64 || a.cols > kWCols || a.cols % 32 != 0 || (d->w_blocked && a.cols != kWCols) ||
      (d->rope_table != nullptr && a.cols % d->hd != 0))
    return -11;
  const int stage_bytes = kWSub * (kWOperandBytes + a.cols / 2 * kBK * 2);
  a.stages = kWMaxStages;
  while (wide_smem(a.stages, stage_bytes, d->G) > kWSmemMax) --a.stages;
  const int smem = wide_smem(a.stages, stage_bytes, d->G);
  a.offs = d->offs;
  a.G = d->G; a.T = d->T; a.F = d->F; a.K = d->K;
  a.w_rows = d->epi == EPI_SWIGLU ? 2 * d->F : d->F;
  a.w_blocked = d->w_blocked != 0;
  a.Y = d->Y; a.ldy = d->ldy; a.y_f32 = d->y_f32;
  a.R = static_cast<const __nv_bfloat16*>(d->R); a.ldr = d->ldr;
  a.recs = static_cast<const int4*>(d->recs);
  a.bases = static_cast<void* const*>(d->bases);
  a.unit_weights = d->unit_weights;
  a.act = d->act; a.act_limit = d->act_limit; a.act_cols = d->act_cols;
  a.rope_table = static_cast<const float2*>(d->rope_table);
  a.positions = d->positions; a.slots = d->slots;
  a.kcache = static_cast<__nv_bfloat16*>(d->kcache); a.vcache = static_cast<__nv_bfloat16*>(d->vcache);
  a.n_q = d->n_q; a.n_kv = d->n_kv; a.hd = d->hd; a.rope_max_pos = d->rope_max_pos;
  a.status = d->status;
  CUtensorMap tmW, tmX, tmY, tmW64, tmX64;
  const long long ldx = d->ldx > 0 ? d->ldx : d->K, rows = static_cast<long long>(d->G) * a.w_rows;
  if (a.w_blocked) {
    if (make_map_2d(&tmW, d->W, rows * (d->K / kBK), kBK, kBK, kBM) != 0) return -20;
  } else if (make_map_2d(&tmW, d->W, rows, d->K, d->K, a.cols / 2) != 0) {
    return -20;
  }
  if (make_map_2d(&tmX, d->X, d->T, d->K, ldx, kBM) != 0) return -21;
  memset(&tmY, 0, sizeof(tmY));
  memset(&tmW64, 0, sizeof(tmW64));
  memset(&tmX64, 0, sizeof(tmX64));
  a.tails = a.cols == kWCols && d->rope_table == nullptr;
  if (a.tails && make_map_2d(&tmX64, d->X, d->T, d->K, ldx, 64) != 0) return -21;
  if (a.tails && d->epi == EPI_SWIGLU) {
    if ((a.w_blocked ? make_map_2d(&tmW64, d->W, rows * (d->K / kBK), kBK, kBK, 64) : make_map_2d(&tmW64, d->W, rows, d->K, d->K, 64)) != 0)
      return -20;
  }
  a.put = d->epi != EPI_COMBINE && !d->y_f32 && d->rope_table == nullptr && d->Y != nullptr;
  if (a.put && make_put_map(&tmY, d->Y, d->T, d->F, d->ldy) != 0) return -22;
  const int feat = d->epi == EPI_SWIGLU ? a.cols / 2 : a.cols;
  // upper bound of the tile count (group sizes live on the device): every group may add one ragged tile
  const long long tiles = static_cast<long long>((d->F + feat - 1) / feat) * ((d->T + kWTokens - 1) / kWTokens + (d->offs ? d->G : 0));
  if (tiles > (1 << 30)) return -11;
  if (d->epi == EPI_PLAIN) return launch_wide<EPI_PLAIN>(tmW, tmX, tmY, tmW64, tmX64, a, smem, static_cast<int>(tiles), stream);
  if (d->epi == EPI_SWIGLU) return launch_wide<EPI_SWIGLU>(tmW, tmX, tmY, tmW64, tmX64, a, smem, static_cast<int>(tiles), stream);
  return launch_wide<EPI_COMBINE>(tmW, tmX, tmY, tmW64, tmX64, a, smem, static_cast<int>(tiles), stream);
}

}  // namespace dmoe
