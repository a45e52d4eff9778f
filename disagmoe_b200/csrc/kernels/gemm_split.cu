// Dense bf16 GEMM for launches that gemm.cu and gemm_wide.cu cannot fill the chip with: one tile per CTA, K cut over a cluster.
//
// gemm.cu is persistent and parks the partial tiles of a split along K in global memory, where the last arriver of an atomic
// counter reads them back; of the 12.4 us that 48 x 2048 x 2048 took there, 7 went by after the last MMA. Here the S CTAs of a
// cluster own a tile of 128 weight rows x bn tokens and a share of K each. When its MMAs are done, a CTA turns its accumulator
// into rows of 128 partial sums per token and sends each CTA of the cluster the rows of the tokens that it owns (bulk copies
// between shared memories, counted on the receiver's barrier). Every CTA then adds S partial rows per token in the order of
// their ranks, applies the epilogue and stores rows of 256 bytes. No counter, no workspace, no second pass; the order of a sum
// depends on the sizes alone.
//
// The weights are the M operand (gemm.cu says why); the token tile is any multiple of 16 up to 256 rows, so that one wave of
// CTAs can be made to fit the chip at any number of tokens. For SwiGLU a tile is 64 gate and the matching 64 up rows: they meet
// again when the partial rows are added up. Up to 128 tokens a CTA takes 112 KB of shared memory, so that two of them share an SM.
//
// A stage holds two K blocks (one from 96 tokens on, where two CTAs share an SM): a round of the issuing warp (wait, MMAs, commit)
// takes about 400 cycles however small the MMAs are. Warp roles as in gemm.cu: warp 0 TMA producer, warp 1 TMEM owner and MMA issuer,
// warps 2..5 accumulator readers; all six add up.
// ops/gemm.py: split_plan holds the rule that chooses bn, S and this kernel, with both sides measured.
#include <string.h>

#include <algorithm>
#include <atomic>

#include "gemm_common.cuh"

namespace dmoe {

constexpr int kSThreads = 192;
constexpr int kSSmallSmem = 112 * 1024 + 512;            // two CTAs per SM
constexpr int kSLargeSmem = 226 * 1024;
constexpr int kSStaticSmem = 256;                        // barriers and the like, at most
constexpr int kSWBytes = kBM * kBK * 2;                  // weights of one K block
constexpr int kSSub = 2;                                 // K blocks per stage (one where two stages of two do not fit)
constexpr int kSMaxStages = 6;
constexpr int kSRow = kBM * 4;                           // bytes of a token's partial sums

struct SplitArgs {
  int T, F, K, bn, splits, per, sub;      // per: K blocks per CTA, sub: per stage
  int stages, recv_off, alias;       // recv_off: partial rows of this CTA's tokens; alias: they lie over the stages
  int tmem_cols;
  void* Y;
  long long ldy;
  int y_f32;
  const __nv_bfloat16* R;
  long long ldr;
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
};

// Contiguous bytes of this CTA's shared memory to a CTA of its cluster, counted on that CTA's barrier.
__device__ __forceinline__ void bulk_to_cluster(uint32_t dst_cluster, uint32_t src, uint32_t bytes, uint32_t bar_cluster) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_cluster), "r"(src),
               "r"(bytes), "r"(bar_cluster)
               : "memory");
}

// Partial rows of the tokens that this CTA owns: its own and those of the others, added in the order of the ranks.
struct PartialRows {
  const float* own;
  const float* recv;
  int rank, splits, stride;      // stride: floats between the rows of two senders
  // 8 consecutive sums, `at` floats behind the first
  __device__ __forceinline__ void sum8(int at, float (&o)[8]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = 0.f;
#pragma unroll 4
    for (int s = 0; s < splits; ++s) {
      const float* p = s == rank ? own + at : recv + (s < rank ? s : s - 1) * stride + at;
      const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
      o[0] += a.x; o[1] += a.y; o[2] += a.z; o[3] += a.w;
      o[4] += b.x; o[5] += b.y; o[6] += b.z; o[7] += b.w;
    }
  }
};

__device__ __forceinline__ uint4 pack_row8(const float (&x)[8]) {
  uint4 pk;
  __nv_bfloat162* pp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
  for (int i = 0; i < 4; ++i) pp[i] = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
  return pk;
}

// QKV: features f0 .. f0 + 7 of token t, whose partial sums are `at` floats behind the first. A tile holds whole heads, so the rotation
// partner of a feature is half a head away in the same partial rows. Sums are rounded to bf16 before the rotation, as the unfused path
// stores and re-reads them.
__device__ __forceinline__ void rope_item(const SplitArgs& a, const PartialRows& rows, int at, int f0, long long t) {
  const int half = a.hd >> 1, d0 = f0 % a.hd, head = f0 / a.hd;
  const bool lower = d0 < half, rot = head < a.n_q + a.n_kv;
  int pos = rot ? __ldg(a.positions + t) : 0;
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.Y) + t * a.ldy + f0;
  if (head >= a.n_q) {
    const long long slot = a.slots != nullptr ? __ldg(a.slots + t) : -1;
    const int kvh = head - a.n_q;
    dst = slot < 0 ? nullptr : (kvh < a.n_kv ? a.kcache : a.vcache) + (slot * a.n_kv + (kvh < a.n_kv ? kvh : kvh - a.n_kv)) * a.hd + d0;
  }
  float o[8], z[8];
  rows.sum8(at, o);
  if (rot) {
    rows.sum8(at + (lower ? half : -half), z);
    pos = pos < 0 ? 0 : (pos >= a.rope_max_pos ? a.rope_max_pos - 1 : pos);
    const float4* cs = reinterpret_cast<const float4*>(a.rope_table + static_cast<long long>(pos) * half + (lower ? d0 : d0 - half));
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 v = __ldg(cs + e);      // (cos, sin) of two consecutive rotation pairs
      const float a0 = __bfloat162float(__float2bfloat16(o[2 * e])), b0 = __bfloat162float(__float2bfloat16(z[2 * e]));
      const float a1 = __bfloat162float(__float2bfloat16(o[2 * e + 1])), b1 = __bfloat162float(__float2bfloat16(z[2 * e + 1]));
      o[2 * e] = lower ? a0 * v.x - b0 * v.y : a0 * v.x + b0 * v.y;
      o[2 * e + 1] = lower ? a1 * v.z - b1 * v.w : a1 * v.z + b1 * v.w;
    }
  }
  if (dst != nullptr) *reinterpret_cast<uint4*>(dst) = pack_row8(o);
}

template <int EPI>
__global__ void __launch_bounds__(kSThreads)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SplitArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kFeat = EPI == EPI_SWIGLU ? kBM / 2 : kBM;      // output features per tile
  const int x_bytes = a.bn * kBK * 2, stage_bytes = a.sub * (kSWBytes + x_bytes);
  __shared__ uint64_t bars[2 * kSMaxStages + 2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  const uint32_t full = smem_u32(bars), empty = full + 8 * kSMaxStages, tfull = empty + 8 * kSMaxStages, rfull = tfull + 8;

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int rank = blockIdx.x, m = blockIdx.y;
  const int row0 = blockIdx.z * a.bn, ntok = min(a.bn, a.T - row0);
  const int tpr = (ntok + a.splits - 1) / a.splits;             // tokens of the tile that a CTA adds up
  const int tok0 = rank * tpr, own = max(0, min(tpr, ntok - tok0));
  const int kblocks = (a.K + kBK - 1) / kBK;
  const int kb0 = rank * a.per, nkb = min(a.per, kblocks - kb0), steps = (nkb + a.sub - 1) / a.sub;
  const bool cluster = a.splits > 1;
  float* parts = reinterpret_cast<float*>(smem);                     // [tokens][kBM], over the stages once these are consumed
  float* recv = reinterpret_cast<float*>(smem + a.recv_off);         // [splits - 1][tpr][kBM]: the others' rows of this CTA's tokens

  if (threadIdx.x == 0) {
    abort_word = 0;
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full + 8 * s, 1);
      mbar_init(empty + 8 * s, 1);
    }
    mbar_init(tfull, 1);
    mbar_init(rfull, 1);
    mbar_fence_init();
    if (cluster && own > 0) mbar_expect_tx(rfull, own * kSRow * (a.splits - 1));
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), a.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  pdl_trigger();      // behind the allocation: a CTA of the next launch never holds TMEM that this one still needs
  // partial rows may be sent to a CTA that runs (or, over the stages, to one whose MMAs are done)
  if (cluster && !a.alias) cluster_arrive_relaxed();
  // all warps: the time limits below count from here, and the launch before may wait for a peer longer than they allow
  pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    const uint64_t pol_w = gridDim.z == 1 ? l2_policy_evict_first() : l2_policy_evict_last(), pol_x = l2_policy_evict_last();
    int stage = 0;
    uint32_t phase = 0;
    for (int i = 0; i < steps; ++i) {
      if (!mbar_wait_warp(empty + 8 * stage, phase ^ 1, &abort_word)) break;
      const uint32_t fb = full + 8 * stage, st = smem_u32(smem) + stage * stage_bytes, sx = st + a.sub * kSWBytes;
      const int x = (kb0 + i * a.sub) * kBK, n = min(a.sub, nkb - i * a.sub);
      if (elect_one()) {
        mbar_expect_tx(fb, n * (kSWBytes + x_bytes));
#pragma unroll
        for (int k = 0; k < kSSub; ++k) {
          if (k < n) {
            tma_load_2d(st + k * kSWBytes, &tmW, x + k * kBK, m * kFeat, fb, pol_w);
            if (EPI == EPI_SWIGLU) tma_load_2d(st + k * kSWBytes + kSWBytes / 2, &tmW, x + k * kBK, a.F + m * kFeat, fb, pol_w);
            tma_load_2d(sx + k * x_bytes, &tmX, x + k * kBK, row0, fb, pol_x);
          }
        }
      }
      __syncwarp();
      if (++stage == a.stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t idesc = umma_idesc_bf16(kBM, (ntok + 15) & ~15);      // ragged tiles pay for the columns they have
    int stage = 0;
    uint32_t phase = 0;
    for (int i = 0; i < steps; ++i) {
      if (!mbar_wait_warp(full + 8 * stage, phase, &abort_word)) break;
      tc_fence_after();
      const uint32_t st = smem_u32(smem) + stage * stage_bytes, sx = st + a.sub * kSWBytes;
      const int n = min(a.sub, nkb - i * a.sub);
      if (elect_one()) {
#pragma unroll
        for (int j = 0; j < kSSub; ++j) {
          if (j < n) {
            const uint64_t da = umma_desc_sw128(st + j * kSWBytes), db = umma_desc_sw128(sx + j * x_bytes);
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; ++k)
              umma_f16(tmem_base, da + 2 * k, db + 2 * k, idesc, (i > 0 || j > 0 || k > 0) ? 1u : 0u);
          }
        }
        umma_commit(empty + 8 * stage);
        if (i == steps - 1) umma_commit(tfull);
      }
      __syncwarp();
      if (++stage == a.stages) { stage = 0; phase ^= 1; }
    }
  } else if (mbar_wait_warp(tfull, 0, &abort_word)) {
    // ------------------------------------------------------------ accumulator to rows of one token (warps 2..5)
    tc_fence_after();
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t t0 = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
    for (int c = 0; c * 32 < ntok; ++c) {
      uint32_t v[32];
      tmem_ld32(t0 + c * 32, v);
      tmem_ld_wait();
      float* p = parts + c * 32 * kBM + row;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (c * 32 + j < ntok) p[j * kBM] = __uint_as_float(v[j]);
      }
    }
    fence_proxy_async_smem();
  }
  __syncthreads();
  if (cluster) {
    if (a.alias) cluster_arrive_relaxed();
    cluster_wait();
    if (warp == 0 && lane < a.splits && lane != rank && *const_cast<volatile int*>(&abort_word) == 0) {
      const int rows = min(tpr, ntok - lane * tpr);
      if (rows > 0)
        bulk_to_cluster(mapa_rank(smem_u32(recv) + (rank < lane ? rank : rank - 1) * tpr * kSRow, lane),
                        smem_u32(parts) + lane * tpr * kSRow, rows * kSRow, mapa_rank(rfull, lane));
    }
    __syncwarp();
  }
  if (cluster && own > 0) mbar_wait(rfull, 0, &abort_word);
  __syncwarp();
  if (cluster) cluster_arrive_relaxed();      // all that this CTA waits for has come

  // ---------------------------------------------------------------- add up, epilogue, store: 8 features of one token per item
  constexpr int kGroups = kFeat / 8;
  const int items = own * kGroups;
  PartialRows rows;
  rows.rank = rank; rows.splits = a.splits; rows.stride = tpr * kBM;
  rows.own = parts + tok0 * kBM;
  rows.recv = recv;
  // one item at a time: two or four at a time were slower at every size (6.8, 6.9 instead of 6.7 us at 37 x 2048 x 2048)
#pragma unroll 1
  for (int i = threadIdx.x; i < items; i += kSThreads) {
    const int j = i / kGroups, f = i % kGroups * 8, f0 = m * kFeat + f, at = j * kBM + f;
    if (f0 >= a.F) continue;
    const long long t = row0 + tok0 + j;
    if (EPI == EPI_PLAIN && a.rope_table != nullptr) {
      rope_item(a, rows, at, f0, t);
      continue;
    }
    uint4 rr = make_uint4(0, 0, 0, 0);
    if (EPI == EPI_PLAIN && a.R != nullptr) rr = *reinterpret_cast<const uint4*>(a.R + t * a.ldr + f0);
    float o[8];
    rows.sum8(at, o);
    if (EPI == EPI_SWIGLU) {
      float u[8];
      rows.sum8(at + kFeat, u);
      gated(o, u, a.act, a.act_limit);
    } else {
      if (a.act == 2) {
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = out_tanh(o[k]);
      } else if (a.act == 4) {
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = f0 + k < a.act_cols ? gate_act<0>(o[k]) : o[k];
      }
      if (a.R != nullptr) {
        const __nv_bfloat162* rp = reinterpret_cast<const __nv_bfloat162*>(&rr);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 rf = __bfloat1622float2(rp[k]);
          o[2 * k] += rf.x;
          o[2 * k + 1] += rf.y;
        }
      }
    }
    if (EPI == EPI_PLAIN && a.y_f32) {
      float4* y = reinterpret_cast<float4*>(static_cast<float*>(a.Y) + t * a.ldy + f0);
      y[0] = make_float4(o[0], o[1], o[2], o[3]);
      y[1] = make_float4(o[4], o[5], o[6], o[7]);
    } else {
      *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.Y) + t * a.ldy + f0) = pack_row8(o);
    }
  }

  // ---------------------------------------------------------------- tear-down
  tc_fence_before();
  __syncthreads();
  if (abort_word) {
    if (threadIdx.x == 0 && a.status != nullptr) atomicCAS(a.status, kStatusOk, kStatusBarrierTimeout);
    // give copies that may still be in flight time to land before shared memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (cluster) cluster_wait();      // the others have what this CTA sent from its shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, a.tmem_cols);
  }
}

template <int EPI>
static int configure_split() {
  static PerDeviceOnce configured;
  return configured.run([] {
    return static_cast<int>(cudaFuncSetAttribute(gemm_split_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSLargeSmem));
  });
}

// What the driver is asked about in place of gemm_split_kernel: of a kernel that allocates tensor memory it counts one CTA per SM
// whatever it needs, where two do share an SM (tiles of 16 tokens, K 512, in L2: 148 CTAs 5.3 us, 149 5.9, 296 6.9, 297 9.2).
__global__ void __launch_bounds__(kSThreads) split_room_kernel() {}

// CTAs in clusters of `splits` that are on the chip at once with the large or the small amount of shared memory (asked for once per
// device: clusters stay inside a group of SMs, whose sizes differ from chip to chip); 0 where the driver does not say
static int split_capacity(int splits, bool large) {
  static std::atomic<int> cache[kMaxDevicesPerProcess][2][9];
  int dev = 0;
  if (splits < 1 || splits > 8 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevicesPerProcess) return 0;
  int n = cache[dev][large][splits].load(std::memory_order_relaxed);
  if (n != 0) return n;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(splits, 1, 1);
  cfg.blockDim = dim3(kSThreads, 1, 1);
  cfg.dynamicSmemBytes = (large ? kSLargeSmem : kSSmallSmem) + kSStaticSmem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  // always the large amount: another thread may ask about the other one at the same time
  if (cudaFuncSetAttribute(split_room_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSLargeSmem + kSStaticSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&clusters, split_room_kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();      // not the error of the next launch
    return 0;
  }
  n = clusters * splits;
  cache[dev][large][splits].store(n, std::memory_order_relaxed);
  return n;
}

template <int EPI>
static int launch_split(const CUtensorMap& tmW, const CUtensorMap& tmX, const SplitArgs& a, dim3 grid, int smem, cudaStream_t stream) {
  const int crc = configure_split<EPI>();
  if (crc != 0) return crc;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kSThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = a.splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.numAttrs = 1;
  if (pdl_enabled()) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  cfg.attrs = attr;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_split_kernel<EPI>, tmW, tmX, a));
}

int gemm_split(const DmoeGemm* d, cudaStream_t stream) {
  const int kblocks = (d->K + kBK - 1) / kBK, bn = d->bn;
  if (bn < 16 || bn > 256 || bn % 16 != 0) return -11;
  const bool gate = d->epi == EPI_SWIGLU;
  const int feat = gate ? kBM / 2 : kBM;
  SplitArgs a;
  memset(&a, 0, sizeof(a));
  a.T = d->T; a.F = d->F; a.K = d->K; a.bn = bn;
  a.splits = std::min({d->cluster, kblocks, 8});
  a.per = (kblocks + a.splits - 1) / a.splits;
  a.splits = (kblocks + a.per - 1) / a.per;      // no share may be empty
  // A CTA's partial rows lie over its stages; those it receives behind them where that leaves all of its share or two stages, else over
  // them too. The large amount of shared memory (one CTA per SM) has more stages in flight, which counts where each is fetched from
  // HBM: 1.1 us per round trip. It is taken where all CTAs find place at once, and where the small one is too small.
  const long long mt = (d->F + feat - 1) / feat, nt = (d->T + bn - 1) / bn;
  const bool spread = a.per > 2 * kSSub && a.splits * mt * nt <= split_capacity(a.splits, true);
  const int parts = bn * kSRow, recv = (a.splits - 1) * ((bn + a.splits - 1) / a.splits) * kSRow;
  const auto fits = [&](int room, int sub) {
    const int stage = sub * (kSWBytes + bn * kBK * 2), steps = (a.per + sub - 1) / sub;
    const int most = std::min(steps, kSMaxStages), want = std::min(steps, sub == 1 ? 3 : 2);
    const int beside = std::min(most, (room - recv) / stage), over = std::min(most, room / stage);
    if (beside >= want && beside * stage >= parts) {
      a.alias = 0; a.stages = beside; a.recv_off = beside * stage;
    } else if (over >= want && parts + recv <= room) {
      a.alias = 1; a.stages = over; a.recv_off = parts;
    } else {
      return false;
    }
    a.sub = sub;
    return true;
  };
  const int small = kSSmallSmem - 1024 /*alignment*/, large = kSLargeSmem - 1024;
  int smem = 0;
  if (!spread && (fits(small, kSSub) || (bn <= 128 && fits(small, 1)))) smem = kSSmallSmem;
  else if (fits(large, kSSub)) smem = kSLargeSmem;
  if (smem == 0) return -11;
  a.tmem_cols = 32;
  while (a.tmem_cols < bn) a.tmem_cols *= 2;
  a.Y = d->Y; a.ldy = d->ldy; a.y_f32 = d->y_f32;
  a.R = static_cast<const __nv_bfloat16*>(d->R); a.ldr = d->ldr;
  a.act = d->act; a.act_limit = d->act_limit; a.act_cols = d->act_cols;
  a.rope_table = static_cast<const float2*>(d->rope_table);
  a.positions = d->positions; a.slots = d->slots;
  a.kcache = static_cast<__nv_bfloat16*>(d->kcache); a.vcache = static_cast<__nv_bfloat16*>(d->vcache);
  a.n_q = d->n_q; a.n_kv = d->n_kv; a.hd = d->hd; a.rope_max_pos = d->rope_max_pos;
  a.status = d->status;
  CUtensorMap tmW, tmX;
  if (make_map_2d(&tmW, d->W, gate ? 2ll * d->F : d->F, d->K, d->K, feat) != 0) return -20;
  if (make_map_2d(&tmX, d->X, d->T, d->K, d->ldx > 0 ? d->ldx : d->K, bn) != 0) return -21;
  if (mt > 65535 || nt > 65535) return -11;
  const dim3 grid(a.splits, static_cast<unsigned>(mt), static_cast<unsigned>(nt));
  return gate ? launch_split<EPI_SWIGLU>(tmW, tmX, a, grid, smem, stream) : launch_split<EPI_PLAIN>(tmW, tmX, a, grid, smem, stream);
}

}  // namespace dmoe

// CTAs of the split GEMM that the current device holds at once in clusters of `splits` (1 .. 8), one per SM (`large`) or two; 0: unknown
extern "C" int dmoe_gemm_split_ctas(int splits, int large) { return dmoe::split_capacity(splits, large != 0); }
