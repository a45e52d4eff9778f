"""bf16 GEMMs on the tcgen05 kernels of ``csrc/kernels``: ``gemm.cu``, for prompt-sized batches ``gemm_wide.cu``, for dense products that
these two cannot fill the chip with ``gemm_split.cu``; :func:`want_wide` and :func:`_dense_plan` choose.

``linear``          y = x @ w.T (+ residual)                         -- reference: disagmoe/models/linear.py:131-136
``grouped_swiglu``  act = silu(x @ w13[g][:I].T) * (x @ w13[g][I:].T)   -- reference: disagmoe/models/experts.py:84-88
                    (or the tanh form of gelu in place of silu)
``grouped_linear``  y = x @ w2[g].T per expert group                   -- reference: disagmoe/models/experts.py:89
``grouped_combine`` the same GEMM whose epilogue scales each row by its router weight and scatters it to the
                    row (and GPU) it came from                         -- reference: disagmoe/frontend/engine.py:731-734

Weights are K-contiguous ``[groups, out, in]``. CPU tensors take a plain PyTorch path (used by the fp32 CPU
configuration and as the numerical reference); CUDA tensors always run the sm_100a kernels: bf16 the tcgen05 kernels, fp32
operands (and bf16 operands whose rows are not 16-byte aligned) the CUDA-core kernel of ``csrc/kernels/layer_ops.cu``.
"""
from __future__ import annotations

import ctypes
from functools import lru_cache
from typing import Optional

import torch

from . import _lib, reference

ACTS = {"silu": 0, "gelu_tanh": 1, "clamped": 3}      # of gated feed-forwards; clamped: min(g, limit) sigmoid(1.702 g) (clamp(u) + 1)
ACT_TANH, ACT_SILU = 2, 4      # of the output of a plain GEMM (silu: of its first columns)
EPI_PLAIN, EPI_SWIGLU, EPI_COMBINE = 0, 1, 2
STREAM_K = True      # default work distribution of every GEMM launched without an explicit split (tests may turn it off)
TRACE = None         # profiling aid: an int64 [8] CUDA tensor that CTA 0 of every launch fills with nanosecond stamps
_num_sms_cache = {}


def num_sms(device=None) -> int:
    """SM count of a CUDA device (read once per device)."""
    idx = None if device is None else device.index if isinstance(device, torch.device) else torch.device(device).index
    if idx is None:
        idx = torch.cuda.current_device() if torch.cuda.is_available() else -1
    if idx not in _num_sms_cache:
        _num_sms_cache[idx] = torch.cuda.get_device_properties(idx).multi_processor_count if idx >= 0 else 148
    return _num_sms_cache[idx]


class _Scratch:
    """Per-device split-K workspace, tile counters and status word (allocated once, reused by every call)."""

    def __init__(self, device):
        self.device = device
        self.ws = torch.empty(64 << 20, dtype=torch.uint8, device=device)
        self.counters = torch.zeros(65536, dtype=torch.int32, device=device)
        self.status = torch.zeros(1, dtype=torch.int32, device=device)

    def ensure(self, nbytes):
        if nbytes > self.ws.numel():
            self.ws = torch.empty(int(nbytes * 1.25), dtype=torch.uint8, device=self.device)


_scratch = {}


def scratch(device) -> _Scratch:
    key = (device.index if isinstance(device, torch.device) else torch.device(device).index) or 0
    if key not in _scratch:
        _scratch[key] = _Scratch(torch.device("cuda", key))
    return _scratch[key]


def check_status(device=None) -> int:
    """Reads (and clears) the device status word; non-zero means a kernel gave up on a bounded wait."""
    s = scratch(device if device is not None else torch.cuda.current_device())
    v = int(s.status.item())
    if v != 0:
        s.status.zero_()
    return v


def pick_splitk(T: int, F: int, K: int, bn: int, sms: int = 0) -> int:
    """Split-K factor of a dense GEMM: enough (tile, split) work items to occupy most of the SMs when the output
    has few tiles (decode-size token counts), never more than one split per 4 K-blocks."""
    sms = sms or num_sms()
    tiles = ((F + 127) // 128) * ((T + bn - 1) // bn)
    kblocks = (K + 63) // 64
    if tiles >= sms * 80 // 148 or kblocks < 8:
        return 1
    return max(1, min((sms * 128 // 148 + tiles // 2) // tiles, kblocks // 4, 16))


@lru_cache(maxsize=4096)
def dense_cost(T: int, F: int, K: int, sms: int):
    """(cost in us, token tile, split-K factor) of a dense GEMM below one wave of tiles, by a cost model fitted to the tile /
    split sweep of benchmark/ops/dense_gemm.py on B200. At these sizes a CTA is bound by what its SM can pull from L2
    (~100 GB/s: 16 KB of weights plus bn x 128 B of tokens per K block), so the model counts, per CTA, the bytes of
    its K range times the number of waves, the parked and re-read partial tiles of a split (the last arriver reads
    them chunk by chunk, latency-bound) and a fixed launch + pipeline-fill cost. It reproduces the order of the
    measured configurations (QKV and o_proj of Mixtral at 64-512 tokens)."""
    kblocks = (K + 63) // 64
    mt = (F + 127) // 128
    best = None
    for bn in (32, 64, 128, 256):
        if bn < 32 or (bn > 32 and bn // 2 >= T):
            continue                      # a tile twice as wide as the batch only adds shared-memory traffic
        nt = (T + bn - 1) // bn
        for sk in (1, 2, 3, 4, 6, 8):
            per = (kblocks + sk - 1) // sk
            if sk > 1 and (per < 8 or (kblocks + per - 1) // per != sk):
                continue
            units = mt * nt * sk
            if sk > 1 and units > sms:
                continue                  # a split that spills into a second wave measured far slower than whole tiles
            waves = (units + sms - 1) // sms
            cost = 6.0 + waves * per * (16384 + bn * 128) / 1e5 + (bn // 32) * 0.3
            if sk > 1:
                cost += 128 * bn * 4 / 1e5 + (bn // 32) * sk * 0.35
            if best is None or cost < best[0] - 1e-9:
                best = (cost, bn, sk)
    return best


def pick_dense(T: int, F: int, K: int, sms: int = 0):
    """(token tile, split-K factor) of :func:`dense_cost`."""
    return dense_cost(T, F, K, sms or num_sms())[1:]


def pick_bn(tokens_per_group: int, epi: int) -> int:
    cap = 128 if epi == EPI_SWIGLU else 256
    bn = 32
    while bn < tokens_per_group and bn < cap:
        bn *= 2
    return bn


def pick_even_bn(tokens: int, F: int, G: int, sms: int = 0) -> int:
    """Token tile of a grouped GEMM whose G groups have ``tokens`` rows each (the per-head maps of latent attention): the
    smallest one whose tiles fit one wave of CTAs; below a wave short loops and epilogues count for more than weight re-reads.
    0 (let the grouped GEMM choose) where :func:`want_wide` takes the groups anyway."""
    if tokens >= 144:
        return 0
    for bn in (32, 64, 128):
        if (F + 127) // 128 * G * ((tokens + bn - 1) // bn) <= (sms or num_sms()):
            return bn
    return 256


def want_streamk(epi: int, F: int, G: int, T: int, bn: int, sms: int) -> bool:
    """Work distribution of a grouped GEMM, from measurements on B200 (benchmark/ops/grouped_gemm.py): the stream-K
    tail pays off when the expected tile count fills the last wave of CTAs badly (few experts with long K loops, the
    down-projection at decode sizes); the SwiGLU up-projection, whose partial tiles carry two accumulators, is faster
    with whole tiles. Group sizes are only known on the device: the estimate assumes even routing. (One Mixtral token, two of
    eight experts: 64 tiles for 148 SMs, 77 us with whole tiles, 47 us with a stream-K tail.)"""
    if not STREAM_K or epi == EPI_SWIGLU:
        return False
    active = G * (1.0 - (1.0 - 1.0 / G) ** max(T, 1))       # groups that T evenly routed rows are expected to reach
    tiles = ((F + 127) // 128) * max(round(active), (T + bn - 1) // bn)
    waves = (tiles + sms - 1) // sms
    return tiles / (waves * sms) < 0.85


@lru_cache(maxsize=4096)
def want_wide(epi: int, T: int, F: int, K: int, G: int, sms: int) -> bool:
    """Should the tokens be the M operand (csrc/kernels/gemm_wide.cu, CTA pairs) instead of the weights (csrc/kernels/gemm.cu)?

    Dense: for launches that fit no :func:`split_plan` (:func:`_dense_plan`; one group of a grouped product counts as well). A cost
    model of both, in us, of an earlier state of the two kernels: tiles of 256 weight rows, 0.31 us per K block of 64 whatever part of
    a tile is used, against what an SM of the other kernel pulls from L2; the pair kernel has become the faster of them since (4096 x
    6144 x 4096 then 201 against 149 us, now 228 against 140), so that the line is on the safe side for it. A few rows of SwiGLU gain
    by the wider tile's faster K blocks (1 row, 2048 x 4096 38 -> 32, 16 rows, 8192 x 7168 82 -> 65), but pay 2 us more per launch (1
    row, 2048 x 256 11.2 -> 12.6, 4096 x 1024 17.4 -> 17.4), and more where the tiles of a wave want more than HBM gives (1 row, 8192 x
    1024 17.4 -> 19.3, 8192 x 7168 69 -> 78; 8 rows, 8192 x 4096 47 -> 49).

    Grouped (only the mean group size is known): up to 128 tokens both kernels read the weights once; the wide one has a half product
    for such groups and no transposing epilogue, the other one smaller units, which counts where few experts have long rows of tiles.
    From 40 tokens per expert on, sweep over 20 shapes at 40 .. 128 (other kernel -> wide, us): SwiGLU with F K to 6 million 0.99 ..
    1.57 times as fast (64 x 1408 x 2048, 104 tokens 133 -> 126; 16 x 2816 x 2048, 96 tokens 69 -> 64), above that 0.93 .. 1.1 (8 x
    14336 x 4096: 40 tokens 290 -> 309, 128: 354 -> 339); down-projections to K 5632 1.00 .. 1.70 (16 x (2048 x 2816), 96 tokens 46 ->
    37), 8 x (4096 x 14336): 64 tokens 155 -> 157, 96: 183 -> 159. Beyond 128 tokens the other kernel needs a second tile per group (8
    x 14336 x 4096, SwiGLU, 160: 533 -> 369). Below 40 tokens short K loops are bound by the other kernel's transposing epilogue:
    sweep over 8 .. 64 experts, F 2048 .. 6144, K 512 .. 7168, before the half products and both kernels' present issue loops: with F
    K to 4.4 million 0.92 .. 1.9 times as fast, 1.17 on average (60 x (2048 x 1408): 16 rows 46 -> 34; 8 x (4096 x 1024): 74 rows 28
    -> 25); above that a badly filled wave of long tiles can make it 0.8 times as fast with few experts (16 x (6144 x 2048): 24 rows
    74 -> 88), while 60 and 64 experts still gain to K 2048; from K 2816 on nothing was gained there (8 x (4096 x 14336): 2 rows 47 ->
    77)."""
    kblocks, pairs = (K + 63) // 64, max(1, sms // 2)
    if G > 1:
        if epi == EPI_SWIGLU:
            return T >= 128 * G or (T >= 40 * G and F * K <= 6_000_000)
        return T >= 88 * G or (T >= 40 * G and K <= 6144) or (K <= 2048 and (F * K <= 4_400_000 or G >= 60))
    if T < 64 and epi != EPI_SWIGLU:
        return False
    if T <= 32 and (K < 1024 or F > 4096 and K < (8192 if T <= 8 else 4096)):      # SwiGLU: see above
        return False
    feat = 128 if epi == EPI_SWIGLU else 256
    tiles = ((F + feat - 1) // feat) * ((T + 255) // 256)
    wide = 8.0 + (tiles + pairs - 1) // pairs * kblocks * 0.31
    bn, mt = pick_bn(T, epi), (F + 127) // 128
    units = mt * ((T + bn - 1) // bn)
    if epi == EPI_SWIGLU:
        return wide < 10.0 + (units + sms - 1) // sms * kblocks * (32768 + bn * 128) / 1e5
    return units >= sms or wide < 1.4 + dense_cost(T, F, K, sms)[0]


@lru_cache(maxsize=4096)
def dense_wide(T: int, F: int, K: int, epi: int, sms: int, hd: int = 0):
    """(us, weight rows per tile) of a dense product in csrc/kernels/gemm_wide.cu: of the tile sizes the one whose count fills whole
    waves of CTA pairs best; ``hd``: heads that a tile has to hold whole. Fitted to a sweep on B200 (42 sizes, T 66 .. 4096, K 16 ..
    10944, harness of benchmark/ops/dense_gemm.py; error 7 %, the choice is 1 % slower than the best size on average). Measured with
    256 rows -> with the choice, us: 2500 x 2048 x 2048 27.8 -> 20.0 (80 tiles for 74 pairs -> 130 smaller ones), 2500 x 2048 x 5632
    62.6 -> 43.6, 3000 x 2048 x 2048 27.5 -> 22.8, 2500 x 4096 x 2048 39.3 -> 33.5, 1111 x 6144 x 2048 29.8 -> 27.6, 724 x 3664 x 2048
    18.3 -> 14.3, SwiGLU 1111 x 2816 x 2048 29.3 -> 26.4.

    The 0.9 us of a tile that do not shrink with it count where K is short: without them 1386 x 26112 x 64 took 128 rows (46.3 us,
    37.4 with 256) and SwiGLU 622 x 19584 x 384 160 (38.2 and 31.9). Over 230 sizes (T 129 .. 4096, F 256 .. 32000, K 64 .. 11000) the
    choice is 0.24 % slower than the best size on average (0.72 % without), 8 % at most (24 %)."""
    pairs, best = max(1, sms // 2), None
    rows = 1.15 if K % 16 else 1.0            # rows that start inside a sector of 32 bytes: 102 sizes
    for cols in (256, 224, 192, 160, 128):
        if hd and cols % hd:
            continue
        waves = -(-(-(-F // (cols // 2 if epi == EPI_SWIGLU else cols)) * -(-T // 256)) // pairs)
        cost = 6.1 + waves * (0.9 + 1.4 * cols / 256 + rows * (0.05 + 0.254 * cols / 256) * -(-K // 64))
        if best is None or cost < best[0]:
            best = (cost, cols)
    return best


# CTAs of csrc/kernels/gemm_split.cu that a B200 held at once in clusters of 1 .. 8, with the small amount of shared memory (two per
# SM) and the large one; fewer than two per SM and one, because a cluster stays inside a group of SMs. For rules without a device
# (:func:`split_ctas` asks the one at hand)
_SPLIT_SMALL = (296, 296, 279, 284, 280, 270, 259, 264)
_SPLIT_LARGE = (148, 148, 135, 132, 130, 132, 105, 120)


_split_ctas_cache = {}


def split_ctas(device):
    """(small, large): the two tables above for a CUDA device, as its driver says (asked for once per device)."""
    idx = device.index if device.index is not None else torch.cuda.current_device()
    if idx not in _split_ctas_cache:
        with torch.cuda.device(idx):
            tables = [tuple(_lib.lib().dmoe_gemm_split_ctas(n, large) for n in range(1, 9)) for large in (0, 1)]
        if min(map(min, tables)) <= 0:
            tables = _scaled_ctas(num_sms(torch.device("cuda", idx)))
        _split_ctas_cache[idx] = tuple(tables)
    return _split_ctas_cache[idx]


@lru_cache(maxsize=16)
def _scaled_ctas(sms: int):
    return tuple(tuple(n * sms // 148 for n in t) for t in (_SPLIT_SMALL, _SPLIT_LARGE))


def _split_tile(T: int) -> int:
    return -(-min(T, 128) // 16) * 16


def split_plan(T: int, F: int, K: int, epi: int, sms: int, ctas=None):
    """(cost in us, token tile, CTAs per cluster) of a dense product in csrc/kernels/gemm_split.cu, or None where other kernels are
    faster: all its CTAs have to find place at once, or it has one tile of up to 128 tokens and the weights stream through it (an LM
    head).

    The cost model is fitted to a sweep on B200 (T 1 .. 4096, F 16 .. 151936, K 16 .. 14336; launches back to back, weights from HBM:
    benchmark/ops/dense_gemm.py); its choice is 2.8 % slower than the best tile and cluster on average. Measured, this module's other
    kernels -> the choice, us: 1 x 4096 x 4096 13.9 -> 9.7, 37 x 2048 x 2048 10.3 -> 6.6, 37 x 6144 x 2048 14.6 -> 9.6, 37 x 2048 x
    5632 14.1 -> 9.1, SwiGLU 37 x 5632 x 2048 17.7 -> 11.8, 96 x 2048 x 10944 22.6 -> 14.5, 256 x 4096 x 4096 22.0 -> 16.0, 576 x 2048 x
    5632 29.4 -> 22.0, 1111 x 2048 x 2048 17.8 -> 14.7, 3 x 32000 x 4096 54.1 -> 42.4, 37 x 151936 x 2048 111 -> 104, 96 x 102400 x 2048
    88.5 -> 78.0, 66 x 151936 x 2048 128 -> 110. A second wave costs as much as the first: 200 x 10944 x 2048 SwiGLU (171 CTAs of one
    per SM) 23.0 -> 40.6, 1111 x 2816 x 2048 SwiGLU 28.6 -> 36.4, 192 x 32000 x 2048 32.5 -> 42.5.

    ``ctas``: :func:`split_ctas`. Sizes are rounded up to a grid of tokens, so that few plans serve prompts of all lengths."""
    grid = 16 if T <= 256 else 32 if T <= 1024 else 64
    return _split_plan(-(-T // grid) * grid, F, K, epi, sms, ctas or _scaled_ctas(sms))


@lru_cache(maxsize=4096)
def _split_plan(T: int, F: int, K: int, epi: int, sms: int, ctas):
    gate = epi == EPI_SWIGLU
    mt, kblocks = -(-F // (64 if gate else 128)), -(-K // 64)
    small, large = ctas
    stream = F * K * (4 if gate else 2) / 6.6e6
    # bytes per us that a CTA loads. Rows that start inside a sector of 32 bytes (K not a multiple of 16) come at 0.57 of the rate (85
    # sizes, root of the mean square error 23 -> 11 %): fewer and larger token tiles then, 58 x 9152 x 5864 35.4 -> 25.9 us
    load = 7.3e4 if K % 16 else 1.27e5
    best = None
    if mt > small[0]:
        shapes = [(1, T)] if T <= 128 and mt <= 65535 else []      # tiles of weight rows are the grid's second dimension
    elif mt * -(-T // 256) > small[0]:
        shapes = []
    else:
        shapes = []
        for S in range(1, min(8, kblocks) + 1):
            lo, hi = -(-T // (256 if S == 1 else 208)), min(small[S - 1] // (mt * S), -(-T // 16))
            # a dozen counts of token tiles at most; partial rows sent and received have to fit shared memory: 208 tokens
            shapes += [(S, -(-(-(-T // nt)) // 16) * 16) for nt in range(lo, hi + 1, max(1, (hi - lo) // 12))]
    for S, bn in shapes:
        per = -(-kblocks // S)
        if -(-kblocks // per) != S:
            continue                      # a smaller cluster has the same shares
        units = mt * S * -(-T // bn)
        one = bn > 128 or (per > 4 and units <= large[S - 1])      # one CTA per SM
        sub = 2 if one or bn <= 80 else 1                          # K blocks per stage
        steps, stage = -(-per // sub), sub * (16384 + 128 * bn)
        cap = (large if one else small)[S - 1]
        if units > cap and (S > 1 or bn < T or T > 128) or not one and bn > 80 and S > 1:
            continue                      # the latter: stages of one K block and the exchange, 256 x 4096 x 4096 16.1 -> 20.6 us
        waves, shared = -(-units // cap), 2 if not one and units > sms else 1
        flight = min(steps, (230400 if one else 114176) // stage, 6)
        body = max(waves * steps * max(0.226, shared * stage / load, 0.81 / flight), stream)
        adds = -(-(-(-bn // S) * (8 if gate else 16)) // 192)
        cost = 3.4 + body + 0.0098 * bn + (0.0167 * bn if S > 1 else 0.0) + waves * adds * 0.285 + (0.51 if shared > 1 else 0.0) + \
            (0.1 if bn < T else 0.0)
        if best is None or cost < best[0]:
            best = (cost, bn, S)
    return best


@lru_cache(maxsize=4096)
def _dense_plan(T: int, F: int, K: int, epi: int, sms: int, hd: int = 0, device: Optional[torch.device] = None):
    """(weight rows per tile of gemm_wide.cu or 0, split plan or None) of a dense launch on one GPU that leaves the choice of kernel to
    this module; ``hd``: see :func:`dense_wide`; ``device``: whose :func:`split_ctas` count, and part of the key under which every launch finds
    its plan (the tables themselves took 0.5 us to hash: 2 % of prompt steps that the host bounds).

    Up to 128 tokens the split kernel where it has a plan: the pair kernel would work half its rows for nothing, and its model leaves out
    that all of the weights come from HBM. Beyond, the cheaper of both models. Sweep of 267 sizes with a plan on B200 (T 2 .. 4096, F 256 ..
    14336, K 256 .. 14336): the choice is 0.5 % slower than the best tile of either kernel on average, 17 % at most. Split -> pairs, us:
    512 x 4096 x 14336 61 -> 52, 1000 x 2048 x 14336 58 -> 49, 512 x 4096 x 11008 49 -> 40, 200 x 12288 x 4096 35 -> 27, SwiGLU 230 x
    4344 x 5768 50 -> 40; the other way 200 x 2048 x 14336 21 and 44, 300 x 2048 x 14336 29 and 44.

    Rows that start inside a sector of 32 bytes (K not a multiple of 16) load more slowly, in the split kernel above all (see the models);
    beyond 64 tokens the pairs can then be the faster ones: SwiGLU 128 x 8024 x 1752 21 -> 19.5, 120 x 11840 x 1304 27 -> 22."""
    plan = split_plan(T, F, K, epi, sms, None if device is None else split_ctas(device))
    if plan is not None and T <= (64 if K % 16 else 128):
        return 0, plan
    if plan is None and not want_wide(epi, T, F, K, 1, sms):
        return 0, None
    cost, cols = dense_wide(T, F, K, epi, sms, hd)
    return (0, plan) if plan is not None and plan[0] < cost else (cols, None)


def _wide_rows(F: int, out: Optional[torch.Tensor], residual: Optional[torch.Tensor], comm: "Optional[GemmComm]") -> bool:
    """Launches of gemm_wide.cu: on one GPU, rows that move 16 bytes at a time (others keep their split of K)."""
    rows16 = lambda t: t is None or (t.stride(0) * t.element_size() % 16 == 0 and t.data_ptr() % 16 == 0)
    alone = comm is None or (comm.seg_cnt is None and not (comm.S or comm.n_wait or comm.n_signal or comm.shard_rows or comm.group_regions)
                             and comm.rs_bases is None and comm.fanout <= 1 and comm.clear is None)
    return alone and F % 8 == 0 and rows16(out) and rows16(residual)


def _group_hint(T: int, G: int) -> int:
    """Token-tile hint for a grouped GEMM whose group sizes are only known on the device: the mean group size plus
    head-room for routing imbalance, so that most groups fit one token tile (a second tile re-reads the weights)."""
    mean = (T + G - 1) // G
    return mean + mean // 2 + 8 if G > 1 else mean


class GemmComm:
    """Multi-GPU hooks of a grouped GEMM launch (see ``DmoeGemm`` in csrc/kernels/dmoe_kernels.h).

    seg_cnt [S, G] int32 (device): rows source s delivered for group g; region s = rows [s*seg_cap, (s+1)*seg_cap).
    wait_flags [n_wait] int32 + wait_epoch [1]: arrival gate. signal_ptrs int64 [n_signal] (peer flag arrays) +
    signal_slot + signal_epoch [1]: completion signal. done_ticket [1]: zero-initialised scratch int.
    """

    def __init__(self, seg_cnt=None, S=0, seg_cap=0, wait_flags=None, n_wait=0, wait_epoch=None, signal_ptrs=None,
                 n_signal=0, signal_slot=0, signal_epoch=None, done_ticket=None, fanout=0, group_regions=False,
                 clear=None, shard_rows=0, rs_bases=None, rs_rows=0, rs_slot=0, rs_cap=0, rope: "Optional[RopeAppend]" = None):
        self.seg_cnt, self.S, self.seg_cap = seg_cnt, S, seg_cap
        self.wait_flags, self.n_wait, self.wait_epoch = wait_flags, n_wait, wait_epoch
        self.signal_ptrs, self.n_signal, self.signal_slot = signal_ptrs, n_signal, signal_slot
        self.signal_epoch, self.done_ticket = signal_epoch, done_ticket
        self.fanout, self.group_regions, self.clear = fanout, group_regions, clear
        # tensor-parallel attention: all-gather prologue (X arrives in shards of shard_rows rows, one wait flag per
        # shard), reduce-scatter epilogue (row t -> rank t // rs_rows, slot rs_slot of its partial buffer)
        self.shard_rows = shard_rows
        self.rs_bases, self.rs_rows, self.rs_slot, self.rs_cap = rs_bases, rs_rows, rs_slot, rs_cap
        self.rope = rope

    def fill(self, d):
        d.seg_cnt, d.S, d.seg_cap = _lib.ptr(self.seg_cnt), self.S, self.seg_cap
        d.wait_flags, d.n_wait, d.wait_epoch = _lib.ptr(self.wait_flags), self.n_wait, _lib.ptr(self.wait_epoch)
        d.signal_ptrs, d.n_signal, d.signal_slot = _lib.ptr(self.signal_ptrs), self.n_signal, self.signal_slot
        d.signal_epoch, d.done_ticket = _lib.ptr(self.signal_epoch), _lib.ptr(self.done_ticket)
        d.fanout = self.fanout
        d.group_regions = int(self.group_regions)
        d.clear_ptr, d.clear_n = _lib.ptr(self.clear), (0 if self.clear is None else self.clear.numel())
        d.shard_rows = self.shard_rows
        d.rs_bases, d.rs_rows, d.rs_slot, d.rs_cap = _lib.ptr(self.rs_bases), self.rs_rows, self.rs_slot, self.rs_cap
        if self.rope is not None:
            r = self.rope
            d.rope_table, d.positions, d.slots = r.table.data_ptr(), r.positions.data_ptr(), _lib.ptr(r.slots)
            d.kcache, d.vcache = r.kcache.data_ptr(), r.vcache.data_ptr()
            d.n_q, d.n_kv, d.hd, d.rope_max_pos = r.n_q, r.n_kv, r.hd, r.table.shape[0]


class RopeAppend:
    """QKV epilogue: neox RoPE on the q / k heads and K / V append to the paged cache (see ``DmoeGemm``).

    table: fp32 [max_pos, hd / 2, 2] from :func:`rope_table`; positions int32 [T]; slots int64 [T] or None;
    kcache / vcache [blocks, block_size, n_kv, hd] bf16."""

    def __init__(self, table, positions, slots, kcache, vcache, n_q, n_kv, hd):
        assert table.dtype == torch.float32 and table.is_contiguous() and table.shape[1] == hd // 2
        assert positions.dtype == torch.int32 and (slots is None or slots.dtype == torch.int64)
        assert kcache.is_contiguous() and vcache.is_contiguous() and kcache.dtype == torch.bfloat16
        self.table, self.positions, self.slots, self.kcache, self.vcache = table, positions, slots, kcache, vcache
        self.n_q, self.n_kv, self.hd = n_q, n_kv, hd


_rope_tables = {}


def rope_table(max_pos: int, hd: int, theta: float, device) -> torch.Tensor:
    """fp32 [max_pos, hd / 2, 2] = (cos, sin)(pos * theta^(-2 d / hd)), computed on the device with the arithmetic
    of the stand-alone RoPE kernel; cached per (device, max_pos, hd, theta)."""
    device = torch.device(device)
    key = (device.index or 0, max_pos, hd, float(theta))
    t = _rope_tables.get(key)
    if t is None:
        t = torch.empty(max_pos, hd // 2, 2, dtype=torch.float32, device=device)
        with torch.cuda.device(device):
            _lib.check(_lib.lib().dmoe_rope_table(ctypes.c_void_p(t.data_ptr()), ctypes.c_int(max_pos), ctypes.c_int(hd),
                                                  ctypes.c_float(theta), ctypes.c_void_p(_lib.stream_ptr())),
                       "dmoe_rope_table")
        _rope_tables[key] = t
    return t


def _launch(W, X, Y, R, offs, recs, bases, G, T, F, K, epi, bn, splitk, ldy, y_f32, comm: Optional[GemmComm] = None,
            streamk: bool = False, pair: bool = False, w_blocked: bool = False, act: int = 0, act_limit: float = 0.0,
            act_cols: int = 0, unit_weights: bool = False, wide: int = 0, cluster: int = 0):
    s = scratch(X.device)
    d = _lib.DmoeGemm()           # zeros: only what a launch has is filled in
    if cluster:
        d.cluster = cluster
    if wide:
        d.wide = int(wide)        # True, or the weight rows per tile
    if act:
        d.act, d.act_limit, d.act_cols = act, act_limit, act_cols
    if unit_weights:
        d.unit_weights = 1
    if w_blocked:
        d.w_blocked = 1
    if TRACE is not None:
        d.trace = TRACE.data_ptr()
    if streamk and splitk <= 1 and not pair:
        d.streamk = 1
    d.n_counters = s.counters.numel()
    if pair:
        d.pair = 1
    if comm is not None:
        comm.fill(d)
    d.W, d.X = W.data_ptr(), X.data_ptr()
    if Y is not None:
        d.Y = Y.data_ptr()
    if R is not None:
        d.R, d.ldr = R.data_ptr(), R.stride(0)
    if offs is not None:
        d.offs = offs.data_ptr()
    if recs is not None:
        d.recs = recs.data_ptr()
    if bases is not None:
        d.bases = bases.data_ptr()
        d.combine_vec = int(epi == EPI_COMBINE and F % 8 == 0 and ldy % 8 == 0 and _bases_aligned(bases))
    if splitk > 1:
        need = _lib.lib().dmoe_gemm_workspace_bytes(T, F, bn, splitk)
        s.ensure(need)
    d.ws, d.counters, d.status, d.ws_bytes = s.ws.data_ptr(), s.counters.data_ptr(), s.status.data_ptr(), s.ws.numel()
    d.ldx, d.ldy = X.stride(0), ldy
    d.G, d.T, d.F, d.K = G, T, F, K
    d.epi, d.bn, d.splitk = epi, bn, splitk
    if y_f32:
        d.y_f32 = 1
    _lib.check(_lib.lib().dmoe_gemm(ctypes.byref(d), _lib.stream_ptr()), "dmoe_gemm")


def _tma_ok(x, w) -> bool:
    """Can the tcgen05 kernel's TMA address these operands (16-byte rows and base addresses)?"""
    return x.shape[1] % 8 == 0 and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0


def _simt_linear(x, w, out, out_dtype, tanh=False, silu_cols=0):
    """fp32 operands (true fp32 arithmetic), or bf16 operands that TMA cannot address: the CUDA-core GEMM."""
    T, K = x.shape
    F = w.shape[0]
    assert w.is_contiguous() and w.dtype == x.dtype and w.shape[1] == K and x.stride(1) == 1
    f32 = x.dtype == torch.float32
    if out is None:
        out = torch.empty(T, F, dtype=out_dtype or x.dtype, device=x.device)
    assert out.stride(1) == 1 and (out.dtype == torch.float32 or not f32)
    v, ll, i = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
    _lib.check(_lib.lib().dmoe_simt_linear(
        i(int(f32)), i(int(out.dtype == torch.float32)), v(x.data_ptr()), ll(x.stride(0)), v(w.data_ptr()), ll(K),
        v(out.data_ptr()), ll(out.stride(0)), i(T), i(F), i(K), i(ACT_TANH if tanh else ACT_SILU if silu_cols else 0), i(silu_cols),
        v(_lib.stream_ptr())), "dmoe_simt_linear")
    return out


def _simt_grouped(x, w, offs, out, recs=None, base=None, ld_out=0, unit_weights=False):
    """The CUDA-core GEMM over row groups: rows offs[g] .. offs[g + 1] of x times w[g].T, into ``out`` or, with ``recs``
    (combine), scaled and scattered to rows of the buffer at ``base[0]`` in x's dtype."""
    T, K = x.shape
    G, F, _ = w.shape
    assert w.is_contiguous() and w.dtype == x.dtype and w.shape[2] == K and x.stride(1) == 1
    assert offs.dtype == torch.int32 and (out is None or out.dtype in (x.dtype, torch.float32))
    v, ll, i = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
    _lib.check(_lib.lib().dmoe_simt_grouped(
        i(int(x.dtype == torch.float32)), i(int((x if out is None else out).dtype == torch.float32)), v(x.data_ptr()), ll(x.stride(0)),
        v(w.data_ptr()), v(offs.data_ptr()), i(G), v(_lib.ptr(out)), ll(out.stride(0) if out is not None else ld_out),
        v(_lib.ptr(recs)), v(_lib.ptr(base)), i(int(unit_weights)), i(T), i(F), i(K), v(_lib.stream_ptr())), "dmoe_simt_grouped")
    return out


def _gate_mul(gu, out, I: int, act: str, limit: float = 0.0, recs=None):
    """out = act(gu[:, :I]) * gu[:, I:], gu scaled by the weights of ``recs`` first where these are given."""
    v, ll, i = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
    _lib.check(_lib.lib().dmoe_gate_mul(i(int(gu.dtype == torch.float32)), i(ACTS[act]), v(gu.data_ptr()), ll(gu.stride(0)),
                                        v(out.data_ptr()), ll(out.stride(0)), i(gu.shape[0]), i(I), ctypes.c_float(limit), v(_lib.ptr(recs)),
                                        v(_lib.stream_ptr())), "dmoe_gate_mul")
    return out


def _check_x(x):
    assert x.dim() == 2 and x.stride(1) == 1 and x.dtype == torch.bfloat16, "x must be [T, K] bf16, K contiguous"
    assert x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0, "x rows must be 16-byte aligned"


def linear(x: torch.Tensor, w: torch.Tensor, residual: Optional[torch.Tensor] = None,
           out: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None, bn: int = 0,
           splitk: int = 0, comm: Optional["GemmComm"] = None, pair: bool = False, tanh: bool = False,
           silu_cols: int = 0, wide: Optional[bool] = None, cluster: Optional[int] = None) -> torch.Tensor:
    """y[T, F] = x[T, K] @ w[F, K].T (+ residual[T, F]); ``tanh``: of the product; ``silu_cols``: silu of the first so
    many columns. ``pair``: CTA pairs (tcgen05 cta_group::2) on tiles of 256 weight rows x ``bn`` (128 / 256) tokens, whole tiles.
    ``cluster``: tiles of 128 weight rows x ``bn`` tokens (any multiple of 16 up to 256, up to 240 from 5 CTAs on, where partial rows sent
    and received share the memory; 0: those of the batch, 128 at most), K cut over so many CTAs (csrc/kernels/gemm_split.cu)."""
    T, K = x.shape
    F = w.shape[0]
    if not x.is_cuda:
        y = torch.nn.functional.linear(x.float(), w.float())
        if tanh:
            y = torch.tanh(y)
        if silu_cols:
            y[:, :silu_cols] = torch.nn.functional.silu(y[:, :silu_cols])
        if residual is not None:
            y = y + residual.float()
        y = y.to(out_dtype or x.dtype)
        if out is not None:
            out.copy_(y)
            return out
        return y
    if x.dtype == torch.float32 or (comm is None and residual is None and not _tma_ok(x, w)):
        assert comm is None and residual is None
        return _simt_linear(x, w, out, out_dtype, tanh, silu_cols)
    _check_x(x)
    assert w.is_contiguous() and w.dtype == torch.bfloat16 and w.shape[1] == K
    odt = out_dtype or torch.bfloat16
    scatter = comm is not None and comm.rs_bases is not None      # reduce-scatter epilogue: rows go to the peers
    if out is None and not scatter:
        out = torch.empty(T, F, dtype=odt, device=x.device)
    assert scatter or (out.stride(1) == 1 and out.dtype in (torch.bfloat16, torch.float32))
    if T == 0:
        return out
    # splitk = 0 (default): with at least one full wave of tiles, whole tiles per CTA plus a stream-K tail (the tiles of
    # the last, partial wave are cut along K into equal shares for all SMs); with fewer tiles than SMs (decode sizes)
    # plain split-K with a factor that fills the SMs. An explicit splitk >= 1 selects split-K with that factor.
    sms = num_sms(x.device)
    auto_sk = 0
    if wide is None and not cluster:
        wide = False
        if not (bn or splitk or pair) and _wide_rows(F, out, residual, comm):
            wide, plan = _dense_plan(T, F, K, EPI_PLAIN, sms, comm.rope.hd if comm is not None and comm.rope is not None else 0, x.device)
            if plan is not None:
                _, bn, cluster = plan
    if cluster:
        bn = bn or _split_tile(T)
        _launch(w, x, out, residual, None, None, None, 1, T, F, K, EPI_PLAIN, bn, 1, out.stride(0), out.dtype == torch.float32, comm,
                act=ACT_TANH if tanh else ACT_SILU if silu_cols else 0, act_cols=silu_cols, cluster=cluster)
        return out
    if not bn:
        bn = pick_bn(T, EPI_PLAIN)
        if ((F + 127) // 128) * ((T + bn - 1) // bn) < sms and not pair:
            bn, auto_sk = pick_dense(T, F, K, sms)
    if pair:
        bn = 256 if bn not in (128, 256) else bn
        splitk = 1
    if wide:
        splitk = 1
    streamk = splitk == 0 and STREAM_K and ((F + 127) // 128) * ((T + bn - 1) // bn) >= sms
    if streamk:
        splitk = 1
    else:
        splitk = splitk or auto_sk or pick_splitk(T, F, K, bn, sms)
    _launch(w, x, out, residual, None, None, None, 1, T, F, K, EPI_PLAIN, bn, splitk,
            F if scatter else out.stride(0), (not scatter) and out.dtype == torch.float32, comm, streamk=streamk,
            pair=pair, act=ACT_TANH if tanh else ACT_SILU if silu_cols else 0, act_cols=silu_cols, wide=wide)
    return out


def _grouped_ref(x, w, offs, swiglu, act="silu", limit=0.0, recs=None):
    offs = offs.tolist()
    G = w.shape[0]
    F = w.shape[1] // 2 if swiglu else w.shape[1]
    y = torch.zeros(x.shape[0], F, dtype=torch.float32, device=x.device)
    for g in range(G):
        a, b = offs[g], offs[g + 1]
        if b <= a:
            continue
        h = x[a:b].float() @ w[g].float().T
        if recs is not None:
            h = h * recs[a:b, 2].contiguous().view(torch.float32)[:, None]
        if swiglu:
            h = reference.swiglu(h, act, limit)
        y[a:b] = h
    return y


def grouped_swiglu(x: torch.Tensor, w13: torch.Tensor, offs: Optional[torch.Tensor], out: Optional[torch.Tensor] = None,
                   bn: int = 0, comm: Optional[GemmComm] = None, streamk: Optional[bool] = None,
                   pair: bool = False, w_blocked: bool = False, act: str = "silu", limit: float = 0.0,
                   recs: Optional[torch.Tensor] = None, wide: Optional[bool] = None) -> torch.Tensor:
    """y[T, I] = act(x @ w13[g, :I].T) * (x @ w13[g, I:].T) for the rows of group g; w13 is [G, 2I, K]. ``recs``: row t of x counts
    with the weight of its record (see :func:`grouped_combine`)."""
    T, K = x.shape
    G, F2, _ = w13.shape
    I = F2 // 2
    if not x.is_cuda:
        y = _grouped_ref(x, w13, offs, True, act, limit, recs).to(x.dtype)
        if out is not None:
            out.copy_(y)
            return out
        return y
    if x.dtype == torch.float32 or (comm is None and not w_blocked and not _tma_ok(x, w13)):
        gu = _simt_grouped(x, w13, offs, torch.empty(T, F2, dtype=x.dtype, device=x.device))
        return _gate_mul(gu, torch.empty(T, I, dtype=x.dtype, device=x.device) if out is None else out, I, act, limit, recs)
    _check_x(x)
    assert w13.is_contiguous() and w13.dtype == torch.bfloat16
    assert recs is None or (recs.dtype == torch.int32 and recs.is_contiguous() and recs.shape[1] == 4)
    assert comm is not None or (offs.dtype == torch.int32 and offs.is_cuda)
    if out is None:
        out = torch.empty(T, I, dtype=torch.bfloat16, device=x.device)
    if T == 0:
        return out
    if wide is None:
        wide = not (bn or pair or streamk or comm is not None) and want_wide(EPI_SWIGLU, T, I, K, G, num_sms(x.device))
    bn = bn or (pick_bn(_group_hint(T, G), EPI_COMBINE) if pair else pick_bn(_group_hint(T, G), EPI_SWIGLU))
    if pair:
        bn = max(bn, 128)
    sk = want_streamk(EPI_SWIGLU, I, G, T, bn, num_sms(x.device)) if streamk is None else streamk
    _launch(w13, x, out, None, offs, recs, None, G, T, I, K, EPI_SWIGLU, bn, 1, out.stride(0), False, comm,
            streamk=sk, pair=pair, w_blocked=w_blocked, act=ACTS[act], act_limit=limit, wide=wide)
    return out


def grouped_linear(x: torch.Tensor, w: torch.Tensor, offs: torch.Tensor, out: Optional[torch.Tensor] = None,
                   bn: int = 0, streamk: Optional[bool] = None, pair: bool = False,
                   w_blocked: bool = False, out_dtype: Optional[torch.dtype] = None, wide: Optional[bool] = None) -> torch.Tensor:
    """y[T, F] = x @ w[g].T for the rows of group g; w is [G, F, K]. ``out_dtype``: that of x, or fp32."""
    T, K = x.shape
    G, F, _ = w.shape
    dt = out.dtype if out is not None else out_dtype or x.dtype
    if not x.is_cuda:
        y = _grouped_ref(x, w, offs, False).to(dt)
        if out is not None:
            out.copy_(y)
            return out
        return y
    if x.dtype == torch.float32 or (not w_blocked and not _tma_ok(x, w)):
        return _simt_grouped(x, w, offs, torch.empty(T, F, dtype=dt, device=x.device) if out is None else out)
    _check_x(x)
    assert w.is_contiguous() and w.dtype == torch.bfloat16 and offs.dtype == torch.int32 and offs.is_cuda
    if out is None:
        out = torch.empty(T, F, dtype=dt, device=x.device)
    if T == 0:
        return out
    if wide is None:
        wide = not (bn or pair or streamk) and want_wide(EPI_PLAIN, T, F, K, G, num_sms(x.device))
    bn = bn or pick_bn(_group_hint(T, G), EPI_PLAIN)
    if pair:
        bn = max(bn, 128)
    sk = want_streamk(EPI_PLAIN, F, G, T, bn, num_sms(x.device)) if streamk is None else streamk
    _launch(w, x, out, None, offs, None, None, G, T, F, K, EPI_PLAIN, bn, 1, out.stride(0), out.dtype == torch.float32,
            streamk=sk, pair=pair, w_blocked=w_blocked, wide=wide)
    return out


def block_weight(w: torch.Tensor) -> torch.Tensor:
    """Re-orders a K-contiguous weight stack [G, R, K] (or [R, K]) tile by tile: [G, R / 128, K / 64, 128, 64], returned
    with the ORIGINAL shape (only the memory order changes), for launches with ``w_blocked=True``. Every 128-row x
    64-column box the GEMM fetches is then 16 KB of consecutive addresses instead of 128 runs of 128 bytes one weight
    row apart. R must be a multiple of 128 (for SwiGLU stacks: the gate and the up half each) and K of 64."""
    shape = w.shape
    w3 = w if w.dim() == 3 else w.unsqueeze(0)
    G, R, K = w3.shape
    assert R % 128 == 0 and K % 64 == 0, "blocked weights need whole 128 x 64 tiles"
    return w3.view(G, R // 128, 128, K // 64, 64).permute(0, 1, 3, 2, 4).contiguous().view(shape)


def unblock_weight(w: torch.Tensor) -> torch.Tensor:
    """Inverse of :func:`block_weight`: a row-major copy of a tile-blocked stack."""
    shape = w.shape
    w3 = w if w.dim() == 3 else w.unsqueeze(0)
    G, R, K = w3.shape
    return w3.view(G, R // 128, K // 64, 128, 64).permute(0, 1, 3, 2, 4).contiguous().view(shape)


_bases_checked = {}


def _bases_aligned(bases: torch.Tensor) -> bool:
    """Are all destination pointers of a combine table 16-byte aligned? Read back once per table (tables are built at
    start-up and never change); a table first seen during a graph capture, where nothing can be read back, counts as
    unaligned and keeps the 2-byte stores."""
    key = (bases.data_ptr(), bases.numel())
    if key not in _bases_checked:
        if torch.cuda.is_current_stream_capturing():
            return False
        _bases_checked[key] = bool((bases % 16 == 0).all().item())
    return _bases_checked[key]


def grouped_combine(x: torch.Tensor, w: torch.Tensor, offs: Optional[torch.Tensor], recs: torch.Tensor,
                    bases: torch.Tensor, ld_out: int, bn: int = 0, outs=None, comm: Optional[GemmComm] = None,
                    streamk: Optional[bool] = None, pair: bool = False, w_blocked: bool = False,
                    unit_weights: bool = False, wide: Optional[bool] = None) -> None:
    """GEMM-2 with the combine epilogue: row t of group g becomes ``weight[t] * (x[t] @ w[g].T)`` written to row
    ``recs[t, 1]`` of the buffer ``bases[recs[t, 0]]`` (row stride ``ld_out`` elements).

    recs: int32 [T, 4] = (dst_rank, dst_row or -1, weight as fp32 bits, 0). bases: int64 [n_ranks] device
    tensor of raw pointers (peer buffers included). ``outs`` (CPU path only) is the list of destination tensors.
    ``unit_weights``: the records' weights are left out.
    """
    T, K = x.shape
    G, F, _ = w.shape
    if not x.is_cuda:
        y = _grouped_ref(x, w, offs, False)
        if not unit_weights:
            y = y * recs[:, 2].contiguous().view(torch.float32)[:, None]
        for r, o in enumerate(outs):
            mine = (recs[:, 0] == r) & (recs[:, 1] >= 0)
            o[recs[mine, 1].long()] = y[mine].to(o.dtype)
        return
    if x.dtype == torch.float32 or (comm is None and not w_blocked and not _tma_ok(x, w)):
        _simt_grouped(x, w, offs, None, recs, bases, ld_out, unit_weights)
        return
    _check_x(x)
    assert recs.dtype == torch.int32 and recs.is_contiguous() and recs.shape[1] == 4 and bases.dtype == torch.int64
    if T == 0:
        return
    if wide is None:
        wide = not (bn or pair or streamk or comm is not None) and want_wide(EPI_COMBINE, T, F, K, G, num_sms(x.device))
    bn = bn or pick_bn(_group_hint(T, G), EPI_COMBINE)
    if pair:
        bn = max(bn, 128)
    sk = want_streamk(EPI_COMBINE, F, G, T, bn, num_sms(x.device)) if streamk is None else streamk
    _launch(w, x, None, None, offs, recs, bases, G, T, F, K, EPI_COMBINE, bn, 1, ld_out, False, comm, streamk=sk,
            pair=pair, w_blocked=w_blocked, unit_weights=unit_weights, wide=wide)


def swiglu_linear(x: torch.Tensor, w13: torch.Tensor, out: Optional[torch.Tensor] = None, bn: int = 0,
                  act: str = "silu", wide: Optional[bool] = None, cluster: Optional[int] = None) -> torch.Tensor:
    """Dense gated up-projection: act(x @ w13[:I].T) * (x @ w13[I:].T); w13 is [2I, K] (a one-group grouped_swiglu)."""
    T, K = x.shape
    I = w13.shape[0] // 2
    if not x.is_cuda:
        y = reference.swiglu(x.float() @ w13.float().T, act).to(x.dtype)
        if out is not None:
            out.copy_(y)
            return out
        return y
    if x.dtype == torch.float32 or not _tma_ok(x, w13):
        gu = _simt_linear(x, w13, None, None)
        return _gate_mul(gu, torch.empty(T, I, dtype=x.dtype, device=x.device) if out is None else out, I, act)
    _check_x(x)
    assert w13.is_contiguous() and w13.dtype == torch.bfloat16
    if out is None:
        out = torch.empty(T, I, dtype=torch.bfloat16, device=x.device)
    if T == 0:
        return out
    if wide is None and not cluster:
        wide = False
        if not bn:
            wide, plan = _dense_plan(T, I, K, EPI_SWIGLU, num_sms(x.device), 0, x.device)
            if plan is not None and _wide_rows(I, out, None, None):
                _, bn, cluster = plan
    if cluster:
        bn = bn or _split_tile(T)
        _launch(w13, x, out, None, None, None, None, 1, T, I, K, EPI_SWIGLU, bn, 1, out.stride(0), False, act=ACTS[act], cluster=cluster)
        return out
    bn = bn or pick_bn(T, EPI_SWIGLU)
    _launch(w13, x, out, None, None, None, None, 1, T, I, K, EPI_SWIGLU, bn, 1, out.stride(0), False,
            act=ACTS[act], wide=wide)
    return out
