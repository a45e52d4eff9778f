"""Which GEMM and which router kernel a call takes: the rules on sizes, rows and multi-GPU hooks (no GPU)."""
import pytest
import torch

from disagmoe_b200.ops import functional as F
from disagmoe_b200.ops import gemm

SMS = 148


@pytest.mark.parametrize("epi,T,F,K,G,wide", [
    (gemm.EPI_PLAIN, 4096, 6144, 4096, 1, True), (gemm.EPI_PLAIN, 1, 32000, 4096, 1, False), (gemm.EPI_PLAIN, 63, 32000, 4096, 1, False),
    (gemm.EPI_PLAIN, 256, 32000, 4096, 1, True), (gemm.EPI_PLAIN, 300, 256, 5632, 1, False), (gemm.EPI_PLAIN, 2048, 2048, 2048, 1, True),
    (gemm.EPI_SWIGLU, 256, 5632, 2048, 1, True), (gemm.EPI_SWIGLU, 64, 14336, 4096, 1, False), (gemm.EPI_SWIGLU, 100, 1408, 2048, 64, False),
    (gemm.EPI_SWIGLU, 144 * 8, 14336, 4096, 8, True), (gemm.EPI_COMBINE, 2, 4096, 14336, 8, False), (gemm.EPI_COMBINE, 148, 2048, 1408, 60, True),
    (gemm.EPI_SWIGLU, 1, 2048, 256, 1, False), (gemm.EPI_SWIGLU, 16, 8192, 1024, 1, False), (gemm.EPI_SWIGLU, 1, 8192, 7168, 1, False),
    (gemm.EPI_SWIGLU, 16, 8192, 7168, 1, True), (gemm.EPI_SWIGLU, 1, 2048, 4096, 1, True), (gemm.EPI_SWIGLU, 37, 5632, 2048, 1, True),
    (gemm.EPI_COMBINE, 24, 6144, 2048, 16, False), (gemm.EPI_COMBINE, 24, 4096, 1408, 16, False), (gemm.EPI_COMBINE, 24, 4096, 1408, 60, True),
    (gemm.EPI_COMBINE, 74, 4096, 1024, 8, True), (gemm.EPI_PLAIN, 96, 2048, 2816, 64, False),
])
def test_measured_choices(epi, T, F, K, G, wide):
    assert gemm.want_wide(epi, T, F, K, G, SMS) is wide


@pytest.mark.parametrize("epi,per,F,K,G,wide", [
    (gemm.EPI_SWIGLU, 104, 1408, 2048, 64, True), (gemm.EPI_SWIGLU, 39, 1408, 2048, 64, False), (gemm.EPI_SWIGLU, 127, 14336, 4096, 8, False),
    (gemm.EPI_SWIGLU, 128, 14336, 4096, 8, True), (gemm.EPI_SWIGLU, 64, 6144, 2048, 16, False), (gemm.EPI_COMBINE, 87, 4096, 14336, 8, False),
    (gemm.EPI_COMBINE, 88, 4096, 14336, 8, True), (gemm.EPI_PLAIN, 40, 6144, 2048, 16, True), (gemm.EPI_COMBINE, 39, 6144, 2048, 16, False),
])
def test_measured_choices_per_expert(epi, per, F, K, G, wide):
    assert gemm.want_wide(epi, per * G, F, K, G, SMS) is wide


@pytest.mark.parametrize("epi,T,F,K,pairs", [
    (gemm.EPI_PLAIN, 512, 4096, 14336, True), (gemm.EPI_PLAIN, 1000, 2048, 14336, True), (gemm.EPI_PLAIN, 512, 4096, 11008, True),
    (gemm.EPI_PLAIN, 200, 12288, 4096, True), (gemm.EPI_SWIGLU, 230, 4344, 5768, True), (gemm.EPI_PLAIN, 660, 3064, 11816, True),
    (gemm.EPI_PLAIN, 200, 2048, 14336, False), (gemm.EPI_PLAIN, 300, 2048, 14336, False), (gemm.EPI_PLAIN, 128, 4096, 14336, False),
    (gemm.EPI_PLAIN, 256, 4096, 4096, False), (gemm.EPI_PLAIN, 4096, 6144, 4096, True), (gemm.EPI_PLAIN, 96, 102400, 2048, False),
])
def test_dense_products_take_the_faster_of_both_kernels(epi, T, F, K, pairs):
    """Sizes that were measured in both: a plan of the split kernel is no reason to leave the pairs' cost out."""
    cols, plan = gemm._dense_plan(T, F, K, epi, SMS)
    assert (cols > 0) is pairs and (plan is None) is pairs


@pytest.mark.parametrize("hd", [64, 128])
def test_pair_tiles_hold_whole_heads(hd):
    for T in (200, 512, 700, 1111, 4096):
        cols, plan = gemm._dense_plan(T, 48 * hd, 14336, gemm.EPI_PLAIN, SMS, hd)
        assert cols % hd == 0 and (cols > 0 or plan is not None)


@pytest.mark.parametrize("G", [1, 2, 8, 64])
def test_stream_k_of_no_expected_rows(G):
    """An expert rank whose share of the arriving rows rounds to none still asks for a rule: 32 tiles leave most SMs idle."""
    assert gemm.want_streamk(gemm.EPI_COMBINE, 4096, G, 0, 32, SMS)


@pytest.mark.parametrize("T,H,E,separate", [
    (1, 2048, 64, True), (1, 2048, 60, True), (37, 2048, 32, True), (96, 1024, 64, True), (1, 4096, 8, False), (256, 4096, 8, False),
    (448, 4096, 8, True), (448, 2048, 8, False), (640, 2048, 8, True), (148, 1024, 24, False), (512, 256, 24, False), (64, 2000, 64, False),
])
def test_measured_router_choices(T, H, E, separate):
    rows, weight = torch.empty(2, H, dtype=torch.bfloat16), torch.empty(E, H, dtype=torch.bfloat16)
    assert F.separate_router(T, H, E, rows, weight) is separate
    assert not F.separate_router(T, H, E, torch.empty(2, H + 8, dtype=torch.bfloat16)[:, 1:H + 1], weight)      # unaligned rows


def test_rows_and_hooks():
    y = torch.empty(4, 64, dtype=torch.bfloat16)
    assert gemm._wide_rows(64, y, y, None) and gemm._wide_rows(64, None, None, gemm.GemmComm())
    assert not gemm._wide_rows(60, None, None, None)                       # rows end inside 16 bytes
    assert not gemm._wide_rows(56, y[:, 1:57], None, None)                 # unaligned rows
    assert not gemm._wide_rows(64, y, torch.empty(4, 65, dtype=torch.bfloat16)[:, :64], None)
    for hooks in (dict(n_wait=1), dict(n_signal=1), dict(shard_rows=4), dict(group_regions=True), dict(fanout=2), dict(rs_bases=y),
                  dict(seg_cnt=y, S=1), dict(clear=torch.ones(4, dtype=torch.int32), done_ticket=torch.zeros(1, dtype=torch.int32))):
        assert not gemm._wide_rows(64, y, None, gemm.GemmComm(**hooks))


def test_reach_of_prompt_tiles():
    """Against the keys of every token of every tile: never less, and no more than the worst place of a window or chunk makes it."""
    tiles, _ = F.build_prefill_tiles([0] * 100 + [1] * 20, list(range(100)) + list(range(40, 60)), 32)
    for window, chunk in ((None, None), (1, None), (10, None), (200, None), (None, 24), (None, 64), (5, 24), (50, 64)):
        first = lambda p: max(p - window + 1 if window else 0, p // chunk * chunk if chunk else 0, 0)
        most = max(pos + n - first(pos) for _, n, _, pos in tiles.tolist())
        reach = F.tile_reach(100, 32, window, chunk)
        assert most <= reach <= min(100, 32 + min(window or 100, chunk or 100) - 1)
    assert F.tile_reach(90, 32) == 90 and F.tile_reach(90, 32, window=10) == 41


@pytest.mark.parametrize("epi,T,F,K,cols", [
    (gemm.EPI_PLAIN, 1386, 26112, 64, (224, 256)), (gemm.EPI_SWIGLU, 622, 19584, 384, (256,)), (gemm.EPI_PLAIN, 1601, 14336, 192, (224, 256)),
    (gemm.EPI_PLAIN, 1601, 14360, 200, (224, 256)), (gemm.EPI_PLAIN, 2500, 2048, 2048, (160,)), (gemm.EPI_PLAIN, 2500, 2048, 5632, (160,)),
])
def test_tile_widths_of_short_and_long_products(epi, T, F, K, cols):
    """Measured: many tiles of short K pay for each tile, whatever its width; long ones gain by tiles that fill their waves."""
    assert gemm.dense_wide(T, F, K, epi, SMS)[1] in cols


@pytest.mark.parametrize("epi,T,F,K,pairs,bn", [
    (gemm.EPI_PLAIN, 58, 9152, 5864, False, 64), (gemm.EPI_PLAIN, 48, 9152, 5864, False, 48),
    (gemm.EPI_SWIGLU, 128, 8024, 1752, True, 0), (gemm.EPI_SWIGLU, 120, 11840, 1304, True, 0), (gemm.EPI_SWIGLU, 64, 8024, 1752, False, 64),
    (gemm.EPI_SWIGLU, 128, 5632, 2048, False, 128), (gemm.EPI_PLAIN, 96, 5120, 88, False, 32), (gemm.EPI_PLAIN, 1, 4104, 4088, False, 16),
])
def test_rows_inside_a_sector_load_more_slowly(epi, T, F, K, pairs, bn):
    """Measured choices where K is not a multiple of 16 (one that is beside them): weights are not loaded once per cut of the tokens."""
    cols, plan = gemm._dense_plan(T, F, K, epi, SMS)
    assert (cols > 0) is pairs and (plan is None or plan[1] == bn)
