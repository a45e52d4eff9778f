"""The rule that chooses tiles and clusters of csrc/kernels/gemm_split.cu keeps the limits of that kernel."""
import random

import pytest

from disagmoe_b200.ops import gemm


def _fits(bn, S, per):
    """Restates the kernel's shared memory: stages of two K blocks, a CTA's partial rows over them, those it receives beside or over."""
    steps, stage, parts, recv = -(-per // 2), 2 * (128 * 64 * 2 + bn * 128), bn * 512, (S - 1) * -(-bn // S) * 512
    room = 226 * 1024 - 1024
    beside, over = min(steps, 6, max(0, room - recv) // stage), min(steps, 6, room // stage)
    return (beside >= min(steps, 2) and beside * stage >= parts) or (over >= min(steps, 2) and parts + recv <= room)


@pytest.mark.parametrize("epi", [gemm.EPI_PLAIN, gemm.EPI_SWIGLU])
def test_plans_fit_the_kernel(epi):
    rng = random.Random(epi)
    found = 0
    for _ in range(1500):
        T, F, K = (int(2 ** rng.uniform(0, hi)) for hi in (12, 17, 14))
        F, K = max(8, F // 8 * 8), max(8, K // 8 * 8)
        plan = gemm.split_plan(T, F, K, epi, 148)
        if plan is None:
            continue
        found += 1
        _, bn, S = plan
        kblocks = -(-K // 64)
        assert 16 <= bn <= 256 and bn % 16 == 0 and 1 <= S <= min(8, kblocks) and _fits(bn, S, -(-kblocks // S))
        tiles = -(-F // (64 if epi == gemm.EPI_SWIGLU else 128)) * -(-T // bn)
        assert S * tiles <= 296 or (S == 1 and T <= 64 and bn >= T)      # one wave, or one tile of tokens that weights stream through
    assert found > 300


def test_refused_where_a_second_wave_would_start():
    assert gemm.split_plan(4096, 4096, 4096, gemm.EPI_PLAIN, 148) is None
    assert gemm.split_plan(192, 32000, 2048, gemm.EPI_PLAIN, 148) is None
    assert gemm.split_plan(96, 10944, 2048, gemm.EPI_SWIGLU, 148) is None
    assert gemm.split_plan(1, 151936, 2048, gemm.EPI_PLAIN, 148)[1:] == (16, 1)
