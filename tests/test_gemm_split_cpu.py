"""The rule that chooses tiles and clusters of csrc/kernels/gemm_split.cu keeps the limits of that kernel."""
import random

import pytest

from disagmoe_b200.ops import gemm


def _fits(bn, S, per):
    """Restates the kernel's shared memory: stages of one or two K blocks, a CTA's partial rows over them, those it receives beside or
    over, in the amount that lets two CTAs share an SM or in the one that does not."""
    parts, recv = bn * 512, (S - 1) * -(-bn // S) * 512
    for room, sub in ((112 * 1024 + 512 - 1024, 2), (112 * 1024 + 512 - 1024, 1), (226 * 1024 - 1024, 2)):
        stage, steps = sub * (16384 + bn * 128), -(-per // sub)
        want, beside, over = min(steps, 3 if sub == 1 else 2), min(steps, 6, max(0, room - recv) // stage), min(steps, 6, room // stage)
        if (beside >= want and beside * stage >= parts) or (over >= want and parts + recv <= room):
            return True
    return False


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
        assert S * tiles <= 296 or (S == 1 and T <= 128 and bn >= T)      # one wave, or one tile of tokens that weights stream through
    assert found > 300


def test_refused_where_a_second_wave_would_start():
    assert gemm.split_plan(4096, 4096, 4096, gemm.EPI_PLAIN, 148) is None
    assert gemm.split_plan(192, 32000, 2048, gemm.EPI_PLAIN, 148) is None
    assert gemm.split_plan(200, 10944, 2048, gemm.EPI_SWIGLU, 148) is None
    assert gemm.split_plan(1, 151936, 2048, gemm.EPI_PLAIN, 148)[1:] == (16, 1)


def test_plans_follow_what_the_device_holds():
    """On a chip whose groups of SMs hold fewer clusters of 4 and 5 no plan asks for more of them than find place at once."""
    small, large = (list(t) for t in (gemm._SPLIT_SMALL, gemm._SPLIT_LARGE))
    for n in (3, 4):
        small[n], large[n] = small[n] // 2, large[n] // 2
    changed = 0
    for T, F, K in ((37, 2048, 5632), (96, 2048, 4096), (128, 1024, 8192), (48, 6144, 4096), (200, 2048, 14336), (16, 4096, 4096)):
        _, bn, S = gemm.split_plan(T, F, K, gemm.EPI_PLAIN, 148, (tuple(small), tuple(large)))
        per = -(-(-(-K // 64)) // S)
        cap = large if bn > 128 or (per > 4 and S * -(-F // 128) * -(-T // bn) <= large[S - 1]) else small
        assert S * -(-F // 128) * -(-T // bn) <= cap[S - 1]
        changed += (bn, S) != gemm.split_plan(T, F, K, gemm.EPI_PLAIN, 148)[1:]
    assert changed > 0


def test_more_weight_rows_than_the_grid_has_tiles_stay_with_the_other_kernel():
    assert gemm.split_plan(1, 65535 * 128, 8, gemm.EPI_PLAIN, 148) is not None and gemm.split_plan(1, 65535 * 128 + 8, 8, gemm.EPI_PLAIN, 148) is None
    assert gemm._dense_plan(1, 65535 * 128 + 8, 8, gemm.EPI_PLAIN, 148) == (0, None)
    assert gemm.split_plan(1, 65535 * 64 + 8, 8, gemm.EPI_SWIGLU, 148) is None
