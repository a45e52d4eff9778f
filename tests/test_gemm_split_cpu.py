"""The rule that chooses tiles and clusters of csrc/kernels/gemm_split.cu keeps the limits of that kernel."""
import random

import pytest

from disagmoe_b200.ops import gemm


def _layout(bn, S, per, units):
    """Restates how the kernel lays out its shared memory, in its order of choice: one CTA per SM where all of a launch find place that way
    and a share is long; else the amount with which two share an SM, stages of two K blocks, or of one up to 128 tokens; else the large
    amount. Partial rows lie over the stages; those received beside them, or over them too. Returns (large, stages), or None: refused."""
    parts, recv = bn * 512, (S - 1) * -(-bn // S) * 512
    small, large = 112 * 1024 + 512 - 1024, 226 * 1024 - 1024

    def fits(room, sub):
        stage, steps = sub * (16384 + bn * 128), -(-per // sub)
        want, beside, over = min(steps, 3 if sub == 1 else 2), min(steps, 6, max(0, room - recv) // stage), min(steps, 6, room // stage)
        if beside >= want and beside * stage >= parts:
            return beside
        return over if over >= want and parts + recv <= room else 0
    spread = per > 4 and units <= gemm._SPLIT_LARGE[S - 1]
    if not spread:
        n = fits(small, 2) or (bn <= 128 and fits(small, 1))
        if n:
            return False, n
    n = fits(large, 2)
    return (True, n) if n else None


@pytest.mark.parametrize("epi", [gemm.EPI_PLAIN, gemm.EPI_SWIGLU])
def test_plans_fit_the_kernel(epi):
    rng = random.Random(epi)
    found, clusters = 0, set()
    for _ in range(3000):
        T, F, K = (int(2 ** rng.uniform(0, hi)) for hi in (12, 17, 14))
        F, K = max(8, F // 8 * 8), max(8, K // 8 * 8)
        plan = gemm.split_plan(T, F, K, epi, 148)
        if plan is None:
            continue
        found += 1
        _, bn, S = plan
        kblocks = -(-K // 64)
        per = -(-kblocks // S)
        units = S * -(-F // (64 if epi == gemm.EPI_SWIGLU else 128)) * -(-T // bn)
        assert 16 <= bn <= 256 and bn % 16 == 0 and 1 <= S <= min(8, kblocks) and -(-kblocks // per) == S
        layout = _layout(bn, S, per, units)
        assert layout is not None, (T, F, K, plan)
        # one wave of what the device holds, or one tile of tokens that weights stream through
        assert units <= (gemm._SPLIT_LARGE if layout[0] else gemm._SPLIT_SMALL)[S - 1] or (S == 1 and T <= 128 and bn >= T), (T, F, K, plan)
        clusters.add(S)
    assert found > 600 and clusters == set(range(1, 9))


def test_limits_of_explicit_tiles():
    """Every tile of up to 240 tokens in every cluster, 256 up to 4 CTAs, whatever the length of a share."""
    for S in range(1, 9):
        for bn in range(16, 257, 16):
            refused = [per for per in range(1, 300) if any(_layout(bn, S, per, u) is None for u in (1, 1000))]
            assert not refused or (bn == 256 and S >= 5)


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


def test_a_launch_finds_its_plan_without_the_tables(monkeypatch):
    """The tables of a device are asked for once per plan, and each device has plans of its own."""
    import torch
    asked = []
    monkeypatch.setattr(gemm, "split_ctas", lambda device: asked.append(device.index) or gemm._scaled_ctas(148 if device.index == 0 else 74))
    gemm._dense_plan.cache_clear()
    try:
        a, b = ([gemm._dense_plan(64, 4096, 4096, gemm.EPI_PLAIN, 148, 0, torch.device("cuda", i)) for _ in range(3)] for i in (0, 1))
    finally:
        gemm._dense_plan.cache_clear()
    assert asked == [0, 1] and a[0] == a[2] and b[0] == b[2] and a[0] != b[0]
