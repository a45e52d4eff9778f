"""Prompt attention on tcgen05 (heads of 128) vs fp32 PyTorch: edges of query and key tiles, page sizes, garbage beyond the keys."""
import math

import pytest
import torch

from disagmoe_b200.config import QueryTemperature
from disagmoe_b200.ops import functional as F
from disagmoe_b200.ops import gemm, reference

pytestmark = pytest.mark.gpu

HD = 128
# (block-table row, first position, tokens)
SEGS = [(0, 0, 300), (1, 0, 128), (2, 137, 70), (3, 0, 8), (4, 31, 129), (5, 255, 9), (6, 127, 257)]


def _run(n_q, n_kv, bs, poison=False, seed=0, segs=SEGS, span=512, **opt):
    torch.manual_seed(seed)
    maxb, rows, pos = span // bs, [], []
    for r, p0, n in segs:
        rows += [r] * n
        pos += list(range(p0, p0 + n))
    T, nb = len(rows), 7 * maxb
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    q, kc, vc = bf(T, n_q * HD), bf(nb, bs, n_kv, HD), bf(nb, bs, n_kv, HD)
    bt = torch.randperm(nb, device="cuda").view(7, maxb).int()
    bt_row = torch.tensor(rows, dtype=torch.int32, device="cuda")
    ctx = torch.tensor(pos, dtype=torch.int32, device="cuda") + 1
    if "gate" in opt:
        opt["gate"] = bf(T, n_q)
    if "sink" in opt:
        opt["sink"] = torch.randn(n_q, device="cuda")
    ref = reference.paged_attention(q, kc, vc, bt, bt_row, ctx, n_q, n_kv, HD, opt.get("scale"), opt.get("window"), opt.get("softcap"),
                                    opt.get("sink"), opt.get("chunk"), opt.get("q_temp"), opt.get("gate"))
    if poison:
        # what a page holds behind the last cached token must not matter
        for r, p0, n in segs:
            for p in range(p0 + n, maxb * bs):
                for c in (kc, vc):
                    c[bt[r, p // bs].long(), p % bs] = float("nan")
    tiles, covered = F.build_prefill_tiles(rows, pos, F.prefill_tile_tokens(n_q, n_kv))
    assert bool(covered.all()) and F.loose_rows(covered) == 0
    out = torch.full((T, n_q * HD), 9.0, dtype=torch.bfloat16, device="cuda")
    assert F._prefill_on_tcgen05(q, kc, vc, out, HD, HD)
    F.prefill_attention(q, kc, vc, bt, tiles.cuda(), len(tiles), n_q, n_kv, HD, out, **opt)
    assert gemm.check_status() == 0
    return out.float(), ref.float()


def _close(y, ref, tol):
    bound = ref.abs() * tol + ref.pow(2).mean().sqrt() * tol
    bad = int(((y - ref).abs() > bound).sum())
    assert bad == 0, f"{bad} of {ref.numel()} off, max {(y - ref).abs().max().item():.4g}"


@pytest.mark.parametrize("n_q,n_kv", [(2, 2), (8, 2), (8, 1), (6, 2), (64, 1)])
@pytest.mark.parametrize("bs", [8, 16, 64, 128])
def test_groups_and_pages(n_q, n_kv, bs):
    # fp32 softmax weights: one rounding of the output, 2^-9 relative, and twice that for the bf16 reference it is compared in
    _close(*_run(n_q, n_kv, bs, poison=True, fp32_weights=True), tol=2 ** -7)


@pytest.mark.parametrize("opt", [
    dict(window=64), dict(window=1, sink=None), dict(window=200, softcap=20.0), dict(chunk=96), dict(chunk=128, window=40),
    dict(sink=None, gate=None), dict(q_temp=QueryTemperature(0.3, 50), scale=0.2), dict(fp32_weights=True, scale=3.0),
])
def test_options(opt):
    # fp32 softmax weights: one rounding of the output, 2^-9 relative, and twice that for the bf16 reference it is compared in
    _close(*_run(8, 2, 16, poison=True, **opt), tol=2 ** -7)


@pytest.mark.parametrize("opt", [dict(window=64), dict(sink=None, gate=None), dict(chunk=96, softcap=20.0)])
def test_short_reach(opt):
    """Prompts of few keys take the mma.sync kernel, two of whose CTAs share a tile of 128 rows."""
    segs = [(0, 0, 90), (1, 0, 8), (2, 30, 33)]
    # fp32 softmax weights: one rounding of the output, 2^-9 relative, and twice that for the bf16 reference it is compared in
    _close(*_run(8, 2, 16, segs=segs, reach=90, **opt), tol=2 ** -7)


@pytest.mark.parametrize("n_q,n_kv", [(2, 2), (8, 2), (8, 1)])
@pytest.mark.parametrize("scale", [None, 0.7])
def test_without_options(n_q, n_kv, scale):
    """Long prompts take this kernel, others (or of unknown reach) the mma.sync one: both round the weights to bf16 in the same places."""
    opt = {} if scale is None else dict(scale=scale)
    (far, ref), (near, _) = (_run(n_q, n_kv, 16, reach=r, **opt) for r in (129, 128))
    # fp32 weights would give 2^-7 as above; bf16 weights add 2^-9 of the absolute sum of the weighted values
    _close(far, ref, tol=2 ** -6)
    # sums in another order: now and then an output on the other side of a tie, one unit of the last place or 2^-7 apart
    _close(far, near, tol=2 ** -7)
    assert float((far != near).float().mean()) < 0.05


def test_many_key_blocks():
    """Two CTAs per SM, each with up to 32 key blocks: scores of a block take the place of the weights before."""
    # fp32 softmax weights: one rounding of the output, 2^-9 relative, and twice that for the bf16 reference it is compared in
    segs = [(0, 3000, 1096), (1, 2047, 300), (2, 0, 2049), (3, 4088, 8)]
    _close(*_run(8, 2, 16, segs=segs, span=4096, scale=0.5, fp32_weights=True), tol=2 ** -7)


@pytest.mark.parametrize("shift", [-120, -127, -130, -133])
def test_weights_below_the_normal_range(shift):
    """A key that is 2^shift of the largest weight still counts: its value is as large as bf16 has them, those of all others are 0."""
    n_q, bs, n = 2, 16, 130
    q, kc, vc = (torch.zeros(s, dtype=torch.bfloat16, device="cuda") for s in ((n, n_q * HD), (9, bs, n_q, HD), (9, bs, n_q, HD)))
    q[:, ::HD] = 1.0
    kc[0, 3, :, 0], vc[0, 3] = float(shift), 2.0 ** 127
    bt, out = torch.arange(9, device="cuda").int()[None], torch.empty(n, n_q * HD, dtype=torch.bfloat16, device="cuda")
    tiles, _ = F.build_prefill_tiles([0] * n, range(n), F.prefill_tile_tokens(n_q, n_q))
    F.prefill_attention(q, kc, vc, bt, tiles.cuda(), len(tiles), n_q, n_q, HD, out, scale=math.log(2.0), fp32_weights=True)
    t = torch.arange(n, device="cuda", dtype=torch.float64)
    want = torch.where(t >= 3, 2.0 ** (127 + shift) / t.clamp(min=1), t * 0)
    # powers of two down to bf16's smallest, 2^-133: one rounding of the output and the fp32 division by the sum
    assert gemm.check_status() == 0
    torch.testing.assert_close(out.double(), want[:, None].expand_as(out), rtol=2.0 ** -7, atol=0.0)


def test_loose_rows():
    assert F.loose_rows(torch.tensor([True, False, True])) == 2 and F.loose_rows(torch.zeros(4, dtype=torch.bool)) == 4
    assert F.loose_rows(torch.ones(3, dtype=torch.bool)) == 0


@pytest.mark.parametrize("window", [None, 1, 64, 200])
@pytest.mark.parametrize("extras", [False, True])
def test_latent(window, extras):
    """Expanded keys and values of several runs, rows of garbage before, between and behind them."""
    torch.manual_seed(3)
    H, rankp, scale = 3, 72, 0.07
    lay = F.LatentLayout(H, 128, 64, 128, rankp)
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    runs = [(0, 0, 300), (1, 50, 129), (2, 400, 16), (3, 0, 128)]      # (row, first position, tokens)
    rows, pos = [], []
    for r, p0, n in runs:
        rows += [r] * n
        pos += list(range(p0, p0 + n))
    T = len(rows)
    tiles, covered = F.build_prefill_tiles(rows, pos, 128, 8)
    assert bool(covered.all())
    lo = {r: max(0, p0 - window + 1) if window else 0 for r, p0, n in runs}
    start, at = {}, 5
    for r, p0, n in runs:
        start[r] = at - lo[r]
        at += p0 + n - lo[r] + 5
    base = torch.tensor([start[int(t[2])] for t in tiles], dtype=torch.int32, device="cuda")
    kv, lat = bf(at, H * 256), bf(at, rankp + 64 + 8)[:, :rankp + 64]
    live = torch.zeros(at, dtype=torch.bool, device="cuda")
    for r, p0, n in runs:
        live[start[r] + lo[r]:start[r] + p0 + n] = True
    kv[~live], lat[~live] = float("nan"), float("nan")
    q = bf(T, H * 192 + 16)
    sink = torch.randn(H, device="cuda") if extras else None
    gate = bf(T, H) if extras else None
    out = torch.full((T, H * 128), 9.0, dtype=torch.bfloat16, device="cuda")
    F.latent_prefill(q, kv, lat, tiles.cuda(), base, len(tiles), lay, scale, window, sink, out, gate)
    assert gemm.check_status() == 0
    t0 = 0
    for r, p0, n in runs:
        keys = torch.arange(lo[r], p0 + n, device="cuda")
        kr, p = (start[r] + keys).long(), torch.arange(p0, p0 + n, device="cuda")
        hide = keys[None] > p[:, None]
        if window:
            hide |= keys[None] <= p[:, None] - window
        for h in range(H):
            k = torch.cat([kv[kr, h * 256:h * 256 + 128], lat[kr, rankp:]], 1).double()
            s = (q[t0:t0 + n, h * 192:(h + 1) * 192].double() @ k.T * scale).masked_fill(hide, -float("inf"))
            if extras:
                s = torch.cat([s, sink[h].double().expand(n, 1)], 1)
            o = torch.softmax(s, -1)[:, :len(keys)] @ kv[kr, h * 256 + 128:(h + 1) * 256].double()
            if extras:
                o = o * torch.sigmoid(gate[t0:t0 + n, h, None].double())
            _close(out[t0:t0 + n, h * 128:(h + 1) * 128].double(), o, tol=2 ** -8)
        t0 += n
