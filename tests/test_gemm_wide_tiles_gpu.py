"""Tiles of 64 .. 256 weight rows of the pair GEMM (csrc/kernels/gemm_wide.cu): edges of tokens, weight rows, K blocks and stages."""
import pytest
import torch

from disagmoe_b200.ops import gemm, reference

pytestmark = pytest.mark.gpu


def _bf(*s):
    return torch.randn(*s, device="cuda").to(torch.bfloat16)


def _close(y, ref, K):
    """One rounding of the output (half a unit: 2^-8 relative) and fp32 sums of K products of size 1 / K in any order."""
    bad = ((y.double() - ref).abs() > ref.abs() * 2.0 ** -8 + 2.0 ** -22 * K ** 0.5 + 1e-6).sum().item()
    assert bad == 0 and gemm.check_status() == 0, f"{bad} of {ref.numel()} off, max {(y.double() - ref).abs().max().item():.3g}"


@pytest.mark.parametrize("cols", [64, 96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("T,N,K", [(1, 8, 8), (129, 168, 64), (257, 520, 136), (700, 1320, 712)])
def test_tile_sizes(T, N, K, cols):
    torch.manual_seed(T + cols)
    x, w, r = _bf(T, K), _bf(N, K) * K ** -0.5, _bf(T, N)
    ref = x.double() @ w.double().T
    out = torch.full((T + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm.linear(x, w, out=out[:T, :N], wide=cols)
    _close(out[:T, :N], ref, K)
    assert bool((out[T] == 7.0).all()) and bool((out[:, N:] == 7.0).all())
    y = r.clone()
    gemm.linear(x, w, residual=y, out=y, wide=cols)
    _close(y, ref + r.double(), K)
    w2 = _bf(2 * N, K) * K ** -0.5
    h = x.double() @ w2.double().T
    out.fill_(7.0)
    gemm.swiglu_linear(x, w2, out=out[:T, :N], wide=cols)
    _close(out[:T, :N], h[:, :N] * torch.sigmoid(h[:, :N]) * h[:, N:], K)
    assert bool((out[T] == 7.0).all()) and bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("cols", [64, 128, 160, 256])
@pytest.mark.parametrize("T,N,K", [(1, 8, 64), (150, 200, 520), (300, 328, 1024)])
def test_other_epilogues(T, N, K, cols):
    torch.manual_seed(T + cols)
    x, w, r, w13 = _bf(T, K), _bf(N, K) * K ** -0.5, _bf(T, N), _bf(2 * N, K) * K ** -0.5
    h = x.double() @ w.double().T
    # the bound's 2^-8 of the output is more than fp32 outputs need; what they add is the order of their sums
    _close(gemm.linear(x, w, wide=cols, tanh=True), torch.tanh(h), K)
    _close(gemm.linear(x, w, wide=cols, tanh=True, out_dtype=torch.float32), torch.tanh(h), K)
    _close(gemm.linear(x, w, wide=cols, residual=r, out_dtype=torch.float32), h + r.double(), K)
    silu = h.clone()
    silu[:, :N // 2] *= torch.sigmoid(silu[:, :N // 2])
    _close(gemm.linear(x, w, wide=cols, silu_cols=N // 2), silu, K)
    g, u = (x.double() @ w13.double().T).split(N, 1)
    # the error of the gate's product counts |u| <= 4 times: 16 K under the root
    _close(gemm.swiglu_linear(x, w13, wide=cols, act="gelu_tanh"), torch.nn.functional.gelu(g, approximate="tanh") * u, 16 * K)
    out, m = torch.empty(T, N, dtype=torch.bfloat16, device="cuda"), g.clamp(max=0.75)
    gemm._launch(w13, x, out, None, None, None, None, 1, T, N, K, gemm.EPI_SWIGLU, 128, 1, N, False, act=gemm.ACTS["clamped"], act_limit=0.75, wide=cols)
    _close(out, m * torch.sigmoid(1.702 * m) * (u.clamp(-0.75, 0.75) + 1.0), 16 * K)


@pytest.mark.parametrize("sizes", [[33, 0, 1, 31, 257, 32, 300], [64, 255, 7]])
def test_rows_of_the_next_group_stay(sizes):
    """Whole warps of a group go out as boxes of 32 rows; a remainder may not reach into the next group or past the last."""
    torch.manual_seed(len(sizes))
    G, N, K, T = len(sizes), 328, 136, sum(sizes) + 40
    x, w13 = _bf(T, K), _bf(G, 2 * N, K) * K ** -0.5
    offs = torch.tensor([0, *sizes], device="cuda").cumsum(0).to(torch.int32)
    for op, w in ((gemm.grouped_linear, w13[:, :N].contiguous()), (gemm.grouped_swiglu, w13)):
        out = torch.full((T + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
        op(x, w, offs, out=out[:T, :N], wide=True)
        for g in range(G):
            a, b = sum(sizes[:g]), sum(sizes[:g + 1])
            h = x[a:b].double() @ w[g].double().T
            _close(out[a:b, :N], h if op is gemm.grouped_linear else h[:, :N] * torch.sigmoid(h[:, :N]) * h[:, N:], K)
        assert bool((out[sum(sizes):] == 7.0).all()) and bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("blocked", [False, True])
@pytest.mark.parametrize("sizes", [[5, 64, 128, 65, 0, 129, 385], [1], [127, 32]])
def test_tail_tiles(sizes, blocked):
    """Tiles of up to 128 tokens (64 per CTA, both halves of the columns in one TMEM): plain, fp32, gated and combining."""
    torch.manual_seed(sum(sizes))
    G, N, K, T = len(sizes), 384, 192, sum(sizes)
    x, w13, w = _bf(T, K), _bf(G, 2 * N, K) * K ** -0.5, _bf(G, N, K) * K ** -0.5
    offs = torch.tensor([0, *sizes], device="cuda").cumsum(0).to(torch.int32)
    lay = gemm.block_weight if blocked else lambda t: t
    kw = dict(wide=True, w_blocked=blocked)
    up, y, y32 = gemm.grouped_swiglu(x, lay(w13), offs, **kw), gemm.grouped_linear(x, lay(w), offs, **kw), \
        gemm.grouped_linear(x, lay(w), offs, out_dtype=torch.float32, **kw)
    recs, weight, to = torch.zeros(T, 4, dtype=torch.int32, device="cuda"), torch.rand(T, device="cuda"), torch.randperm(T, device="cuda")
    recs[:, 1], recs[:, 2] = to.int(), weight.view(torch.int32)
    out = torch.full((T + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm.grouped_combine(x, lay(w), offs, recs, torch.tensor([out.data_ptr()], device="cuda"), N, **kw)
    assert bool((out[T] == 7.0).all())
    for g in range(G):
        a, b = sum(sizes[:g]), sum(sizes[:g + 1])
        h, r = x[a:b].double() @ w13[g].double().T, x[a:b].double() @ w[g].double().T
        _close(up[a:b], h[:, :N] * torch.sigmoid(h[:, :N]) * h[:, N:], K)
        _close(y[a:b], r, K)
        _close(y32[a:b], r, K)
        _close(out[to[a:b]], r * weight[a:b, None].double(), K)


@pytest.mark.parametrize("hd,cols", [(64, 64), (64, 192), (64, 256), (128, 128), (128, 256)])
def test_heads_stay_whole(hd, cols):
    torch.manual_seed(cols)
    T, K, n_q, n_kv, bs = 300, 256, 5, 2, 16
    N = (n_q + 2 * n_kv) * hd
    x, w = _bf(T, K), _bf(N, K) * K ** -0.5
    pos = torch.randint(0, 500, (T,), device="cuda", dtype=torch.int32)
    slots = torch.randperm(400, device="cuda")[:T]
    caches = [torch.zeros(25, bs, n_kv, hd, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    table, y = gemm.rope_table(512, hd, 1e4, "cuda"), torch.zeros(T, N, dtype=torch.bfloat16, device="cuda")
    gemm.linear(x, w, out=y, wide=cols, comm=gemm.GemmComm(rope=gemm.RopeAppend(table, pos, slots, *caches[:2], n_q, n_kv, hd)))
    z = gemm.linear(x, w, wide=256)
    reference.rope_kv_append(z, pos, slots, *caches[2:], n_q, n_kv, hd, 1e4)
    # the reference rotates in fp32 with its own sines: a unit of the last place of bf16
    for a, b in ((y[:, :n_q * hd], z[:, :n_q * hd]), (caches[0], caches[2]), (caches[1], caches[3])):
        torch.testing.assert_close(a.float(), b.float(), rtol=2 ** -7, atol=2 ** -7)
    assert gemm.check_status() == 0


def test_chosen_tiles():
    assert gemm.dense_wide(2500, 2048, 2048, gemm.EPI_PLAIN, 148)[1] == 160      # 130 tiles in two waves of 74 pairs, 80 of 256 rows
    assert gemm.dense_wide(4096, 4096, 4096, gemm.EPI_PLAIN, 148, 128)[1] % 128 == 0
    x, w = _bf(2500, 512), _bf(2048, 512) * 512 ** -0.5
    _close(gemm.linear(x, w), x.double() @ w.double().T, 512)
