"""The router on the tensor cores, greedy sampling over several CTAs per row and the gated shared expert vs PyTorch."""
import pytest
import torch

from disagmoe_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _bf(*s, scale=1.0):
    return (torch.randn(*s, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("T", [1, 15, 16, 17, 300])
@pytest.mark.parametrize("H,E,K", [(256, 17, 3), (2048, 60, 4), (4096, 64, 8), (512, 256, 8), (2048, 33, 1)])
def test_softmax_router(T, H, E, K, monkeypatch):
    monkeypatch.setattr(F, "separate_router", lambda *a: True)
    torch.manual_seed(T)
    x, nw, gw = _bf(T, H), _bf(H), _bf(E, H, scale=H ** -0.5)
    bias = torch.randn(E, device="cuda")
    counts = torch.zeros(E, dtype=torch.int32, device="cuda")
    y, ids, w, logits = F.route(x, nw, 1e-5, gw, K, True, counts=counts, want_logits=True, logit_bias=bias)
    exact = y.double() @ gw.double().T + bias.double()
    # fp32 sums of exact products: a few units of 2^-24 of the sum of their sizes (the tensor core truncates when it aligns them)
    bound = (y.double().abs() @ gw.double().abs().T + bias.double().abs()) * 2.0 ** -20
    assert bool(((logits.double() - exact).abs() <= bound).all())
    s, want = torch.softmax(logits.double(), -1).sort(dim=-1, descending=True, stable=True)
    assert torch.equal(ids.long(), want[:, :K])
    torch.testing.assert_close(w.double(), s[:, :K] / s[:, :K].sum(-1, keepdim=True), rtol=1e-5, atol=1e-7)
    assert torch.equal(counts.long(), torch.bincount(ids.reshape(-1).long(), minlength=E))


@pytest.mark.parametrize("kind", ["normal", "outliers", "offset"])
@pytest.mark.parametrize("T,H,E", [(1111, 2048, 64), (37, 2048, 60), (2048, 4096, 8), (300, 256, 33), (300, 8192, 17), (300, 1024, 256)])
def test_logits_no_less_exact_than_on_the_cuda_cores(T, H, E, kind, monkeypatch):
    """Errors against fp64 of the same rows on the tensor cores and in the fused kernel's fp32 multiply-adds."""
    torch.manual_seed(H + E)
    x, gw = torch.randn(T, H, device="cuda"), torch.randn(E, H, device="cuda") * H ** -0.5
    if kind == "outliers":
        x[:, ::97] *= 30
    if kind == "offset":
        x, gw = x + 3, gw + 0.05
    x, gw, nw, err = x.bfloat16(), gw.bfloat16(), _bf(H).abs() + 0.5, []
    for separate in (True, False):
        monkeypatch.setattr(F, "separate_router", lambda *a: separate)
        y, _, _, logits = F.route(x, nw, 1e-5, gw, 2, want_logits=True)
        err.append((logits.double() - y.double() @ gw.double().T).pow(2).mean().sqrt())
    # the errors are sums of many rounding errors: their mean square over some thousand logits moves by a few percent
    assert float(err[0]) <= 1.05 * float(err[1])


@pytest.mark.parametrize("T", [3, 161, 700])
@pytest.mark.parametrize("E,top,groups,keep,sigmoid", [(64, 6, 8, 3, True), (24, 2, 1, 1, True), (64, 6, 1, 1, False)])
def test_router_behind_sum_norm(T, E, top, groups, keep, sigmoid, monkeypatch):
    """The same rows through the fused kernel: only nearly equal scores may be chosen differently."""
    torch.manual_seed(E)
    W = 1024
    resid, y, w = torch.randn(T, W, device="cuda"), _bf(T, W), torch.rand(W, device="cuda") + 0.5
    corr = torch.randn(E, device="cuda") * 0.1 if sigmoid else None
    weight, out = _bf(E, W, scale=W ** -0.5), []
    for fused in (False, True):
        monkeypatch.setattr(F, "separate_router", lambda *a: not fused)
        r = F.Router(weight, top, sigmoid, torch.zeros(E, dtype=torch.int32, device="cuda"), sigmoid, corr, groups, keep, 2.5)
        h, ids, wts = F.sum_norm(resid.clone(), y, None, w, 1e-6, torch.bfloat16, False, router=r)
        assert torch.equal(r.counts.long(), torch.bincount(ids.reshape(-1).long(), minlength=E))
        out.append((h, ids, wts))
    # the fused kernel sums a row's squares in another order (fp32): the last bf16 bit at most
    torch.testing.assert_close(out[0][0].float(), out[1][0].float(), rtol=2.0 ** -7, atol=1e-6)
    same = out[0][1] == out[1][1]
    assert float(same.float().mean()) > 0.99
    rows = same.all(-1)
    torch.testing.assert_close(out[0][2][rows], out[1][2][rows], rtol=2e-3, atol=1e-6)


def test_refusals_stay():
    x, gw = _bf(4, 256), _bf(64, 256)
    with pytest.raises(Exception):
        F.route(x, None, 1e-5, gw, 9)                   # more than 8 choices
    with pytest.raises(Exception):
        F.route(_bf(4, 256), None, 1e-5, _bf(300, 256), 2)


@pytest.mark.parametrize("T,V,dtype,off", [(1, 151936, torch.float32, 0), (37, 32000, torch.float32, 0), (3, 8193, torch.float32, 1),
                                           (400, 1000, torch.float32, 0), (5, 9001, torch.bfloat16, 0), (2, 5, torch.float32, 0)])
def test_argmax(T, V, dtype, off):
    torch.manual_seed(V)
    x = torch.randint(-50, 50, (T, V + off), device="cuda").to(dtype)[:, off:]      # many ties: the first one wins
    x[0, :] = -float("inf")
    if T > 2:
        x[1, :] = float("nan")
        x[1, V // 2] = 1.0
        x[2, -1] = 99.0
    got = F.argmax(x).long()
    want = torch.stack([(r == r[~r.isnan()].max()).nonzero()[0, 0] for r in x])
    assert torch.equal(got, want)


@pytest.mark.parametrize("T", [1, 37, 38, 74, 75, 148, 149, 300])
@pytest.mark.parametrize("V,dtype", [(8192, torch.float32), (24011, torch.bfloat16), (32000, torch.float32)])
def test_argmax_over_the_runs_of_a_row(T, V, dtype):
    """Rows that 8, 4, 2 CTAs of a cluster share, and those that one CTA scans: the maximum stands in every run in turn."""
    x = torch.zeros(T, V, dtype=dtype, device="cuda")
    at = (torch.arange(T, device="cuda") * 1031 + 17) % V
    x[torch.arange(T, device="cuda"), at] = 1.0
    for _ in range(20):
        assert torch.equal(F.argmax(x).long(), at)


@pytest.mark.parametrize("T,H", [(1, 8), (37, 2048), (300, 264)])
def test_gated_add(T, H):
    torch.manual_seed(H)
    resid, sh, y, w = _bf(T, H), _bf(T, H), _bf(T, H), _bf(1, H, scale=H ** -0.5)
    want = resid.double() + sh.double() * torch.sigmoid(y.double() @ w.double().T)
    got = F.gated_add(resid.clone(), sh, y, w).double()
    # one bf16 rounding of the sum (half a unit in the last of 8 bits) and the fp32 gate
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -7.99 + 1e-5).all())
    # unaligned rows take the general path
    base = torch.cat([resid, resid], 1)
    v = base[:, 1:H + 1]
    assert v.data_ptr() % 16 != 0
    want = v.double() + sh.double() * torch.sigmoid(y.double() @ w.double().T)
    got = F.gated_add(v, sh, y, w).double()
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -7.99 + 1e-5).all())
