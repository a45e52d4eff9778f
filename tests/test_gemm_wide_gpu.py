"""The GEMM with the tokens as the M operand (CTA pairs on 256 x 256 tiles) vs fp32 PyTorch: edges of tiles, remainders, epilogues."""
import pytest
import torch

from disagmoe_b200.ops import functional as F
from disagmoe_b200.ops import gemm

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _close(y, ref, tol=2 ** -7):
    """A bf16 result of an fp32 accumulation is off by at most 2^-9 relative; an intermediate rounding doubles that."""
    assert gemm.check_status() == 0
    y, ref = y.float(), ref.float()
    bound = ref.abs() * tol + ref.pow(2).mean().sqrt() * tol
    bad = int(((y - ref).abs() > bound).sum())
    assert bad == 0, f"{bad} of {ref.numel()} elements off, max {(y - ref).abs().max().item():.4g}"


@pytest.mark.parametrize("T", [1, 127, 128, 129, 256, 257, 700])
@pytest.mark.parametrize("O,K", [(8, 8), (264, 72), (512, 1000)])
def test_linear_variants(T, O, K):
    torch.manual_seed(T)
    x, w, r = _rand(T, K), _rand(O, K, scale=K ** -0.5), _rand(T, O)
    ref = x.float() @ w.float().T
    _close(gemm.linear(x, w, wide=True), ref)
    _close(gemm.linear(x, w, out_dtype=torch.float32, wide=True), ref, tol=2 ** -12)
    _close(gemm.linear(x, w, tanh=True, wide=True), torch.tanh(ref))
    silu = torch.cat([torch.nn.functional.silu(ref[:, :O // 2 + 1]), ref[:, O // 2 + 1:]], 1)
    _close(gemm.linear(x, w, silu_cols=O // 2 + 1, wide=True), silu)
    out = r.clone()
    gemm.linear(x, w, residual=out, out=out, wide=True)
    _close(out, ref + r.float())


@pytest.mark.parametrize("wide", [False, True])
def test_silu_divides_exactly(wide):
    """Of a product with the identity the activation is all that rounds: the quotient to nearest (0.5 units of 2^-24), its denominator
    and the exponential. Their errors' root mean square measured 0.77 units, and 0.93 with an approximate quotient."""
    torch.manual_seed(0)
    x = _rand(4096, 256, scale=0.1)
    y = gemm.linear(x, torch.eye(256, device="cuda").bfloat16(), out_dtype=torch.float32, silu_cols=256, wide=wide).double()
    want = torch.nn.functional.silu(x.double())
    err = ((y - want) / want)[want != 0] * 2.0 ** 24
    assert float(err.pow(2).mean().sqrt()) < 0.85 and float(err.abs().max()) < 5
    # signed zeros, infinities and NaN as the division has them
    edge = torch.tensor([0.0, -0.0, float("inf"), float("nan"), -200.0, 300.0, -88.0, 1.0], device="cuda").bfloat16()
    y = gemm.linear(edge.repeat(8).diag(), torch.eye(64, device="cuda").bfloat16(), out_dtype=torch.float32, silu_cols=64, wide=wide)
    assert bool(y[3].isnan().all()) and bool(y[2, 2].isposinf()) and float(y[5, 5]) == 300.0
    assert -1e-35 < float(y[6, 6]) < 0 and float(y[4, 4]) == 0 and float(y[0].abs().max()) == 0


@pytest.mark.parametrize("wide", [None, True])
def test_counters_to_clear(wide):
    """Only the other kernel zeroes the counters that a launch is given: it keeps such a launch, whatever is asked for."""
    x, w = _rand(1024, 512), _rand(2048, 512, scale=512 ** -0.5)
    cnt, ticket = torch.full((37,), 5, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    _close(gemm.linear(x, w, wide=wide, comm=gemm.GemmComm(done_ticket=ticket, clear=cnt)), x.float() @ w.float().T)
    assert int(cnt.abs().sum()) == 0 and int(ticket) == 0


@pytest.mark.parametrize("counts,I,K,blocked", [
    ([1, 0, 255, 256], 128, 64, True), ([257, 128, 0, 129], 264, 200, False), ([0, 0, 0], 128, 64, True),
    ([600, 3, 40, 512, 0, 90] * 11, 256, 192, True),
])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "clamped"])
def test_grouped(counts, I, K, blocked, act):
    torch.manual_seed(1)
    G, T = len(counts), sum(counts)
    offs = torch.tensor([0] + counts).cumsum(0).int().cuda()
    x, w13, w2 = _rand(T + 5, K)[:T], _rand(G, 2 * I, K, scale=2 * K ** -0.5), _rand(G, K, I, scale=I ** -0.5)
    recs = torch.zeros(T, 4, dtype=torch.int32, device="cuda")
    recs[:, 1] = torch.randperm(T, device="cuda").int()
    recs[::5, 1] = -1
    recs[:, 2] = torch.rand(T, device="cuda").view(torch.int32)
    block = gemm.block_weight if blocked else (lambda w: w)
    rows = recs if act == "clamped" else None
    y = gemm.grouped_swiglu(x, block(w13), offs, w_blocked=blocked, act=act, limit=1.5, recs=rows, wide=True)
    ref = gemm._grouped_ref(x, w13, offs, True, act, 1.5, rows)
    if T:
        _close(y, ref)
    ref2 = gemm._grouped_ref(y, w2, offs, False)
    if T:
        _close(gemm.grouped_linear(y, w2, offs, wide=True), ref2)
    out = torch.full((T + 1, K), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm.grouped_combine(y, w2, offs, recs, torch.tensor([out.data_ptr()], device="cuda"), K, wide=True)
    want, kept = torch.full_like(out, 7.0).float(), recs[:, 1] >= 0
    want[recs[kept, 1].long()] = (ref2 * recs[:, 2].contiguous().view(torch.float32)[:, None])[kept]
    _close(out, want)


@pytest.mark.parametrize("n_q,n_kv,hd,T", [(4, 1, 128, 300), (3, 3, 64, 129), (8, 2, 64, 513)])
def test_qkv_epilogue(n_q, n_kv, hd, T):
    torch.manual_seed(2)
    H, heads = 256, n_q + 2 * n_kv
    x, w = _rand(T, H), _rand(heads * hd, H, scale=H ** -0.5)
    pos = torch.randint(0, 900, (T,), device="cuda", dtype=torch.int32)
    slots = torch.randperm(2 * T, device="cuda")[:T].long()
    slots[::9] = -1
    kc, vc = (torch.zeros((2 * T + 15) // 16, 16, n_kv, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    rope = gemm.RopeAppend(gemm.rope_table(1024, hd, 1e4, "cuda"), pos, slots, kc, vc, n_q, n_kv, hd)
    q = gemm.linear(x, w, comm=gemm.GemmComm(rope=rope), wide=True)[:, :n_q * hd]
    kc2, vc2 = torch.zeros_like(kc), torch.zeros_like(vc)
    ref = gemm.linear(x, w, wide=True)
    F.rope_kv_append(ref, pos, slots, kc2, vc2, n_q, n_kv, hd, 1e4)
    # both rotate the same bf16 values in fp32, in another order of operations: at most the last bf16 bit, 2^-8 relative
    for a, b in ((q, ref[:, :n_q * hd]), (kc, kc2), (vc, vc2)):
        _close(a, b, tol=2 ** -8)
    assert torch.equal(vc, vc2)
