"""Chunks of linear recurrences (csrc/kernels/recurrent_chunk.cu) where the decay of a chunk's tokens decides how its factors are formed:
ordinary, fading so far before the middle that e^(b - m) e^m is no fp32 product, and so fast that pairs are evaluated one by one."""
import pytest
import torch

from disagmoe_b200.ops.recurrent import Recurrence, build_segments, recurrent_attention

pytestmark = pytest.mark.gpu


def _z(fade, T, n):
    z = 0.3 + 0.2 * torch.rand(T, n, device="cuda")
    if fade == "faint":
        z[::64] = 60.0        # 2^-86 at a chunk's first token, 2^-40 from there to the middle, 2^-43 from the middle to the end
    elif fade == "fast":
        z += 3.0
    return z


@pytest.mark.parametrize("fade", ["even", "faint", "fast"])
@pytest.mark.parametrize("delta,H,G,D,V", [(False, 2, 2, 128, 128), (False, 3, 3, 40, 24), (False, 2, 2, 32, 8), (True, 4, 2, 128, 128),
                                           (True, 3, 1, 72, 40), (True, 2, 2, 24, 64)])
@pytest.mark.parametrize("T", [2, 65, 240])
def test_fading(delta, H, G, D, V, T, fade):
    torch.manual_seed(T + D)
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    q, k, v, gate, beta = bf(T, G * D), bf(T, G * D), bf(T, H * V), bf(T, H * V), bf(T, H)
    z, zero = _z(fade, T, H * D), torch.zeros(H * D, device="cuda")
    # the plain write's logits count the other way round: log sigmoid(-z) is -softplus(z)
    r = Recurrence(H, G, D, V, delta, zero, torch.ones(V, device="cuda"), 1e-6, a_log=torch.zeros(H, device="cuda") if delta else None)
    state = r.new_state(1, torch.bfloat16, "cuda")
    out = recurrent_attention(r, q, k, v, gate, beta if delta else None, z if delta else -z, state, build_segments([0] * T, range(T), "cuda"))
    qq, kk = (t.view(T, G, D).double().repeat_interleave(H // G, 1) for t in (q, k))
    if delta:
        qq, kk = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (qq, kk))
    keep = 1 / (1 + torch.exp(z.double().view(T, H, D, 1)))
    vv, b, S, o = v.view(T, H, V).double(), torch.sigmoid(beta.double()), torch.zeros(H, D, V, device="cuda", dtype=torch.double), []
    for t in range(T):
        S = S * keep[t]
        u = b[t, :, None] * (vv[t] - torch.einsum("hd,hdv->hv", kk[t], S)) if delta else vv[t]
        S = S + kk[t][..., None] * u[:, None]
        o.append(torch.einsum("hd,hdv->hv", qq[t], S))
    # factors of 17 bits, three products per product, up to four in a row (T, W, u, state): 12 x 2^-17 of the largest
    assert (state.S[0].double() - S).abs().max() < 2.0 ** -13 * S.abs().max()
    o = torch.stack(o) * D ** -0.5
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6)
    g = gate.view(T, H, V).double()
    o = o * torch.sigmoid(g) * g
    assert (out.view(T, H, V).double() - o).norm() < 2.0 ** -8 * o.norm()      # one rounding to bf16: at most 2^-8 of every value


@pytest.mark.parametrize("drops", [{1: 75.0, 40: 16.0}, {1: 45.0, 40: 46.0}])
@pytest.mark.parametrize("kind,D,V", [("plain", 128, 16), ("plain", 40, 24), ("bonus", 128, 16), ("bonus", 64, 40), ("delta", 72, 16)])
def test_decays_below_the_normal_range(kind, D, V, drops):
    """A state and a write that fade by 2^-131 within a chunk (to a subnormal factor) still count: both are as large as fp32 and bf16 have
    them. The first drops leave pairs of tokens to products, the second ones are evaluated pair by pair."""
    torch.manual_seed(D)
    T, H, pos0 = 64, 2, 100
    bf = lambda *s: (1.0 + torch.rand(*s, device="cuda")).to(torch.bfloat16)
    q, k, v, gate, beta = 2.0 ** 20 * bf(T, H * D), 2.0 ** 20 * bf(T, H * D), torch.zeros(T, H * V, device="cuda").bfloat16(), bf(T, H * V), bf(T, H)
    v[0] = 2.0 ** 100 * bf(H * V)
    q[0] = 0.0                                             # its read-out would be no fp32 number
    if kind == "delta":
        k.zero_()                                          # nothing written or taken back: the state fades
    z = torch.full((T, H * D), -80.0, device="cuda")       # a factor of 1
    for t, x in drops.items():
        z[t] = x
    bonus = torch.rand(H, D, device="cuda") if kind == "bonus" else None
    r = Recurrence(H, H, D, V, kind == "delta", torch.zeros(H * D, device="cuda"), torch.ones(V, device="cuda"), 1e-30, bonus=bonus,
                   a_log=torch.zeros(H, device="cuda") if kind == "delta" else None)
    state = r.new_state(1, torch.bfloat16, "cuda")
    state.S[0] = 2.0 ** 120 * (1.0 + torch.rand(H, D, V, device="cuda"))
    S = state.S[0].double()
    out = recurrent_attention(r, q, k, v, gate, beta if kind == "delta" else None, z if kind == "delta" else -z, state,
                              build_segments([0] * T, range(pos0, pos0 + T), "cuda"))
    qq, kk, vv = q.view(T, H, D).double(), k.view(T, H, D).double(), v.view(T, H, V).double()
    keep, o = 1 / (1 + torch.exp(z.double().view(T, H, D, 1))), []
    for t in range(T):
        if bonus is not None:
            o.append(torch.einsum("hd,hdv->hv", qq[t], S + (bonus.double() * kk[t])[..., None] * vv[t][:, None]))
        S = S * keep[t] + kk[t][..., None] * vv[t][:, None]
        if bonus is None:
            o.append(torch.einsum("hd,hdv->hv", qq[t], S))
    # running sums of 131 in fp32 are off by 2^-17 (relative, in the power), the power itself keeps 18 bits below the normal range, and
    # both factors of a product 16 or more
    assert float(((state.S[0].double() - S).abs() / S).max()) < 2.0 ** -12
    if kind != "delta":
        o = torch.stack(o)[41:]                            # behind the second drop
        o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-30)
        g = gate.view(T, H, V).double()[41:]
        o = o * torch.sigmoid(g) * g
        assert float(((out.view(T, H, V)[41:].double() - o).abs() / o).max()) < 2.0 ** -7


@pytest.mark.parametrize("delta", [False, True])
def test_value_tiles_agree(delta):
    """20 heads take value tiles of 32 columns (one wave of CTAs), 10 heads those of 16: the same sums in the same order."""
    torch.manual_seed(3)
    T, H, D, V = 150, 20, 72, 120
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    q, k, v, gate, beta, z = bf(T, H * D), bf(T, H * D), bf(T, H * V), bf(T, H * V), bf(T, H), torch.randn(T, H * D, device="cuda")
    bias, log = torch.randn(H * D, device="cuda"), 0.3 * torch.randn(H, device="cuda")

    def run(a, b):
        d, e = slice(a * D, b * D), slice(a * V, b * V)
        r = Recurrence(b - a, b - a, D, V, delta, bias[d], torch.ones(V, device="cuda"), 1e-6, a_log=log[a:b] if delta else None)
        s = r.new_state(1, torch.bfloat16, "cuda")
        return recurrent_attention(r, q[:, d], k[:, d], v[:, e], gate[:, e], beta[:, a:b] if delta else None, z[:, d], s,
                                   build_segments([0] * T, range(T), "cuda")), s.S[0]
    out, S = run(0, H)
    for a in (0, 10):
        o, s = run(a, a + 10)
        assert torch.equal(o, out[:, a * V:(a + 10) * V]) and torch.equal(s, S[a:a + 10])


def test_operands_asked_for_ahead():
    """A workspace of more than 32 MB (asked for ahead of its turn) gives what its heads give alone."""
    torch.manual_seed(4)
    T, H, D, V = 1600, 17, 128, 16
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    q, k, v, gate, z = bf(T, H * D), bf(T, H * D), bf(T, H * V), bf(T, H * V), torch.randn(T, H * D, device="cuda") + 3.0

    def run(a, b):
        d, e = slice(a * D, b * D), slice(a * V, b * V)
        r = Recurrence(b - a, b - a, D, V, False, torch.zeros((b - a) * D, device="cuda"), torch.ones(V, device="cuda"), 1e-6)
        s = r.new_state(1, torch.bfloat16, "cuda")
        return recurrent_attention(r, q[:, d].contiguous(), k[:, d].contiguous(), v[:, e].contiguous(), gate[:, e].contiguous(), None,
                                   z[:, d].contiguous(), s, build_segments([0] * T, range(T), "cuda")), s.S[0]
    out, S = run(0, H)
    for a in (0, 16):
        o, s = run(a, a + 1)
        assert torch.equal(o, out[:, a * V:(a + 1) * V]) and torch.equal(s, S[a:a + 1])
