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
