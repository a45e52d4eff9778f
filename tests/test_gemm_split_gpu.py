"""Dense GEMM with K cut over a cluster (csrc/kernels/gemm_split.cu) vs fp64 PyTorch: edges of tiles, shares and shared memory."""
import pytest
import torch

from disagmoe_b200.ops import functional as F
from disagmoe_b200.ops import gemm, reference

pytestmark = pytest.mark.gpu


def _bf(*s):
    return torch.randn(*s, device="cuda").to(torch.bfloat16)


def _close(y, ref, K, bits=8):
    """One rounding of the output (half a unit: 2^-8 relative in bf16, 2^-24 in fp32) and fp32 sums of K products of size 1 / K in any order."""
    bound = ref.abs() * 2.0 ** -bits + 2.0 ** -22 * K ** 0.5 + 1e-6
    bad = ((y.double() - ref).abs() > bound).sum().item()
    assert bad == 0 and gemm.check_status() == 0, f"{bad} of {ref.numel()} off, max {(y.double() - ref).abs().max().item():.3g}"


@pytest.mark.parametrize("bn,cluster", [(16, 1), (16, 8), (32, 4), (48, 5), (80, 2), (96, 1), (96, 3), (112, 8), (128, 1), (128, 2), (208, 8), (256, 1)])
@pytest.mark.parametrize("T,N,K", [(1, 8, 8), (15, 136, 72), (17, 128, 64), (97, 264, 520), (300, 144, 1096), (33, 1024, 2048)])
def test_tiles_and_clusters(T, N, K, bn, cluster):
    torch.manual_seed(T + N + K)
    x, w, r = _bf(T, K), _bf(N, K) * K ** -0.5, _bf(T, N)
    ref = x.double() @ w.double().T
    wide_x = torch.cat([x, _bf(T, 16)], 1)[:, :K]                        # rows further apart than they are long
    out = torch.full((T + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm.linear(wide_x, w, out=out[:T, :N], bn=bn, cluster=cluster)
    _close(out[:T, :N], ref, K)
    assert bool((out[T] == 7.0).all()) and bool((out[:, N:] == 7.0).all())
    y = r.clone()
    gemm.linear(x, w, residual=y, out=y, bn=bn, cluster=cluster)         # in place
    _close(y, ref + r.double(), K)
    _close(gemm.linear(x, w, bn=bn, cluster=cluster, out_dtype=torch.float32), ref, K, bits=22)
    s = ref.clone()
    s[:, :N // 2] *= torch.sigmoid(s[:, :N // 2])
    # the activation adds the error of its exponential, 2^-21 relative
    _close(gemm.linear(x, w, bn=bn, cluster=cluster, silu_cols=N // 2, out_dtype=torch.float32), s, K, bits=19)


@pytest.mark.parametrize("bn,cluster", [(16, 2), (48, 8), (144, 3), (256, 1)])
@pytest.mark.parametrize("T,I,K", [(1, 8, 64), (37, 72, 520), (150, 200, 1024)])
def test_gated(T, I, K, bn, cluster):
    torch.manual_seed(T)
    x, w = _bf(T, K), _bf(2 * I, K) * K ** -0.5
    h = x.double() @ w.double().T
    ref = h[:, :I] * torch.sigmoid(h[:, :I]) * h[:, I:]
    _close(gemm.swiglu_linear(x, w, bn=bn, cluster=cluster), ref, K)


@pytest.mark.parametrize("T,N,K,bn,cluster", [(1, 8, 64, 16, 1), (37, 72, 520, 48, 3), (150, 200, 1024, 144, 4)])
def test_other_epilogues(T, N, K, bn, cluster):
    torch.manual_seed(T)
    kw = dict(bn=bn, cluster=cluster)
    x, w, r, w13 = _bf(T, K), _bf(N, K) * K ** -0.5, _bf(T, N), _bf(2 * N, K) * K ** -0.5
    h = x.double() @ w.double().T
    _close(gemm.linear(x, w, tanh=True, **kw), torch.tanh(h), K)
    # out_tanh is good to 2^-22 (1 - 2 / (e + 1), e to 2^-21): within the absolute part of the bound
    _close(gemm.linear(x, w, tanh=True, out_dtype=torch.float32, **kw), torch.tanh(h), K, bits=22)
    _close(gemm.linear(x, w, residual=r, out_dtype=torch.float32, **kw), h + r.double(), K, bits=22)
    g, u = (x.double() @ w13.double().T).split(N, 1)
    # the error of the gate's product counts |u| <= 4 times: 16 K under the root
    _close(gemm.swiglu_linear(x, w13, act="gelu_tanh", **kw), torch.nn.functional.gelu(g, approximate="tanh") * u, 16 * K)
    out, m = torch.empty(T, N, dtype=torch.bfloat16, device="cuda"), g.clamp(max=0.75)
    gemm._launch(w13, x, out, None, None, None, None, 1, T, N, K, gemm.EPI_SWIGLU, bn, 1, N, False, act=gemm.ACTS["clamped"], act_limit=0.75, cluster=cluster)
    _close(out, m * torch.sigmoid(1.702 * m) * (u.clamp(-0.75, 0.75) + 1.0), 16 * K)


@pytest.mark.parametrize("hd,n_q,n_kv", [(128, 4, 1), (64, 6, 2)])
@pytest.mark.parametrize("T,bn,cluster", [(1, 16, 4), (50, 32, 3), (200, 112, 2)])
def test_rope_append(T, bn, cluster, hd, n_q, n_kv):
    torch.manual_seed(T)
    K, bs, N = 512, 16, (n_q + 2 * n_kv) * hd
    x, w = _bf(T, K), _bf(N, K) * K ** -0.5
    pos = torch.randint(0, 500, (T,), device="cuda", dtype=torch.int32)
    slots = torch.randperm(400, device="cuda")[:T]
    slots[::7] = -1
    caches = [torch.full((25, bs, n_kv, hd), 5.0, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    table = gemm.rope_table(512, hd, 1e4, "cuda")
    y = torch.zeros(T, N, dtype=torch.bfloat16, device="cuda")
    gemm.linear(x, w, out=y, bn=bn, cluster=cluster, comm=gemm.GemmComm(rope=gemm.RopeAppend(table, pos, slots, *caches[:2], n_q, n_kv, hd)))
    z = gemm.linear(x, w, bn=bn, cluster=cluster)
    reference.rope_kv_append(z, pos, slots, *caches[2:], n_q, n_kv, hd, 1e4)
    # the reference rotates in fp32 with its own sines: a unit of the last place of bf16
    for a, b in ((y[:, :n_q * hd], z[:, :n_q * hd]), (caches[0], caches[2]), (caches[1], caches[3])):
        torch.testing.assert_close(a.float(), b.float(), rtol=2 ** -7, atol=2 ** -7)
    assert gemm.check_status() == 0


@pytest.mark.parametrize("T,N,K,gate", [(1, 4096, 4096, False), (37, 6144, 2048, False), (64, 32000, 512, False), (65, 2816, 1024, True),
                                        (300, 2048, 1096, False), (1111, 1024, 256, False), (37, 2048, 2048, False), (96, 1024, 4096, False),
                                        (200, 2048, 4096, False), (65, 1408, 2048, True), (150, 704, 4096, True), (20, 256, 11008, False)])
def test_chosen_plan_agrees_with_the_other_kernels(T, N, K, gate):
    torch.manual_seed(N)
    assert gemm.split_plan(T, N, K, gemm.EPI_SWIGLU if gate else gemm.EPI_PLAIN, gemm.num_sms("cuda"),
                           gemm.split_ctas(torch.device("cuda"))) is not None
    x, w = _bf(T, K), _bf(2 * N if gate else N, K) * K ** -0.5
    y, z = (gemm.swiglu_linear(x, w), gemm.swiglu_linear(x, w, wide=False)) if gate else (gemm.linear(x, w), gemm.linear(x, w, wide=False))
    torch.testing.assert_close(y.float(), z.float(), rtol=2 ** -7, atol=2 ** -9)      # two roundings of nearly equal sums
    assert gemm.check_status() == 0


def test_rule_and_kernel_agree_on_what_the_device_holds():
    """The rule counts waves with the driver's answers; an answer that the driver does not give is no error of a later launch."""
    small, large = gemm.split_ctas(torch.device("cuda"))
    sms = gemm.num_sms("cuda")
    assert small[0] == 2 * sms and large[0] == sms
    for n in range(1, 9):
        assert sms // 2 < large[n - 1] <= sms and large[n - 1] % n == 0 and sms < small[n - 1] <= 2 * sms and small[n - 1] % n == 0
    from disagmoe_b200.ops import _lib
    assert [_lib.lib().dmoe_gemm_split_ctas(n, 1) for n in (0, 9, -1)] == [0, 0, 0]
    x, w = _bf(4, 64), _bf(8, 64)
    _close(gemm.linear(x, w), x.double() @ w.double().T, 64 * 64)


@pytest.mark.parametrize("T", [1, 37, 300])
def test_tile_of_its_own_choice(T):
    x, w, w13 = _bf(T, 520), _bf(264, 520), _bf(528, 520)
    bn = min(-(-T // 16) * 16, 128)
    assert torch.equal(gemm.linear(x, w, cluster=3), gemm.linear(x, w, bn=bn, cluster=3))
    assert torch.equal(gemm.swiglu_linear(x, w13, cluster=3), gemm.swiglu_linear(x, w13, bn=bn, cluster=3))
    for S in range(1, 9):                                  # the widest tile that every cluster takes
        _close(gemm.linear(x, w, bn=256 if S < 5 else 240, cluster=S, out_dtype=torch.float32), x.double() @ w.double().T, 520 * 520, bits=20)


def test_launch_that_does_not_qualify():
    """Rows that do not move 16 bytes at a time keep the kernel that stores them one by one."""
    x, w = _bf(9, 128), _bf(20, 128)
    _close(gemm.linear(x, w, bn=16, cluster=2, out_dtype=torch.float32), x.double() @ w.double().T, 128 * 128, bits=20)


LATE = """
import torch
from disagmoe_b200.ops import _lib, functional as F, gemm
bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
z = lambda n: torch.zeros(n, dtype=torch.int32, device="cuda")
x, w, resid, dst, status = bf(37, 512), bf(1024, 512), bf(4, 256), bf(4, 256), z(1)
ptr, flags, epoch, ticket = torch.tensor([dst.data_ptr()], device="cuda"), z(1), z(1), z(1)
want = [gemm.linear(x, w, bn=48, cluster=c) for c in (1, 4)]
_lib.lib().dmoe_set_flag_wait_cycles(2_300_000_000)
for c, y in zip((1, 4), want):
    status.zero_()
    torch.cuda.synchronize()
    F.norm_gather(resid, None, bf(256), 1e-6, None, ptr, 1, 0, 256, 4, 256, wait_flags=flags, n_wait=1, wait_epoch=epoch, ticket=ticket, status=status)
    got = gemm.linear(x, w, bn=48, cluster=c)
    assert int(status) == 2 and gemm.check_status() == 0 and torch.equal(got, y), (c, int(status))
"""


def test_limits_count_from_the_end_of_the_launch_before():
    """Started while its predecessor still waits for a peer (here for a flag that nothing sets, until its own limit of 1.2 s), the kernel
    does not count that time against its barriers' limits of a second."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", LATE], env={**os.environ, "DMOE_PDL": "1", "PYTHONPATH": root}, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
