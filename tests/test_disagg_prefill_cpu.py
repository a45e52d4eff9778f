"""Prompt tiles of a disaggregated attention rank: what the attention call gets (no GPU; launches are recorded)."""
from types import SimpleNamespace

import torch

from disagmoe_b200.ops import functional as F
from disagmoe_b200.ops import gemm
from disagmoe_b200.parallel.disagg import AttentionRank


def test_prompt_attention_knows_its_reach(monkeypatch):
    """Without the longest context the call would stay on another kernel than the one that the colocated executor takes for the same
    prompts, and differ from it on ties of bf16. Decode rows with longer contexts do not count."""
    z = lambda *s: torch.zeros(*s, dtype=torch.int32)
    layer = SimpleNamespace(num_heads=4, num_kv_heads=2, head_dim=8, q_size=32, qkv_w=None, o_w=None)
    mb = [dict(pre_tiles=z(400, 4), ctx_dec=z(400), ctx_len=z(400), positions=z(400), slots=z(400), bt_row=z(400), hs=torch.zeros(400, 32),
               qkv=torch.zeros(400, 64), attn=torch.zeros(400, 32), resid=torch.zeros(400, 32)) for _ in range(2)]
    cfg = SimpleNamespace(max_seq_len=1024)
    rank = SimpleNamespace(layers=[layer], l0=0, mb=mb, n_pre=[0, 0], reach=[0, 0], active=[230, 230], tp=1, tp_rank=0, shape=None, cfg=cfg,
                           kv_cache=torch.zeros(1, 2, 4, 16, 2, 8), block_tables=z(8, 64), block_size=16, rope=None)
    rank.rows = lambda m: (rank.active[m], rank.active[m], 0, rank.active[m])
    rank._meta = lambda m: AttentionRank._meta(rank, m)
    seen = []
    monkeypatch.setattr(F, "prefill_attention", lambda *a, reach=None, **k: seen.append(reach))
    monkeypatch.setattr(F, "paged_attention", lambda *a, **k: None)
    monkeypatch.setattr(F, "pick_attn_splits", lambda *a: 1)
    monkeypatch.setattr(gemm, "linear", lambda *a, **k: None)
    monkeypatch.setattr(gemm, "RopeAppend", lambda *a: None)
    pos = torch.cat([torch.tensor([900, 700]), torch.arange(60, 260), torch.arange(28)])      # two decode rows, two prompts
    rows = torch.cat([torch.tensor([0, 1]), torch.full((200,), 2), torch.full((28,), 3)])
    assert AttentionRank.set_prefill_tiles(rank, 1, rows, pos, pos + 1) > 0
    AttentionRank.layer_attn(rank, 0, 1)
    assert seen == [260] and mb[1]["ctx_dec"][:3].tolist() == [901, 701, 0]
    AttentionRank.layer_attn(rank, 0, 0)                                                      # the other micro-batch has no tiles
    AttentionRank.set_prefill_tiles(rank, 1, None, None, None)
    AttentionRank.layer_attn(rank, 0, 1)
    assert seen == [260]
