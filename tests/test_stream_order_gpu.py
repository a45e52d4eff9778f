"""What a step leaves behind is complete for other streams and for the host, also when the GPU is far behind."""
import pytest
import torch

from disagmoe_b200.config import CacheConfig, tiny_config
from disagmoe_b200.models.registry import make_executor, supinex_config_from_json
from disagmoe_b200.ops import gemm
from oracles import parallel_stack as oracle
from parallel_block_util import MODELS, make_engine

pytestmark = pytest.mark.gpu


def _busy():
    torch.cuda._sleep(400_000_000)      # about 0.2 s of the current stream


def test_kept_decode_tables_are_complete_for_every_stream():
    """The tables of a batch size are made by whichever stream needs them first and then serve all of them."""
    raw = MODELS["even"]
    ex = make_engine(raw, oracle.random_weights(raw, seed=3), "cuda", torch.bfloat16).executor
    flat = lambda tables: [x for t in tables[0].values() for x in (t.offs, t.recs)] + list(tables[1].values())
    want = [t.cpu() for t in flat(ex._decode_tables(5))]
    ex.decode_tables.clear()
    first, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        junk = [torch.full((n,), -7, dtype=torch.int32, device="cuda") for n in (8, 16, 64, 256) for _ in range(50)]
        torch.cuda.synchronize()
        del junk
        _busy()
        tables = flat(ex._decode_tables(5))
    with torch.cuda.stream(other):
        got = [t.clone() for t in tables]
    torch.cuda.synchronize()
    assert all(torch.equal(g.cpu(), w) for g, w in zip(got, want))


@pytest.mark.parametrize("kind", ["fused", "layer_list"])
def test_inputs_are_free_when_prefill_returns(kind):
    """A caller may refill its pinned inputs as soon as the call is back, whatever is still queued before it."""
    n = 40
    if kind == "fused":
        cfg = tiny_config.clone(dtype=torch.bfloat16)
        ex = make_executor(cfg, CacheConfig(block_size=16), device="cuda", max_batch_size=2, max_prefill_tokens=64, num_blocks=8)
    else:
        raw = MODELS["even"]
        cfg = supinex_config_from_json(raw, {}, dtype=torch.bfloat16, max_seq_len=64)
        ex = make_executor(cfg, CacheConfig(block_size=16), device="cuda", max_batch_size=2, max_prefill_tokens=64, num_blocks=8,
                           state_dict=oracle.random_weights(raw, seed=3), dtype=torch.bfloat16)
    ex.set_block_table_row(0, [3, 1, 2])
    pos = torch.arange(n)
    page = torch.tensor([3, 1, 2])
    ids = (pos * 7 + 1) % cfg.vocab_size
    args = [t.pin_memory() for t in (ids.int(), pos.int(), page[pos // 16] * 16 + pos % 16, (pos + 1).int(), torch.zeros(n).int())]
    want = ex.prefill(*args, want_logits=True, out_rows=[n - 1])[1].clone()
    torch.cuda.synchronize()
    _busy()
    got = ex.prefill(*args, want_logits=True, out_rows=[n - 1])[1]
    args[0].zero_()
    got = got.clone()
    torch.cuda.synchronize()
    torch.testing.assert_close(got, want)
    assert gemm.check_status() == 0
