"""What a step leaves behind is complete for other streams and for the host, also when the GPU is far behind."""
import pytest
import torch

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
