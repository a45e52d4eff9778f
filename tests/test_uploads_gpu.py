"""Host tables of a step in one copy: places, alignment, tables that do not fit the room that is left."""
import numpy as np
import pytest
import torch

from disagmoe_b200.ops import _lib
from disagmoe_b200.ops._lib import Uploads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("room", [4, 64, 1 << 14])
def test_tables_arrive(room):
    rng = np.random.default_rng(room)
    arrays = [rng.integers(-2 ** 31, 2 ** 31, shape, dtype=np.int32) for shape in ((1,), (7, 4), (0,), (33,), (5, 2), (300,), (2,))]
    arrays.append(np.arange(24, dtype=np.int32).reshape(6, 4)[:, 1])                 # not contiguous
    up = Uploads("cuda", room)
    views = [up(a) for a in arrays]
    up.flush()
    for a, t in zip(arrays, views):
        assert t.shape == a.shape and t.is_contiguous() and (a.size == 0 or t.data_ptr() % 16 == 0)
        assert torch.equal(t.cpu(), torch.from_numpy(np.ascontiguousarray(a)))
    again = up(arrays[1])                                                             # after a flush: memory of its own
    up.flush()
    assert torch.equal(again.cpu(), views[1].cpu()) and again.data_ptr() != views[1].data_ptr()


def test_a_second_step_of_the_same_size_is_one_copy(monkeypatch):
    """Three tables that together need more room than the first step has, each less; then small steps, after which the room is small again."""
    from disagmoe_b200.executor.step import StepExecutor
    least = 1 << 14
    copies, rooms, flush, init = [], [], Uploads.flush, Uploads.__init__

    def flushed(up):
        copies[-1] += up.at > 0
        flush(up)

    def made(up, device, ints):
        rooms.append(ints)
        init(up, device, ints)
    monkeypatch.setattr(_lib.Uploads, "flush", flushed)
    monkeypatch.setattr(_lib.Uploads, "__init__", made)
    ids, sizes = torch.zeros(4, dtype=torch.int32), []

    class Tables(StepExecutor):
        def __init__(self):
            self.device, self.table_ints = torch.device("cuda"), least
            self.prefill_buf = type("Buffers", (), dict(cap=4, copied=None, out_rows=None))()

        def _fill(self, *a):
            pass

        def _begin_prefill(self, buf, T, positions, ctx_len, bt_row, up):
            for n in sizes:
                up(np.zeros(n, dtype=np.int32))

        def _forward(self, *a):
            pass
    ex = Tables()
    for sizes in [[6001, 9000, 9001]] * 2 + [[10]] * 3:
        copies.append(0)
        ex.prefill(ids, ids, ids, ids, ids, out_rows=[0])
    assert copies == [2, 1, 1, 1, 1] and rooms[1] == 6004 + 9000 + 9004 + 4 and rooms[-1] == least
