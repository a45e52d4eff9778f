"""Host tables of a step in one copy: places, alignment, tables that do not fit the room that is left."""
import numpy as np
import pytest
import torch

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
