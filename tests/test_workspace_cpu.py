"""A workspace hands out the view it handed out last for the same name, type and shape, and one on the buffer as it is now for another shape."""
import pytest
import torch

from arle_b200.engine.batch import Workspace


def test_views_are_kept_and_follow_their_buffer():
    ws = Workspace("cpu")
    a = ws.get("x", (2, 3), torch.float32)
    assert ws.get("x", (2, 3), torch.float32) is a and ws.generation == 1
    b = ws.get("x", (3, 2), torch.float32)
    assert b.shape == (3, 2) and b.data_ptr() == a.data_ptr() and ws.get("x", (2, 3), torch.float32).shape == (2, 3)
    assert ws.get("x", (2, 3), torch.bfloat16).dtype == torch.bfloat16 and ws.get("y", (2, 3), torch.float32).data_ptr() != a.data_ptr()
    big = ws.get("x", (8, 8), torch.float32)                    # another buffer: no view of the old one comes back
    small = ws.get("x", (2, 3), torch.float32)
    assert small.data_ptr() == big.data_ptr() and small is not a
    ws.frozen = True
    assert ws.get("x", (2, 3), torch.float32) is small
    with pytest.raises(RuntimeError):
        ws.get("x", (9, 9), torch.float32)
    z = Workspace("cpu").get_zeroed("f", (4,), torch.int32)
    assert (z == 0).all()
