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


def test_cuts_are_kept_as_long_as_their_view():
    ws = Workspace("cpu")
    a = ws.get("x", (2, 6), torch.float32)
    left = ws.cut("x", a, 0, 2)
    assert ws.cut("x", a, 0, 2) is left and torch.equal(left, a[:, :2]) and left.data_ptr() == a.data_ptr()
    assert ws.cut("x", a, 2, 6).stride() == a[:, 2:].stride() and ws.cut("x", a, 2, 6).data_ptr() == a[:, 2:].data_ptr()
    b = ws.get("x", (3, 4), torch.float32)
    assert ws.cut("x", b, 0, 2).shape == (3, 2) and ws.cut("x", a, 0, 2).shape == (2, 2) and ws.cut("x", a, 0, 2) is not left
    big = ws.get("x", (50, 4), torch.float32)                   # another buffer
    assert ws.cut("x", big, 1, 3).data_ptr() == big[:, 1:].data_ptr() and ws.cut("x", b, 0, 2).data_ptr() == b.data_ptr()
    z = ws.get_zeroed("z", (2, 4), torch.float32)
    kept = ws.cut("z", z, 0, 2)
    y = ws.get_zeroed("z", (4, 4), torch.float32)
    assert ws.cut("z", y, 0, 2).shape == (4, 2) and ws.cut("z", z, 0, 2) is not kept
    assert ws.cut("unknown", a, 0, 1).shape == (2, 1)
