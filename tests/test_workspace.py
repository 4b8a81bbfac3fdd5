"""The engine's work buffers: one per name and row shape, kept views, any sequence as a shape."""

import torch

from freetoken_b200.parts import Workspace


def test_buffers_and_views():
    ws = Workspace(torch.device("cpu"))
    a = ws.get("x", (3, 4), torch.float32, (10, 4))
    assert a.shape == (3, 4) and ws.nbytes() == 160
    assert ws.get("x", [3, 4], torch.float32, (10, 4)).data_ptr() == a.data_ptr()  # (a list too)
    assert ws.get("x", torch.Size((10, 4)), torch.float32).data_ptr() == a.data_ptr()
    assert ws.get("x", (3, 5), torch.float32).data_ptr() != a.data_ptr()  # another row shape: a buffer of its own
    b = ws.get("x", (12, 4), torch.float32)  # more than there was room for
    assert ws.get("x", (3, 4), torch.float32).data_ptr() == b.data_ptr()  # no view of the buffer before is handed out
    assert ws.get("x", (3, 4), torch.int32).dtype == torch.int32
    for n in range(3000):  # (steps of ever other lengths: views are bounded)
        ws.get("y", (n,), torch.uint8, (3000,))
    assert len(ws._views) <= 1024 and ws.get("y", (2999,), torch.uint8).shape == (2999,)
