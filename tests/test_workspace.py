"""The workspace that parts take their scratch buffers from."""
import pytest
import torch

from cpi_b200.parts import Workspace


@pytest.mark.parametrize("shape", [(2, 3), [2, 3], torch.Size([2, 3]), range(2, 4)])
def test_a_shape_is_any_sequence_of_sizes(shape):
    ws = Workspace("cpu")
    for _ in range(2):
        assert ws.get("a", shape, torch.float32).shape == (2, 3)
    assert ws.get("a", [4], torch.float32).data_ptr() == ws.get("a", (2, 2), torch.float32).data_ptr()


def test_views_follow_a_buffer_that_grew():
    ws = Workspace("cpu")
    small, other = ws.get("a", (4,), torch.float32), ws.get("b", (4,), torch.float32)
    assert ws.get("a", (4,), torch.float32).data_ptr() == small.data_ptr()
    assert ws.get("a", (4,), torch.float32) is ws.get("a", (4,), torch.float32)
    before = ws.generation
    ws.get("a", (8, 2), torch.float32).fill_(1)
    assert ws.generation == before + 1
    again = ws.get("a", (4,), torch.float32)
    assert again.data_ptr() == ws.get("a", (8, 2), torch.float32).data_ptr() != small.data_ptr() and bool((again == 1).all())
    assert ws.get("b", (4,), torch.float32).data_ptr() == other.data_ptr()


def test_views_of_many_shapes_stay_right():
    ws = Workspace("cpu")
    for i in range(3000):
        assert ws.get("a", (1 + i % 1500, 2), torch.float32).shape == (1 + i % 1500, 2)


def test_scratch_is_not_kept_and_moves_no_buffer():
    ws = Workspace("cpu")
    ws.get("a", (4,), torch.float32)
    before = ws.generation
    for n in (1, 5, 97, 1000, 4097):
        t = ws.scratch(n, torch.float32)
        assert t.shape == (n,) and n * 4 <= t.untyped_storage().nbytes() <= max(8, 4 * (3 * n // 2 + 2))
    assert ws.generation == before and len(ws._buffers) == 1


def test_scratch_without_room_is_none(monkeypatch):
    """Where the allocator has no room, nothing is raised, and for a while nothing of that size is asked for again."""
    ws, asked, empty = Workspace("cpu"), [], torch.empty

    def full(size, **kw):
        asked.append(size)
        if size > 1024:
            raise torch.OutOfMemoryError("no room")
        return empty(size, **kw)
    monkeypatch.setattr(torch, "empty", full)
    assert ws.scratch(2000, torch.float32) is None and ws.scratch(2000, torch.float32) is None and ws.scratch(9000, torch.float32) is None
    assert asked == [2048] and ws.scratch(1000, torch.float32).numel() == 1000
    monkeypatch.setattr(torch, "empty", empty)
    got = [ws.scratch(2000, torch.float32) is not None for _ in range(80)]
    assert not got[0] and got[-1]
