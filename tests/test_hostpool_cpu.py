"""Result buffers on the host: a block is used again only when the last tensor over it is gone, and what waits is bounded."""
import pytest
import torch

from trspmm import _hostpool


@pytest.fixture(autouse=True)
def clean():
    _hostpool.release()
    yield
    _hostpool.release()


@pytest.mark.parametrize("shape,dtype", [((3,), torch.float32), ((1 << 18, 1), torch.float32), ((1 << 20,), torch.int8),
                                         ((3 << 19, 2), torch.float16), ((0, 4), torch.int64), ((1 << 18,), torch.int64)])
def test_shapes_and_types(shape, dtype):
    t = _hostpool.empty(shape, dtype)
    assert t.shape == torch.Size(shape) and t.dtype == dtype and t.is_contiguous() and t.device.type == "cpu"
    assert torch.equal(t.fill_(1), torch.ones(shape, dtype=dtype))


def test_blocks_in_use_are_left_alone():
    a = _hostpool.empty((1 << 20,), torch.float32).fill_(1)
    at, view = a.data_ptr(), a[100:200]
    del a
    b = _hostpool.empty((1 << 20,), torch.float32).fill_(2)
    assert b.data_ptr() != at and bool((view == 1).all())
    del view
    c = _hostpool.empty((1 << 20,), torch.float32)
    assert c.data_ptr() == at


def test_waiting_memory_is_bounded(monkeypatch):
    monkeypatch.setattr(_hostpool, "KEEP_BYTES", 8 << 20)
    held = [_hostpool.empty((1 << 20,), torch.float32) for _ in range(4)]
    held.clear()
    assert sum(b.bytes for b in _hostpool._idle) <= 8 << 20
    assert _hostpool.empty((3 << 20,), torch.float32).numel() == 3 << 20   # beyond the bound: ordinary memory
