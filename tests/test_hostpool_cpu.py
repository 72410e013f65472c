"""Result buffers on the host: a block is used again only when the last tensor over it is gone, and what waits is bounded."""
import gc
import os

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


def _address_again(shape=(1 << 20,)):
    return _hostpool.empty(shape, torch.float32).data_ptr()


@pytest.mark.parametrize("hold", [lambda t: t.untyped_storage(), lambda t: t[5:9], lambda t: t.numpy(), lambda t: memoryview(t.numpy()),
                                  lambda t: torch.utils.dlpack.to_dlpack(t), lambda t: (t.requires_grad_() * 2).sum()])
def test_held_in_other_ways(hold):
    a = _hostpool.empty((1 << 20,), torch.float32).fill_(1)
    at, held = a.data_ptr(), hold(a)
    del a
    assert _address_again() != at
    del held
    gc.collect()


def test_a_result_is_an_ordinary_tensor():
    a = _hostpool.empty((1 << 20,), torch.float32).fill_(1)
    assert not a._is_view() and not a.is_pinned()
    assert torch.equal(a.resize_(3 << 20)[:1 << 20], torch.ones(1 << 20))   # grown in place
    at = a.data_ptr()
    del a
    assert _hostpool.empty((1 << 20,), torch.float32).untyped_storage().nbytes() == 4 << 20
    b = _hostpool.empty((2 << 20,), torch.float32).fill_(2).share_memory_()
    shared = b.data_ptr()
    del b
    assert _hostpool.empty((2 << 20,), torch.float32).data_ptr() != shared
    c = _hostpool.empty((1 << 20,), torch.float32)
    del c
    d = _hostpool.empty((1 << 20,), torch.float32)
    assert d.untyped_storage().resizable() and not d.untyped_storage().is_shared() and d.data_ptr() != at


def test_private_after_a_fork():
    """What a child process writes stays its own, and what it reads does not change when the parent goes on."""
    a = _hostpool.empty((1 << 20,), torch.float32).fill_(1)
    del a
    a = _hostpool.empty((1 << 20,), torch.float32).fill_(1)   # memory that has been handed out before
    at = a.data_ptr()
    to_child, to_parent = os.pipe(), os.pipe()
    pid = os.fork()
    if pid == 0:
        a[:10] = 7
        os.write(to_parent[1], b"w")
        os.read(to_child[0], 1)
        os._exit(0 if float(a[10]) == 1 and float(a[9]) == 7 else 1)
    os.read(to_parent[0], 1)
    same = bool((a == 1).all())
    del a
    b = _hostpool.empty((1 << 20,), torch.float32).fill_(3)
    os.write(to_child[1], b"w")
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0 and same and b.data_ptr() == at


def test_allocates_what_it_returns(monkeypatch):
    """A new block makes no allocation but its own, once given back: the heap's policy follows the results' sizes."""
    sizes, empty = [], torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: sizes.append(a[0]) or empty(*a, **k))
    monkeypatch.setattr(_hostpool, "_adapted", False, raising=False)
    _hostpool.empty((1 << 20,), torch.float32)
    assert sorted(sizes) == [0, 4 << 20, 4 << 20]
