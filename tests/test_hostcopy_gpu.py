"""Copies between pageable host arrays and the device: sizes around a chunk and around the whole pinned ring, many
arrays in one call, two threads at once."""
import subprocess
import sys
import threading

import pytest
import torch

from trspmm import _lib

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.mark.parametrize("sizes", [[1], [MB // 2 - 1], [MB - 1], [MB], [MB + 1], [31 * MB + 7], [32 * MB], [33 * MB + 1], [80 * MB + 5],
                                   [0, 3, 5 * MB + 1, 0, MB, 17, 2 * MB - 1]])
def test_round_trip(sizes):
    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(sum(sizes))
    host = [torch.randint(0, 256, (n,), generator=g, dtype=torch.uint8) for n in sizes]
    up = _lib.copy_to_device(host, dev)
    for a, b in zip(up, host):
        assert torch.equal(a, b.cuda())
    for a, b in zip(_lib.copy_to_host(up, dev), host):
        assert torch.equal(a, b)


def test_results_in_reused_blocks():
    """Result blocks are used again and stay ordinary memory, beside small arrays that are not pooled."""
    from trspmm import _hostpool
    dev = torch.device("cuda", 0)
    _hostpool.release()
    src = [torch.arange(n, dtype=torch.int32, device=dev) for n in (3 * MB, 100, MB // 8, 2 * MB + 3)]
    for k in range(4):
        got = _lib.copy_to_host([s + k for s in src], dev)
        for a, b in zip(got, src):
            assert torch.equal(a, (b + k).cpu())
        assert not any(t.is_pinned() for t in got)
        del got, a
    _hostpool.release()


def test_results_beyond_the_pool():
    """More than the pool keeps, in one array and in several."""
    from trspmm import _hostpool
    dev = torch.device("cuda", 0)
    _hostpool.release()
    src = [torch.arange(n, dtype=torch.int32, device=dev) for n in (70 * MB + 3, 30 * MB, 30 * MB + 1, 20 * MB)]
    for k in range(2):
        got = _lib.copy_to_host([s + k for s in src], dev)
        for a, b in zip(got, src):
            assert torch.equal(a, (b + k).cpu())
        assert sum(b.bytes for b in _hostpool._idle) <= _hostpool.KEEP_BYTES
    _hostpool.release()


def test_result_dropped_while_it_is_copied():
    """A caller queues a copy of a result behind work on a stream of its own and drops the result: the next results
    must not reach the copy."""
    dev = torch.device("cuda", 0)
    side, src, copies = torch.cuda.Stream(), torch.arange(4 * MB, dtype=torch.int32, device=dev), []
    for k in range(6):
        got = _lib.copy_to_host([src + k], dev)
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)
            copies.append(got[0].to(dev, non_blocking=True))
        del got
    torch.cuda.synchronize()
    for k, c in enumerate(copies):
        assert torch.equal(c, src + k)


def test_page_locked_arrays():
    """Arrays that the caller has page-locked, as torch does or through the library, beside pageable ones."""
    dev, lib = torch.device("cuda", 0), _lib.load()
    host = [torch.arange(n, dtype=torch.int32) for n in (MB, 2 * MB + 5, 100)]
    host[0] = host[0].pin_memory()
    _lib.check(lib.trs_host_register(host[1].data_ptr(), host[1].numel() * 4))
    for a, b in zip(_lib.copy_to_device(host, dev), host):
        assert torch.equal(a, b.cuda())
    _lib.check(lib.trs_host_unregister(host[1].data_ptr()))


@pytest.mark.parametrize("n", [100, MB // 8 - 1, MB // 8])
def test_page_locked_array_written_after_the_upload(n):
    """An upload has read its arrays when it returns, small page-locked ones behind earlier work too."""
    dev = torch.device("cuda", 0)
    host = torch.arange(n, dtype=torch.int32).pin_memory()
    torch.cuda._sleep(50_000_000)
    up = _lib.copy_to_device([host], dev)[0]
    host.zero_()
    assert torch.equal(up.cpu(), torch.arange(n, dtype=torch.int32))


def test_two_threads():
    dev = torch.device("cuda", 0)
    data = [torch.arange(9 * MB + i, dtype=torch.int32) for i in range(2)]
    bad = []

    def go(i):
        for _ in range(5):
            if not torch.equal(_lib.copy_to_host(_lib.copy_to_device([data[i]], dev), dev)[0], data[i]):
                bad.append(i)

    threads = [threading.Thread(target=go, args=(i,)) for i in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
    assert _lib.load().trs_pool_trim() == 0
    assert torch.equal(_lib.copy_to_host([data[0].cuda()], dev)[0], data[0])   # the ring comes back after a trim


def test_no_threads_to_be_had():
    """Where the system gives no threads, copies and the host entries go without.  (A child process whose default thread
    stack is larger than the address space.)"""
    code = """
import ctypes, sys
sys.path[:0] = [%r, %r]
import torch
from trspmm import SpmmPlan, _lib, build_format, graphs, spmm_forward_host
rp, col, val = graphs.uniform_graph(1 << 15, 8, seed=1, device="cuda")
n = rp.numel() - 1
fmt = build_format(rp, col, val)[0]
B = torch.randn(n, 64).half()
want = SpmmPlan(fmt, n, n).run(B.cuda(), out_dtype=torch.float32).cpu()
host = fmt.half_values().to("cpu")
torch.cuda.synchronize()
libc, attr = ctypes.CDLL(None), ctypes.create_string_buffer(256)
assert libc.pthread_attr_init(attr) == 0
assert libc.pthread_attr_setstacksize(attr, ctypes.c_size_t(1 << 48)) == 0
assert libc.pthread_setattr_default_np(attr) == 0
data = torch.arange(3 << 20, dtype=torch.int32)
dev = torch.device("cuda", 0)
assert torch.equal(_lib.copy_to_host(_lib.copy_to_device([data], dev), dev)[0], data)
assert torch.equal(spmm_forward_host(host, B, 64, n, n)[0], want)
print("done")
""" % (str(_lib.PKG_ROOT), str(_lib.PKG_ROOT.parent))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "done", r.stderr[-2000:]
