"""SDDMM at widths around the kernels' 32-feature chunks (planned: up to 256 in registers; entry-parallel beyond), rows
off 16-byte boundaries, and patterns with long runs of empty rows."""
import pytest
import torch

from oracle import oracle as O
from trspmm import SddmmPlan, TrsError, graphs, sddmm

pytestmark = pytest.mark.gpu


def _pattern(kind):
    if kind == "rmat":
        return graphs.rmat_graph(10, 12, seed=4)[:2]
    g = torch.Generator().manual_seed(6)                       # 5000 rows, a few of them with entries
    rows = torch.randint(0, 40, (3000,), generator=g) * 123
    return graphs.coo_to_csr(rows, torch.randint(0, 700, (3000,), generator=g), 5000, 700)[:2]


@pytest.mark.parametrize("kind", ["rmat", "gaps"])
@pytest.mark.parametrize("K", [1, 8, 31, 32, 33, 48, 72, 96, 100, 127, 128, 136, 160, 192, 200, 224, 256, 264, 300])
def test_widths(kind, K):
    rp, col = _pattern(kind)
    n, m = rp.numel() - 1, 1024 if kind == "rmat" else 700
    g = torch.Generator().manual_seed(K)
    X, Y = torch.randn(n, K, generator=g).half(), torch.randn(m, K, generator=g).half()
    ref = O.sddmm_csr(rp, col, X, Y).float()
    scale = float(ref.abs().max())
    rp, col, X, Y = rp.cuda(), col.cuda(), X.cuda(), Y.cuda()
    plan = SddmmPlan(rp, col, m)
    for run in (lambda out: sddmm(rp, col, X, Y, out=out), lambda out: plan.run(X, Y, out=out)):
        out = run(torch.full((col.numel(),), float("nan"), dtype=torch.float16, device="cuda")).float().cpu()
        assert float((out - ref).abs().max()) <= 2e-3 * scale
    assert torch.equal(plan.run(X, Y, out_dtype=torch.float32), plan.run(X, Y).float())
    base = torch.empty(n * K + 8, dtype=torch.float16, device="cuda")   # X one element off its boundary
    Xo = base[1:1 + n * K].view(n, K).copy_(X)
    assert torch.equal(plan.run(Xo, Y), plan.run(X, Y)) and torch.equal(sddmm(rp, col, Xo, Y), sddmm(rp, col, X, Y))


def test_plan_refuses_decreasing_row_pointers():
    rp = torch.tensor([0, 40, 20] + [60] * 30, dtype=torch.int32)
    col = torch.arange(60, dtype=torch.int32)
    with pytest.raises(TrsError) as e:
        SddmmPlan(rp.cuda(), col.cuda(), 64)
    assert e.value.code == -3


def test_results_are_vectors():
    """Columns given as a matrix of one column, as COO files have them."""
    rp, col = (t.cuda() for t in _pattern("rmat"))
    X = torch.randn(1024, 32, generator=torch.Generator().manual_seed(1)).half().cuda()
    for run in (lambda c: sddmm(rp, c, X, X), lambda c: SddmmPlan(rp, c, 1024).run(X, X),
                lambda c: SddmmPlan(rp, c, 1024).run(X, X, out_dtype=torch.float32)):
        assert run(col[:, None]).shape == (col.numel(),)
        assert torch.equal(run(col[:, None]), run(col))


@pytest.mark.parametrize("K", [32, 47, 64, 300])
def test_under_capture(K):
    """A plan's product can be captured at any width, with the copies that some of them make of X and Y."""
    rp, col = (t.cuda() for t in _pattern("rmat"))
    plan = SddmmPlan(rp, col, 1024)
    g = torch.Generator().manual_seed(K)
    X, Y = (torch.randn(1024, K, generator=g).half().cuda() for _ in range(2))
    want = plan.run(X, Y)
    out = torch.zeros_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run(X, Y, out=out)
    for scale in (1, 2, 4):
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want * scale)
        X *= 2


def test_as_many_entries_as_an_int_counts():
    """2^31 - 1 entries: the last step of the entry-parallel kernel ends at the last one."""
    n, K, nnz = 1 << 16, 8, 2 ** 31 - 1
    if torch.cuda.mem_get_info()[0] < 20 << 30:
        pytest.skip("needs 20 GB")
    rp = torch.arange(n + 1, dtype=torch.int64) << 15
    rp[-1] = nnz
    col = torch.arange(nnz, dtype=torch.int32, device="cuda").bitwise_and_(1023)
    g = torch.Generator().manual_seed(3)
    X, Y = torch.randn(n, K, generator=g).half(), torch.randn(1024, K, generator=g).half()
    out = sddmm(rp.to(torch.int32).cuda(), col, X.cuda(), Y.cuda())
    at = torch.cat([torch.arange(nnz - 70, nnz), torch.arange(70), torch.randint(nnz, (1000,), generator=g)])
    want = (X.float()[at >> 15] * Y.float()[at & 1023]).sum(1)
    assert float((out[at.cuda()].float().cpu() - want).abs().max()) <= 2e-3 * float(want.abs().max())


@pytest.mark.parametrize("K", [3, 47, 300])
def test_no_memory_for_copies(K):
    """Rows off 16-byte boundaries where the GPU has no room for padded copies of them."""
    from trspmm import _lib
    n = 1 << 21
    rp, col = (t.cuda() for t in graphs.coo_to_csr(torch.arange(0, n, 5), torch.arange(0, n, 5).flip(0), n, n)[:2])
    X, Y = (torch.randn(n, K, device="cuda", dtype=torch.float16) for _ in range(2))
    plan = SddmmPlan(rp, col, n)
    want = sddmm(rp, col, X, Y)
    out = [torch.empty_like(want) for _ in range(2)]
    torch.cuda.empty_cache()
    _lib.check(_lib.load().trs_pool_trim())
    hog = [torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")]
    while True:
        try:
            hog.append(torch.empty(4 << 20, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            break
    try:
        sddmm(rp, col, X, Y, out=out[0])
        plan.run(X, Y, out=out[1])
        torch.cuda.synchronize()
    finally:
        del hog
        torch.cuda.empty_cache()
    scale = float(want.abs().max())
    for o in out:
        assert float((o.float() - want.float()).abs().max()) <= 2e-3 * scale


def test_windows_beyond_the_entry_lists():
    """A window with more entries than the lists of a plan can place runs the entry-parallel kernel."""
    n_cols, K = 600_000, 16
    rp = torch.arange(33, dtype=torch.int32) * n_cols
    rp[17:] = rp[16] + torch.arange(16, dtype=torch.int32)
    col = torch.cat([torch.arange(n_cols, dtype=torch.int32).repeat(16), torch.arange(15, dtype=torch.int32)]).cuda()
    rp = rp.cuda()
    g = torch.Generator().manual_seed(7)
    X, Y = torch.randn(32, K, generator=g).half().cuda(), torch.randn(n_cols, K, generator=g).half().cuda()
    plan = SddmmPlan(rp, col, n_cols)
    want = torch.cat([(X[:16].float() @ Y.float().T).flatten(), (X[17:].float() * Y[:15].float()).sum(1)])
    for dtype in (torch.float16, torch.float32):
        got = plan.run(X, Y, out_dtype=dtype).float()
        assert float((got - want).abs().max()) <= 2e-3 * float(want.abs().max())
    assert torch.equal(plan.run(X, Y), sddmm(rp, col, X, Y))


@pytest.mark.parametrize("K", [24, 64, 160, 256])
@pytest.mark.parametrize("shape", ["hubs first", "hubs last", "even", "one window"])
def test_shares_of_equal_cost(shape, K):
    """Patterns whose quads cost the same (equal numbers per warp) and very different amounts (a table of first quads): every
    entry is written once, whichever warp has it.  The plan says which of the two it is."""
    g = torch.Generator().manual_seed(K)
    n, m = (16, 60000) if shape == "one window" else (240000, 6000)
    if shape == "one window":
        rows, cols = torch.randint(0, n, (400000,), generator=g), torch.randint(0, m, (400000,), generator=g)
    else:
        rows, cols = torch.arange(n).repeat_interleave(9), torch.randint(0, m, (9 * n,), generator=g)
        if shape != "even":
            hub = torch.arange(1600) + (n - 1600 if shape == "hubs last" else 0)
            rows = torch.cat([rows, hub.repeat_interleave(m)])
            cols = torch.cat([cols, torch.arange(m).repeat(1600)])
    rp, col = graphs.coo_to_csr(rows.cuda(), cols.cuda(), n, m)[:2]
    X, Y = torch.randn(n, K, generator=g).half().cuda(), torch.randn(m, K, generator=g).half().cuda()
    r = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
    plan = SddmmPlan(rp, col, m)
    warps, number, cost, table = _shares(plan, K)
    assert table == shape.startswith("hubs") and (number > 1.5 * cost) == table, (warps, number, cost)
    out = plan.run(X, Y, out=torch.full((col.numel(),), float("nan"), dtype=torch.float16, device="cuda")).float()
    ref = torch.empty_like(out)
    for a in range(0, col.numel(), 1 << 18):
        ref[a:a + (1 << 18)] = (X[r[a:a + (1 << 18)]].float() * Y[col[a:a + (1 << 18)].long()].float()).sum(1)
    # fp16 results (2^-11) of fp32 sums, whose order differs by less than that
    assert float((out - ref).abs().max()) <= 2e-3 * float(ref.abs().max())


def test_row_pointer_ends():
    """What the product's kernel says about the ends of the row pointers: errors, no entries, and calls from several threads and
    streams at a time, each of which gets what its own row pointers say."""
    from concurrent.futures import ThreadPoolExecutor
    rp, col = (t.cuda() for t in _pattern("rmat"))
    X = torch.randn(1024, 64, generator=torch.Generator().manual_seed(2)).half().cuda()
    want = sddmm(rp, col, X, X)
    for bad in (rp + 1, -rp):
        with pytest.raises(TrsError) as e:
            sddmm(bad, col, X, X)
        assert e.value.code == -3
    assert sddmm(torch.zeros_like(rp), col[:0], X, X).numel() == 0
    own = []   # threads 0, 3: the whole pattern; 1, 4: its first rows; 2, 5: row pointers that are an error
    for k in range(6):
        rows = 1024 if k % 3 == 0 else 100 + k
        own.append((rp[:rows + 1] + (1 if k % 3 == 2 else 0), X[:rows], want[:int(rp[rows])]))

    def calls(k):
        ptr, x, mine = own[k]
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda._sleep(100000 * k)
            for i in range(50):
                try:
                    got = sddmm(ptr, col, x, X, out=torch.zeros_like(want))
                except TrsError as e:
                    if k % 3 != 2 or e.code != -3:
                        raise
                else:
                    assert k % 3 != 2 and torch.equal(got[:mine.numel()], mine) and not got[mine.numel():].any()
        return i + 1

    torch.cuda.synchronize()
    with ThreadPoolExecutor(6) as pool:
        assert list(pool.map(calls, range(6))) == [50] * 6


def _runtime():
    """The CUDA runtime that the library and torch share: what one of them leaves as a thread's last error, the other finds."""
    import ctypes
    return ctypes.CDLL("libcudart.so.12")


def test_refused_under_capture():
    """A one-use product under capture is an error (its row pointers cannot be looked at); the error is that call's and is not
    found by a later launch."""
    rp, col = (t.cuda() for t in _pattern("rmat"))
    X = torch.randn(1024, 64, generator=torch.Generator().manual_seed(3)).half().cuda()
    want = sddmm(rp, col, X, X)
    out = torch.zeros_like(want)
    for _ in range(3):
        with pytest.raises(TrsError) as e:
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                try:
                    sddmm(rp, col, X, X, out=out)
                finally:
                    left = _runtime().cudaPeekAtLastError()
        assert e.value.code == 900 and left == 0   # cudaErrorStreamCaptureUnsupported
        assert torch.equal(sddmm(rp, col, X, X), want)
        with pytest.raises(TrsError) as e:
            sddmm(rp + 1, col, X, X)
        assert e.value.code == -3
    torch.cuda.synchronize()
    assert not out.any()


def test_error_of_an_earlier_call():
    """An error that another call left with the thread is not the product's: it runs, behind work that takes a while, and the calls
    after it get their own row pointers."""
    rp, col = (t.cuda() for t in _pattern("rmat"))
    X = torch.randn(1024, 64, generator=torch.Generator().manual_seed(4)).half().cuda()
    want, out = sddmm(rp, col, X, X), torch.zeros(col.numel(), dtype=torch.float16, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(20):
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1000000)
            assert _runtime().cudaSetDevice(4096) == 101   # cudaErrorInvalidDevice, now the thread's last error
            sddmm(rp, col, X, X, out=out)
        with pytest.raises(TrsError) as e:
            sddmm(rp + 1, col, X, X)
        assert e.value.code == -3
        stream.synchronize()
        assert torch.equal(out, want)
        out.zero_()
        torch.cuda.synchronize()


def test_no_memory_for_copies_and_no_wait():
    """The product without copies tells the row pointers' ends as it begins as well: the call does not wait for its end."""
    import time
    from trspmm import _lib
    n, K = 1 << 20, 47
    rp = torch.arange(n + 1, dtype=torch.int32, device="cuda") * 24
    col = torch.randint(0, n, (24 * n,), device="cuda", dtype=torch.int32)
    X = torch.randn(n, K, device="cuda", dtype=torch.float16)
    out = torch.empty(col.numel(), dtype=torch.float16, device="cuda")
    sddmm(rp, col, X, X, out=out)
    want = out.clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    _lib.check(_lib.load().trs_pool_trim())
    hog = [torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")]
    while True:
        try:
            hog.append(torch.empty(4 << 20, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            break
    try:
        times = []
        for _ in range(5):
            out.zero_()
            torch.cuda.synchronize()
            t = [time.perf_counter()]
            sddmm(rp, col, X, X, out=out)
            t.append(time.perf_counter())
            torch.cuda.synchronize()
            t.append(time.perf_counter())
            times.append((t[1] - t[0]) / (t[2] - t[0]))
    finally:
        del hog
        torch.cuda.empty_cache()
    assert float((out.float() - want.float()).abs().max()) <= 2e-3 * float(want.abs().max())
    assert min(times) < 0.5, times   # a tenth; all of it where the call waits for the product's end


def test_wait_behind_a_long_queue():
    """A call that waits for earlier work of its stream leaves the core to others, and is not late when the work ends."""
    import time
    rp, col = (t.cuda() for t in _pattern("rmat"))
    X = torch.randn(1024, 64, generator=torch.Generator().manual_seed(5)).half().cuda()
    want = sddmm(rp, col, X, X)
    torch.cuda.synchronize()
    for cycles in (100_000, 3_000_000, 500_000_000):   # 50 us, 2 ms, 0.3 s
        done = torch.cuda.Event()
        wall, cpu = time.perf_counter(), time.thread_time()
        torch.cuda._sleep(cycles)
        done.record()
        got = sddmm(rp, col, X, X)
        wall, cpu = time.perf_counter() - wall, time.thread_time() - cpu
        assert done.query() and torch.equal(got, want)
    assert wall > 0.1 and cpu < 0.25 * wall, (wall, cpu)


def _shares(plan, K):
    """(warps, largest share by number of quads, by cost, goes by cost) of a plan at width K."""
    import ctypes
    warps, table = ctypes.c_int(), ctypes.c_int()
    number, cost = ctypes.c_uint(), ctypes.c_uint()
    assert plan.lib.trs_sddmm_plan_shares(plan._handle, K, ctypes.byref(warps), ctypes.byref(number), ctypes.byref(cost),
                                          ctypes.byref(table)) == 0
    return warps.value, number.value, cost.value, bool(table.value)


def test_shares_are_looked_at_where_they_can_be_used():
    """Patterns of one quad a window, around the number of quads from which the smallest wave gets two a warp: the shares of a
    wave are those of its quads (16 each: one block, up to 32 entries, a new window), and not looked at below."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    least = 12 * sms
    for n_quads in (1, 2 * least - 1, 2 * least, 2 * least + 1, 40 * sms, 2 * 32 * sms):
        rp = torch.arange(16 * n_quads + 1, dtype=torch.int32, device="cuda")
        col = (torch.arange(16 * n_quads, dtype=torch.int32, device="cuda") // 2) % 8   # 16 entries, 8 columns a window
        plan = SddmmPlan(rp, col, 8)
        for K in (24, 64, 96, 128, 160, 192, 224, 256):
            warps, number, cost, table = _shares(plan, K)
            assert warps % (4 * sms) == 0 and warps >= least and not table
            if n_quads // 2 < warps:
                assert (number, cost) == (0, 0)
            else:
                assert number == 16 * -(-n_quads // warps) and cost in (number, number - 16, number + 16)
        X = torch.randn(16 * n_quads, 64, device="cuda").half()
        out, want = plan.run(X, X[:8].contiguous()).float(), (X.float() * X.float()[col.long()]).sum(1)
        # fp16 results (2^-11) of fp32 sums, whose order differs by less than that
        assert float((out - want).abs().max()) <= 2e-3 * float(want.abs().max())
