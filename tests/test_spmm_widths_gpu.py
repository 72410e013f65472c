"""Feature widths around the kernel's slab sizes (multiples of 16 up to 128), rows of B that do not start on
16-byte boundaries (padded copy, or plain loads when no workspace can hold one), and windows whose
steps are of all three kinds and split over several items."""
import pytest
import torch

from oracle import oracle as O
from trspmm import Format, SpmmPlan, _lib, build_format, graphs

pytestmark = pytest.mark.gpu
MAX_ERR_F32 = 2e-5


def _err(x, ref):   # scaled by the largest output: a narrow row may cancel to almost nothing
    return float((x.cpu() - ref).abs().max() / ref.abs().max())


def _case():
    rp, col, val = graphs.rmat_graph(10, 16, seed=3)
    n = rp.numel() - 1
    arrays, _ = O.build_format(rp, col, val, density=4)
    return arrays, n


@pytest.mark.parametrize("chunk", ["256", "8"])
@pytest.mark.parametrize("F", [1, 7, 8, 15, 16, 17, 24, 31, 40, 47, 48, 56, 72, 80, 95, 96, 112, 120, 127, 128, 129, 136, 200, 257])
def test_widths(F, chunk, monkeypatch):
    monkeypatch.setenv("TRS_CHUNK_STEPS", chunk)
    arrays, n = _case()
    B = torch.randn(n, F, generator=torch.Generator().manual_seed(F)).half()
    ref = O.spmm_from_format(arrays, B, n)
    plan = SpmmPlan(Format(arrays).to("cuda"), n, n)
    out = plan.run(B.cuda(), out_dtype=torch.float32)
    assert _err(out, ref) <= MAX_ERR_F32
    assert torch.equal(out, plan.run(B.cuda(), out_dtype=torch.float32))
    assert _err(plan.run(B.cuda(), out_dtype=torch.float16).float(), ref) <= 1e-3
    r = plan.run(B.cuda(), out_dtype=torch.float32, relu=True)
    assert _err(r, torch.relu(ref)) <= MAX_ERR_F32


@pytest.mark.parametrize("F", [104, 152, 168, 184, 208, 224, 232, 264, 320, 392])
def test_slabs_that_rows_do_not_fill(F, monkeypatch):
    test_widths(F, "8", monkeypatch)


@pytest.mark.parametrize("F,offset", [(64, 4), (47, 1), (128, 2), (33, 0)])
def test_no_room_for_a_padded_copy(F, offset):
    """B off a 16-byte boundary and a workspace that holds the partial sums only."""
    arrays, n = _case()
    base = torch.randn(n * F + 8, generator=torch.Generator().manual_seed(1)).half().cuda()
    B = base[offset:offset + n * F].view(n, F)
    ref = O.spmm_from_format(arrays, B.cpu(), n)
    plan = SpmmPlan(Format(arrays).to("cuda"), n, n)
    out = torch.empty(n, F, device="cuda")
    ws = torch.empty(max(plan.static_scratch_bytes(F), 16), dtype=torch.uint8, device="cuda")
    _lib.check(plan.lib.trs_spmm_run(plan._handle, B.data_ptr(), out.data_ptr(), F, 0, ws.data_ptr(), ws.numel(),
                                     _lib.current_stream_ptr(out.device)))
    assert _err(out, ref) <= MAX_ERR_F32


@pytest.mark.parametrize("rows", [16, 1500, 16 * 1024, 16 * 1025 + 3, 16 * 5000])
@pytest.mark.parametrize("F", [64, 47])
def test_ranges_of_windows(rows, F):
    """Ranges on both sides of the samples at which a plan knows where windows begin, with and without hub windows; every
    one writes its own rows, with the bits of the whole run."""
    for rp, col, val in (graphs.uniform_graph(rows, 5, seed=2, device="cuda"),
                         graphs.coo_to_csr(torch.cat([torch.arange(rows), torch.zeros(9000, dtype=torch.long)]),
                                           torch.cat([torch.arange(rows), torch.arange(9000)]), rows, max(rows, 9000))[:2] + (None,)):
        rp, col = rp.cuda(), col.cuda()
        val = torch.rand(col.numel(), device="cuda") if val is None else val
        k = max(rows, 9000)
        plan = SpmmPlan(build_format(rp, col, val)[0], rows, k)
        W = plan.num_windows
        B = torch.randn(k, F, generator=torch.Generator().manual_seed(F)).half().cuda()
        want = plan.run(B, out_dtype=torch.float32)
        out = torch.full_like(want, float("nan"))
        cuts = sorted({0, 1, min(5, W), W // 2, W // 2 + 1 if W > 1 else W, W - 1, W} - {-1})
        for w0, w1 in zip(cuts[:-1], cuts[1:]):
            before = out.clone()
            plan.run_windows(B, out, w0, w1)
            mine = slice(16 * w0, min(16 * w1, rows))
            before[mine] = want[mine]
            assert torch.equal(torch.nan_to_num(out, nan=-7.0), torch.nan_to_num(before, nan=-7.0)), (w0, w1)
        assert torch.equal(out, want)


def test_packed_values_off_their_boundary():
    """Packed tiles that begin 4 bytes behind an 8-byte boundary."""
    arrays, n = _case()
    fmt = Format(arrays).to("cuda")
    B = torch.randn(n, 64, generator=torch.Generator().manual_seed(2)).half().cuda()
    want = SpmmPlan(fmt, n, n).run(B, out_dtype=torch.float32)
    moved = torch.empty(fmt.s_packed_a.numel() + 1, dtype=fmt.s_packed_a.dtype, device="cuda")[1:].view(fmt.s_packed_a.shape)
    fmt.s_packed_a = moved.copy_(fmt.s_packed_a)
    assert moved.data_ptr() % 8 == 4
    assert torch.equal(SpmmPlan(fmt, n, n).run(B, out_dtype=torch.float32), want)


def test_one_plan_on_two_streams():
    """Widths whose rows are copied, no split windows: calls on several streams share nothing that is written."""
    rp, col, val = graphs.uniform_graph(1 << 17, 8, seed=1, device="cuda")
    n = rp.numel() - 1
    plan = SpmmPlan(build_format(rp, col, val)[0], n, n)
    assert plan.launches == 1
    for F in (47, 31):
        B = [torch.randn(n, F, generator=torch.Generator().manual_seed(i)).half().cuda() for i in range(3)]
        want = [plan.run(b) for b in B]
        streams = [torch.cuda.Stream() for _ in B]
        torch.cuda.synchronize()
        got = [[] for _ in B]
        for _ in range(10):
            for i, s in enumerate(streams):
                with torch.cuda.stream(s):
                    got[i].append(plan.run(B[i]))
        torch.cuda.synchronize()
        for i in range(len(B)):
            assert all(torch.equal(g, want[i]) for g in got[i])


def test_copies_of_B_do_not_pile_up():
    arrays, n = _case()
    plan = SpmmPlan(Format(arrays).to("cuda"), n, n)
    B = torch.randn(n, 63, generator=torch.Generator().manual_seed(2)).half().cuda()
    before = torch.cuda.memory_allocated()
    for F in range(1, 63, 2):
        plan.run(B[:, :F].contiguous())
    assert torch.cuda.memory_allocated() - before <= plan.workspace_bytes(61) + 4096   # the last one


def test_captured_call_keeps_its_own_copy():
    """Calls of other widths between replays do not write where the captured call does, nor free it."""
    arrays, n = _case()
    plan = SpmmPlan(Format(arrays).to("cuda"), n, n)
    B = torch.randn(n, 47, generator=torch.Generator().manual_seed(2)).half().cuda()
    want, out = plan.run(B), torch.empty(n, 47, dtype=torch.float16, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run(B, out=out)
    for F in (47, 45, 33, 47):
        other = torch.randn(n, F, generator=torch.Generator().manual_seed(F)).half().cuda()
        a = plan.run(other)
        out.zero_()
        graph.replay()
        assert torch.equal(plan.run(other), a)
        torch.cuda.synchronize()
        assert torch.equal(out, want)


@pytest.mark.parametrize("entries", [400, 6400, 64000])
def test_nearly_empty_matrices(entries):
    """Odd widths where a copy of B would cost more than the product, and ranges of windows on both sides of that."""
    n, F = 1 << 16, 45
    g = torch.Generator().manual_seed(entries)
    rows = torch.cat([torch.randint(n, (entries // 2,), generator=g), torch.randint(n // 16, (entries // 2,), generator=g)])
    rp, col = graphs.coo_to_csr(rows, torch.randint(n, (entries,), generator=g), n, n)[:2]
    val = torch.rand(col.numel(), generator=g)
    plan = SpmmPlan(build_format(rp.cuda(), col.cuda(), val.cuda(), strict=True)[0], n, n)
    B = torch.randn(n, F, generator=g).half()
    ref = O.spmm_csr(rp, col, val, B)
    assert (plan.workspace_bytes(F) < n * F) == (entries < 64000)
    out = plan.run(B.cuda(), out_dtype=torch.float32)
    assert _err(out, ref) <= MAX_ERR_F32
    parts = torch.empty_like(out)
    for w0, w1 in ((0, 300), (300, 4000), (4000, n // 16)):
        plan.run_windows(B.cuda(), parts, w0, w1)
    assert torch.equal(parts, out)


@pytest.mark.parametrize("F", [50, 64])
@pytest.mark.parametrize("per_row", [1, 3, 9, 40])
def test_first_column_ids(F, per_row):
    """Enough items for a warp each, with less than a block of eight steps, a block, and more; windows without entries between
    them: the ids beside the items are those of the stream."""
    n = 40000
    g = torch.Generator().manual_seed(per_row)
    rows = torch.arange(n).repeat_interleave(per_row)
    rows = rows[(rows // 16) % 5 != 2]
    rp, col, _ = graphs.coo_to_csr(rows, torch.randint(0, n, (rows.numel(),), generator=g), n, n)
    val = torch.randn(col.numel(), generator=g)
    B = torch.randn(n, F, generator=g).half()
    fmt = build_format(rp.cuda(), col.cuda(), val.cuda(), strict=True)[0]
    out = SpmmPlan(fmt, n, n).run(B.cuda(), out_dtype=torch.float32).cpu()
    ref = torch.sparse_csr_tensor(rp.long(), col.long(), val.half().double(), (n, n)) @ B.double()
    # fp32 sums of exact products of fp16 values
    assert float((out - ref).abs().max()) <= 2e-5 * float(ref.abs().max())


@pytest.mark.parametrize("windows", [1 << 16, 1 << 20])
def test_plan_without_room_for_first_column_ids(windows):
    """A plan fits where its arrays fit: the ids beside the items (512 bytes an item, more than the rest of this plan) are left out,
    and the results are the same."""
    n, g = 16 * windows, torch.Generator(device="cuda").manual_seed(1)
    rp = torch.arange(n + 1, dtype=torch.int32, device="cuda") * 3
    col = torch.randint(0, 1 << 12, (n, 3), generator=g, device="cuda") + (torch.arange(3, device="cuda") << 12)
    fmt = build_format(rp, col.flatten().to(torch.int32), torch.randn(3 * n, generator=g, device="cuda"))[0]
    B = torch.randn(3 << 12, 64, generator=g, device="cuda").half()
    want = SpmmPlan(fmt, n, 3 << 12).run(B)
    del rp, col
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    _lib.check(_lib.load().trs_pool_trim())
    hog = torch.empty(torch.cuda.mem_get_info()[0] - 640 * windows, dtype=torch.uint8, device="cuda")
    try:
        plan = SpmmPlan(fmt, n, 3 << 12)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert torch.equal(plan.run(B), want)
    assert torch.equal(plan.run(B[:, :50].contiguous()), want[:, :50])
