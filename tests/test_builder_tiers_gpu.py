"""Windows at the borders of the builder's matching tiers (a warp, a block, a block with the units outside shared
memory), with long runs of equal units and with mixed ones, and key widths on both sides of 32 bits."""
import pytest
import torch

from oracle import oracle as O
from trspmm import TrsError, build_format, graphs
from window_slices import compare_window, slice_window, window_segment

pytestmark = pytest.mark.gpu


def _window(n_units, mixed, n_cols, seed):
    """One 16-row window with 2 * n_units distinct columns; `mixed`: counts 1 to 5, otherwise 1 for nearly all."""
    g = torch.Generator().manual_seed(seed)
    d = 2 * n_units - seed % 2
    cols = torch.randperm(n_cols, generator=g)[:d].sort().values
    count = torch.randint(1, 6, (d,), generator=g) if mixed else 1 + (torch.rand(d, generator=g) < 0.001).long()
    rows = torch.rand(d, 16, generator=g).argsort(dim=1)
    keep = torch.arange(16)[None, :] < count[:, None]
    r, c = rows[keep], cols[:, None].expand(-1, 16)[keep]
    order = torch.argsort(r * n_cols + c)
    r, c = r[order], c[order]
    rowptr = torch.zeros(17, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(torch.bincount(r, minlength=16), 0)
    return rowptr.to(torch.int32), c.to(torch.int32), torch.randn(c.numel(), generator=g)


def _check(rp, col, val, **kw):
    want, info = O.build_format(rp, col, val, **kw)
    fmt, stats = build_format(rp.cuda(), col.cuda(), val.cuda(), **kw)
    for name, a, b in zip(O.FORMAT_NAMES, fmt.arrays(), want):
        assert torch.equal(a.cpu(), b), name
    assert stats["dropped_nnz"] == info["dropped_nnz"]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("units", [1, 16, 17, 31, 33, 64, 1023, 2048, 2049, 14336, 14337])
def test_tier_borders(units, mixed):
    _check(*_window(units, mixed, 1 << 20, units))


def test_units_beyond_shared_memory():
    _check(*_window(53000, True, 1 << 20, 1))


@pytest.mark.parametrize("bits", [14, 22])   # one window: under 32 key bits; with 40001 windows 30 and 38
def test_key_widths(bits):
    rp, col, val = _window(40, True, 1 << bits, 3)
    for empty_rows in (0, 16 * 40000):
        _check(torch.cat([rp, rp[-1:].expand(empty_rows)]), col, val)


@pytest.mark.parametrize("window", [16, 5])
@pytest.mark.parametrize("entries", [1, 63, 255, 256, 257, 1023, 1024, 1025, 4095, 4096, 4097, 8191, 8192, 8193, 9000, 20000])
def test_sort_class_borders(entries, window):
    """A window with exactly that many entries between small and empty ones: sorted by a CTA of the class, or (beyond 8192)
    by the device-wide passes; columns shared by many rows and columns of one row."""
    g = torch.Generator().manual_seed(entries)
    n_cols = max(2 * entries // window, 3 * window)
    rows = torch.arange(entries) % window + window                       # the second window
    cols = torch.empty(entries, dtype=torch.int64)
    for r in range(window):
        at = rows == window + r
        cols[at] = torch.randperm(n_cols, generator=g)[:int(at.sum())]
    rows = torch.cat([rows, torch.tensor([0, 3 * window, 4 * window + 1])])
    cols = torch.cat([cols, torch.tensor([n_cols - 1, 0, 5])])
    order = torch.argsort(rows * n_cols + cols)
    rowptr = torch.zeros(6 * window + 1, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(torch.bincount(rows, minlength=6 * window), 0)
    _check(rowptr.to(torch.int32), cols[order].to(torch.int32), torch.randn(entries + 3, generator=g), window=window)


@pytest.mark.parametrize("rows", [1, 255, 256, 257, 512, 1025])
def test_part_block_borders(rows):
    """Rows on both sides of the blocks that count the CUDA-core parts; windows with a unit that is not kept."""
    g = torch.Generator().manual_seed(rows)
    hit = torch.rand(rows, 90, generator=g) < 0.06
    hit[:, :3] |= torch.rand(rows, 3, generator=g) < 0.5
    rowptr = torch.zeros(rows + 1, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(hit.sum(1), 0)
    col = hit.nonzero()[:, 1]
    _check(rowptr.to(torch.int32), col.to(torch.int32), torch.randn(col.numel(), generator=g), window=7, unit_min_nnz=4)


@pytest.mark.parametrize("entries", [12, 20, 40, 100, 200, 500, 600])
def test_repeated_columns_are_refused(entries):
    """A column repeated in every row, in windows sorted by a warp (up to 64 a row), by a CTA and in a hub window (600): more entries of
    one column than the window has rows must not get as far as the records."""
    rp = torch.arange(17, dtype=torch.int32) * entries
    col = torch.full((16 * entries,), 5, dtype=torch.int32)
    with pytest.raises(TrsError) as e:
        build_format(rp.cuda(), col.cuda(), torch.ones(16 * entries).cuda())
    assert e.value.code == -8


# rows of the window, and the place in the first of them whose column does not ascend
_ORDERS = {"warp of 8 a lane, inside a lane": ([12] * 16, 3), "warp of 8 a lane, two lanes of a row": ([12] * 16, 8),
           "warp of 8 a lane, rows that do not fit": ([40] + [10] * 15, 33), "warp of 16 a lane, inside a lane": ([20] * 16, 19),
           "warp of 16 a lane, two lanes of a row": ([20] * 16, 16), "warp of 32 a lane, inside a lane": ([40] * 16, 31),
           "warp of 32 a lane, two lanes of a row": ([40] * 16, 32), "CTA of 1024": ([400] + [10] * 15, 256),
           "CTA of 2048": ([100] * 16, 64), "CTA of 4096": ([200] * 16, 128), "CTA of 8192": ([400] * 16, 399), "hub": ([600] * 16, 300)}


@pytest.mark.parametrize("fault", ["repeated", "descending", "negative"])
@pytest.mark.parametrize("where", _ORDERS)
@pytest.mark.parametrize("bits", [16, 24])   # 24: keys of 64 bits, which a warp does not sort
def test_one_column_out_of_order(where, fault, bits):
    """One entry of one row of the middle one of three windows: refused at every place where a sort looks, and the next build is
    right."""
    rows, at = _ORDERS[where]
    g = torch.Generator().manual_seed(len(rows) * at)
    per_row = torch.tensor(rows * 3)
    col = torch.cat([torch.randperm(1 << 12, generator=g)[:k].sort().values + 1 for k in per_row.tolist()]).to(torch.int32)
    col[-1] = (1 << bits) - 1
    rowptr = torch.zeros(49, dtype=torch.int32)
    rowptr[1:] = torch.cumsum(per_row, 0)
    val = torch.randn(col.numel(), generator=g)
    bad = col.clone()
    e = int(rowptr[16]) + at
    if fault == "negative":
        e -= at
    bad[e] = {"repeated": bad[e - 1], "descending": bad[e - 1] - 1, "negative": -1}[fault]
    with pytest.raises(TrsError) as err:
        build_format(rowptr.cuda(), bad.cuda(), val.cuda())
    assert err.value.code == -8
    _check(rowptr, col, val)


def test_entries_without_arrays_are_refused():
    empty = torch.zeros(0, dtype=torch.int32).cuda()
    with pytest.raises(TrsError) as e:
        build_format(torch.arange(17, dtype=torch.int32).cuda(), empty, empty.float())
    assert e.value.code == -1


@pytest.mark.parametrize("error", [MemoryError, KeyboardInterrupt])
@pytest.mark.parametrize("strict", [False, True])
def test_array_that_cannot_be_had(error, strict, monkeypatch):
    """Memory for the k-th array fails, while other streams are at work on the build or not: the caller's exception comes
    out, and the next build is right."""
    rp, col, val = (t.cuda() for t in graphs.rmat_graph(13, 16, seed=8))   # hub windows and all classes
    want = build_format(rp, col, val, strict=strict)[0].arrays()
    empty = torch.empty
    for k in range(40):
        calls = [0]

        def failing(*a, **kw):
            calls[0] += 1
            if calls[0] == k + 1:
                raise error("no room")
            return empty(*a, **kw)

        with monkeypatch.context() as m:
            m.setattr(torch, "empty", failing)
            try:
                got = build_format(rp, col, val, strict=strict)[0].arrays()
            except error:
                got = None
        if got is None:
            got = build_format(rp, col, val, strict=strict)[0].arrays()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), k
        if calls[0] <= k:
            break
    assert 10 < k < 40


@pytest.mark.parametrize("long_row", [0, 33, 0.6])
@pytest.mark.parametrize("entries,bits", [(entries, bits) for cap, bits in ((256, 23), (512, 22), (1024, 21), (2048, 20))
                                          for entries in (cap - 1, cap, cap + 1) for bits in (bits, bits + 1)])
def test_warp_sort_borders(entries, bits, long_row):
    """Windows on both sides of the classes that a warp sorts, with equal rows (each takes two lanes), with rows longer than
    that, and columns up to the last one of the widest that fit into its keys and of the next power of two."""
    g = torch.Generator().manual_seed(entries + bits)
    per_row = torch.full((16,), entries // 16)
    per_row[:entries % 16] += 1
    more = int(long_row * entries) if long_row < 1 else long_row
    for r in range(15):   # the last row takes from the others
        take = min(int(per_row[r]) - 1, -(-more // 15))
        per_row[r] -= take
        per_row[15] += take
    shared = torch.randint(0, 1 << bits, (entries // 2,), generator=g)
    cols = []
    for r in range(16):
        few = torch.cat([shared[torch.randperm(shared.numel(), generator=g)][:int(per_row[r]) // 2],
                         torch.randint(0, 1 << bits, (3 * int(per_row[r]) + 64,), generator=g)]).unique()
        cols.append(few[torch.randperm(few.numel(), generator=g)][:int(per_row[r])].sort().values)
    cols[15][-1] = (1 << bits) - 1
    rowptr = torch.zeros(17, dtype=torch.int32)
    rowptr[1:] = torch.cumsum(per_row, 0)
    _check(rowptr, torch.cat(cols).to(torch.int32), torch.randn(entries, generator=g))


@pytest.mark.parametrize("windows", [1, 1023, 1024, 4095, 4096, 4607, 4608, 9000])
def test_scan_borders(windows):
    """Sums over windows on both sides of a round of the one-CTA scan, and of its largest number of values."""
    g = torch.Generator().manual_seed(windows)
    n = 16 * windows - 3
    rows = torch.cat([torch.arange(0, n, 5), torch.randint(0, n, (n,), generator=g)])
    cols = torch.randint(0, 300, (rows.numel(),), generator=g)
    rp, col, _ = graphs.coo_to_csr(rows, cols, n, 300)
    _check(rp, col, torch.randn(col.numel(), generator=g))


def _hub_windows(windows):
    """Windows of 16 x 513 entries, more than a CTA sorts, over 600 columns."""
    g = torch.Generator(device="cuda").manual_seed(windows)
    n = 16 * windows
    col = torch.cat([torch.rand(a.numel(), 600, generator=g, device="cuda").argsort(1)[:, :513].sort(1).values.to(torch.int32).flatten()
                     for a in torch.arange(n).split(1 << 15)])
    rp = torch.arange(n + 1, dtype=torch.int32, device="cuda") * 513
    return rp, col, torch.randn(col.numel(), generator=g, device="cuda")


@pytest.mark.parametrize("windows", [4607, 4608])
def test_many_hub_windows(windows):
    """As many hub windows as the one-CTA scan adds up, and one more."""
    rp, col, val = _hub_windows(windows)
    named = dict(zip(O.FORMAT_NAMES, build_format(rp, col, val)[0].arrays()))
    rp = rp.cpu()
    for w in (0, 1, 1023, 2500, windows - 2, windows - 1):
        compare_window(window_segment(named, w), O.build_format(*slice_window(rp, col, val, w))[0], f"window {w}")
