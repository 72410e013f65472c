"""Infinities and NaN in B: a step of the kernel multiplies zeros with the columns that its tile has, as the format says,
but never with anything in the place of a column that it does not have."""
import pytest
import torch

from oracle import oracle as O
from trspmm import Format, SpmmPlan, build_format, graphs

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def _expected(fmt, B, m):
    """The format's own arithmetic in fp64: packed tiles multiply the two positions that a row names in each group of
    four, a pair of TC blocks and a group of 16 CSR entries all of their columns, and unused column slots are zero."""
    B, out = B.double(), torch.zeros(m, B.shape[1], dtype=torch.float64)

    def add(rows, a, cols):   # a [rows, columns]
        b = torch.where((cols >= 0)[:, None], B[cols.clamp(min=0).long()], torch.zeros((), dtype=torch.float64))
        out[rows] += (a[:, :, None] * b[None]).sum(1)[:len(out[rows])]

    W = fmt.s_window_tile_offset.numel() - 1
    for w in range(W):
        rows = slice(16 * w, min(16 * w + 16, m))
        for t in range(int(fmt.s_window_tile_offset[w]), int(fmt.s_window_tile_offset[w + 1])):
            cols = fmt.s_tile_column.view(-1, 16)[t]
            val = fmt.s_packed_a.view(-1, 64)[t].contiguous().view(torch.float16).double().view(8, 4, 2, 2)
            meta = fmt.s_packed_meta.view(-1, 8)[t].long() & 0xffffffff
            for g in range(8):
                for h in range(2):
                    if 16 * w + g + 8 * h >= m:
                        continue
                    for q in range(4):
                        nibble = int(meta[g]) >> (16 * h + 4 * q) & 15
                        for i, p in enumerate((nibble & 3, nibble >> 2)):
                            if cols[4 * q + p] >= 0:
                                out[16 * w + g + 8 * h] += val[g, q, h, i] * B[int(cols[4 * q + p])]
        parts = (fmt.t_window_row == 16 * w).nonzero().flatten().tolist()
        if parts:
            b0, b1 = int(fmt.t_row_offset[parts[0]]), int(fmt.t_row_offset[parts[-1] + 1])
            for b in range(b0, b1, 2):
                a, cols = torch.zeros(16, 16, dtype=torch.float64), torch.full((16,), -1)
                for i in range(min(2, b1 - b)):
                    cols[8 * i:8 * i + 8] = fmt.t_column.view(-1, 8)[b + i]
                    v = iter(fmt.t_value[int(fmt.t_block_offset[b + i]):int(fmt.t_block_offset[b + i + 1])].half().double())
                    for half in range(2):
                        bits = int(fmt.t_binary.view(-1, 2)[b + i, half]) & ((1 << 64) - 1)
                        for k in range(64):
                            if bits >> k & 1:
                                a[8 * half + k // 8, 8 * i + k % 8] = next(v)
                add(rows, a, cols)
        entries = []
        for off, row, col, val in ((fmt.c_row_offset, fmt.c_row, fmt.c_column, fmt.c_value),
                                   (fmt.cs_row_offset, fmt.cs_row, fmt.cs_column, fmt.cs_value)):
            for p in ((row // 16) == w).nonzero().flatten().tolist():
                entries += [(int(row[p]) % 16, int(col[e]), float(val[e].half())) for e in range(int(off[p]), int(off[p + 1]))]
        for e in range(0, len(entries), 16):
            a, cols = torch.zeros(16, 16, dtype=torch.float64), torch.full((16,), -1)
            for k, (r, c, v) in enumerate(entries[e:e + 16]):
                a[r, k], cols[k] = v, c
            add(rows, a, cols)
    return out


def _check(arrays, B, m):
    fmt = Format(arrays)
    want = _expected(fmt, B, m)
    got = SpmmPlan(Format(arrays).to("cuda"), m, B.shape[0]).run(B.cuda(), out_dtype=torch.float32).cpu().double()
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    if bool(finite.any()):
        assert float((got - want)[finite].abs().max()) <= 2e-5 * float(want[finite].abs().max())
    return want


@pytest.mark.parametrize("F", [16, 24, 47, 64, 128, 136])
@pytest.mark.parametrize("chunk", ["256", "8"])
@pytest.mark.parametrize("kind", ["rmat", "strict", "clustered"])
def test_nonfinite_rows(kind, chunk, F, monkeypatch):
    monkeypatch.setenv("TRS_CHUNK_STEPS", chunk)
    rp, col, val = graphs.clustered_graph(256, 64, 12, 2, seed=2) if kind == "clustered" else graphs.rmat_graph(8, 6, seed=5)
    n = rp.numel() - 1
    if kind == "strict":   # CSR remainders in most windows
        arrays = [a.cpu() for a in build_format(rp.cuda(), col.cuda(), val.cuda(), strict=True)[0].arrays()]
    else:
        arrays = O.build_format(rp, col, val, density=4)[0]
    g = torch.Generator().manual_seed(F)
    B = torch.randn(n, F, generator=g).half()
    B[torch.randint(n, (5,), generator=g), torch.randint(F, (5,), generator=g)] = INF
    B[torch.randint(n, (3,), generator=g), torch.randint(F, (3,), generator=g)] = NAN
    B[0, F - 1] = -INF
    want = _check(arrays, B, n)
    assert bool(torch.isinf(want).any()) and bool(torch.isnan(want).any()) and bool(torch.isfinite(want).any())


def test_one_column_of_infinities():
    """A TC block of one column: every row of the window is an infinity, none is NaN."""
    rp, col = torch.arange(17, dtype=torch.int32), torch.full((16,), 3, dtype=torch.int32)
    arrays = O.build_format(rp, col, torch.arange(1, 17).float())[0]
    B = torch.full((20, 32), INF, dtype=torch.float16)
    assert bool(torch.isinf(_check(arrays, B, 16)).all())
