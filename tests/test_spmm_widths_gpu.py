"""Feature widths around the kernel's slab sizes (multiples of 16 up to 128), rows of B that do not start on
16-byte boundaries (padded copy, or plain loads when no workspace can hold one), and windows whose
steps are of all three kinds and split over several items."""
import pytest
import torch

from oracle import oracle as O
from trspmm import Format, SpmmPlan, _lib, graphs

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
