"""The resident handle where a call fails, and with operands of every kind."""
import pytest
import torch

from trspmm import ResidentSpmm, SpmmPlan, TrsError, _lib, build_format, graphs

pytestmark = pytest.mark.gpu


def _case(n=1 << 18):
    rp, col, val = graphs.uniform_graph(n, 4, seed=1, device="cuda")
    return build_format(rp, col, val)[0], n


def test_call_after_one_that_found_no_memory():
    """A width that needs a larger workspace than there is memory for fails, and the handle goes on afterwards."""
    fmt, n = _case()
    op = ResidentSpmm(fmt, n, n, max_dimN=128)
    plan = SpmmPlan(fmt, n, n)
    B = {F: torch.randn(n, F, generator=torch.Generator().manual_seed(F)).half() for F in (47, 128)}
    want = {F: plan.run(b.cuda(), out_dtype=torch.float32).cpu() for F, b in B.items()}
    out = {F: torch.empty(n, F) for F in B}
    torch.cuda.empty_cache()
    _lib.check(op.lib.trs_pool_trim())
    free = torch.cuda.mem_get_info()[0]
    hog = [torch.empty(free - (64 << 20), dtype=torch.uint8, device="cuda")]   # the padded copy takes 25 MB, in chunks of 32
    while True:
        try:
            hog.append(torch.empty(4 << 20, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            break
    try:
        op.forward(B[47], out[47])
        failed = False
    except TrsError as e:
        failed = e.code == 2
    del hog
    torch.cuda.empty_cache()
    assert failed
    for F in (47, 128, 47):
        op.forward(B[F], out[F])
        assert torch.equal(out[F], want[F])
