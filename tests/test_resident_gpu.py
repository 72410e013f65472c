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


@pytest.mark.parametrize("pinned", [(True, True), (False, False), (True, False), (False, True)])
@pytest.mark.parametrize("F", [128, 130, 160, 200, 256])
def test_kinds_of_host_memory(F, pinned):
    """Blocking calls of a size that goes in slabs, on page-locked and pageable operands, and on rows off 64-byte boundaries."""
    fmt, n = _case(1 << 16)
    op, plan = ResidentSpmm(fmt, n, n, max_dimN=256), SpmmPlan(fmt, n, n)
    B = torch.randn(n, F, generator=torch.Generator().manual_seed(F)).half()
    for dtype in (torch.float32, torch.float16):
        want = plan.run(B.cuda(), out_dtype=dtype).cpu()
        for offset in (0, 2):
            rhs, out = torch.empty(n * F + offset, dtype=torch.float16), torch.empty(n * F + offset, dtype=dtype)
            rhs, out = rhs.pin_memory() if pinned[0] else rhs, out.pin_memory() if pinned[1] else out
            rhs, out = rhs[offset:].view(n, F).copy_(B), out[offset:].view(n, F)
            op.forward(rhs, out)
            assert torch.equal(out, want)


def test_kernel_time_leaves_the_copies_out():
    """total_ms is the kernels' time: for a nearly empty matrix a small part of the copies', in slabs too."""
    fmt, n = _case()
    op = ResidentSpmm(fmt, n, n, max_dimN=256)
    rhs, out = torch.zeros(n, 256, dtype=torch.float16).pin_memory(), torch.empty(n, 256).pin_memory()
    times = [op.forward(rhs, out)[1] for _ in range(5)]
    assert min(t.total_ms / t.h2d_ms for t in times) < 0.4
