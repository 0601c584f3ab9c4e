"""Solves on a device whose memory is nearly full: they end with the solution or with an error that says
so, and the context is as good afterwards."""
import numpy as np
import pytest

import gpu_util as G
import rhmc_b200 as rb
from rhmc_b200 import fields as F

pytestmark = pytest.mark.gpu

SHIFTS = np.array([1e-3, 0.05, 1.0, 30.0])


def _free_links(torch, dims):
    """The free field with the staggered phases, on the device."""
    eta = torch.from_numpy(F.eta_phases(dims).astype(np.float64)).cuda()
    return (eta[:, None, None] * torch.eye(3, dtype=torch.complex128, device="cuda")).contiguous()


def _source(torch, ctx, n, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.randn(n * 6 * ctx.Vh, generator=gen, device="cuda", dtype=torch.float64)


def _solve(torch, ctx, b, n, res, shifts=SHIFTS, **kw):
    x = torch.full((n * len(shifts) * 6 * ctx.Vh,), 7.0, dtype=torch.float64, device="cuda")
    info = ctx.msolve(x, b, shifts, res, nrhs=n, **kw)
    torch.cuda.synchronize()
    return x, info


def _fill(torch, left):
    """All free device memory but `left` bytes."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")


def test_no_room_for_the_half_links(torch_cuda):
    """The refinement's half links (42 MB) do not fit beside the vectors of an earlier FP32 solve."""
    dims = (24, 24, 24, 32)
    ctx = G.new_ctx(dims, mass=0.3)
    ctx.set_gauge(_free_links(torch_cuda, dims))
    b = _source(torch_cuda, ctx, 2, 81)
    kw = dict(mode=rb.MSOLVE_MIXED)
    want, _ = _solve(torch_cuda, ctx, b, 2, 1e-6, fmt=rb.LINKS_F32_12, **kw)
    x = torch_cuda.empty_like(want)
    fill = _fill(torch_cuda, 30 << 20)
    try:
        ctx.msolve(x, b, SHIFTS, 1e-6, nrhs=2, fmt=rb.LINKS_F16_12, **kw)
    except rb.RhmcError as err:
        assert "out of memory" in str(err)
    else:
        assert ctx.true_residuals(x, b, SHIFTS, nrhs=2).max() <= 1e-6
    del fill
    torch_cuda.cuda.empty_cache()
    x, info = _solve(torch_cuda, ctx, b, 2, 1e-6, fmt=rb.LINKS_F16_12, **kw)
    assert info["status"] == 0 and ctx.true_residuals(x, b, SHIFTS, nrhs=2).max() <= 1e-6
    x, _ = _solve(torch_cuda, ctx, b, 2, 1e-6, fmt=rb.LINKS_F32_12, **kw)
    assert float((x - want).norm() / want.norm()) < 1e-13


def _used(torch):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free


# 16^3x32: the free memory is asked for; 12^2x16^2: it is not (all that a solve takes is below 256 MB)
@pytest.mark.parametrize("dims", [(16, 16, 16, 32), (12, 12, 16, 16)])
def test_precision_schedule_that_fits_with_half_windows(torch_cuda, dims):
    """A mixed solve in the memory that it takes with half windows, a little more and a little less than with
    whole ones: it solves, to the same solution but for rounding."""
    n, shifts = 4, np.geomspace(1e-4, 50.0, 12)
    ctx = G.new_ctx(dims, mass=0.02)
    ctx.set_gauge(F.random_links(dims, seed=91))
    b = _source(torch_cuda, ctx, n, 92)
    res = 1e-10 * float(b[:6 * ctx.Vh].norm())
    kw = dict(mode=rb.MSOLVE_MIXED, fmt=rb.LINKS_F32_12)
    want, info = _solve(torch_cuda, ctx, b, n, res, shifts, **kw)
    whole = ctx.workspace_bytes()
    assert info["systems_refined"] >= 4 and ctx.msolve_window() == 16
    spinor = 48 * ctx.Vh
    before = _used(torch_cuda)
    ctx.call("rhmc_workspace_release")
    held = before - _used(torch_cuda)  # of the workspaces, as the device counts it
    x = torch_cuda.empty_like(want)
    # whole windows take 8 n FP64 and 8 n FP32 residuals more than half ones
    for less in (0.25, 0.5, 0.9):
        fill = _fill(torch_cuda, held - int(less * 12 * n * spinor))
        info = ctx.msolve(x, b, shifts, res, nrhs=n, **kw)
        del fill
        torch_cuda.cuda.empty_cache()
        assert info["status"] == 0 and ctx.true_residuals(x, b, shifts, nrhs=n).max() <= res
        assert float((x - want).norm() / want.norm()) < 1e-4  # both within res of the solution
        assert ctx.workspace_bytes() < whole
        again, _ = _solve(torch_cuda, ctx, b, n, res, shifts, **kw)  # with all memory free again the choice stands
        assert torch_cuda.equal(x, again)
        ctx.call("rhmc_workspace_release")
    again, _ = _solve(torch_cuda, ctx, b, n, res, shifts, **kw)
    assert torch_cuda.equal(again, want) and ctx.msolve_window() == 16


def test_other_calls_take_the_rings_memory(torch_cuda):
    """What does not fit beside the residuals of an earlier solve gets their memory; the next solve makes
    its own again."""
    dims = (24, 24, 24, 32)
    ctx = G.new_ctx(dims, mass=0.3)
    ctx.set_gauge(_free_links(torch_cuda, dims))
    n = 4
    b = _source(torch_cuda, ctx, n, 95)
    kw = dict(mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_18)
    want, _ = _solve(torch_cuda, ctx, b, n, 1e-6, **kw)
    ref, out = torch_cuda.empty_like(b), torch_cuda.empty_like(b)
    other = G.new_ctx(dims, mass=0.3)
    other.set_gauge(_free_links(torch_cuda, dims))
    other.mdagm(rb.LINKS_F64_18, ref, b, 0.1, n)
    other.sync()
    fill = _fill(torch_cuda, 16 << 20)  # mdagm's own scratch is 42 MB
    ctx.mdagm(rb.LINKS_F64_18, out, b, 0.1, n)
    ctx.sync()
    assert torch_cuda.equal(out, ref)
    del fill
    torch_cuda.cuda.empty_cache()
    x, _ = _solve(torch_cuda, ctx, b, n, 1e-6, **kw)
    assert torch_cuda.equal(x, want)
