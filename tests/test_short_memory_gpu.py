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


def _solve(torch, ctx, b, n, res, **kw):
    x = torch.full((n * len(SHIFTS) * 6 * ctx.Vh,), 7.0, dtype=torch.float64, device="cuda")
    info = ctx.msolve(x, b, SHIFTS, res, nrhs=n, **kw)
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
