"""How far the refinement takes a system that the multi-shift left above its target: until its residual
has fallen by ru_delta, also when it starts just above the target."""
import numpy as np
import pytest

import gpu_util as G
import rhmc_b200 as rb
from rhmc_b200 import fields as F

pytestmark = pytest.mark.gpu

DIMS = (8, 8, 8, 8)
SHIFTS = np.geomspace(1e-4, 50.0, 12)


def _ctx(n):
    ctx = G.new_ctx(DIMS, mass=0.02)
    ctx.set_gauge(F.random_links(DIMS, seed=71))
    return ctx, G.to_internal(ctx, rb.LINKS_F64_18, F.random_spinor(DIMS, seed=72, n=n))


def _residuals(torch, ctx, b, n, res, **kw):
    x = torch.empty(n * len(SHIFTS) * 6 * ctx.Vh, dtype=torch.float64, device="cuda")
    info = ctx.msolve(x, b, SHIFTS, res, nrhs=n, **kw)
    return x.view(n, len(SHIFTS), -1), ctx.true_residuals(x, b, SHIFTS, nrhs=n), info


def test_certified_systems(torch_cuda):
    """FP64: every system above its target is iterated until its residual has fallen twentyfold (the
    recomputed residual within 5 % of the iterated one)."""
    ctx, b = _ctx(4)
    kw = dict(mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_18)
    refined = 0
    for res in np.geomspace(1e-8, 1e-5, 13):
        _, before, _ = _residuals(torch_cuda, ctx, b, 4, res, **kw)
        _, after, info = _residuals(torch_cuda, ctx, b, 4, res, certify=1, **kw)
        above = before > res
        assert info["systems_refined"] == above.sum()
        assert (after[above] <= 0.0525 * before[above]).all(), (res, before[above], after[above])
        assert (after[~above] == before[~above]).all()
        refined += int(above.sum())
    assert refined > 0


@pytest.mark.parametrize("fmt", [rb.LINKS_F32_12, rb.LINKS_F32_18])
def test_delta_decides_how_far(torch_cuda, fmt):
    """Mixed: with ru_delta a hundred times smaller every refined system, and no other, comes out at
    least twenty times further down."""
    ctx, b = _ctx(4)
    refined = 0
    for res in np.geomspace(1e-9, 1e-7, 5):
        x1, r1, info = _residuals(torch_cuda, ctx, b, 4, res, mode=rb.MSOLVE_MIXED, fmt=fmt, ru_delta=0.2)
        x2, r2, _ = _residuals(torch_cuda, ctx, b, 4, res, mode=rb.MSOLVE_MIXED, fmt=fmt, ru_delta=2e-3)
        other = (x1 != x2).any(-1).cpu().numpy()
        assert r1.max() <= res and r2.max() <= res
        assert other.sum() == info["systems_refined"]
        assert (r2[other] <= 0.05 * r1[other]).all(), (res, r1[other], r2[other])
        refined += info["systems_refined"]
    assert refined > 0
