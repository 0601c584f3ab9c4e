"""The one-kernel multi-shift solve of small lattices: the same bits whichever way a right-hand side is
solved (one kernel with one or two right-hand sides a block, alone or in a batch, or launch by
launch), over every way that its blocks meet and the edges between them, ragged lattices and solves
longer than one launch."""
import numpy as np
import pytest

import gpu_util as G
import rhmc_b200 as rb
from rhmc_b200 import fields as F

pytestmark = pytest.mark.gpu

SHIFTS = np.array([2e-3, 0.04, 0.5, 9.0, 40.0])


def _case(dims, mass, n, seed):
    ctx = G.new_ctx(dims, mass=mass)
    ctx.set_gauge(F.random_links(dims, seed=seed, kind="near1"))
    return ctx, F.random_spinor(dims, seed=seed + 1, n=n)


# chunks of 128 sites: 1; 2 (ragged), 15 and 16, which meet as a cluster; 17 (ragged) and 32, by slots; 33
# (ragged), 81 and 217 (ragged), by counted arrivals
CHUNKS = [(4, 4, 4, 4), (6, 4, 4, 4), (8, 8, 6, 10), (8, 8, 8, 8), (6, 6, 10, 12), (8, 8, 8, 16), (10, 10, 6, 14), (12, 12, 12, 12),
          (18, 14, 10, 22)]


@pytest.mark.parametrize("dims", CHUNKS)
@pytest.mark.parametrize("mode,fmt,res", [(rb.MSOLVE_FP64, rb.LINKS_F64_18, 1e-8), (rb.MSOLVE_FP64, rb.LINKS_F64_12, 1e-8),
                                          (rb.MSOLVE_FP32, rb.LINKS_F32_18, 1e-4), (rb.MSOLVE_MIXED, rb.LINKS_F32_12, 1e-8)])
def test_same_bits_launch_by_launch(torch_cuda, dims, mode, fmt, res):
    """Against the launched kernels (mixed mode: its FP64 part, which an FP32 phase continues)."""
    ctx, b = _case(dims, 0.2, 3, 21)
    for n in (1, 2, 3):
        launched = []
        for one in (1, 0):
            ctx.msolve_one_kernel(one)
            before = ctx.launch_count()
            x, info = ctx.msolve_host(b[:n], SHIFTS, res, mode=mode, fmt=fmt)
            launched.append((ctx.launch_count() - before, x, info["iters"][:n]))
        if n < 3 or dims != CHUNKS[-1]:  # three right-hand sides of 217 chunks do not fit as one kernel
            assert launched[0][0] < launched[1][0]
        assert launched[0][2] == launched[1][2]
        assert np.array_equal(launched[0][1], launched[1][1]), (dims, n)


# batches of one kernel beside each other, and for the last two lattices of 8 launched
@pytest.mark.parametrize("dims", [(4, 4, 4, 4), (6, 4, 4, 4), (8, 8, 8, 16), (10, 10, 6, 14), (12, 12, 12, 12), (18, 14, 10, 22)])
@pytest.mark.parametrize("mode,fmt,res", [(rb.MSOLVE_FP64, rb.LINKS_F64_18, 1e-8), (rb.MSOLVE_FP64, rb.LINKS_F64_12, 1e-8)])
def test_same_bits_in_any_batch(torch_cuda, dims, mode, fmt, res):
    ctx, b = _case(dims, 0.2, 8, 31)
    x8, info = ctx.msolve_host(b, SHIFTS, res, mode=mode, fmt=fmt)
    assert info["status"] == 0
    for n in (1, 2, 3):
        x, one = ctx.msolve_host(b[:n], SHIFTS, res, mode=mode, fmt=fmt)
        assert one["iters"][:n] == info["iters"][:n]
        assert np.array_equal(x, x8[:n]), (dims, n)
    xi = G.to_internal(ctx, rb.LINKS_F64_18, x8.reshape(-1, ctx.Vh, 3))
    bi = G.to_internal(ctx, rb.LINKS_F64_18, b)
    # the stopping test is the reference's lagged one: its true residuals end within twice the target
    assert ctx.true_residuals(xi, bi, SHIFTS, nrhs=8).max() <= 2.0 * res


def test_two_right_hand_sides_a_block(torch_cuda):
    """16^4: 256 chunks, so two right-hand sides share a block, and four are launched."""
    ctx, b = _case((16, 16, 16, 16), 0.3, 4, 41)
    x4, _ = ctx.msolve_host(b, SHIFTS, 1e-7, mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_18)
    for lo in (0, 2):
        x2, _ = ctx.msolve_host(b[lo:lo + 2], SHIFTS, 1e-7, mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_18)
        assert np.array_equal(x2, x4[lo:lo + 2])


def test_fp32_batches(torch_cuda):
    ctx, b = _case((12, 12, 12, 12), 0.3, 8, 51)
    x8, _ = ctx.msolve_host(b, SHIFTS, 1e-4, mode=rb.MSOLVE_FP32, fmt=rb.LINKS_F32_12)
    for n in (1, 2):
        x, _ = ctx.msolve_host(b[:n], SHIFTS, 1e-4, mode=rb.MSOLVE_FP32, fmt=rb.LINKS_F32_12)
        assert np.array_equal(x, x8[:n])


def test_longer_than_one_launch(torch_cuda):
    """More than 1024 iterations (the solve continues in a second launch), and the iteration cap there."""
    ctx, b = _case((8, 8, 8, 8), 0.004, 1, 61)
    ctx.set_gauge(F.random_links((8, 8, 8, 8), seed=62))  # Haar links: no spectral gap
    res = 1e-7
    x, info = ctx.msolve_host(b, SHIFTS * 1e-2, res, mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_18)
    assert info["iters"][0] > 1024, info
    xi = G.to_internal(ctx, rb.LINKS_F64_18, x.reshape(-1, ctx.Vh, 3))
    bi = G.to_internal(ctx, rb.LINKS_F64_18, b)
    assert ctx.true_residuals(xi, bi, SHIFTS * 1e-2).max() <= 20.0 * res  # iterated residual, kappa 4e5
    with pytest.raises(rb.RhmcError, match="cap 1030"):
        ctx.msolve_host(b, SHIFTS * 1e-2, res, max_iter=1030, mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_18)


def test_longer_than_one_launch_launch_by_launch(torch_cuda):
    """The state that one launch of 1024 iterations leaves to the next."""
    ctx, b = _case((8, 8, 8, 8), 0.004, 2, 71)
    ctx.set_gauge(F.random_links((8, 8, 8, 8), seed=72))
    out = []
    for one in (1, 0):
        ctx.msolve_one_kernel(one)
        out.append(ctx.msolve_host(b, SHIFTS * 1e-2, 1e-7, mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_18))
    assert out[0][1]["iters"][0] > 1024 and out[0][1]["iters"] == out[1][1]["iters"]
    assert np.array_equal(out[0][0], out[1][0])
