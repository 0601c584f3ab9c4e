"""The delayed-update window of the multi-shift solver: solves that stop in the first window, exactly at
a window's end and just past it, with frozen shifts, and with the shorter window that the solver
falls back to when the longer residual ring would not leave it enough device memory."""
import numpy as np
import pytest

import gpu_util as G
import rhmc_b200 as rb
from rhmc_b200 import fields as F

pytestmark = pytest.mark.gpu

SHIFTS = np.array([1e-3, 0.05, 1.0, 30.0])


def _solve(ctx, b, nrhs, mode, fmt, residual):
    import torch
    x = torch.full((nrhs * len(SHIFTS) * 6 * ctx.Vh,), 7.0, dtype=torch.float64, device="cuda")
    info = ctx.msolve(x, b, SHIFTS, residual, nrhs=nrhs, mode=mode, fmt=fmt)
    torch.cuda.synchronize()
    return x, info


@pytest.mark.parametrize("nrhs,mode,fmt", [(1, rb.MSOLVE_FP64, rb.LINKS_F64_18), (4, rb.MSOLVE_FP64, rb.LINKS_F64_12),
                                           (8, rb.MSOLVE_MIXED, rb.LINKS_F32_12), (3, rb.MSOLVE_FP32, rb.LINKS_F32_18)])
def test_residuals_over_window_positions(torch_cuda, nrhs, mode, fmt):
    dims = (6, 4, 4, 8)
    ctx = G.new_ctx(dims, mass=0.3)
    ctx.set_gauge(F.random_links(dims, seed=11))
    b = G.to_internal(ctx, rb.LINKS_F64_18, F.random_spinor(dims, seed=12, n=nrhs))
    nb = np.sqrt(ctx.Vh * 3.0)
    seen = set()
    # from a solve of a few iterations to one of several windows
    for res in nb * 10.0 ** -np.arange(0.5, 5.0 if mode == rb.MSOLVE_FP32 else 9.0, 0.5):
        x, info = _solve(ctx, b, nrhs, mode, fmt, float(res))
        assert torch_cuda.isfinite(x).all()
        tr = ctx.true_residuals(x, b, SHIFTS, nrhs=nrhs)
        # FP64 and FP32 stop on the iterated residual, frozen shifts on their lagged one
        assert tr.max() <= res * (1.0 + 1e-12 if mode == rb.MSOLVE_MIXED else 2.0), (res, tr, info["iters"])
        seen.update(i % 16 for i in info["iters"][:nrhs])
    assert len(seen) > 4


def test_zero_rhs_in_a_batch(torch_cuda):
    dims = (4, 4, 4, 4)
    ctx = G.new_ctx(dims, mass=0.3)
    ctx.set_gauge(F.random_links(dims, seed=21))
    src = F.random_spinor(dims, seed=22, n=2)
    src[0] = 0.0
    b = G.to_internal(ctx, rb.LINKS_F64_18, src)
    x, _ = _solve(ctx, b, 2, rb.MSOLVE_FP64, rb.LINKS_F64_18, 1e-9)
    assert (x[:x.numel() // 2] == 0).all()
    one, _ = _solve(ctx, G.to_internal(ctx, rb.LINKS_F64_18, src[1]), 1, rb.MSOLVE_FP64, rb.LINKS_F64_18, 1e-9)
    assert torch_cuda.equal(x[x.numel() // 2:], one)


def test_short_window_when_memory_is_short(torch_cuda):
    """With too little free memory for the long ring the solve runs windows of half the length; only
    the composition of the shifted updates differs (rounding)."""
    dims = (24, 24, 24, 32)
    nrhs = 4
    spinor = 48 * (24 * 24 * 24 * 32 // 2)
    gen = torch_cuda.Generator(device="cuda")
    gen.manual_seed(5)
    b = torch_cuda.randn(nrhs * 3 * spinor // 48 * 2, generator=gen, device="cuda", dtype=torch_cuda.float64)
    eta = torch_cuda.from_numpy(F.eta_phases(dims).astype(np.float64)).cuda()
    u = eta[:, None, None] * torch_cuda.eye(3, dtype=torch_cuda.complex128, device="cuda")
    out, held = [], []
    for short in (False, True):
        ctx = G.new_ctx(dims, mass=0.3)
        ctx.set_gauge(u.contiguous())
        x = torch_cuda.empty(nrhs * len(SHIFTS) * spinor // 8, dtype=torch_cuda.float64, device="cuda")
        fill = None
        if short:
            # room for the vectors, the short ring and the refinement's reserve, not for the long ring
            need = nrhs * (3 + len(SHIFTS)) * spinor + ctx.Vh * 8 * 96
            ctx.dslash(rb.LINKS_F64_12, 1, x, b, nrhs)  # derived links and launch shapes made beforehand
            ctx.sync()
            torch_cuda.cuda.empty_cache()
            free = torch_cuda.cuda.mem_get_info()[0]
            fill = torch_cuda.empty(free - need - (8 * nrhs + 68 + 16) * spinor, dtype=torch_cuda.uint8, device="cuda")
        ctx.msolve(x, b, SHIFTS, 1e-6, nrhs=nrhs, mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_12)
        torch_cuda.cuda.synchronize()
        held.append(ctx.workspace_bytes())
        out.append(x)
        del fill
        ctx.close()
    assert held[0] - held[1] == 8 * nrhs * spinor  # the ring: 16 or 8 slots
    assert float((out[0] - out[1]).norm() / out[0].norm()) < 1e-13


def test_zero_product_in_the_first_iteration(torch_cuda):
    """A right-hand side that is zero in FP32 but not in FP64 gives <p,s> = 0 in the very first iteration:
    the batch ends with the non-finite error, and the context solves on as if it had not happened."""
    dims = (24, 16, 16, 16)  # too large for one kernel
    ctx = G.new_ctx(dims, mass=0.3)
    ctx.set_gauge(F.random_links(dims, seed=31, kind="near1"))
    src = F.random_spinor(dims, seed=32, n=4)
    b = G.to_internal(ctx, rb.LINKS_F64_18, src)
    args = (4, rb.MSOLVE_FP32, rb.LINKS_F32_12, 1e-3)
    want, _ = _solve(ctx, b, *args)
    src[1] *= 1e-60
    with pytest.raises(rb.RhmcError, match="non-finite"):
        _solve(ctx, G.to_internal(ctx, rb.LINKS_F64_18, src), *args)
    again, _ = _solve(ctx, b, *args)
    assert torch_cuda.equal(want, again)


# two right-hand sides a block (256 chunks), launched FP64, launched FP32 in packs of four
@pytest.mark.parametrize("dims,nrhs,mode,fmt,res", [((16, 16, 16, 16), 2, rb.MSOLVE_FP64, rb.LINKS_F64_18, 1e-8),
                                                    ((16, 16, 16, 16), 4, rb.MSOLVE_FP64, rb.LINKS_F64_12, 1e-8),
                                                    ((24, 16, 16, 16), 4, rb.MSOLVE_FP32, rb.LINKS_F32_12, 1e-4)])
@pytest.mark.parametrize("scale", [0.0, 1e-12])
def test_slots_a_right_hand_side_did_not_write(torch_cuda, dims, nrhs, mode, fmt, res, scale):
    """A right-hand side that is zero (scale 0) or stops after one iteration, beside others that go on, over a
    ring that holds NaN in a later slot of it: its solutions are those of a solve in a new context."""
    if scale and mode == rb.MSOLVE_FP32:
        scale = 1e-8
    src = F.random_spinor(dims, seed=42, n=nrhs)
    src[-1] *= scale
    links = F.random_links(dims, seed=41, kind="near1")
    out = []
    for poison in (False, True):
        ctx = G.new_ctx(dims, mass=0.3)
        ctx.set_gauge(links)
        b = G.to_internal(ctx, rb.LINKS_F64_18, src)
        x, info = _solve(ctx, b, nrhs, mode, fmt, res)
        if poison:
            # the initial residual of a single solve lies in slot 15, which in the ring of nrhs right-hand
            # sides is slot 15 // nrhs of number 15 % nrhs = nrhs - 1
            bad = torch_cuda.full((6 * ctx.Vh,), float("nan"), dtype=torch_cuda.float64, device="cuda")
            with pytest.raises(rb.RhmcError, match="non-finite"):
                _solve(ctx, bad, 1, mode, fmt, res)
            x, info = _solve(ctx, b, nrhs, mode, fmt, res)
        assert info["status"] == 0 and info["iters"][nrhs - 1] == (1 if scale else 0) and info["iters"][0] > 8
        out.append(x)
        ctx.close()
    assert torch_cuda.isfinite(out[0]).all()
    assert torch_cuda.equal(out[0], out[1])
    if not scale:
        assert (out[1][-out[1].numel() // nrhs:] == 0).all()


def test_two_threads_with_different_pole_counts(torch_cuda):
    """Eight right-hand sides with 24 and with 32 poles, both above the default limit of shared memory, in two
    contexts and threads that each capture their solver graph anew."""
    import threading
    dims = (12, 12, 12, 12)
    links = F.random_links(dims, seed=51, kind="near1")
    src = F.random_spinor(dims, seed=52, n=8)
    failed = []

    def work(poles):
        try:
            ctx = G.new_ctx(dims, mass=0.5)
            ctx.set_gauge(links)
            b = G.to_internal(ctx, rb.LINKS_F64_18, src)
            x = torch_cuda.empty(8 * poles * 6 * ctx.Vh, dtype=torch_cuda.float64, device="cuda")
            torch_cuda.cuda.synchronize()
            shifts = np.geomspace(0.1, 50.0, poles)
            for _ in range(40):
                info = ctx.msolve(x, b, shifts, 1e-6, nrhs=8, mode=rb.MSOLVE_FP64, fmt=rb.LINKS_F64_18)
                assert info["status"] == 0
                ctx.call("rhmc_workspace_release")
            ctx.close()
        except Exception as err:
            failed.append(err)

    threads = [threading.Thread(target=work, args=(n,)) for n in (24, 32)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
