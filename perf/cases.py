"""The work a lattice-QCD program has this library do, as cases that can be timed and checked.

Every case goes through ``rhmc_b200.Context`` with device buffers of the caller, on one stream of
the caller, as a molecular-dynamics program does.  Links are exp(i 0.3 H) per link (plaquette
near 0.6, the ordered phase a run spends its time in) with the staggered phases folded in;
spinors and momenta are Gaussian.  Kinds:

  dslash       out = D in onto one parity, n right-hand sides           (operator, every format)
  mdagm        out = (M^dag M + shift) in, n right-hand sides           (operator, every format)
  dslash_host  the same operator on host arrays                         (the reference's own call)
  msolve       multi-shift CG for n pseudofermions and all poles        (force, heatbath, action)
  gauge_steps  the inner gauge sub-steps of a multistep integrator: force, momentum, link update
  fermion_force  the force of all pseudofermions and poles from their shifted solutions
  action       the gauge, momentum and pseudofermion actions of the Metropolis step
  update       one whole RHMC trajectory, heatbath to accept/reject
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rhmc-on-gpu_b200"))
import rhmc_b200 as rb  # noqa: E402
from rhmc_b200 import rational  # noqa: E402

FMT = {name: code for code, name in rb.FMT_NAMES.items()}
MODE = {"fp64": rb.MSOLVE_FP64, "mixed": rb.MSOLVE_MIXED, "fp32": rb.MSOLVE_FP32}
BETA = 5.8


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the operator alone at the size its published rate is quoted on, one right-hand side
        dict(name="dslash_f64_18_n1_32x32x32x32", kind="dslash", dims="32 32 32 32", fmt="f64_18", n=1, parity=1),
        # a ragged lattice (no extent a power of two, no multiple of a thread block), eight right-hand sides
        dict(name="dslash_f32_12_n8_18x14x10x22", kind="dslash", dims="18 14 10 22", fmt="f32_12", n=8, parity=0),
        # the operator of an outside Krylov solver, a batch of four
        dict(name="mdagm_f64_12_n4_24x24x24x32", kind="mdagm", dims="24 24 24 32", fmt="f64_12", n=4),
        # a host program that keeps its fields and calls the operator as the reference's Doe
        dict(name="dslash_host_24x24x24x32", kind="dslash_host", dims="24 24 24 32", parity=1),
        # the smallest solve: the 4^4 lattice of the reference's own run, one pseudofermion
        dict(name="msolve_fp64_n1_4x4x4x4", kind="msolve", dims="4 4 4 4", mode="fp64", fmt="f64_18", n=1, nshift=8, mass=0.1),
        # a medium lattice, two pseudofermions, the reference's algorithm in double precision
        dict(name="msolve_fp64_n2_12x12x12x24", kind="msolve", dims="12 12 12 24", mode="fp64", fmt="f64_18", n=2, nshift=15,
             mass=0.05),
        # four pseudofermions batched, double-precision vectors, compressed links, certified residuals
        dict(name="msolve_mixed_f64_12_n4_24x24x24x32", kind="msolve", dims="24 24 24 32", mode="mixed", fmt="f64_12", n=4,
             nshift=16, mass=0.03),
        # the precision-scheduled solve at the largest everyday size
        dict(name="msolve_mixed_f32_12_n4_32x32x32x32", kind="msolve", dims="32 32 32 32", mode="mixed", fmt="f32_12", n=4,
             nshift=16, mass=0.02),
        # five gauge sub-steps between two fermion kicks
        dict(name="gauge_steps_32x32x32x32", kind="gauge_steps", dims="32 32 32 32", steps=5),
        # the force of two pseudofermions with a degree-15 approximation
        dict(name="fermion_force_n2_s15_24x24x24x32", kind="fermion_force", dims="24 24 24 32", n=2, nshift=15),
        # the three actions before and after a trajectory
        dict(name="action_32x32x32x32", kind="action", dims="32 32 32 32", n=2),
        # a whole small trajectory, where launches and latency count
        dict(name="update_leapfrog_8x8x8x8", kind="update", dims="8 8 8 8", n=1, order=8, steps=6, integrator=rb.INT_LEAPFROG),
    ]


def _dims(rng, lo, hi, most):
    """Even extents in [lo, hi], mostly unequal, at most `most` sites, spread over log volume."""
    target = math.exp(rng.uniform(math.log(lo ** 4), math.log(most)))
    while True:
        d = [2 * max(lo // 2, min(hi // 2, round(target ** 0.25 * rng.uniform(0.7, 1.45) / 2))) for _ in range(4)]
        v = d[0] * d[1] * d[2] * d[3]
        if v <= most and 0.5 * target <= v <= 2 * target:
            return " ".join(map(str, d))


def draw(rng):
    kind = rng.choice(["dslash", "mdagm", "dslash_host", "msolve", "msolve", "gauge_steps", "fermion_force", "action", "update"])
    fmts = ["f64_18", "f64_12", "f32_18", "f32_12"]
    if kind == "dslash":
        return dict(kind=kind, dims=_dims(rng, 4, 40, 32 ** 4), fmt=rng.choice(fmts), n=rng.randint(1, 8), parity=rng.randint(0, 1))
    if kind == "mdagm":
        return dict(kind=kind, dims=_dims(rng, 4, 40, 32 ** 4), fmt=rng.choice(fmts), n=rng.randint(1, 8))
    if kind == "dslash_host":
        return dict(kind=kind, dims=_dims(rng, 4, 40, 32 ** 4), parity=rng.randint(0, 1))
    if kind == "msolve":
        mode, fmt = rng.choice([("fp64", "f64_18"), ("fp64", "f64_12"), ("mixed", "f64_12"), ("mixed", "f32_12"), ("mixed", "f16_12")])
        n = rng.choice([1, 2, 3, 4, 8])
        return dict(kind=kind, dims=_dims(rng, 4, 32, min(24 ** 3 * 32, 1800000 // n)), mode=mode, fmt=fmt, n=n,
                    nshift=rng.randint(1, 20), mass=round(math.exp(rng.uniform(math.log(0.02), math.log(0.2))), 4))
    if kind == "gauge_steps":
        return dict(kind=kind, dims=_dims(rng, 4, 40, 32 ** 4), steps=rng.randint(1, 5))
    if kind == "fermion_force":
        return dict(kind=kind, dims=_dims(rng, 4, 40, 24 ** 3 * 32), n=rng.randint(1, 4), nshift=rng.randint(4, 20))
    if kind == "action":
        return dict(kind=kind, dims=_dims(rng, 4, 40, 32 ** 4), n=rng.randint(1, 4))
    return dict(kind=kind, dims=_dims(rng, 4, 12, 10 ** 4), n=rng.randint(1, 2), order=rng.randint(7, 10), steps=rng.randint(4, 6),
                integrator=rng.choice([rb.INT_LEAPFROG, rb.INT_2MN]))


# ------------------------------------------------------------------ inputs
def _ext(case):
    return tuple(int(v) for v in case["dims"].split())


@functools.lru_cache(maxsize=8)
def _geometry(dims):
    """Even-first site order on the GPU: fwd/bwd[parity][mu] half indices of the neighbours, eta[mu][V]."""
    nx, ny, nz, nt = dims
    V = nx * ny * nz * nt
    lex = torch.arange(V, device="cuda")
    c = [lex % nx, lex // nx % ny, lex // (nx * ny) % nz, lex // (nx * ny * nz)]
    par = (c[0] + c[1] + c[2] + c[3]) % 2
    num = par * (V // 2) + lex // 2
    site = torch.empty_like(lex)
    site[num] = lex
    c = [a[site] for a in c]  # coordinates by site number

    def half(mu, step):
        d = list(c)
        d[mu] = (d[mu] + step) % dims[mu]
        return (d[0] + nx * (d[1] + ny * (d[2] + nz * d[3]))) // 2

    fwd = [half(mu, 1) for mu in range(4)]
    bwd = [half(mu, -1) for mu in range(4)]
    one = torch.ones(V, device="cuda", dtype=torch.float64)
    eta = [one, one - 2 * (c[0] % 2), one - 2 * ((c[0] + c[1]) % 2), one - 2 * ((c[0] + c[1] + c[2]) % 2)]
    eta[3] = torch.where(c[3] == nt - 1, -eta[3], eta[3])  # antiperiodic in time
    Vh = V // 2
    split = lambda t: [[a[:Vh] for a in t], [a[Vh:] for a in t]]
    return split(fwd), split(bwd), torch.stack(eta)


def _unitary(u, eta):
    """Rows orthonormalised in order, row 2 = eta conj(row0 x row1); u (..., 3, 3), eta (...)."""
    r0 = u[..., 0, :] / torch.linalg.vector_norm(u[..., 0, :], dim=-1, keepdim=True)
    r1 = u[..., 1, :] - (r0.conj() * u[..., 1, :]).sum(-1, keepdim=True) * r0
    r1 = r1 / torch.linalg.vector_norm(r1, dim=-1, keepdim=True)
    r2 = eta[..., None] * torch.linalg.cross(r0, r1, dim=-1).conj()
    return torch.stack([r0, r1, r2], dim=-2)


def _algebra(n, gen):
    """n traceless Hermitian matrices sum_a w_a lambda_a, w_a ~ N(0, 1/2)."""
    w = torch.randn(n, 8, generator=gen, device="cuda", dtype=torch.float64) * math.sqrt(0.5)
    m = torch.zeros(n, 3, 3, dtype=torch.complex128, device="cuda")
    s3 = 1 / math.sqrt(3.0)
    m[:, 0, 0], m[:, 1, 1], m[:, 2, 2] = (w[:, 2] + s3 * w[:, 7]).to(m.dtype), (s3 * w[:, 7] - w[:, 2]).to(m.dtype), (-2 * s3 * w[:, 7]).to(m.dtype)
    for (i, j), a in (((0, 1), 0), ((0, 2), 3), ((1, 2), 5)):
        m[:, i, j] = torch.complex(w[:, a], -w[:, a + 1])
        m[:, j, i] = torch.complex(w[:, a], w[:, a + 1])
    return m


def _taylor(x, order):
    r = torch.eye(3, dtype=x.dtype, device=x.device) + x
    t = x
    for k in range(2, order + 1):
        t = _mm(t, x) / k
        r = r + t
    return r


def _inputs(case, seed):
    """Links (4V, 3, 3), momenta (4V, 3, 3) and spinors (m, 3, Vh), made from the seed on the GPU."""
    dims = _ext(case)
    V = dims[0] * dims[1] * dims[2] * dims[3]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000003 * seed + 17)
    eta = _geometry(dims)[2].reshape(-1)
    h = _taylor(0.3j * _algebra(4 * V, gen), 12)
    u = _unitary(h, torch.ones_like(eta)) * eta[:, None, None]
    mom = _algebra(4 * V, gen) if case["kind"] in ("gauge_steps", "action", "update") else None
    m = case.get("n", 1) * (case["nshift"] if case["kind"] == "fermion_force" else 1)
    s = torch.randn(m, 3, V // 2, generator=gen, device="cuda", dtype=torch.complex128)
    if case.get("fmt", "f64").startswith("f32") and case["kind"] in ("dslash", "mdagm"):
        s = s.to(torch.complex64)
    return u, mom, s


def _shifts(case):
    """The poles of a rational approximation are spread evenly over the logarithm of the spectrum."""
    return np.geomspace(1e-4, 50.0, case["nshift"]) if case["nshift"] > 1 else np.array([1e-3])


def _residual(case):
    """Absolute target of a solve, 1e-10 of the right-hand side's expected norm."""
    d = _ext(case)
    return 1e-10 * math.sqrt(1.5 * d[0] * d[1] * d[2] * d[3])


def _numerators(case):
    return np.geomspace(1e-3, 2.0, case["nshift"])


@functools.lru_cache(maxsize=32)
def _approximations(order, n):
    """N_f = 2, n pseudofermions, am = 0.1: heatbath, force and action approximations."""
    eps = 0.9 * 0.01 / (1.05 * 16.01)
    power = (1 / (4 * n), -1 / (2 * n), -1 / (2 * n))
    return tuple(rational.rational_power(p, order, eps) for p in power)


@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()


def prepare(case, seed):
    kind, dims = case["kind"], _ext(case)
    u, mom, s = _inputs(case, seed)
    mass = case.get("mass", 0.1)
    ctx = rb.Context(dims, mass=mass, beta=BETA)
    ctx.set_stream(_stream().cuda_stream)
    torch.cuda.synchronize()
    ctx.set_gauge(u)
    st = dict(case=case, ctx=ctx, u=u, spinors=s)
    if kind in ("dslash", "mdagm"):
        st["out"] = torch.empty_like(s)
    elif kind == "dslash_host":
        st["inp"] = s[0].t().contiguous().cpu().pin_memory().numpy()
        st["out"] = torch.empty(s.shape[2], 3, dtype=torch.complex128).pin_memory().numpy()
    elif kind == "msolve":
        st["x"] = torch.empty(case["n"] * case["nshift"], 3, s.shape[2], dtype=torch.complex128, device="cuda")
    elif kind == "fermion_force":
        st["ip"] = torch.empty_like(u)
    elif kind == "action":
        ctx.set_momenta(mom)
    elif kind in ("gauge_steps", "update"):
        st["mom"], st["u_out"], st["p_out"] = mom, torch.empty_like(u), torch.empty_like(u)
    if kind == "update":
        st["phi"] = s.transpose(1, 2).contiguous().cpu().numpy()
        ctx.driver_setup(no_flavours=2, no_ps=case["n"], no_md=case["steps"], integrator=case["integrator"], residue_metro=1e-10,
                         residue_md=1e-8)
        for which, ap in enumerate(_approximations(case["order"], case["n"])):
            ctx.set_approx(which, ap)
        ctx.set_eig_bounds(0.01, 16.01)
    ctx.sync()
    return st


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "dslash":
        ctx.dslash(FMT[case["fmt"]], case["parity"], st["out"], st["spinors"], case["n"])
        return st["out"]
    if kind == "mdagm":
        ctx.mdagm(FMT[case["fmt"]], st["out"], st["spinors"], 0.05, case["n"])
        return st["out"]
    if kind == "dslash_host":
        ctx.dslash_host(case["parity"], st["out"], st["inp"])
        return st["out"]
    if kind == "msolve":
        ctx.msolve(st["x"], st["spinors"], _shifts(case), _residual(case), nrhs=case["n"], mode=MODE[case["mode"]],
                   fmt=FMT[case["fmt"]])
        return st["x"]
    if kind == "fermion_force":
        ctx.fermion_force(st["spinors"], _numerators(case), nrhs=case["n"])
        ctx.get_ipdot(st["ip"])
        return st["ip"]
    if kind == "action":
        return [ctx.gauge_action(), ctx.momentum_action(), ctx.rdot(st["spinors"], st["spinors"], case["n"])]
    ctx.set_gauge(st["u"])
    ctx.set_momenta(st["mom"])
    if kind == "gauge_steps":
        for _ in range(case["steps"]):
            ctx.gauge_force()
            ctx.mom_update(-0.02)
            ctx.link_update(0.02)
        ctx.get_gauge(st["u_out"])
        ctx.get_momenta(st["p_out"])
        return [st["u_out"], st["p_out"]]
    ctx.set_phi(st["phi"])
    delta_s, _ = ctx.update(0.0)  # accepted unless exp(-delta_s) is zero
    ctx.get_gauge(st["u_out"])
    ctx.get_momenta(st["p_out"])
    return [delta_s, st["u_out"], st["p_out"]]


# ------------------------------------------------------------------ work and tolerances
def _cg_iterations(mass, shift, reduction):
    """The classical count for conjugate gradients on a spectrum m^2 + [0.007, 6] (what these links give)."""
    kappa = (mass * mass + shift + 6.0) / (mass * mass + shift + 0.007)
    return 0.5 * math.sqrt(kappa) * math.log(2.0 / reduction)


def _solve_work(V, n, nshift, its, link, real):
    """An iteration reads the links twice (both half operators); direction, residual and product vectors pass
    the smallest number of times; what the L2 can hold is read from memory once."""
    site = 3 * 2 * real
    per = 2 * 4 * V * link + n * (V // 2) * site * 10
    if per > 100e6:
        dram = its * per + n * nshift * (V // 2) * 48 * 2
    else:
        dram = 4 * V * link + n * (nshift + 1) * (V // 2) * 48
    return {"bytes": dram, "flops": its * n * V * 576.0 + its * n * (V // 2) * 60.0}


def work(case):
    kind, d = case["kind"], _ext(case)
    V = d[0] * d[1] * d[2] * d[3]
    Vh, n = V // 2, case.get("n", 1)
    if kind in ("dslash", "mdagm"):
        real = 8 if case["fmt"].startswith("f64") else 4
        link = real * (18 if case["fmt"].endswith("18") else 12)
        return {"bytes": 4 * V * link + 2 * n * Vh * 6 * real, "flops": n * Vh * 573.0 * (2 if kind == "mdagm" else 1)}
    if kind == "dslash_host":
        return {"bytes": 4 * V * 144 + 2 * Vh * 48, "flops": Vh * 573.0}
    if kind == "msolve":
        sh = _shifts(case)
        base = sh[0] if case["mode"] != "fp64" else 0.0
        its = _cg_iterations(case["mass"], base, 1e-10)
        low = case["fmt"] in ("f32_12", "f16_12")
        return _solve_work(V, n, case["nshift"], its, 48 if low else (144 if case["fmt"] == "f64_18" else 96), 4 if low else 8)
    force = V * 46 * 198.0 + 4 * V * 100.0  # seven products per plane (the two upper staples share one), U S, TA
    if kind == "gauge_steps":
        per = 4 * V * (144 + 128 + 64 + 288)  # force and momentum in one pass, then the links
        return {"bytes": case["steps"] * per, "flops": case["steps"] * (force + 4 * V * 1500.0)}
    if kind == "fermion_force":
        m = n * case["nshift"]
        return {"bytes": 4 * V * 144 + m * Vh * 48 + 4 * V * 144, "flops": m * (Vh * 573.0 + 4 * V * 72.0)}
    if kind == "action":
        return {"bytes": 4 * V * (144 + 64) + n * Vh * 48, "flops": V * 6 * (2 * 198.0 + 36)}
    its = _cg_iterations(0.1, 0.0, 1e-9)
    solves = 2 + case["steps"] * (2 if case["integrator"] == rb.INT_2MN else 1)
    w = _solve_work(V, n, case["order"], its, 144, 8)
    return {"bytes": solves * (w["bytes"] + 4 * V * 700), "flops": solves * (w["flops"] + force)}


def tolerance(case):
    """About four times the error against exact() over the ranges of draw()."""
    kind = case["kind"]
    if kind in ("dslash", "mdagm"):
        return {"rel": 1.5e-15 if case["fmt"].startswith("f64") else 5e-7}
    if kind == "dslash_host":
        return {"rel": 1.5e-15}
    if kind == "msolve":
        # the target is 1e-10 |b|; the smallest pole's solution carries it over the smallest eigenvalue
        return {"rel": 3e-9}
    if kind == "action":
        return {"rel": 2e-14}
    if kind == "update":
        return {"rel": 5e-10, "max": 2e-8}
    return {"rel": 2e-15}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _mm(a, b):
    """Product of stacks of 3x3 matrices."""
    return (a[..., :, :, None] * b[..., None, :, :]).sum(-2) if a.numel() < 4e6 else _mm_big(a, b)


def _mm_big(a, b):
    r = a[..., :, 0:1] * b[..., 0:1, :]
    r += a[..., :, 1:2] * b[..., 1:2, :]
    r += a[..., :, 2:3] * b[..., 2:3, :]
    return r


def _dag(a):
    return a.conj().transpose(-1, -2)


class _Exact:
    """The operator, solver, forces and updates on links u (4V, 3, 3)."""

    def __init__(self, dims, u, mass):
        self.dims, self.m2 = dims, mass * mass
        self.fwd, self.bwd, self.eta = _geometry(dims)
        self.V = dims[0] * dims[1] * dims[2] * dims[3]
        self.Vh = self.V // 2
        self.set(u)

    def set(self, u):
        self.u = u.reshape(4, 2, self.Vh, 3, 3)
        self.planes = None

    def hop(self, p, v):
        """1/2 sum_mu [U_mu(x) v(x+mu) - U_mu(x-mu)^dag v(x-mu)] on parity p; v (n, 3, Vh)."""
        if self.planes is None:
            self.planes = self.u.permute(0, 1, 3, 4, 2).contiguous()
        out = torch.zeros_like(v)
        for mu in range(4):
            f, b = self.fwd[p][mu], self.bwd[p][mu]
            vf, vb, uf, ub = v[:, :, f], v[:, :, b], self.planes[mu, p], self.planes[mu, 1 - p][:, :, b].conj()
            for i in range(3):
                for j in range(3):
                    out[:, i].addcmul_(uf[i, j], vf[:, j])
                    out[:, i].addcmul_(ub[j, i], vb[:, j], value=-1)
        return out.mul_(0.5)

    def mdagm(self, v, shift=0.0):
        return (self.m2 + shift) * v - self.hop(0, self.hop(1, v))

    def solve(self, b, shifts, target=1e-13):
        """(M^dag M + s) x = b for every s and right-hand side: multi-shift CG on the smallest shift."""
        s0 = min(shifts)
        n, S = b.shape[0], len(shifts)
        col = lambda a: a[:, None, None]
        dot = lambda x, y: (x.conj() * y).sum((1, 2)).real
        x = torch.zeros((S,) + tuple(b.shape), dtype=b.dtype, device=b.device)
        ps = b.expand_as(x).clone()
        r, p = b.clone(), b.clone()
        rr = dot(r, r)
        stop = float((target * rr.max().sqrt()) ** 2)
        z, zo = torch.ones(S, n, dtype=torch.float64, device=b.device), torch.ones(S, n, dtype=torch.float64, device=b.device)
        ao, be = torch.ones_like(rr), torch.zeros_like(rr)
        rel = torch.tensor([s - s0 for s in shifts], dtype=torch.float64, device=b.device)[:, None]
        for it in range(20000):
            q = self.mdagm(p, s0)
            al = rr / dot(p, q)
            zn = z * zo * ao / (al * be * (zo - z) + zo * ao * (1 + rel * al))
            x += (al * zn / z)[:, :, None, None] * ps
            r = r - col(al) * q
            rn = dot(r, r)
            bn = rn / rr
            ps.mul_((bn * (zn / z) ** 2)[:, :, None, None]).add_(zn[:, :, None, None] * r)
            p = r + col(bn) * p
            zo, z, ao, be, rr = z, zn, al, bn, rn
            if it % 8 == 7 and float(rr.max()) <= stop:
                break
            z, zo = z.clamp_min(1e-150), zo.clamp_min(1e-150)
        return x.transpose(0, 1).contiguous()  # [rhs][shift]

    def at(self, mu, field, step):
        """field (2, Vh, ...) at x + step mu, by parity of x."""
        t = self.fwd if step > 0 else self.bwd
        return torch.stack([field[1][t[0][mu]], field[0][t[1][mu]]])

    def gauge_force(self):
        u, out = self.u, []
        for mu in range(4):
            S = torch.zeros_like(u[0])
            for nu in range(4):
                if nu == mu:
                    continue
                un = self.at(mu, u[nu], +1)
                S += _mm(_mm(un, _dag(self.at(nu, u[mu], +1))), _dag(u[nu]))
                low = _mm(_dag(_mm(u[mu], un)), u[nu])
                S += self.at(nu, low, -1)
            out.append((BETA / 3) * _mm(u[mu], S))
        return torch.stack(out)

    def fermion_force(self, x, num):
        """U F from the solutions x (m, 3, Vh) with numerators num (m,)."""
        h = self.hop(1, x)
        out = []
        for mu in range(4):
            F = torch.zeros(2, 3, 3, self.Vh, dtype=torch.complex128, device="cuda")
            for v in range(x.shape[0]):
                le, lo = num[v] * h[v][:, self.fwd[0][mu]], -num[v] * x[v][:, self.fwd[1][mu]]
                F[0] += le[:, None] * x[v].conj()[None]
                F[1] += lo[:, None] * h[v].conj()[None]
            out.append(_mm(self.u[mu], F.permute(0, 3, 1, 2)))
        return torch.stack(out)

    @staticmethod
    def ta(m):
        a = 0.5 * (m - _dag(m))
        tr = torch.diagonal(a, dim1=-2, dim2=-1).sum(-1) / 3
        return a - tr[..., None, None] * torch.eye(3, dtype=m.dtype, device=m.device)

    def drift(self, p, step):
        e = _unitary(_taylor(1j * step * p, 6), torch.ones(p.shape[:-2], dtype=torch.float64, device=p.device))
        self.set(_unitary(_mm(e, self.u), self.eta.reshape(4, 2, self.Vh)))

    def plaquettes(self):
        t = 0.0
        for mu in range(4):
            for nu in range(mu):
                a = _mm(self.u[nu], self.at(nu, self.u[mu], +1))
                b = _mm(self.u[mu], self.at(mu, self.u[nu], +1))
                t += float((a * b.conj()).real.sum())
        return BETA / 3 * t


def exact(case, seed):
    kind, dims = case["kind"], _ext(case)
    V = dims[0] * dims[1] * dims[2] * dims[3]
    n = case.get("n", 1)
    if kind == "msolve":
        its = 1.2 * _cg_iterations(case["mass"], _shifts(case)[0], 1e-13)
        if its * (6e-3 + V * n * (2 + 0.1 * case["nshift"]) * 1e-9) > 15:
            return None
    u, mom, s = _inputs(case, seed)
    mass = case.get("mass", 0.1)
    E = _Exact(dims, u, mass)
    s = s.to(torch.complex128)
    if kind == "dslash":
        return E.hop(case["parity"], s)
    if kind == "mdagm":
        return E.mdagm(s, 0.05)
    if kind == "dslash_host":
        return E.hop(case["parity"], s)[0].t().contiguous().cpu().numpy()
    if kind == "msolve":
        x = E.solve(s, [float(v) for v in _shifts(case)])
        return x.reshape(n * case["nshift"], 3, V // 2)
    if kind == "fermion_force":
        return E.ta(E.fermion_force(s, list(_numerators(case)) * n)).reshape(4 * V, 3, 3)
    if kind == "action":
        return [E.plaquettes(), 0.5 * float((mom.abs() ** 2).sum()), float((s.abs() ** 2).sum())]
    p = mom.reshape(4, 2, V // 2, 3, 3)
    if kind == "gauge_steps":
        for _ in range(case["steps"]):
            p = p + 1j * (-0.02) * E.ta(E.gauge_force())
            E.drift(p, 0.02)
        return [E.u.reshape(4 * V, 3, 3), p.reshape(4 * V, 3, 3)]
    aps = _approximations(case["order"], n)
    power = (1 / (4 * n), -1 / (2 * n), -1 / (2 * n))
    mx = 1.05 * 16.01
    aps = [dict(a0=a["a0"] * mx ** e, a=[v * mx * mx ** e for v in a["a"]], b=[v * mx for v in a["b"]]) for a, e in zip(aps, power)]

    def apply(ap, v):
        x = E.solve(v, ap["b"], 1e-14)
        return ap["a0"] * v + (torch.tensor(ap["a"], dtype=v.dtype, device=v.device)[None, :, None, None] * x).sum(1)

    def force():
        x = E.solve(chi, aps[1]["b"], 1e-14).reshape(-1, 3, V // 2)
        return E.ta(E.gauge_force() + E.fermion_force(x, list(aps[1]["a"]) * n))

    chi = apply(aps[0], s)
    s0 = E.plaquettes() + 0.5 * float((p.abs() ** 2).sum()) + float((s.abs() ** 2).sum())
    eps, L = 1.0 / case["steps"], 0.1931833275037836
    if case["integrator"] == rb.INT_LEAPFROG:
        plan = [("u", eps / 2)] + [("p", eps), ("u", eps)] * (case["steps"] - 1) + [("p", eps), ("u", eps / 2)]
    else:
        body = [("p", eps / 2), ("u", eps * (1 - 2 * L)), ("p", eps / 2)]
        plan = [("u", eps * L)] + (body + [("u", 2 * eps * L)]) * (case["steps"] - 1) + body + [("u", eps * L)]
    for what, c in plan:
        if what == "u":
            E.drift(p, c)
        else:
            p = p - 1j * c * force()
    phi = apply(aps[2], chi)
    s1 = E.plaquettes() + 0.5 * float((p.abs() ** 2).sum()) + float((phi.conj() * chi).sum().real)
    new = E.u.reshape(4 * V, 3, 3) if s1 < s0 or math.exp(s0 - s1) > 0.0 else u
    return [s1 - s0, new, p.reshape(4 * V, 3, 3)]
