"""Performance cases of the BSE solvers: what is timed, on which inputs, and what
the results are in plain 64-bit arithmetic.

A case is one call that a spectrum calculation makes, through the library's own
bindings: a Haydock run of a core-level or a valence Hamiltonian, one H psi with
host vectors (the drop-in for OCEAN_xact), a batch of core sites, or a GMRES
spectrum with its gradient.  Sizes are those of the benchmark and test workloads
(ocean_gb300/workloads.py) and ragged ones between them: k-meshes 2..8 per axis,
cubic or not, 24 to 128 bands, x-meshes 6^3 to 12^3, 1s and 2p edges, one or
three polarisations, one or two spins, both precisions.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  contexts and start vectors as a user's program holds them
  run(state)           one pass
  work(case)           bytes and flops one pass cannot do without
  exact(case, seed)    the same results from torch in complex128

The Bloch functions are orthonormal per k-point, the screened potential is
erf(r/a)/(eps r), energies are spread over 30 eV and the lowest states of the
window are masked out, as in a run on a real material.
"""
import itertools
import math
import random
import types

import numpy as np
import torch

from ocean_gb300 import adjoint, capi
from ocean_gb300 import workloads as WL

EV = WL.EV2HARTREE
A_BOHR = 4.0 / WL.BOHR
CELVOL = A_BOHR ** 3
EPS0 = 4.0
DEV = "cuda:0"


# ------------------------------------------------------------------- the cases

def _core(name, kmesh, nb, xmesh, prec, call, niter=0, nv=1, lc=0, mult=False, nspn=1):
    return dict(name=name, call=call, k1=kmesh[0], k2=kmesh[1], k3=kmesh[2], nb=nb, x1=xmesh[0], x2=xmesh[1],
                x3=xmesh[2], prec=prec, niter=niter, nv=nv, lc=lc, mult=mult, nspn=nspn)


def _val(name, kmesh, nc, nvb, xmesh, prec, niter):
    return dict(name=name, call="val_haydock", k1=kmesh[0], k2=kmesh[1], k3=kmesh[2], nc=nc, nvb=nvb, x1=xmesh[0],
                x2=xmesh[1], x3=xmesh[2], prec=prec, niter=niter)


def listed():
    return [
        # the plain 1s example (4^3 k, 32 bands): a short mixed-precision run and its spectrum, where launches count
        _core("k4_1s_mixed_spectrum", (4, 4, 4), 32, (8, 8, 8), "mixed", "spectrum", niter=60),
        # the same example through the drop-in call of OCEAN_xact: FP64 (the default precision), host vectors
        _core("k4_1s_fp64_xact", (4, 4, 4), 32, (8, 8, 8), "fp64", "xact"),
        # the benchmark's 1s workload (8^3 k, 100 bands, 12^3 x), mixed precision and FP64
        _core("k8_1s_mixed", (8, 8, 8), 100, (12, 12, 12), "mixed", "haydock", niter=45),
        _core("k8_1s_fp64", (8, 8, 8), 100, (12, 12, 12), "fp64", "haydock", niter=6),
        # the 2p edge with multiplet and spin-orbit terms (12 channels), both precisions
        _core("k6_2p_mult_mixed", (6, 6, 6), 64, (10, 10, 10), "mixed", "haydock", niter=45, lc=1, mult=True),
        _core("k6_2p_mult_fp64", (6, 6, 6), 64, (10, 10, 10), "fp64", "haydock", niter=9, lc=1, mult=True),
        # three polarisations of one site on a mesh without symmetry, FP64
        _core("k765_3pol_fp64", (7, 6, 5), 53, (9, 10, 11), "fp64", "haydock", niter=9, nv=3),
        # a block of three host vectors, spin-polarised Bloch functions, ragged sizes, mixed precision
        _core("k465_spin_block_mixed", (4, 6, 5), 75, (10, 9, 8), "mixed", "xact", nv=3, nspn=2),
        # a batch of uneven sites, three polarisations each, in shared launches
        dict(name="batch12_mixed", call="batch", count=12, mix=1, niter=30, prec="mixed"),
        # differentiable GMRES spectrum: forward solves and the adjoint solves behind the gradient, FP64
        dict(name="k4_gmres_grad_fp64", call="gmres_grad", k1=4, k2=4, k3=4, nb=32, x1=8, x2=8, x3=8, prec="fp64",
             nomega=12, lc=0, nspn=1, nv=1, mult=False),
        # valence BSE: the benchmark's silicon-like case in mixed precision, a smaller one in FP64
        _val("val_k8_mixed", (8, 8, 8), 8, 4, (10, 10, 10), "mixed", 5),
        _val("val_k6_fp64", (6, 6, 6), 6, 4, (7, 7, 7), "fp64", 5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    prec = rng.choice(["fp64", "mixed"])
    what = rng.choice(["haydock", "haydock", "haydock", "xact", "xact", "batch", "gmres_grad", "val", "val"])
    if what == "batch":
        return dict(call="batch", count=rng.randint(3, 12), mix=rng.randint(2, 10 ** 6), niter=3 * rng.randint(3, 8),
                    prec="mixed")
    cubic = rng.random() < 0.5 or what == "gmres_grad"
    while True:
        n = rng.choice([3, 4, 5, 6, 8])
        km = (n, n, n) if cubic else tuple(rng.randint(2, 8) for _ in range(3))
        if math.prod(km) >= 12:
            break
    if what == "val":
        nvb, nc = rng.randint(1, 4), rng.randint(2, 10)
        most = 400 if prec == "fp64" else 1000
        while True:
            xm = tuple(rng.randint(4, 10) for _ in range(3))
            if 4 * (nvb + nc) <= math.prod(xm) <= most and math.prod(xm) ** 2 * math.prod(km) <= 3e8:
                break
            if math.prod(km) > 300 and prec == "fp64":
                most = 300
        c = _val("", km, nc, nvb, xm, prec, rng.randint(2, 5))
        del c["name"]
        return c
    if what == "gmres_grad":
        n = rng.choice([3, 4, 5])
        m = rng.randint(6, 9)
        return dict(call="gmres_grad", k1=n, k2=n, k3=n, nb=_log_int(rng, 16, 40), x1=m, x2=m, x3=m, prec=prec,
                    nomega=rng.randint(4, 10), lc=0, nspn=1, nv=1, mult=False)
    lc = 1 if rng.random() < 0.3 else 0
    nb = _log_int(rng, 24, 128)
    while True:
        xm = tuple(rng.randint(6, 12) for _ in range(3))
        if math.prod(xm) >= 2 * nb and math.prod(xm) * math.prod(km) * nb * (3 if lc else 1) <= 8.8e7:
            break
        nb = max(24, nb - 8)
    c = _core("", km, nb, xm, prec, what, niter=rng.randint(4, 12) if what == "haydock" else 0,
              nv=rng.choice([1, 1, 2, 3]), lc=lc, mult=bool(lc) and rng.random() < 0.5, nspn=rng.choice([1, 1, 1, 2]))
    del c["name"]
    return c


# -------------------------------------------------------------- core-level inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + 11)
    return g


def _randn_c(g, *shape):
    return torch.complex(torch.randn(shape, generator=g, device=DEV, dtype=torch.float64),
                         torch.randn(shape, generator=g, device=DEV, dtype=torch.float64))


def _orthonormal(g, nk, nx, nb):
    """(nk, nx, nb): nb orthonormal columns per k-point (Cholesky QR of a Gaussian)."""
    a = _randn_c(g, nk, nx, nb)
    low = torch.linalg.cholesky(a.mH @ a)
    return torch.linalg.solve_triangular(low.mH.contiguous(), a, upper=True, left=False)


def _core_inputs(c, seed):
    """Everything a core-level case is made of: torch tensors on the device, spin-major."""
    g = _gen(seed)
    km, xm = (c["k1"], c["k2"], c["k3"]), (c["x1"], c["x2"], c["x3"])
    nk, nx, nb, na = math.prod(km), math.prod(xm), c["nb"], 4 * (2 * c["lc"] + 1)
    d = types.SimpleNamespace(km=km, xm=xm, nk=nk, nx=nx, nb=nb, na=na, nspn=c["nspn"], lc=c["lc"], nv=c["nv"])
    d.u = torch.stack([_orthonormal(g, nk, nx, nb) for _ in range(c["nspn"])])  # (s, k, x, n)
    e = torch.sort(30.0 * torch.rand((nk, nb), generator=g, device=DEV, dtype=torch.float64), dim=1).values * EV
    d.er = e[None].expand(na, nk, nb).contiguous()
    d.allow = (d.er > 0.2 * EV).double()
    psi = _randn_c(g, c["nv"], na, nk, nb)
    norm = torch.linalg.vector_norm(psi.reshape(c["nv"], -1), dim=1)
    d.kpref = 4.0 * math.pi * float(norm[0]) ** 2 / (nk * CELVOL ** 2)
    d.psi = psi / norm[:, None, None, None]
    d.rtab, d.ptab = WL.w_table(EPS0)
    d.mult = None
    d.so_xi = 0.0
    if c["mult"]:
        lmax, npl = 3, 8
        nm = 2 * lmax + 1
        m = _randn_c(g, c["nspn"], lmax + 1, nm, npl, nk, nb) / math.sqrt(2.0 * nb * nk)
        for l in range(lmax + 1):
            m[:, l, :lmax - l] = 0.0
            m[:, l, lmax + l + 1:] = 0.0
        mono = 0.5 + 7.5 * torch.rand((lmax + 1, npl, npl), generator=g, device=DEV, dtype=torch.float64)
        d.mpm = 0.5 * (mono + mono.mT) * EV
        d.mh = []
        for l in range(lmax + 1):
            h = _randn_c(g, *(2 * (na * (2 * l + 1) * npl,))) * (0.05 * EV)
            d.mh.append(0.5 * (h + h.mH))
        d.mult, d.mpc, d.lmax, d.npl = True, m, lmax, npl
        d.so_xi = 5.0 * EV
    return d


def _flat(t):
    return t.contiguous().reshape(-1).cpu().numpy()


def _core_workload(d):
    """The workload record the bindings take, in the reference's (Fortran) orders."""
    avec = np.zeros(9)
    avec[0] = avec[4] = avec[8] = A_BOHR
    u = d.u.permute(0, 2, 1, 3)  # (s, x, k, n)
    psi = d.psi[0]
    w = WL.Workload(name="case", nb=d.nb, kmesh=d.km, xmesh=d.xm, na=d.na, nspn=d.nspn, core_l=d.lc, celvol=CELVOL,
                    avec=avec, tau=np.zeros(3), epsilon0=EPS0, interaction_scale=1.0, rtab=d.rtab, ptab=d.ptab,
                    er=_flat(d.er), ei=np.zeros(d.er.numel()), allow=_flat(d.allow), ur=_flat(u.real), ui=_flat(u.imag),
                    psi_r=_flat(psi.real), psi_i=_flat(psi.imag), kpref=d.kpref)
    if d.mult:
        mh = torch.cat([h.reshape(-1) for h in d.mh])
        w.mult = dict(lmin=0, lmax=d.lmax, nproj=np.full(d.lmax + 1, d.npl, dtype=np.int32), npmax=d.npl,
                      mpcr=_flat(d.mpc.real), mpci=_flat(d.mpc.imag), mpm=_flat(d.mpm), mhr=_flat(mh.real),
                      mhi=_flat(mh.imag))
        w.so_xi = d.so_xi
    return w


def _planes(psi):
    """(nv, npsi) complex -> nv blocks of (re plane, im plane), the device layout of a block."""
    f = psi.reshape(psi.shape[0], -1)
    return torch.stack([f.real, f.imag], dim=1).contiguous()


def _prec(c):
    return capi.OCN_PREC_FP64 if c["prec"] == "fp64" else capi.OCN_PREC_MIXED


def _core_context(c, seed):
    d = _core_inputs(c, seed)
    w = _core_workload(d)
    ctx = capi.Context(w, precision=_prec(c), nvec=c["nv"])
    w.ur = w.ui = None  # the context keeps its own copy
    return types.SimpleNamespace(case=c, w=w, ctx=ctx, psi=_planes(d.psi), host=(
        np.ascontiguousarray(_flat(d.psi.real).reshape(c["nv"], -1)),
        np.ascontiguousarray(_flat(d.psi.imag).reshape(c["nv"], -1))))


def _batch_members(c):
    """Member shapes of a batch: k-mesh n^3, n in {4, 5, 6, 8}, 24..128 bands, x-mesh 8^3..10^3, 1s or 2p."""
    r = random.Random(c["mix"])
    out = []
    for i in range(c["count"]):
        n, m = r.choice([4, 5, 6, 8]), r.randint(8, 10)
        nb = r.randint(24, 128)
        lc = r.randint(0, 1) if n < 8 else 0
        out.append(dict(k1=n, k2=n, k3=n, nb=nb, x1=m, x2=m, x3=m, prec=c["prec"], nv=3, lc=lc, mult=False, nspn=1))
    return out


# ------------------------------------------------------------------- valence inputs

def _lattice_r(km):
    """Integer lattice vectors of the k-mesh in FFT order, k3 fastest, with the images of a Nyquist index."""
    axes = [[[j - n, j] if 2 * j == n else [j if j < (n + 1) // 2 else j - n] for j in range(n)] for n in km]
    return [list(itertools.product(*o)) for o in itertools.product(*axes)]


def _val_ladder(km, xm):
    """ladder(k, x, y) as (y, x, k): the smoothed screened interaction W(|R + x - y|) of the synthetic workloads."""
    nk = math.prod(km)
    a = 0.5 / WL.BOHR
    q = (6.0 * math.pi ** 2 / (CELVOL * nk)) ** (1.0 / 3.0)
    images = _lattice_r(km)
    most = max(len(i) for i in images)
    R = torch.zeros((nk, most, 3), dtype=torch.float64, device=DEV)
    wt = torch.zeros((nk, most), dtype=torch.float64, device=DEV)
    rows = torch.tensor([list(i) + [(0, 0, 0)] * (most - len(i)) for i in images], dtype=torch.float64)
    R.copy_(rows)
    wt.copy_(torch.tensor([[1.0 / len(i)] * len(i) + [0.0] * (most - len(i)) for i in images], dtype=torch.float64))
    spans = [torch.arange(-(n - 1), n, dtype=torch.float64, device=DEV) / n for n in xm]
    diff = torch.stack(torch.meshgrid(*spans, indexing="ij"), dim=-1).reshape(-1, 3)  # every x - y
    table = torch.empty((diff.shape[0], nk), dtype=torch.float64, device=DEV)
    for lo in range(0, diff.shape[0], 512):
        r = A_BOHR * torch.linalg.vector_norm(diff[lo:lo + 512, None, None, :] + R[None], dim=-1)
        s = r.clamp_min(1e-9)
        pot = torch.where(r > 0, torch.erf(s / a) / (EPS0 * s), torch.full_like(r, 2.0 / (a * math.sqrt(math.pi) * EPS0)))
        t = (q * r).clamp_min(1e-6)
        f = torch.where(q * r > 1e-6, 3.0 * (torch.sin(t) - t * torch.cos(t)) / t ** 3, torch.ones_like(r))
        table[lo:lo + 512] = (pot * f * f * wt).sum(-1)
    pos = torch.stack(torch.meshgrid(*[torch.arange(n, device=DEV) for n in xm], indexing="ij"), dim=-1).reshape(-1, 3)
    d = pos[None, :, :] - pos[:, None, :] + torch.tensor([n - 1 for n in xm], device=DEV)  # (y, x, 3)
    flat = (d[..., 0] * (2 * xm[1] - 1) + d[..., 1]) * (2 * xm[2] - 1) + d[..., 2]
    return table[flat.reshape(-1)].reshape(len(pos), len(pos), nk)


def _val_bubble(xm, nk):
    """4 pi / (V Nk G^2) in FFT order, G = 0 removed."""
    ax = [np.fft.fftfreq(n, 1.0 / n) for n in xm]
    g2 = sum(v ** 2 for v in np.meshgrid(*ax, indexing="ij")) * (2.0 * math.pi / A_BOHR) ** 2
    b = np.zeros(xm)
    b[g2 > 0] = 4.0 * math.pi / (CELVOL * nk * g2[g2 > 0])
    return b.reshape(-1)


def _val_inputs(c, seed):
    g = _gen(seed)
    km, xm = (c["k1"], c["k2"], c["k3"]), (c["x1"], c["x2"], c["x3"])
    nk, nx, nc, nv = math.prod(km), math.prod(xm), c["nc"], c["nvb"]
    d = types.SimpleNamespace(km=km, xm=xm, nk=nk, nx=nx, nc=nc, nv=nv)
    st = _orthonormal(g, nk, nx, nc + nv).mT  # (k, band, x)
    d.val, d.con = st[:, :nv].contiguous(), st[:, nv:].contiguous()
    ev = torch.sort(-8.0 * torch.rand((nk, nv), generator=g, device=DEV, dtype=torch.float64), dim=1).values
    ec = torch.sort(1.0 + 15.0 * torch.rand((nk, nc), generator=g, device=DEV, dtype=torch.float64), dim=1).values
    d.er = (ec[:, None, :] - ev[:, :, None]) * EV  # (k, v, c)
    d.allow = torch.ones_like(d.er)
    psi = _randn_c(g, nk, nv, nc)
    norm = float(torch.linalg.vector_norm(psi.reshape(-1)))
    d.kpref = 4.0 * math.pi * norm ** 2 / (nk * CELVOL ** 2)
    d.psi = psi / norm
    d.ladder = _val_ladder(km, xm)
    d.bubble = _val_bubble(xm, nk)
    return d


def _val_context(c, seed):
    d = _val_inputs(c, seed)
    avec, bvec = np.zeros(9), np.zeros(9)
    avec[0] = avec[4] = avec[8] = A_BOHR
    bvec[0] = bvec[4] = bvec[8] = 2.0 * math.pi / A_BOHR
    w = WL.ValWorkload(name="case", nc=d.nc, nv=d.nv, kmesh=d.km, xmesh=d.xm, celvol=CELVOL, avec=avec, bvec=bvec,
                       qinb=np.zeros(3), epsilon0=EPS0, er=_flat(d.er), ei=np.zeros(d.er.numel()), allow=_flat(d.allow),
                       conr=None, coni=None, valr=None, vali=None, ladder=None, psi_r=_flat(d.psi.real),
                       psi_i=_flat(d.psi.imag), kpref=d.kpref)
    w.device_arrays = dict(valr=d.val.real.contiguous(), vali=d.val.imag.contiguous(), conr=d.con.real.contiguous(),
                           coni=d.con.imag.contiguous(), ladder=d.ladder.contiguous())
    torch.cuda.synchronize()
    ctx = capi.ValContext(w, precision=_prec(c))
    ctx._chk(ctx.lib.ocn_val_set_bubble(ctx.ptr, capi._dp(d.bubble)))
    w.device_arrays = {}
    return types.SimpleNamespace(case=c, w=w, ctx=ctx, psi=_planes(d.psi[None]))


# ------------------------------------------------------------------- prepare / run

def prepare(case, seed):
    c = case
    if c["call"] == "val_haydock":
        s = _val_context(c, seed)
    elif c["call"] == "batch":
        s = types.SimpleNamespace(case=c, members=[_core_context(m, 1000 * int(seed) + i)
                                                   for i, m in enumerate(_batch_members(c))])
        for m in s.members:
            m.host = None
    elif c["call"] == "gmres_grad":
        d = _core_inputs(c, seed)
        w = _core_workload(d)
        e = np.linspace(-3.0, 27.0, c["nomega"])
        prob = adjoint.GmresProblem(w, e, precision=_prec(c))
        w.ur = w.ui = None
        g = torch.Generator()
        g.manual_seed(int(seed))
        s = types.SimpleNamespace(case=c, prob=prob, ptab=torch.from_numpy(d.ptab.copy()), cot=[
            torch.randn(c["nomega"], generator=g, dtype=torch.float64) for _ in range(2)])
    else:
        s = _core_context(c, seed)
    torch.cuda.synchronize()
    return s


def _coefficients(ra, ia, rb, done):
    """Lanczos a (complex: its imaginary part is rounding noise of a Hermitian run), b and the step counts."""
    return {"a": ra + 1j * ia, "b": rb, "done": done}


def run(state):
    c = state.case
    if c["call"] == "val_haydock":
        return _coefficients(*state.ctx.haydock_dev(c["niter"], state.psi.data_ptr()))
    if c["call"] == "batch":
        m = state.members
        got = capi.haydock_batch([x.ctx for x in m], [x.psi.data_ptr() for x in m], [3] * len(m), c["niter"])
        return [_coefficients(*g) for g in got]
    if c["call"] == "gmres_grad":
        p = [torch.tensor(1.0, dtype=torch.float64, requires_grad=True), state.ptab.clone().requires_grad_(True),
             torch.tensor(0.5 * EV, dtype=torch.float64, requires_grad=True),
             torch.tensor(0.0, dtype=torch.float64, requires_grad=True)]
        o = adjoint.gmres_spectrum(state.prob, *p)
        grads = torch.autograd.grad(o, p, grad_outputs=state.cot)
        return {"re": o[0].detach(), "im": o[1].detach(), "grad": list(grads)}
    ctx, w = state.ctx, state.w
    if c["call"] == "xact":
        if c["nv"] > 1:
            return list(ctx.apply_H_block(*state.host))
        return list(ctx.apply_H(state.host[0][0], state.host[1][0]))
    if c["nv"] > 1:
        return _coefficients(*ctx.haydock_block_dev(c["niter"], c["nv"], state.psi.data_ptr()))
    n8 = 8 * w.npsi
    ra, ia, rb, done = ctx.haydock_dev(c["niter"], state.psi.data_ptr(), state.psi.data_ptr() + n8)
    out = _coefficients(ra, ia, rb, done)
    if c["call"] == "spectrum":
        out["spectrum"] = capi.spectrum_cf(ra, ia, rb, done, w.kpref, w.el, w.eh, w.ne, w.gam0, ucvol=CELVOL)
    return out


# ------------------------------------------------------------------- work

def _action_work(c):
    """One H psi of nv vectors: Bloch functions read once, vectors in and out, the x-mesh transform's arithmetic."""
    nk, nx = c["k1"] * c["k2"] * c["k3"], c["x1"] * c["x2"] * c["x3"]
    na = 4 * (2 * c["lc"] + 1)
    t = na * c["nv"]
    cb = 16 if c["prec"] == "fp64" else 8
    by = c["nspn"] * nk * nx * c["nb"] * cb + 8.0 * nk * nx + 4 * 16.0 * t * nk * c["nb"]
    fl = 16.0 * t * nk * nx * c["nb"] + nx * t * 10.0 * nk * math.log2(nk)
    if c["mult"]:
        by += 128 * nk * c["nb"] * cb * c["nspn"]
        fl += 16.0 * 128 * t * nk * c["nb"]
    return by, fl


def work(case):
    c = case
    if c["call"] == "val_haydock":
        nk, nx = c["k1"] * c["k2"] * c["k3"], c["x1"] * c["x2"] * c["x3"]
        by = float(nk) * nx * nx * (8 if c["prec"] == "fp64" else 4)
        fl = float(nx) * nx * (16.0 * c["nvb"] * nk + 10.0 * nk * math.log2(nk) + 2.0 * nk)
        return {"bytes": by * c["niter"], "flops": fl * c["niter"]}
    if c["call"] == "batch":
        w = [_action_work(m) for m in _batch_members(c)]
        return {"bytes": c["niter"] * sum(x[0] for x in w), "flops": c["niter"] * sum(x[1] for x in w)}
    by, fl = _action_work(c)
    # a GMRES spectrum and its adjoint: at least two actions per energy and direction
    n = c["niter"] if c["call"] in ("haydock", "spectrum") else (4 * c["nomega"] if c["call"] == "gmres_grad" else 1)
    return {"bytes": by * n, "flops": fl * n}


# ------------------------------------------------------------------- exact (complex128 torch)

def _shift(d):
    """x-mesh shift of the core site at the origin: none on an even k-mesh axis, half a cell on an odd one."""
    return [math.floor(m * (0.0 if k % 2 == 0 else -0.5)) for k, m in zip(d.km, d.xm)]


def _phase_and_radius(d):
    sh = _shift(d)
    pos = [p.reshape(-1) for p in np.meshgrid(*[np.arange(1, m + 1) for m in d.xm], indexing="ij")]
    order = np.lexsort((pos[0], pos[1], pos[2]))  # x1 fastest
    pos = [p[order] for p in pos]
    kk = [k.reshape(-1) for k in np.meshgrid(*[np.arange(n) for n in d.km], indexing="ij")]  # k3 fastest
    angle = np.zeros((d.nx, d.nk))
    r2 = np.zeros((d.nx, d.nk))
    for i in range(3):
        m, n = d.xm[i], d.km[i]
        t = pos[i] - sh[i]
        turn = np.where(t > m, -m, np.where(t < 1, m, 0))
        angle += 2.0 * math.pi * np.outer(turn + pos[i] - 1, kk[i]) / (m * n)
        frac = (t + turn - 1) / m
        cell = kk[i] if n == 1 else np.where(kk[i] >= (n + 1) // 2, kk[i] - n, kk[i])
        r2 += (A_BOHR * (frac[:, None] + cell[None, :] + sh[i] / m)) ** 2
    return np.exp(1j * angle), np.sqrt(r2)


class _CoreH:
    """H of a core-level case on (v, a, k, n) complex128 tensors."""

    def __init__(self, d):
        self.d = d
        ph, self.r = _phase_and_radius(d)
        inside = self.r <= d.rtab[-1]
        w = np.where(inside, np.interp(self.r, d.rtab, d.ptab), 1.0 / (EPS0 * np.maximum(self.r, 1e-30)))
        self.W = torch.from_numpy(w).to(DEV)  # (x, k)
        self.u = d.u * torch.from_numpy(ph).to(DEV).T[None, :, :, None]  # (s, k, x, n)
        self.so = None
        if d.mult:
            self.mul = 1.0 / (d.nk * CELVOL)
            self.so = torch.from_numpy(self._spin_orbit()).to(DEV).to(torch.complex128)

    def _spin_orbit(self):
        l, xi = self.d.lc, self.d.so_xi

        def ang(j):
            m = np.arange(-j, j + 1)
            up = np.diag(np.sqrt(j * (j + 1) - m[:-1] * (m[:-1] + 1)), -1)
            return 0.5 * (up + up.T), -0.5j * (up - up.T), np.diag(m)

        ls = sum(np.kron(s, o) for s, o in zip(ang(0.5), ang(l)))
        return -xi * np.kron(ls.real, np.eye(2))

    def to_x(self, q):
        """phi (v, a, k, x) of q (v, a, k, n)."""
        u = self.u
        if len(u) == 1:
            t = q.permute(2, 3, 0, 1).reshape(self.d.nk, self.d.nb, -1)
            return (u[0] @ t).reshape(self.d.nk, self.d.nx, *q.shape[:2]).permute(2, 3, 0, 1)
        out = torch.empty(*q.shape[:3], self.d.nx, dtype=q.dtype, device=DEV)
        for s in range(2):
            t = q[:, s::2].permute(2, 3, 0, 1)
            sh = t.shape[2:]
            out[:, s::2] = (u[s] @ t.reshape(self.d.nk, self.d.nb, -1)).reshape(self.d.nk, self.d.nx, *sh).permute(2, 3, 0, 1)
        return out

    def to_band(self, f):
        u = self.u
        out = torch.empty(*f.shape[:3], self.d.nb, dtype=f.dtype, device=DEV)
        for s in range(len(u)):
            t = f[:, s::len(u)].permute(2, 3, 0, 1)
            sh = t.shape[2:]
            out[:, s::len(u)] = (u[s].mH @ t.reshape(self.d.nk, self.d.nx, -1)).reshape(self.d.nk, self.d.nb, *sh).permute(2, 3, 0, 1)
        return out

    def back(self, f):
        """Unnormalised transform k -> R (sign +) of (v, a, k, x)."""
        g = f.reshape(*f.shape[:2], *self.d.km, self.d.nx)
        return torch.fft.ifftn(g, dim=(2, 3, 4), norm="forward").reshape(f.shape)

    def fwd(self, f):
        g = f.reshape(*f.shape[:2], *self.d.km, self.d.nx)
        return torch.fft.fftn(g, dim=(2, 3, 4)).reshape(f.shape)

    def multiplet(self, q):
        d = self.d
        out = torch.zeros_like(q)
        spin = [a % 2 if d.nspn == 2 else 0 for a in range(d.na)]
        for l in range(d.lmax + 1):
            m = d.mpc[:, l, d.lmax - l:d.lmax + l + 1]  # (s, m, nu, k, n)
            ms = m[spin]  # (a, m, nu, k, n)
            amp = torch.einsum("amukn,vakn->vamu", ms, q)
            h = -torch.einsum("uw,vamw->vamu", d.mpm[l].to(amp.dtype), amp)
            h = h + (amp.reshape(len(q), -1) @ d.mh[l].T).reshape(amp.shape)
            out += torch.einsum("amukn,vamu->vakn", ms.conj(), h * self.mul)
        return out

    def __call__(self, psi):
        d = self.d
        q = d.allow * psi
        f = self.fwd(self.back(self.to_x(q)) * self.W.T) / d.nk
        acc = -self.to_band(f)
        if d.mult:
            acc = acc + self.multiplet(q)
        out = d.er * psi + d.allow * acc
        if self.so is not None:
            out = out + torch.einsum("ij,vjkn->vikn", self.so, psi)
        return out


def _lanczos(h, psi, niter):
    """Two-term recurrence of nv vectors (leading axis); arrays (nv, niter + 1)."""
    nv = psi.shape[0]
    a = np.zeros((nv, niter + 1), dtype=complex)
    b = np.zeros((nv, niter + 1))
    dims = tuple(range(1, psi.dim()))
    old = torch.zeros_like(psi)
    one = (slice(None),) + (None,) * len(dims)
    for i in range(1, niter + 1):
        hp = h(psi) - torch.from_numpy(b[:, i - 1]).to(DEV)[one] * old
        ai = (hp.conj() * psi).sum(dims)
        a[:, i - 1] = ai.cpu().numpy()
        hp = hp - ai.real[one] * psi
        nb = torch.sqrt((hp.abs() ** 2).sum(dims))
        b[:, i] = nb.cpu().numpy()
        old, psi = psi, hp / nb[one]
    return a, b


def _exact_gmres(c, seed):
    """<b|x>, x = (w + i Gamma - H)^-1 b, and its gradient, in a fully orthogonalised Krylov basis."""
    d = _core_inputs(c, seed)
    H = _CoreH(d)
    gam = 0.5 * EV
    om = torch.from_numpy(np.linspace(-3.0, 27.0, c["nomega"]) * EV).to(DEV)
    b = (d.allow * d.psi).reshape(-1)
    n, m = b.numel(), min(480, b.numel() - 1)
    V = torch.zeros((m, n), dtype=torch.complex128, device=DEV)
    T = torch.zeros((m, m), dtype=torch.float64, device=DEV)
    bn = torch.linalg.vector_norm(b)
    V[0] = b / bn
    for j in range(m):
        hv = H(V[j].reshape(d.psi.shape)).reshape(-1)
        for _ in range(2):
            pr = V[:j + 1].conj() @ hv
            hv = hv - pr @ V[:j + 1]
            T[j, j] += pr[j].real
        if j + 1 < m:
            beta = torch.linalg.vector_norm(hv)
            T[j, j + 1] = T[j + 1, j] = beta
            V[j + 1] = hv / beta
    lam, Q = torch.linalg.eigh(T)
    Qc = Q.to(torch.complex128)
    z = torch.complex(om, torch.full_like(om, gam))

    def solve(zz):
        return ((Qc @ (Qc[0][:, None] * bn / (zz[None, :] - lam[:, None]))).T @ V)  # (w, n)

    x, y = solve(z), solve(z.conj())
    F = (x @ b.conj())
    g = torch.Generator()
    g.manual_seed(int(seed))
    cot = [torch.randn(c["nomega"], generator=g, dtype=torch.float64).to(DEV) for _ in range(2)]
    yx = (y.conj() * x).sum(1)

    def pull(df):  # d out_re = -kpref Re dF, d out_im = -kpref Im dF
        return float((-d.kpref * (cot[0] * df.real + cot[1] * df.imag)).sum())

    gW = torch.zeros_like(H.W)
    for w in range(c["nomega"]):
        ax = H.back(H.to_x(d.allow * x[w].reshape(d.psi.shape)))
        ay = H.back(H.to_x(d.allow * y[w].reshape(d.psi.shape)))
        dw = -(ay.conj() * ax).sum((0, 1)).T / d.nk  # (x, k)
        gW += -d.kpref * (cot[0][w] * dw.real + cot[1][w] * dw.imag)
    gW, r = gW.cpu().numpy().reshape(-1), H.r.reshape(-1)
    inside = r <= d.rtab[-1]
    i = np.clip(np.searchsorted(d.rtab, r[inside], side="left") - 1, 0, len(d.rtab) - 2)
    t = (r[inside] - d.rtab[i]) / (d.rtab[i + 1] - d.rtab[i])
    gp = np.bincount(i, gW[inside] * (1 - t), len(d.rtab)) + np.bincount(i + 1, gW[inside] * t, len(d.rtab))
    gs = float((gW * H.W.cpu().numpy().reshape(-1)).sum())
    return {"re": (1.0 - d.kpref * F.real).cpu(), "im": (-d.kpref * F.imag).cpu(),
            "grad": [torch.tensor(gs, dtype=torch.float64), torch.from_numpy(gp),
                     torch.tensor(pull(-1j * yx), dtype=torch.float64), torch.tensor(pull(yx), dtype=torch.float64)]}


def _exact_val(c, seed):
    d = _val_inputs(c, seed)
    vol = math.prod(d.xm)
    bub = torch.from_numpy(d.bubble.reshape(d.xm)).to(DEV)
    chunk = max(1, min(vol, int(4e8 // (16 * vol * d.nk))))

    def h(psi):
        q = d.allow * psi[0]  # (k, v, c)
        A = q @ d.con  # (k, v, x)
        l = (d.val.conj() * A).sum((0, 1)).reshape(d.xm)
        s = torch.fft.fftn(torch.fft.ifftn(l, norm="forward") * bub).reshape(-1)
        B = torch.zeros_like(A)
        for y0 in range(0, vol, chunk):
            vy = d.val[:, :, y0:y0 + chunk]
            t = A.mT @ vy.conj()  # (k, x, y)
            sh = t.shape
            t = torch.fft.fftn(t.reshape(*d.km, *sh[1:]), dim=(0, 1, 2)).reshape(sh)
            t = t * d.ladder[y0:y0 + chunk].permute(2, 1, 0)
            t = torch.fft.ifftn(t.reshape(*d.km, *sh[1:]), dim=(0, 1, 2)).reshape(sh)
            B += vy @ t.mT
        out = (2.0 * s[None, None, :] * d.val - B) @ d.con.mH
        return (d.er * psi[0] + d.allow * out)[None]

    a, b = _lanczos(h, d.psi[None], c["niter"])
    return {"a": a[0], "b": b[0], "done": None}


def _exact_spectrum(c, d, a, b):
    """write_core's continued fraction with its square-root terminator, kept in 64 bits throughout."""
    w = types.SimpleNamespace(el=-10.0 * EV, eh=40.0 * EV, ne=2000, gam0=0.5 * EV)
    n = c["niter"]
    e = w.el + (w.eh - w.el) * np.arange(w.ne + 1) / w.ne
    ct = e - a[n - 1].real + 1j * (w.gam0 + a[n - 1].imag)
    disc = np.sqrt(ct * ct - 4.0 * b[n] ** 2)
    delta = 0.5 * (ct + np.where(disc.imag > 0.0, disc, -disc))
    for j in range(n - 1, -1, -1):
        delta = e - a[j].real + 1j * (w.gam0 + a[j].imag) - b[j + 1] ** 2 / delta
    den = np.abs(delta) ** 2
    s, k = d.kpref * np.abs(delta.imag) / den, d.kpref * delta.real / den
    al, bohr2 = 0.0072973525643, (WL.BOHR * WL.BOHR * 1e-16)
    ener = WL.HARTREE2EV * e
    sig = EV * al * CELVOL * ener * s
    tpa = al * al * 2.0 * math.pi * CELVOL
    return np.stack([ener, s, s, k, k, sig, sig * bohr2, s * tpa, s * tpa * bohr2 * bohr2 * 2.4188843265864e-17], axis=1)


def exact(case, seed):
    c = case
    if c["call"] == "val_haydock":
        return _exact_val(c, seed)
    if c["call"] == "gmres_grad":
        return _exact_gmres(c, seed)
    if c["call"] == "batch":
        out = []
        for i, m in enumerate(_batch_members(c)):
            d = _core_inputs(m, 1000 * int(seed) + i)
            a, b = _lanczos(_CoreH(d), d.psi, c["niter"])
            out.append({"a": a, "b": b, "done": None})
        return out
    d = _core_inputs(c, seed)
    H = _CoreH(d)
    if c["call"] == "xact":
        o = H(d.psi).reshape(c["nv"], -1)
        o = o if c["nv"] > 1 else o[0]
        return [o.real.contiguous(), o.imag.contiguous()]
    a, b = _lanczos(H, d.psi, c["niter"])
    if c["nv"] > 1:
        return {"a": a, "b": b, "done": None}
    out = {"a": a[0], "b": b[0], "done": None}
    if c["call"] == "spectrum":
        out["spectrum"] = _exact_spectrum(c, d, a[0], b[0])
    return out
