"""Accuracy of single elements of the FP64 action when rows and columns of a contraction are
graded oppositely: large elements of one meet small elements of the other.

Each element's error is measured against B, the same sums over absolute values: a binary64
sum of K products in any order is off by 0.3 to 0.5 eps/2 of that (rms, K = 4..1000; eps/2
= 2^-53), and two nested sums, a transform and a few roundings follow each other, so 4 eps/2
is allowed for the long-range term and 8 eps/2 for the three nested sums of the multiplet
term.  Digit sums that end at 2^-60 of the largest products of row and column maxima are off
by 50 eps/2 and more from four decades on.  The exact values are numpy's in extended precision.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LD, CLD = np.longdouble, np.clongdouble


def _dft(n, sign):
    j = np.arange(n).astype(LD)
    return np.exp(sign * 2j * (np.arccos(LD(-1.0)) * (np.outer(j, j) % n) / n).astype(CLD))


def _gauss(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _long_range(u, W, q, km):
    """-sum_x conj(u) FFT[W FFT[sum_n u q]] / Nk for one spin: u (x, k, n), W (x, k), q (a, k, n)."""
    nx, nk, nb = u.shape
    phi = np.einsum("xkn,akn->axk", u, q).reshape(-1, nx, *km)
    for ax in range(3):
        phi = np.moveaxis(np.tensordot(phi, _dft(km[ax], 1), axes=([2 + ax], [0])), -1, 2 + ax)
    phi = phi * (W.reshape(1, nx, *km) / LD(nk))
    for ax in range(3):
        phi = np.moveaxis(np.tensordot(phi, _dft(km[ax], -1), axes=([2 + ax], [0])), -1, 2 + ax)
    return -np.einsum("xkn,axk->akn", u.conj(), phi.reshape(-1, nx, nk))


def _bound(u, W, q):
    s = np.einsum("xkn,akn->ax", np.abs(u), np.abs(q))  # over k as well: the transforms mix the k
    return np.einsum("xkn,ax->akn", np.abs(u), s * np.abs(W).sum(1)[None] / W.shape[1])


CASES = [  # kmesh, bands, xmesh, core_l, nspn, vectors
    ((1, 1, 1), 40, (6, 7, 8), 0, 1, 1),
    ((1, 1, 1), 9, (5, 4, 3), 0, 2, 3),
    ((1, 1, 1), 150, (5, 6, 7), 1, 1, 1),
    ((2, 1, 2), 33, (5, 5, 5), 0, 1, 2),
    ((3, 2, 1), 17, (4, 3, 5), 1, 2, 1),
    ((9, 1, 1), 5, (3, 3, 3), 0, 1, 1),    # phi' in binary64
]


@pytest.mark.parametrize("kmesh,nb,xmesh,core_l,nspn,nv", CASES)
@pytest.mark.parametrize("over,decades", [("n", 0), ("n", 2), ("n", 5), ("x", 2), ("x", 4), ("both", 4)])
def test_long_range(lib_built, kmesh, nb, xmesh, core_l, nspn, nv, over, decades):
    capi.load(lib_built)
    w = WL.make("tiny", seed=1, nb=nb, kmesh=kmesh, xmesh=xmesh, core_l=core_l, with_mult=False)
    w.nspn = nspn
    rng = np.random.default_rng(11)
    nk, nx, na = w.nk, w.nx, w.na
    gn = 10.0 ** (-decades * np.arange(nb) / max(nb - 1, 1)) if over != "x" else np.ones(nb)
    gx = 10.0 ** (-decades * rng.permutation(nx) / (nx - 1)) if over != "n" else np.ones(nx)
    u = _gauss(rng, nspn, nx, nk, nb) * gn * gx[:, None, None]
    w.ur, w.ui = u.real.reshape(-1).copy(), u.imag.reshape(-1).copy()
    w.er[:] = 0.0
    W = rng.uniform(0.5, 1.0, (nx, nk)) * gx[:, None] ** -3
    psi = _gauss(rng, nv, na, nk, nb) / gn
    pr, pi = psi.real.reshape(nv, -1).copy(), psi.imag.reshape(nv, -1).copy()
    ctx = capi.Context(w, nvec=nv)
    try:
        ctx.set_W(W.reshape(-1))
        b = [x.reshape(nspn, nx, nk, nb) for x in ctx.get_bloch()]
        got = ctx.apply_H_block(pr, pi)
    finally:
        ctx.close()
    b = b[0] + 1j * b[1]
    h = (got[0] + 1j * got[1]).reshape(nv, na, nk, nb)
    for v in range(nv):
        for s in range(nspn):
            mine = [a for a in range(na) if nspn == 1 or a % 2 == s]
            want = _long_range(b[s].astype(CLD), W.astype(LD), psi[v, mine].astype(CLD), kmesh)
            err = np.abs(h[v, mine].astype(CLD) - want)
            assert float(np.max(err / _bound(b[s], W, psi[v, mine]))) < 4.0 * U


def test_more_open_tiles_than_a_cta_remembers(lib_built):
    """82 row tiles per CTA, every one with open sums: the digits' path against the FP64 pipe's,
    whose errors add up."""
    capi.load(lib_built)
    kmesh, nb, xmesh = (14, 14, 16), 2, (5, 8, 10)
    w = WL.make("tiny", seed=1, nb=nb, kmesh=kmesh, xmesh=xmesh, core_l=0, with_mult=False)
    rng = np.random.default_rng(14)
    gn = np.array([1.0, 1e-5])
    u = _gauss(rng, 1, w.nx, w.nk, nb) * gn
    w.ur, w.ui = u.real.reshape(-1).copy(), u.imag.reshape(-1).copy()
    w.er[:] = 0.0
    psi = _gauss(rng, w.na, w.nk, nb) / gn
    pr, pi = psi.real.reshape(-1).copy(), psi.imag.reshape(-1).copy()
    W = rng.uniform(0.5, 1.0, (w.nx, w.nk))
    ctx = capi.Context(w)
    try:
        ctx.set_W(W.reshape(-1))
        b = [x.reshape(w.nx, w.nk, nb) for x in ctx.get_bloch()]
        h = []
        for mask in (1, 0):
            ctx.set_fp64_digits(mask)
            r, i = ctx.apply_H(pr, pi)
            h.append((r + 1j * i).reshape(w.na, w.nk, nb))
    finally:
        ctx.close()
    assert float(np.max(np.abs(h[0] - h[1]) / _bound(b[0] + 1j * b[1], W, psi))) < 8.0 * U


@pytest.mark.parametrize("kmesh,nb,core_l,nspn,npl", [((2, 1, 2), 33, 0, 1, 20), ((1, 1, 1), 150, 1, 2, 7)])
@pytest.mark.parametrize("decades", [0, 3, 6])
def test_multiplet(lib_built, kmesh, nb, core_l, nspn, npl, decades):
    """One angular momentum without exchange matrices: mpc^H (-mpm (mpc q)) / (Nk V)."""
    capi.load(lib_built)
    w = WL.make("tiny", seed=1, nb=nb, kmesh=kmesh, xmesh=(6, 6, 6), core_l=core_l, with_mult=False)
    w.nspn = nspn
    rng = np.random.default_rng(12)
    nk, na = w.nk, w.na
    u = _gauss(rng, nspn, w.nx, nk, nb)
    w.ur, w.ui = u.real.reshape(-1).copy(), u.imag.reshape(-1).copy()
    w.er[:] = 0.0
    gn = 10.0 ** (-decades * np.arange(nb) / (nb - 1))
    gp = 10.0 ** (-decades * np.arange(npl) / (npl - 1))
    mpc = _gauss(rng, nspn, npl, nk, nb) * gn * gp[:, None, None]
    mpm = rng.uniform(0.5, 1.0, (npl, npl))
    mpm = (mpm + mpm.T) / np.outer(gp, gp)
    w.mult = dict(lmin=0, lmax=0, nproj=np.array([npl], dtype=np.int32), npmax=npl, mpcr=mpc.real.reshape(-1).copy(),
                  mpci=mpc.imag.reshape(-1).copy(), mpm=mpm.reshape(-1).copy(), mhr=np.zeros((na * npl) ** 2),
                  mhi=np.zeros((na * npl) ** 2))
    w.so_xi = 0.0
    q = _gauss(rng, na, nk, nb) / gn
    ctx = capi.Context(w, hflag=(0, 1, 1, 1, 1, 1))
    try:
        got = ctx.apply_H(q.real.reshape(-1).copy(), q.imag.reshape(-1).copy())
    finally:
        ctx.close()
    h = (got[0] + 1j * got[1]).reshape(na, nk, nb)
    for s in range(nspn):
        mine = [a for a in range(na) if nspn == 1 or a % 2 == s]
        m, c = mpc[s].astype(CLD), q[mine].astype(CLD)
        mul = LD(w.interaction_scale) / (LD(nk) * LD(w.celvol))
        hamp = -mul * np.einsum("pr,ra->pa", mpm.astype(LD), np.einsum("rkn,akn->ra", m, c))
        want = np.einsum("pkn,pa->akn", m.conj(), hamp)
        bound = float(mul) * np.einsum("pkn,pa->akn", np.abs(mpc[s]),
                                       np.einsum("pr,ra->pa", mpm, np.einsum("rkn,akn->ra", np.abs(mpc[s]), np.abs(q[mine]))))
        err = np.abs(h[mine].astype(CLD) - want)
        assert float(np.max(err / bound)) < 8.0 * U
