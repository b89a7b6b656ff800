"""Accuracy of single elements of the FP64 direct term of the valence action when its factors
are graded oppositely: A large in the bands in which the states at y are small, or the
ladder large where they are small.

Each element's error is measured against the same sums over absolute values.  Nested sums
over Nc, Nv, Nx and Nx products follow each other (0.3 to 0.5 eps/2 rms each in binary64, eps/2
= 2^-53) with a transform pair between them: 8 eps/2 is allowed.  The exact values are numpy's
in extended precision.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL
from test_gpu_graded import CLD, LD, U, _dft, _gauss

pytestmark = pytest.mark.gpu


def _direct(con, val, lad, psi, km):
    """-sum_x conj(con) sum_y val FFT^-1[ladder FFT[sum_v A conj(val)]]: con (k, c, x), val (k, v, x),
    lad (y, x, k), psi (k, v, c)."""
    A = np.einsum("kcx,kvc->kvx", con, psi)
    t = np.einsum("kvx,kvy->yxk", A, val.conj())
    sh = t.shape
    t = t.reshape(sh[0], sh[1], *km)
    for ax in range(3):
        t = np.moveaxis(np.tensordot(t, _dft(km[ax], -1), axes=([2 + ax], [0])), -1, 2 + ax)
    t = t * (lad.reshape(t.shape) / LD(np.prod(km)))
    for ax in range(3):
        t = np.moveaxis(np.tensordot(t, _dft(km[ax], 1), axes=([2 + ax], [0])), -1, 2 + ax)
    B = np.einsum("yxk,kvy->kvx", t.reshape(sh), val)
    return -np.einsum("kvx,kcx->kvc", B, con.conj())


def _bound(con, val, lad, psi):
    con, val, lad, psi = [np.abs(a) for a in (con, val, lad, psi)]
    A = np.einsum("kcx,kvc->kvx", con, psi)
    t = np.einsum("kvx,kvy->yx", A, val) * lad.sum(2) / lad.shape[2]  # over k: the transforms mix the k
    return np.einsum("yx,kvy,kcx->kvc", t, val, con)


CASES = [  # kmesh, xmesh, nc, nv
    ((1, 1, 1), (3, 3, 2), 3, 4),
    ((2, 1, 3), (3, 2, 2), 2, 3),
    ((3, 3, 3), (2, 3, 3), 3, 4),
    ((2, 2, 2), (3, 3, 3), 2, 8),
    ((8, 1, 2), (2, 2, 3), 3, 5),
    ((4, 4, 4), (2, 2, 3), 2, 2),
]


@pytest.mark.parametrize("kmesh,xmesh,nc,nv", CASES)
@pytest.mark.parametrize("over,decades", [("v", 0), ("v", 3), ("v", 6), ("y", 3), ("both", 4)])
def test_direct_term(lib_built, kmesh, xmesh, nc, nv, over, decades):
    capi.load(lib_built)
    w = WL.make_val("vtiny", seed=4, nc=nc, nv=nv, kmesh=kmesh, xmesh=xmesh)
    rng = np.random.default_rng(13)
    nk, nx = w.nk, w.nx
    gv = 10.0 ** (-decades * np.arange(nv) / max(nv - 1, 1)) if over != "y" else np.ones(nv)
    gy = 10.0 ** (-decades * rng.permutation(nx) / (nx - 1)) if over != "v" else np.ones(nx)
    con = _gauss(rng, nk, nc, nx)
    val = _gauss(rng, nk, nv, nx) * gv[:, None] * gy
    lad = rng.uniform(0.2, 1.0, (nx, nx, nk)) * gy[:, None, None] ** -3
    psi = _gauss(rng, nk, nv, nc) * gv[:, None] ** -2
    for name, a in (("con", con), ("val", val)):
        setattr(w, name + "r", a.real.reshape(-1).copy())
        setattr(w, name + "i", a.imag.reshape(-1).copy())
    w.ladder = lad.reshape(-1).copy()
    ctx = capi.ValContext(w)
    try:
        got = ctx.apply_H(psi.real.reshape(-1).copy(), psi.imag.reshape(-1).copy(), flags=(0, 0, 1))
    finally:
        ctx.close()
    h = (got[0] + 1j * got[1]).reshape(nk, nv, nc)
    want = _direct(con.astype(CLD), val.astype(CLD), lad.astype(LD), psi.astype(CLD), kmesh)
    err = np.abs(h.astype(CLD) - want)
    assert float(np.max(err / _bound(con, val, lad, psi))) < 8.0 * U
