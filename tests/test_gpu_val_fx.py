"""The FP64 direct term of the valence action in 64-bit fixed point against the oracle.

The kernel's own error is below 2^-56 of a block's largest element per step; the
comparison is limited by the oracle's binary64 sums over Nx * Nv <= 700 products
(sqrt(700) * 1.1e-16 = 3e-15 of the result's 2-norm) and its transforms: 3e-14
is allowed.  Sizes cover every line length 1..8, cubic and mixed meshes, 1..8
valence bands (one and two line-band pairs per thread), x-meshes that leave a
partial tile of y, and meshes and band counts that keep the FP64-pipe kernel.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu

TOL = 3e-14


@pytest.fixture(scope="module")
def built(lib_built, oracle_lib):
    return capi.load(lib_built), oracle_lib


def _direct(w, O):
    P = O.OracleVal(w)
    ctx = capi.ValContext(w)
    try:
        rng = np.random.default_rng(3)
        x = rng.standard_normal(w.npsi) + 1j * rng.standard_normal(w.npsi)
        got = ctx.apply_H(x.real, x.imag, flags=(0, 0, 1))
        want = P.act(x.real, x.imag, flags=(0, 0, 1))
    finally:
        ctx.close()
    g, r = got[0] + 1j * got[1], want[0] + 1j * want[1]
    return np.linalg.norm(g - r) / np.linalg.norm(r)


CASES = [  # kmesh, xmesh, nc, nv
    ((1, 1, 2), (2, 2, 2), 2, 1),
    ((3, 3, 3), (3, 3, 3), 4, 4),
    ((4, 4, 4), (3, 3, 5), 3, 5),
    ((5, 5, 5), (3, 2, 3), 2, 8),
    ((6, 6, 6), (2, 3, 3), 3, 4),
    ((8, 8, 8), (2, 2, 3), 3, 4),
    ((8, 8, 8), (3, 2, 3), 3, 7),   # two line-band pairs per thread
    ((7, 1, 8), (3, 3, 2), 4, 3),
    ((2, 8, 5), (3, 3, 3), 4, 2),
    ((7, 7, 7), (2, 2, 2), 2, 2),
    ((9, 2, 1), (3, 2, 2), 2, 2),   # an axis beyond 8: the FP64-pipe kernel
    ((2, 2, 2), (4, 3, 2), 3, 9),   # more than 8 bands: the FP64-pipe kernel
]


@pytest.mark.parametrize("kmesh,xmesh,nc,nv", CASES)
def test_direct_term(built, kmesh, xmesh, nc, nv):
    if nc + nv > np.prod(xmesh):
        pytest.skip("more bands than x-points")
    w = WL.make_val("vtiny", seed=4, nc=nc, nv=nv, kmesh=kmesh, xmesh=xmesh)
    assert _direct(w, built[1]) < TOL


def test_scales_per_x_and_y(built):
    """States over nine decades in x (one x-point zero) and ladder rows over six: every
    row keeps its own scale."""
    w = WL.make_val("vtiny", seed=6, nc=3, nv=3, kmesh=(4, 3, 2), xmesh=(3, 3, 3))
    f = 10.0 ** (-9.0 * np.arange(w.nx) / (w.nx - 1))
    f[5] = 0.0
    for name in ("conr", "coni", "valr", "vali"):
        a = getattr(w, name).reshape(-1, w.nx)
        setattr(w, name, (a * f).reshape(-1))
    lad = w.ladder.reshape(w.nx, w.nx, w.nk)
    g = 10.0 ** (-6.0 * np.arange(w.nx) / (w.nx - 1))
    w.ladder = (lad * g[:, None, None] * g[None, :, None]).reshape(-1)
    assert _direct(w, built[1]) < TOL


@pytest.mark.parametrize("where", ["ladder", "valr", "psi"])
def test_nan_reaches_the_result(built, where):
    w = WL.make_val("vtiny", seed=8)
    pr = w.psi_r.copy()
    if where == "psi":
        pr[1] = np.nan
    else:
        getattr(w, where)[3] = np.nan
    ctx = capi.ValContext(w)
    try:
        hr, hi = ctx.apply_H(pr, w.psi_i, flags=(0, 0, 1))
        assert np.isnan(hr).any() and np.isnan(hi).any()
    finally:
        ctx.close()
