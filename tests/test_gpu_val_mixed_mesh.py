"""The mixed-precision direct term on cubic k-meshes of every size the cubic kernel
takes, against the oracle: even and odd lines (two, one k3 value per load), one and two
(line, band) pairs per thread, an odd number of x-points (a padding x-point), and band
counts beyond the kernel's range.

Binary32 sums of Nx * Nv <= 250 products and six transforms of <= 24 additions per
element: (sqrt(250) + sqrt(6 * 24)) * 6e-8 = 1.7e-6 of the result's 2-norm; 1e-5 is
allowed.  A value at a wrong place is an error of order one.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu

CASES = [  # kmesh, xmesh, nc, nv
    (2, (3, 3, 3), 2, 1),
    (2, (3, 3, 3), 2, 7),
    (3, (3, 3, 3), 3, 4),
    (4, (3, 3, 4), 3, 3),
    (5, (3, 3, 3), 2, 5),
    (5, (4, 3, 3), 2, 12),  # two pairs per thread
    (6, (3, 3, 3), 2, 4),
    (6, (3, 3, 3), 2, 9),   # two pairs per thread
    (8, (3, 3, 3), 2, 3),
    (8, (3, 2, 3), 2, 6),   # two pairs per thread
    (8, (3, 3, 3), 2, 9),   # beyond the cubic kernel
]


@pytest.mark.parametrize("n,xmesh,nc,nv", CASES)
def test_direct_term_mixed(lib_built, oracle_lib, n, xmesh, nc, nv):
    capi.load(lib_built)
    w = WL.make_val("vtiny", seed=8, nc=nc, nv=nv, kmesh=(n, n, n), xmesh=xmesh)
    P = oracle_lib.OracleVal(w)
    ctx = capi.ValContext(w, precision=capi.OCN_PREC_MIXED)
    try:
        rng = np.random.default_rng(n)
        x = rng.standard_normal(w.npsi) + 1j * rng.standard_normal(w.npsi)
        got = ctx.apply_H(x.real, x.imag, flags=(0, 0, 1))
        want = P.act(x.real, x.imag, flags=(0, 0, 1))
    finally:
        ctx.close()
    g, r = got[0] + 1j * got[1], want[0] + 1j * want[1]
    assert np.linalg.norm(g - r) < 1e-5 * np.linalg.norm(r)
