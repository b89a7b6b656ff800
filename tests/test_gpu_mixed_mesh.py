"""The mixed-precision action on k-meshes without symmetry, every axis length 1 to 8 at
every place, 4 and 12 channels, blocks of one and three vectors, against the oracle; a mesh
with an axis beyond 8 keeps the general transform.

1e-4 of the result is the bound of the mixed action everywhere (split-BF16 products); a
value at a wrong place is an error of order one.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu

CASES = [  # kmesh, bands, xmesh, core_l, nv
    ((1, 2, 3), 5, (3, 3, 3), 0, 1),
    ((3, 1, 4), 5, (3, 3, 3), 1, 1),
    ((4, 5, 1), 7, (3, 3, 5), 0, 3),
    ((5, 4, 6), 6, (3, 3, 3), 1, 1),
    ((6, 7, 5), 4, (2, 3, 3), 0, 3),
    ((7, 8, 2), 4, (2, 3, 3), 0, 1),
    ((8, 6, 7), 3, (2, 2, 2), 1, 1),
    ((2, 3, 8), 6, (3, 5, 5), 1, 3),
    ((7, 7, 7), 3, (2, 2, 2), 0, 1),
    ((9, 2, 3), 5, (3, 3, 3), 0, 1),
]


@pytest.mark.parametrize("kmesh,nb,xmesh,core_l,nv", CASES)
def test_mixed_action(lib_built, oracle_lib, kmesh, nb, xmesh, core_l, nv):
    capi.load(lib_built)
    w = WL.make("batch", seed=nb, nb=nb, kmesh=kmesh, xmesh=xmesh, core_l=core_l, with_mult=False)
    w.er[:] = 0.0  # the long-range term alone
    P = oracle_lib.OracleProblem(w)
    rng = np.random.default_rng(nb)
    pr, pi = rng.standard_normal((nv, w.npsi)), rng.standard_normal((nv, w.npsi))
    ctx = capi.Context(w, precision=capi.OCN_PREC_MIXED, nvec=nv)
    try:
        hr, hi = ctx.apply_H_block(pr, pi)
    finally:
        ctx.close()
    for v in range(nv):
        wr, wi = P.xact(pr[v], pi[v])
        want = wr + 1j * wi
        assert np.linalg.norm(hr[v] + 1j * hi[v] - want) < 1e-4 * np.linalg.norm(want)
