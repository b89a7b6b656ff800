"""The action on host vectors at both sides of the staging limit (49152 doubles in and
out): blocks of growing and shrinking size through one context's kept buffers.

The bound is that of the FP64 action against the oracle: 2e-14 of the result.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built(lib_built, oracle_lib):
    return capi.load(lib_built), oracle_lib


@pytest.mark.parametrize("nb,order", [(16, (2, 1, 3, 1)), (24, (1, 3)), (1, (3, 2))])
def test_blocks_of_host_vectors(built, nb, order):
    _, O = built
    w = WL.make("batch", seed=nb, nb=nb, kmesh=(6, 6, 4), xmesh=(3, 3, 3), core_l=0, with_mult=False)
    P = O.OracleProblem(w)
    ctx = capi.Context(w, nvec=3)
    try:
        rng = np.random.default_rng(nb)
        for nv in order:
            pr, pi = rng.standard_normal((nv, w.npsi)), rng.standard_normal((nv, w.npsi))
            hr, hi = ctx.apply_H_block(pr, pi)
            for v in range(nv):
                wr, wi = P.xact(pr[v], pi[v])
                want = wr + 1j * wi
                assert np.linalg.norm(hr[v] + 1j * hi[v] - want) < 2e-14 * np.linalg.norm(want)
            if nv == 1:
                sr, si = ctx.apply_H(pr[0], pi[0])
                assert np.array_equal(sr, hr[0]) and np.array_equal(si, hi[0])
    finally:
        ctx.close()
