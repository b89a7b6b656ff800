"""FP64 contexts whose contractions run on the FP64 pipe, as they do where the digit
operands do not fit, and contexts with one of the two terms on either path.

The action agrees with the oracle to 1e-12 (the bound of the other FP64 comparisons), a
block's vectors to the bits of the single actions, and the path in use is reported.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built(lib_built, oracle_lib):
    return capi.load(lib_built), oracle_lib


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


CASES = [  # kmesh, bands, xmesh, core_l, multiplet, nspn, nvec
    ((4, 4, 4), 11, (4, 4, 4), 0, False, 1, 3),   # 8 x-splits on the pipe where the digits take fewer
    ((3, 2, 4), 37, (5, 4, 3), 0, False, 2, 2),
    ((1, 1, 1), 40, (9, 10, 11), 0, False, 1, 1),
    ((2, 2, 3), 16, (4, 4, 4), 1, True, 1, 1),
    ((2, 3, 1), 20, (4, 4, 4), 1, True, 2, 2),
    ((9, 2, 1), 7, (3, 2, 2), 0, False, 1, 2),    # the transform on the FP64 pipe as well
]


@pytest.mark.parametrize("kmesh,nb,xmesh,core_l,mult,nspn,nvec", CASES)
def test_action_on_every_path(built, kmesh, nb, xmesh, core_l, mult, nspn, nvec):
    _, O = built
    w = WL.make("batch", seed=nb, nb=nb, kmesh=kmesh, xmesh=xmesh, core_l=core_l, with_mult=mult, nspn=nspn)
    P = O.OracleProblem(w)
    rng = np.random.default_rng(4)
    pr, pi = rng.standard_normal((nvec, w.npsi)), rng.standard_normal((nvec, w.npsi))
    want = [np.asarray(r) + 1j * np.asarray(i) for r, i in (P.xact(pr[v], pi[v]) for v in range(nvec))]
    every = 3 if mult else 1
    ctx = capi.Context(w, nvec=nvec)
    try:
        assert ctx.fp64_digits() == every
        for mask in ((0, 1, 2, 3) if mult else (0, 1)):
            ctx.set_fp64_digits(mask)
            assert ctx.fp64_digits() == mask
            br, bi = ctx.apply_H_block(pr, pi)
            for v in range(nvec):
                assert _rel(br[v] + 1j * bi[v], want[v]) < 1e-12
                sr, si = ctx.apply_H(pr[v], pi[v])
                assert np.array_equal(br[v], sr) and np.array_equal(bi[v], si)
    finally:
        ctx.close()


def test_haydock_follows_a_change_of_path(built):
    """A captured Haydock loop does not outlive the path that it was captured on."""
    _, O = built
    w = WL.make("c3small", seed=7)
    _, ora, oia, orb, _ = O.OracleProblem(w).haydock(12)
    ctx = capi.Context(w)
    try:
        for mask in (3, 0, 2, 1, 3):
            ctx.set_fp64_digits(mask)
            ra, ia, rb, done = ctx.haydock(12)
            assert done == 12
            assert np.max(np.abs(ra[:10] - ora[:10]) / np.abs(ora[:10])) < 1e-12
            assert np.max(np.abs(rb[1:10] - orb[1:10]) / np.abs(orb[1:10])) < 1e-12
    finally:
        ctx.close()


def test_choice_is_for_fp64_contexts(built):
    w = WL.make("tiny", seed=1)
    ctx = capi.Context(w, precision=capi.OCN_PREC_MIXED)
    try:
        assert ctx.fp64_digits() == 0
        with pytest.raises(capi.OcnError):
            ctx.set_fp64_digits(0)
    finally:
        ctx.close()
