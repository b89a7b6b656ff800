"""FP64 contractions on the FP8 tensor cores (digit slices) and the fixed-point
k-mesh transform against the oracle.

The digit sums are exact up to 2^-60 of a row's largest element, so the
difference is the oracle's own rounding: a sum of K products in binary64 is off by
about sqrt(K) eps of its terms' 2-norm, here K <= 2 * 300 bands or 2 * 1400
x-points, i.e. 50 * 1.1e-16 = 6e-15 of the long-range term; 2e-14 is allowed.
Sizes sit at the edges of the tiles: 128 rows (x-points, bands), 16-wide K
granules, 8-row groups, K chunks and splits, one and two valence spins, 4 and 12
channels.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu

TOL = 2e-14


@pytest.fixture(scope="module")
def built(lib_built, oracle_lib):
    return capi.load(lib_built), oracle_lib


def _rel(got, want):
    g, w = got[0] + 1j * got[1], want[0] + 1j * want[1]
    return np.linalg.norm(g - w) / np.linalg.norm(w)


CASES = [  # kmesh, bands, xmesh, core_l, nspn
    ((2, 2, 2), 1, (1, 1, 2), 0, 1),
    ((1, 1, 1), 8, (4, 4, 8), 0, 1),      # one k-point; 128 x: one full row tile
    ((2, 2, 2), 9, (3, 43, 1), 0, 1),     # 129 x: a last tile of one row; odd granule count
    ((3, 2, 2), 40, (5, 5, 5), 1, 1),     # 12 channels: one MMA per part
    ((2, 1, 3), 128, (7, 9, 4), 0, 2),    # two spins, a full band tile
    ((2, 2, 1), 137, (6, 6, 8), 1, 2),    # a second band tile of 9 rows
    ((2, 1, 1), 300, (10, 7, 20), 0, 1),  # several K chunks in both contractions, three band tiles
    # the fixed-point k-mesh transform: every line length, cubic and mixed meshes
    ((7, 5, 3), 6, (3, 2, 2), 0, 1),
    ((8, 4, 6), 5, (2, 3, 2), 1, 1),
    ((1, 8, 7), 5, (2, 2, 3), 0, 1),
    ((3, 3, 3), 7, (2, 2, 3), 0, 1),
    ((4, 4, 4), 7, (2, 2, 3), 1, 1),
    ((5, 5, 5), 7, (2, 2, 3), 0, 1),
    ((6, 6, 6), 7, (2, 2, 3), 0, 1),
    ((7, 7, 7), 5, (2, 2, 2), 0, 1),
    ((8, 8, 8), 5, (2, 2, 2), 1, 1),
    ((9, 2, 3), 5, (2, 2, 2), 0, 1),      # an axis beyond 8: the FP64-pipe transform
]


@pytest.mark.parametrize("kmesh,nb,xmesh,core_l,nspn", CASES)
def test_action_matches_oracle(built, kmesh, nb, xmesh, core_l, nspn):
    _, O = built
    if nb > np.prod(xmesh):
        pytest.skip("more bands than x-points")
    w = WL.make("batch", seed=nb, nb=nb, kmesh=kmesh, xmesh=xmesh, core_l=core_l, with_mult=False, nspn=nspn)
    w.er[:] = 0.0  # the long-range term alone
    P = O.OracleProblem(w)
    ctx = capi.Context(w)
    try:
        want = P.xact(w.psi_r, w.psi_i)
        assert _rel(ctx.apply_H(w.psi_r, w.psi_i), want) < TOL
    finally:
        ctx.close()


def test_wide_dynamic_range_zero_and_extreme_columns(built):
    """Bands over six decades, a zero channel, channels of 1e-200 and 1e150: every
    column keeps its own scale."""
    _, O = built
    w = WL.make("batch", seed=5, nb=33, kmesh=(2, 3, 2), xmesh=(5, 6, 7), core_l=0, with_mult=False)
    w.er[:] = 0.0
    f = np.tile(10.0 ** (-6.0 * np.arange(33) / 32), w.nk * w.nx)
    w.ur, w.ui = w.ur * f, w.ui * f
    P = O.OracleProblem(w)
    ctx = capi.Context(w)
    try:
        rng = np.random.default_rng(7)
        shape = (w.na, w.nk, w.nb)
        pr, pi = rng.standard_normal(shape), rng.standard_normal(shape)
        for a, s in enumerate((0.0, 1.0, 1e-200, 1e150)):
            pr[a] *= s
            pi[a] *= s
        got = [x.reshape(shape) for x in ctx.apply_H(pr.reshape(-1), pi.reshape(-1))]
        want = [x.reshape(shape) for x in P.xact(pr.reshape(-1), pi.reshape(-1))]
        assert not got[0][0].any() and not got[1][0].any()
        for a in (1, 2, 3):
            s = (1.0, 1e200, 1e-150)[a - 1]
            assert _rel([x[a] * s for x in got], [x[a] * s for x in want]) < TOL
    finally:
        ctx.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_input_stays_visible(built, bad):
    """A NaN or Inf in psi reaches the Lanczos a, which the run reports, as FP64 arithmetic would."""
    w = WL.make("tiny", seed=2)
    ctx = capi.Context(w)
    try:
        pr = w.psi_r.copy()
        pr[3] = bad
        hr, hi = ctx.apply_H(pr, w.psi_i)
        assert not np.all(np.isfinite(hr)) and not np.all(np.isfinite(hi))
        with pytest.raises(capi.OcnError) as exc:
            ctx.haydock(6, pr, w.psi_i)
        assert exc.value.code == capi.OCN_ERR_NAN
        good = ctx.apply_H(w.psi_r, w.psi_i)  # nothing of it stays behind
        assert np.all(np.isfinite(good[0])) and np.all(np.isfinite(good[1]))
    finally:
        ctx.close()


@pytest.mark.parametrize("kmesh,nb,xmesh,nspn,nvec,nv", [
    ((3, 2, 4), 19, (5, 4, 3), 1, 3, 3),   # 12 columns in one launch
    ((4, 4, 4), 11, (4, 4, 4), 2, 2, 2),   # 8 columns, two spins
    ((2, 2, 3), 21, (4, 3, 3), 1, 5, 5),   # groups of three and two
    ((9, 2, 1), 7, (3, 2, 2), 1, 2, 2),    # FP64-pipe transform: vector by vector
])
def test_block_of_vectors(built, kmesh, nb, xmesh, nspn, nvec, nv):
    """Vectors that share launches give the action of each alone, bit for bit, and match the oracle."""
    _, O = built
    w = WL.make("batch", seed=nb, nb=nb, kmesh=kmesh, xmesh=xmesh, core_l=0, with_mult=False, nspn=nspn)
    w.er[:] = 0.0
    P = O.OracleProblem(w)
    rng = np.random.default_rng(9)
    pr, pi = rng.standard_normal((nv, w.npsi)), rng.standard_normal((nv, w.npsi))
    pr[1] *= 1e-30
    pi[1] *= 1e-30
    ctx = capi.Context(w, nvec=nvec)
    try:
        br, bi = ctx.apply_H_block(pr, pi)
        for v in range(nv):
            sr, si = ctx.apply_H(pr[v], pi[v])
            assert np.array_equal(br[v], sr) and np.array_equal(bi[v], si)
            assert _rel((br[v], bi[v]), P.xact(pr[v], pi[v])) < TOL
    finally:
        ctx.close()
