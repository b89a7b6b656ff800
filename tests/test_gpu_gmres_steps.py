"""GMRES inner steps that are started before their residual is read back, against the
oracle's sequential sweep.

Both sides take the same iterates in exact arithmetic, so with a threshold far above
the FP64 floor the iteration counts are equal, step for step, also where a step that was
started early is void because the residual before it had already converged.  The spectra
then differ by rounding only; 1e-8 is the bound of the other GMRES comparisons.  The depths
reach a restart at every few steps and a basis of more than 128 vectors (the longest
coefficient list that travels with a launch).
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from test_gpu_parity import problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built(lib_built, oracle_lib):
    return capi.load(lib_built), oracle_lib


@pytest.mark.parametrize("depth,tol", [(2, 1e-3), (4, 1e-8), (16, 1e-2), (16, 1e-12)])
def test_gmres_steps_match_oracle(built, depth, tol):
    _, O = built
    w, P = problem("small", O, seed=21)
    E = np.array([3.0, 3.1, 3.2, 9.0, 9.05])
    ctx = capi.Context(w)
    try:
        ore, oim, rel, its = ctx.gmres(E, depth=depth, tol=tol, max_restarts=2000)
    finally:
        ctx.close()
    rc, ore2, oim2, rel2, its2, tot = P.gmres(E, depth=depth, ffff=tol, max_restarts=2000)
    assert rc == 0
    assert np.array_equal(its, its2)
    assert np.max(np.abs(oim - oim2) / np.abs(oim2)) < 1e-8
    assert np.max(np.abs(ore - ore2) / np.abs(ore2)) < 1e-8


def test_gmres_long_basis(built):
    """A second energy that goes on with the first one's 124 vectors."""
    _, O = built
    w, P = problem("small", O, seed=21)
    E = np.array([14.0, 14.05])
    ctx = capi.Context(w)
    try:
        ore, oim, rel, its = ctx.gmres(E, depth=400, tol=1e-18)
    finally:
        ctx.close()
    rc, ore2, oim2, rel2, its2, tot = P.gmres(E, depth=400, ffff=1e-18)
    assert rc == 0
    assert its.sum() > 150  # of 222 steps in the oracle
    assert np.max(np.abs(oim - oim2) / np.abs(oim2)) < 1e-8
    assert np.max(np.abs(ore - ore2) / np.abs(ore2)) < 1e-8
