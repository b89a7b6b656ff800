"""Energy lanes of the GMRES sweep against one sweep per lane's chunk of energies.

A lane takes the steps that a single sweep over its chunk takes, whatever the other lanes
do meanwhile.  The shallow bases and loose thresholds make lanes converge on a restart while
a later lane has already started its next step: the order of the input slots in a block
action then differs from the order of the lanes, and a slot that is reused before it is
read changes steps and spectra by 1e-3 and more.  The FP64 action of a block has the bits
of the single actions, so the runs differ at most by rounding (1e-16 a step, some hundred
steps): 1e-10 is allowed.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,tol,lanes", [(2, 1e-3, 2), (3, 1e-3, 2), (4, 1e-2, 2), (3, 1e-4, 3), (2, 1e-3, 4)])
@pytest.mark.parametrize("nvec", [1, 4])
def test_lanes_take_the_steps_of_their_chunks(lib_built, depth, tol, lanes, nvec):
    capi.load(lib_built)
    w = WL.make("tiny", seed=3)
    E = np.linspace(3.0, 9.0, 12)
    ctx = capi.Context(w, nvec=nvec)
    try:
        ctx.set_gmres_lanes(lanes)
        got = ctx.gmres(E, depth=depth, tol=tol, max_restarts=5000)
        ctx.set_gmres_lanes(1)
        want = [ctx.gmres(E[len(E) * l // lanes:len(E) * (l + 1) // lanes], depth=depth, tol=tol, max_restarts=5000)
                for l in range(lanes)]
    finally:
        ctx.close()
    ore, oim, rel, its = [np.concatenate(v) for v in zip(*want)]
    assert np.array_equal(got[3], its)
    assert np.max(np.abs(got[1] - oim) / np.abs(oim)) < 1e-10
    assert np.max(np.abs(got[0] - ore) / np.abs(ore)) < 1e-10
