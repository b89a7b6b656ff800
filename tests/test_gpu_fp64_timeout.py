"""The bounded waits of the FP64 digit contractions, made to run out on purpose.

As for the mixed-precision contractions: with the test hook on, the load warp issues no
copies, the MMA warp's wait (bounded at about one second) runs out, and the kernel records
that, frees its tensor memory and returns with nothing in flight.  Every kind of call on
the FP64 path must report OCN_ERR_TIMEOUT, and the context must then give the bits that it
gave before.
"""
import numpy as np
import pytest

from ocean_gb300 import capi
from ocean_gb300 import workloads as WL

pytestmark = pytest.mark.gpu

OCN_ERR_TIMEOUT = 5


@pytest.mark.parametrize("name,call", [("tiny", "apply"), ("tiny", "haydock"), ("c3small", "apply")])
def test_starved_fp64_contraction_reports_timeout_and_context_recovers(lib_built, name, call):
    capi.load(lib_built)
    w = WL.make(name, seed=3)
    ctx = capi.Context(w)
    try:
        go = (lambda: ctx.apply_H(w.psi_r, w.psi_i)) if call == "apply" else (lambda: ctx.haydock(2)[:3])
        before = go()
        assert ctx.fp64_digits() > 0
        ctx.starve_tc(True)
        with pytest.raises(capi.OcnError) as exc:
            go()
        assert exc.value.code == OCN_ERR_TIMEOUT
        ctx.starve_tc(False)
        for a, b in zip(before, go()):
            assert np.array_equal(a, b)
    finally:
        ctx.close()
