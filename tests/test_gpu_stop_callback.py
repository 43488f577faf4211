"""A stop requested from the residual callback (needs a B200): the callback runs on
the solving thread between two batches of iterations, and no further iteration
runs after it.
"""
import ctypes as C

import numpy as np
import pytest

from axisim import cases
import axisim.abi as abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("when", [0, 2, 5, 11])
@pytest.mark.parametrize("geom", ["steady", "transient"])
def test_no_iteration_after_the_callback_that_stops(geom, when):
    if geom == "steady":
        c = cases.expansion(scale=1 / 32, max_iter=40, tol=1e-30)
    else:
        c = cases.pulsatile_expansion(scale=1 / 32)
        c.settings.update(maxIter=40, resTol=[1e-30] * 3)
    s = abi.Solver(abi.multiblock(c.blocks), c.bc_fields(), c.settings)
    seen = []

    def on_residual(_, iteration, values):
        seen.append(iteration)
        if len(seen) == when + 1:
            s.request_stop()

    fn = abi.RESIDUAL_FN(on_residual)
    abi.lib().axisim_set_log(s.h, C.cast(None, abi.LOG_FN), fn, None)
    r = s.solve(allow=(abi.E_STOPPED,))
    # iterations run in batches of 4, 8, 16, ...: the one that holds the stopping iteration is the last
    assert r["iterations"] == next(n for n in (4, 12, 28) if when < n)
    assert len(seen) == r["iterations"] and seen == sorted(seen)
    fields = {f: s.get(f) for f in ("u", "v", "p", "mDot")}
    s.close()
    if geom == "steady":
        c.settings.update(maxIter=r["iterations"])
        one = abi.Solver(abi.multiblock(c.blocks), c.bc_fields(), c.settings)
        one.solve()
        for f, a in fields.items():
            np.testing.assert_array_equal(a, one.get(f), err_msg=f)
        one.close()
