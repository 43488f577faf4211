"""A batch with a case whose fields are not finite (needs a B200): the case's
statistics are what its standalone solve reports, in every norm, and the batch
ends as diverged. A maximum over cells that are all NaN is the empty maximum,
-inf, never a converged 0.
"""
import numpy as np
import pytest

from axisim import batch, cases
import axisim.abi as abi

pytestmark = pytest.mark.gpu

SIZES = [(4, 8), (8, 32), (16, 20)]  # fewer cells than lanes, as many, more


@pytest.mark.parametrize("norm", [0, 1, 2], ids=["L1", "L2", "LINF"])
@pytest.mark.parametrize("bad", range(len(SIZES)))
def test_statistics_of_a_case_of_nans(bad, norm):
    members = [cases.pipe(nr=a, nz=b, max_iter=12, tol=0.0, U0=float("nan") if i == bad else 0.05)
               for i, (a, b) in enumerate(SIZES)]
    for c in members:
        # U and V alone are monitored: a sum over the cells would show the NaN in the continuity
        c.settings.update(linearType=cases.LINEAR_JACOBI, resNorm=[norm, norm, 0], resScale=[0, 0, 0],
                          resEnabled=[1, 1, 0])
    meshes = [abi.multiblock(c.blocks) for c in members]
    union, start, bcs = batch.pack_union(meshes, [c.groups for c in members])
    s = abi.Solver(union, bcs, members[0].settings)
    s.set_batch(start)
    r = s.solve(allow=(abi.OK, abi.E_DIVERGED))
    _, res = s.batch_status()
    u = s.get("u")
    s.close()
    assert r["status"] == abi.E_DIVERGED and not r["converged"]
    assert np.isnan(u[start[bad]:start[bad + 1]]).any()
    alone = abi.Solver(meshes[bad], members[bad].bc_fields(), dict(members[bad].settings, maxIter=r["iterations"]))
    ra = alone.solve(allow=(abi.OK, abi.E_DIVERGED))
    alone.close()
    assert ra["iterations"] == r["iterations"]
    np.testing.assert_array_equal(res[bad, :2], ra["residual"][:2])
    assert np.isfinite(np.delete(res[:, :2], bad, axis=0)).all()
