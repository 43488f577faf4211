"""Per-case residual statistics of a batch (needs a B200) against the per-cell
residual arrays, for case sizes at the edges of the reduction's rounds (fewer
cells than lanes, one short of and one past 32 rounds of 256 lanes) and every
norm. A sum of n non-negative terms in any order is within n eps of another
order; maxima are exact.
"""
import numpy as np
import pytest

from axisim import batch, cases
import axisim.abi as abi

pytestmark = pytest.mark.gpu

SIZES = [(4, 8), (8, 32), (16, 511), (16, 512), (3, 2731), (20, 700)]  # 32, 256, 8176, 8192, 8193, 14,000 cells


@pytest.mark.parametrize("norm", [0, 1, 2], ids=["L1", "L2", "LINF"])
def test_case_statistics_match_the_cells(norm):
    members = [cases.pipe(nr=a, nz=b, max_iter=3, tol=1e-30) for a, b in SIZES]
    union, start, bcs = batch.pack_union([abi.multiblock(c.blocks) for c in members], [c.groups for c in members])
    st = dict(members[0].settings, linearType=cases.LINEAR_JACOBI, resNorm=[norm, norm, 0], resScale=[0, 0, 0])
    s = abi.Solver(union, bcs, st)
    s.set_batch(start)
    s.solve()
    _, res = s.batch_status()
    ru, rv = s.get("res_U"), s.get("res_V")
    s.close()
    for c in range(len(SIZES)):
        for q, r in ((0, ru), (1, rv)):
            x = r[start[c]:start[c + 1]]
            want = (x.sum(), np.sqrt((x * x).sum()), x.max())[norm]
            if norm == 2:
                assert res[c, q] == want
            else:
                np.testing.assert_allclose(res[c, q], want, rtol=4 * len(x) * 2.3e-16)
