"""Cases of a batch that end above its deepest level run their coarsest-level
sweeps beside the deeper levels when nothing reads the level in between (at most
one pre-smoothing sweep), else in line (needs a B200). The first gather's sweep
is also left out (no pre-sweep). Either way each case evolves as it does alone,
bit for bit, over several cycles an iteration and a second solve on the same
solver.
"""
import numpy as np
import pytest

from axisim import batch, cases
import axisim.abi as abi

pytestmark = pytest.mark.gpu

SIZES = [(8, 24), (12, 30), (16, 100), (40, 160)]  # 192 to 6,400 cells: coarsest levels at different depths


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("pre", [0, 1, 2])
def test_each_case_evolves_as_alone(pre, precision):
    members = [cases.pipe(nr=a, nz=b, max_iter=4, tol=1e-30) for a, b in SIZES]
    meshes = [abi.multiblock(c.blocks) for c in members]
    union, start, bcs = batch.pack_union(meshes, [c.groups for c in members])
    _, term = abi.mg_batch_levels_host(union, start)
    assert (term > 0).sum() >= 2
    st = dict(members[0].settings, mgPreSweep=pre)
    s = abi.Solver(union, bcs, st, precision=precision)
    s.set_batch(start)
    s.solve()
    s.solve(cont=True)
    got = {f: batch.split_fields(s.get(f), start) for f in ("u", "v", "p")}
    s.close()
    for i, c in enumerate(members):
        alone = abi.Solver(meshes[i], c.bc_fields(), dict(c.settings, mgPreSweep=pre), precision=precision)
        alone.solve()
        alone.solve(cont=True)
        for f in got:
            np.testing.assert_array_equal(got[f][i], alone.get(f), err_msg=f"{i} {f}")
        alone.close()
