"""Cases in one mesh on the deep multigrid levels' cluster (needs a B200). Batches
whose cases' coarsest levels, merged, are larger than it has threads: every case
equals its standalone solve bit for bit, in FP64 and mixed precision, on both
sides of 512 and of 1,024 rows. Small cases that share one hierarchy, with whole
slices of isolated coarse cells, and meshes with a single coarse level: the
oracle's fields bit for bit.
"""
import numpy as np
import pytest

from axisim import batch, cases
import axisim.abi as abi
import oracle
from test_cluster_plan_cpu import BATCHES, SMALL, SORTED

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "p", "mDot")


def _member(i, nr, nz):
    c = cases.pipe(nr=nr, nz=nz, max_iter=2, tol=1e-30, U0=0.02 + 0.001 * i)
    c.settings.update(linearType=cases.LINEAR_JACOBI)
    return c


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("rows", list(BATCHES))
def test_every_case_equals_its_own_solve(rows, precision):
    sizes = [(nr, nz) for n, nr, nz in BATCHES[rows] for _ in range(n)]
    members = [_member(i, *s) for i, s in enumerate(sizes)]
    meshes = [abi.multiblock(c.blocks) for c in members]
    union, start, bcs = batch.pack_union(meshes, [c.groups for c in members])
    s = abi.Solver(union, bcs, members[0].settings, precision=precision)
    s.set_batch(start)
    s.solve()
    got = {f: s.get(f) for f in FIELDS}
    s.close()
    faces = np.cumsum([0] + [m["nFaces"] for m in meshes])
    for i in sorted({0, 1, len(members) // 2, len(members) - 1}):
        one = abi.Solver(meshes[i], members[i].bc_fields(), members[i].settings, precision=precision)
        one.solve()
        for f in FIELDS:
            at = faces if f == "mDot" else start
            np.testing.assert_array_equal(got[f][at[i]:at[i + 1]], one.get(f), err_msg=f"{f} of case {i}")
        one.close()


@pytest.mark.parametrize("name", ["small", "sorted", "mixed"])
def test_isolated_cells_match_the_oracle(name):
    # cases that share one hierarchy: a case down to one cell is a coarse cell without a neighbour
    sizes = {"small": SMALL, "sorted": SORTED, "mixed": [(2, 4)] * 40 + [(40, 200)]}[name]
    members = [_member(i % 8, *s) for i, s in enumerate(sizes)]
    union, _, bcs = batch.pack_union([abi.multiblock(c.blocks) for c in members], [c.groups for c in members])
    gpu = abi.Solver(union, bcs, members[0].settings)
    gpu.solve()
    orc = oracle.Oracle(union, bcs, members[0].settings)
    orc.run()
    for f in FIELDS + ("pp",):
        np.testing.assert_array_equal(gpu.get(f), orc.get(f), err_msg=f)
    gpu.close()
    orc.close()


@pytest.mark.parametrize("coarse", [0, 1, 2, 30])
@pytest.mark.parametrize("nr,nz", [(8, 16), (10, 10), (5, 37)])
def test_a_single_coarse_level_matches_the_oracle(nr, nz, coarse):
    c = _member(0, nr, nz)
    c.settings.update(mgLinearSweep=coarse)
    mesh = abi.multiblock(c.blocks)
    plan = abi.vcycle_cluster_host(mesh, coarse=coarse)
    assert (plan["first"], plan["count"]) == (1, 1)
    gpu = abi.Solver(mesh, c.bc_fields(), c.settings)
    gpu.solve()
    orc = oracle.Oracle(mesh, c.bc_fields(), c.settings)
    orc.run()
    for f in FIELDS + ("pp",):
        np.testing.assert_array_equal(gpu.get(f), orc.get(f), err_msg=f)
    gpu.close()
    orc.close()
