"""Cycles with more sweeps than the deep levels' cluster launch takes (needs a
B200): the small levels run in the single-CTA tail, and the fields are the
oracle's bit for bit.
"""
import numpy as np
import pytest

from axisim import cases
import axisim.abi as abi
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nz,pre,post", [(8, 64, 70, 1), (64, 100, 40, 1), (64, 100, 1, 40), (64, 100, 8, 8)])
def test_more_sweeps_than_steps(nr, nz, pre, post):
    c = cases.pipe(nr=nr, nz=nz, max_iter=2, tol=1e-30)
    c.settings.update(linearType=cases.LINEAR_JACOBI, mgPreSweep=pre, mgPostSweep=post)
    mesh = abi.multiblock(c.blocks)
    plan = abi.vcycle_cluster_host(mesh, pre=pre, post=post)
    assert len(plan["steps"]) == 0 and len(abi.vcycle_cluster_host(mesh)["steps"]) > 0
    gpu = abi.Solver(mesh, c.bc_fields(), c.settings)
    gpu.solve()
    orc = oracle.Oracle(mesh, c.bc_fields(), c.settings)
    orc.run()
    for f in ("u", "v", "p", "pp", "mDot"):
        np.testing.assert_array_equal(gpu.get(f), orc.get(f), err_msg=f)
    names = {k["name"] for k in gpu.profile(1)}
    assert "mg_tail" in names and "mg_smooth_cluster" not in names
    gpu.close()
    orc.close()
