"""Cycles that the deep levels' cluster launch does not take (needs a B200): with
more sweeps than it lists, the small levels run in the single-CTA tail; with the
resident V-cycle switched on and off on one handle, also between solves. The
fields are the oracle's bit for bit.
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


@pytest.mark.parametrize("modes", ["rp", "pr", "rpr"])
@pytest.mark.parametrize("geom", ["pipe", "triangles"])
def test_switching_the_kernel_of_the_cycle(geom, modes):
    c = cases.pipe(nr=64, nz=100) if geom == "pipe" else cases.bullet(scale=0.1)
    c.settings.update(linearType=cases.LINEAR_JACOBI, maxIter=2, resTol=[1e-30] * 3)
    mesh = c.packed(abi.multiblock)
    orc = oracle.Oracle(mesh, c.bc_fields(), c.settings)
    orc.run()
    gpu = abi.Solver(mesh, c.bc_fields(), c.settings)
    for m in modes:
        gpu.set_vcycle_kernel(abi.VCYCLE_RESIDENT if m == "r" else abi.VCYCLE_PER_PHASE)
        gpu.solve()
        for f in ("u", "v", "p", "pp", "mDot"):
            np.testing.assert_array_equal(gpu.get(f), orc.get(f), err_msg=f"{f} {m}")
    gpu.close()
    orc.close()
