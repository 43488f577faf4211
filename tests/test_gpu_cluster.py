"""The V-cycle's deep levels in one thread-block cluster (needs a B200): bit
for bit the oracle in FP64 and the per-phase arithmetic of the resident kernel
in mixed precision, on hierarchies at the edges of the kernel's layout (a level
just below and above the single-CTA size 1024 and the cluster's size 15,360,
partial slices, a single level) and over the sweep counts that change its steps.
"""
import numpy as np
import pytest

from axisim import cases
import axisim.abi as abi
import oracle

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "p", "pp", "mDot")
# (radial, axial) cells of a pipe -> cells of its first coarse levels
SIZES = {(8, 40): 80, (10, 37): 97, (63, 65): 1021, (64, 64): 1025, (64, 66): 1056, (128, 240): 7680,
         (128, 479): 15331, (128, 480): 15362}


def _pipe(nr, nz, its=2, **settings):
    c = cases.pipe(nr=nr, nz=nz, max_iter=its, tol=1e-30)
    c.settings.update(linearType=cases.LINEAR_JACOBI, **settings)
    return c, abi.multiblock(c.blocks)


@pytest.mark.parametrize("nr,nz", sorted(SIZES), ids=lambda v: str(v))
def test_sizes_match_the_oracle(nr, nz):
    c, mesh = _pipe(nr, nz)
    gpu = abi.Solver(mesh, c.bc_fields(), c.settings)
    gpu.solve()
    orc = oracle.Oracle(mesh, c.bc_fields(), c.settings)
    orc.run()
    for f in FIELDS:
        np.testing.assert_array_equal(gpu.get(f), orc.get(f), err_msg=f)
    assert any(k["name"] == "mg_smooth_cluster" for k in gpu.profile(1))
    gpu.close()
    orc.close()


@pytest.mark.parametrize("pre,post,coarse", [(0, 1, 30), (1, 0, 30), (2, 1, 29), (1, 2, 1), (3, 3, 0), (0, 2, 2)])
@pytest.mark.parametrize("geom", ["pipe", "triangles"])
def test_sweep_counts_match_the_oracle(geom, pre, post, coarse):
    if geom == "pipe":
        c, mesh = _pipe(64, 100)
    else:
        c = cases.bullet(scale=0.2, max_iter=2, tol=1e-30)
        mesh = c.mesh
    c.settings.update(mgPreSweep=pre, mgPostSweep=post, mgLinearSweep=coarse, mgMaxIter=2)
    gpu = abi.Solver(mesh, c.bc_fields(), c.settings)
    gpu.solve()
    orc = oracle.Oracle(mesh, c.bc_fields(), c.settings)
    orc.run()
    for f in FIELDS:
        np.testing.assert_array_equal(gpu.get(f), orc.get(f), err_msg=f)
    gpu.close()
    orc.close()


@pytest.mark.parametrize("nr,nz", [(8, 40), (63, 65), (64, 66), (128, 480)])
def test_mixed_precision_equals_the_per_phase_arithmetic(nr, nz):
    c, mesh = _pipe(nr, nz)
    got = []
    for mode in (abi.VCYCLE_PER_PHASE, abi.VCYCLE_RESIDENT):
        s = abi.Solver(mesh, c.bc_fields(), c.settings, precision=abi.PREC_MIXED)
        s.set_vcycle_kernel(mode)
        s.solve()
        got.append([s.get(f) for f in FIELDS])
        s.close()
    for f, a, b in zip(FIELDS, *got):
        np.testing.assert_array_equal(a, b, err_msg=f)
