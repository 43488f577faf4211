"""Linear sweeps that run in one launch with the system on the chip (needs a
B200): bit for bit the oracle in FP64, and the tiled launches' fields in mixed
precision, on both sides of the single-CTA (2,048 cells) and cluster (16,384
cells) sizes, with odd, single and few sweeps, quads and triangles, Jacobi and
multicolour Gauss-Seidel, flow and scalars.
"""
import numpy as np
import pytest

from axisim import cases
import axisim.abi as abi
import oracle

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "p", "mDot")


def _case(nr, nz, linear, sweeps, its=2):
    c = cases.pipe(nr=nr, nz=nz, max_iter=its, tol=1e-30)
    c.settings.update(linearType=linear, linearMaxIter=sweeps)
    return c, abi.multiblock(c.blocks)


def _equal_to_oracle(c, mesh, fields=FIELDS):
    gpu = abi.Solver(mesh, c.bc_fields(), c.settings)
    gpu.solve()
    orc = oracle.Oracle(mesh, c.bc_fields(), c.settings)
    orc.run()
    for f in fields:
        np.testing.assert_array_equal(gpu.get(f), orc.get(f), err_msg=f)
    gpu.close()
    orc.close()


@pytest.mark.parametrize("linear", [cases.LINEAR_JACOBI, cases.LINEAR_GS_RB], ids=["jacobi", "gs"])
@pytest.mark.parametrize("nr,nz", [(2, 3), (16, 32), (32, 64), (31, 67), (64, 256), (113, 145)],
                         ids=["6", "512", "2048", "2077", "16384", "16385"])
def test_sizes_match_the_oracle(nr, nz, linear):
    _equal_to_oracle(*_case(nr, nz, linear, 20))


@pytest.mark.parametrize("linear", [cases.LINEAR_JACOBI, cases.LINEAR_GS_RB], ids=["jacobi", "gs"])
@pytest.mark.parametrize("sweeps", [1, 2, 3])
@pytest.mark.parametrize("nr,nz", [(8, 40), (40, 100)])
def test_few_sweeps_match_the_oracle(nr, nz, sweeps, linear):
    _equal_to_oracle(*_case(nr, nz, linear, sweeps))


@pytest.mark.parametrize("linear", [cases.LINEAR_JACOBI, cases.LINEAR_GS_RB], ids=["jacobi", "gs"])
def test_triangles_match_the_oracle(linear):
    c = cases.bullet(scale=0.12, max_iter=2, tol=1e-30)
    c.settings.update(linearType=linear)
    _equal_to_oracle(c, c.mesh)


@pytest.mark.parametrize("linear", [cases.LINEAR_JACOBI, cases.LINEAR_GS_RB], ids=["jacobi", "gs"])
@pytest.mark.parametrize("scale", [0.03, 0.1, 0.15])
def test_scalars_match_the_oracle(scale, linear):
    c = cases.with_scalars(cases.expansion(scale=scale, max_iter=2, tol=1e-30), wall_c=cases.michaelis_menten(1e-3, 0.2),
                           wall_layers=[(1e-6, 1e-4)], D=1e-6)
    c.settings.update(linearType=linear)
    _equal_to_oracle(c, abi.multiblock(c.blocks), FIELDS + ("T", "C"))


@pytest.mark.parametrize("scale", [0.03, 0.04, 0.06, 0.13])
def test_mixed_precision_equals_the_tiled_launches(scale):
    c = cases.expansion(scale=scale, max_iter=3, tol=1e-30)
    mesh = abi.multiblock(c.blocks)
    got = []
    for sweeps in (1, 3):
        s = abi.Solver(mesh, c.bc_fields(), c.settings, precision=abi.PREC_MIXED)
        s.set_momentum_sweeps(sweeps)
        s.solve()
        assert (s.sweep_tiles() > 0) == (sweeps > 1)
        got.append([s.get(f) for f in FIELDS])
        s.close()
    for f, a, b in zip(FIELDS, *got):
        np.testing.assert_array_equal(a, b, err_msg=f)
