"""Flexible CG on row counts off its blocks of 256 cells and four rows a thread
(needs a B200): run to a tolerance of 1e-8, the solve must leave a p' whose true
residual, formed from the device's own system in float64, meets it. The recursive
and the true residual drift apart by rounding of about cond(A) eps relative to
|A||p'|, far below 1e-8 of |b| on these meshes of at most a few thousand cells;
twice the tolerance is allowed.
"""
import numpy as np
import pytest

from axisim import cases
import axisim.abi as abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nr,nz", [(5, 51), (16, 16), (11, 93), (32, 32), (25, 41)],
                         ids=["255", "256", "1023", "1024", "1025"])
def test_solve_meets_its_tolerance(nr, nz, precision):
    c = cases.pipe(nr=nr, nz=nz, max_iter=2, tol=1e-30)
    c.settings.update(linearType=cases.LINEAR_JACOBI, mgMaxIter=400)
    mesh = abi.multiblock(c.blocks)
    s = abi.Solver(mesh, c.bc_fields(), c.settings, precision=precision, pressure_solver=abi.PSOLVE_FCG,
                   pressure_tol=1e-8, prolong_scale=2.0)
    s.solve()
    x, b, ac, af = s.get("pp"), s.get("b_pp"), s.get("AC_pp"), s.get("AF_pp")
    solves, its = s.pressure_stats()
    s.close()
    start, ids = mesh["cellFaceStart"], mesh["cellFaceIDs"]
    row = np.repeat(np.arange(len(x)), np.diff(start))
    own, nb = mesh["faceOwner"][ids], mesh["faceNeighbor"][ids]
    other = np.where(own == row, nb, own)
    inner = nb >= 0
    r = b - ac * x - np.bincount(row[inner], weights=(af * x[np.where(inner, other, 0)])[inner], minlength=len(x))
    assert solves == 2 and its < 800
    assert np.linalg.norm(r) <= 2e-8 * np.linalg.norm(b)


def test_triangles_meet_the_tolerance():
    c = cases.bullet(scale=0.1, max_iter=1, tol=1e-30)
    c.settings.update(useNonOrthCorrector=0, mgMaxIter=400)
    s = abi.Solver(c.mesh, c.bc_fields(), c.settings, pressure_solver=abi.PSOLVE_FCG, pressure_tol=1e-8,
                   prolong_scale=2.0)
    s.solve()
    x, b, ac, af = s.get("pp"), s.get("b_pp"), s.get("AC_pp"), s.get("AF_pp")
    s.close()
    m = c.mesh
    row = np.repeat(np.arange(len(x)), np.diff(m["cellFaceStart"]))
    own, nb = m["faceOwner"][m["cellFaceIDs"]], m["faceNeighbor"][m["cellFaceIDs"]]
    other, inner = np.where(own == row, nb, own), nb >= 0
    r = b - ac * x - np.bincount(row[inner], weights=(af * x[np.where(inner, other, 0)])[inner], minlength=len(x))
    assert np.linalg.norm(r) <= 2e-8 * np.linalg.norm(b)
