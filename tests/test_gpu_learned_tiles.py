"""The network's layers at row counts off their 16-row tiles and on both sides
of their dispatch (needs a B200), against the float64 oracle of the network on
the same rounded weights. With BF16 weights every product is exact and sums run
in FP32, so a prediction differs by roundings of 2^-24 through some 20 layers of
at most 256 terms: 1e-4 relative L2 leaves an order of magnitude. Losses and
gradients keep the bounds of the FP32 network (1e-5, 1e-4).
"""
import numpy as np
import pytest

from axisim import cases
import axisim.abi as abi
import learned_ref as LR

pytestmark = pytest.mark.gpu


def _bf16_round(x):
    u = np.asarray(x, np.float32).view(np.uint32).astype(np.uint64)
    u = (u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000
    return u.astype(np.uint32).view(np.float32)


# 15, 65, 1,023 and 66,049 cells: one level below a tile, odd remainders on every
# level, and a finest coarse level on the other side of the 16,384-row rule
@pytest.mark.parametrize("nr,nz", [(3, 5), (5, 13), (31, 33), (257, 257)], ids=lambda v: str(v))
def test_prediction_and_gradient_match_the_oracle(nr, nz):
    case = cases.pipe(nr=nr, nz=nz, max_iter=1, tol=1e-30)
    mesh = abi.multiblock(case.blocks)
    s = abi.Solver(mesh, case.bc_fields(), case.settings)
    s.learned_init(abi.NET_BF16_WEIGHTS, seed=nr)
    levels = s.mg_levels()
    net = LR.NetRef(LR.hierarchy(mesh, s.mg_level_maps, len(levels)))
    p = s.learned_params()
    p[np.abs(p) == 0] = 0.01  # biases off zero
    s.learned_set_params(p)
    p64 = _bf16_round(p).astype(np.float64)
    rng = np.random.default_rng(nz)
    n = int(mesh["nCells"])
    ac, af = LR.random_spd_system(mesh, rng)
    A = LR.matrix(mesh, ac.astype(np.float32), af.astype(np.float32))
    t = rng.standard_normal(n)
    b = A @ t
    d = 1.0 - (np.asarray(abs(A).sum(1)).ravel() - ac) / ac
    want = net.predict(p64, b.astype(np.float32), ac.astype(np.float32), d.astype(np.float32))
    got = s.learned_predict(b, ac, d)
    assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want)
    s.learned_harvest(0, 1)
    s.learned_add_sample(b, t, ac, d, af)
    b32, t32, ac32, d32, af32, _ = s.learned_get_sample(0)
    loss_ref, g_ref = net.loss_and_grad(p64, b32, t32, ac32, d32, LR.matrix(mesh, ac32, af32))
    loss, g = s.learned_grad(0)
    assert abs(loss - loss_ref) <= 1e-5 * max(loss_ref, 1e-3)
    assert np.linalg.norm(g - g_ref) <= 1e-4 * np.linalg.norm(g_ref)
    s.close()
