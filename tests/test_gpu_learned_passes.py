"""The network's two forward passes (needs a B200): a prediction's and the one that
a solve applies and a loss is formed on, at odd row counts and with BF16 and
FP32 activations. The prediction against the float64 oracle on the same rounded
weights, d apart at most in relative L2: 1e-4 with FP32 activations, 30 layers of
2^-9 with BF16 ones. The loss 1 - (y.b)^2 / ((y.A y)(b.t)) of the prediction
against that of the other pass (FP32 activations): one minus the squared cosine
of y and t in the energy norm, which d in relative L2 turns into at most
d sqrt(cond A), and the squared cosine by twice that, a pass.
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


@pytest.mark.parametrize("prec,d", [(abi.NET_BF16_WEIGHTS, 1e-4), (abi.NET_BF16, 30 * 2.0 ** -9)], ids=["fp32", "bf16"])
@pytest.mark.parametrize("nr,nz", [(3, 5), (5, 13), (31, 33), (101, 99)], ids=lambda v: str(v))
def test_prediction_and_its_loss(nr, nz, prec, d):
    case = cases.pipe(nr=nr, nz=nz, max_iter=1, tol=1e-30)
    mesh = abi.multiblock(case.blocks)
    s = abi.Solver(mesh, case.bc_fields(), case.settings)
    s.learned_init(prec, seed=nr)
    levels = s.mg_levels()
    net = LR.NetRef(LR.hierarchy(mesh, s.mg_level_maps, len(levels)))
    params = _bf16_round(s.learned_params()).astype(np.float64)
    rng = np.random.default_rng(nz)
    ac, af = LR.random_spd_system(mesh, rng)
    A = LR.matrix(mesh, ac, af)
    t = rng.standard_normal(int(mesh["nCells"]))
    b = A @ t
    off = np.asarray(abs(A).sum(1)).ravel() - ac
    s.learned_harvest(0, 1)
    s.learned_add_sample(b, t, ac, 1.0 - off / ac, af)
    b, t, ac, deficit, af, _ = (np.asarray(v, np.float64) for v in s.learned_get_sample(0))
    A = LR.matrix(mesh, ac, af)
    loss, _ = s.learned_grad(0)
    y = s.learned_predict(b, ac, deficit).astype(np.float64)
    s.close()
    ref = net.predict(params, b, ac, deficit)
    assert np.linalg.norm(y - ref) <= d * np.linalg.norm(ref)
    if prec == abi.NET_BF16:
        return
    want = 1.0 - (y @ b) ** 2 / ((y @ (A @ y)) * (b @ t))
    cond = (ac + off).max() / (ac - off).min()  # Gershgorin
    assert abs(loss - want) <= 2 * 2 * d * np.sqrt(cond)
