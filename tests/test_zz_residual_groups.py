"""axisim_residual_static at the edges of its blocks (needs a B200): cell counts
around a group of 256 and around the size from which a block takes several
groups, arrays off their 16-byte boundaries, and cells of three slots, which
take its general slot loop. Per-cell outputs are the same operations in the same
order without contraction, so they are equal bit for bit; a sum of n terms in
another order is within n eps of the largest partial sum, here of the sum of
magnitudes.
"""
import ctypes as C

import numpy as np
import pytest

from axisim import cases
import axisim.abi as abi

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MESHES = {"255": (15, 17), "256": (16, 16), "257": (1, 257), "151552": (256, 592), "151553": (43, 3525)}


def _mesh(name):
    if name == "triangles":
        return cases.bullet(scale=0.1).mesh
    nr, nz = MESHES[name]
    return abi.multiblock(cases.pipe(nr=nr, nz=nz).blocks)


def _device(a, shift):
    """`a` on the device, starting `shift` elements past an aligned address."""
    t = torch.zeros(len(a) + shift, dtype=torch.from_numpy(a[:0]).dtype, device="cuda")
    t[shift:] = torch.from_numpy(a).cuda()
    return t[shift:]


@pytest.mark.parametrize("norm", [0, 1, 2], ids=["L1", "L2", "LINF"])
@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "shifted"])
@pytest.mark.parametrize("name", list(MESHES) + ["triangles"])
def test_outputs_equal_the_same_operations(name, shift, norm):
    m = _mesh(name)
    n, f, slots = int(m["nCells"]), int(m["nFaces"]), len(m["cellFaceIDs"])
    rng = np.random.default_rng(n + norm)
    ids = m["cellFaceIDs"]
    own, nb = m["faceOwner"], m["faceNeighbor"]
    af = np.where(nb[ids] >= 0, -rng.uniform(0.1, 1.0, slots), 0.0)
    d = dict(AF=af, ACu=rng.uniform(2, 5, n), ACv=rng.uniform(2, 5, n), bu=rng.standard_normal(n),
             bv=rng.standard_normal(n), u=rng.standard_normal(n), v=rng.standard_normal(n), mDot=rng.standard_normal(f))
    dev = {k: _device(np.ascontiguousarray(a), shift) for k, a in d.items()}
    dev.update({k: _device(np.ascontiguousarray(m[k]), shift)
                for k in ("cellFaceStart", "cellFaceIDs", "faceOwner", "faceNeighbor")})
    out = {k: torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for k in ("resU", "resV", "resC")}
    out["sums"] = torch.zeros(5, dtype=torch.float64, device="cuda")
    err = C.create_string_buffer(256)
    st = abi.lib().axisim_residual_static(
        n, f, slots, *(dev[k].data_ptr() for k in ("cellFaceStart", "cellFaceIDs", "faceOwner", "faceNeighbor", "AF",
                                                   "ACu", "ACv", "bu", "bv", "u", "v", "mDot")),
        norm, norm, *(out[k].data_ptr() for k in ("resU", "resV", "resC", "sums")),
        torch.cuda.current_stream().cuda_stream, err, len(err))
    assert st == abi.OK, err.value
    W = slots // n
    face = ids.reshape(n, W)
    me = np.arange(n)
    ax = {k: d["AC" + k] * d[k] for k in "uv"}
    scale = {k: np.abs(ax[k]).sum() for k in "uv"}
    imb = np.zeros(n)
    for j in range(W):
        g = face[:, j]
        mine, inner = own[g] == me, nb[g] >= 0
        other = np.where(mine, nb[g], own[g])
        for k in "uv":
            ax[k] = np.where(inner, ax[k] + af.reshape(n, W)[:, j] * d[k][np.where(inner, other, 0)], ax[k])
        imb = np.where(mine, imb + d["mDot"][g], imb - d["mDot"][g])
    ru, rv = np.abs(d["bu"] - ax["u"]), np.abs(d["bv"] - ax["v"])
    for key, want in (("resU", ru), ("resV", rv), ("resC", imb)):
        np.testing.assert_array_equal(out[key].cpu().numpy(), want, err_msg=key)
    stat = (np.sum, lambda x: np.sum(x * x), np.max)[norm]
    want = np.array([stat(ru), scale["u"], stat(rv), scale["v"], np.abs(imb).sum()])
    np.testing.assert_allclose(out["sums"].cpu().numpy(), want, rtol=2 * n * 2.3e-16)
