"""Workloads of the solver library, each through the entry points a program
calls: whole SIMPLE runs (structured, unstructured, transient, batched, with
scalars), the learned preconditioner's inference and training gradient, and
the residuals of caller-owned device arrays.

A case is a dict of plain values; `prepare` builds what a program holds before
the call (mesh, handle, boundary conditions, initial fields, network weights)
and `run` makes the call.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("axisim-software_b200"))  # the package lies one folder below the repository's root

from axisim import abi, batch, cases  # noqa: E402

FULL = 874_496           # cells of the expansion at scale 1
TRANSIENT = 1.512        # scale of the 2M-cell pulsatile expansion


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # The smallest call: a coarse preview of the expansion, where launches are everything.
        dict(name="expansion_864_fp64", kind="run", geom="expansion", scale=1 / 32, precision="fp64", iters=10),
        # Laminar pipe on 40 x 200 cells, multicolour Gauss-Seidel and Green-Gauss: the case a new user
        # starts with and runs to convergence (thousands of iterations of this size).
        dict(name="pipe_8000_fp64_gs", kind="run", geom="pipe", nr=40, nz=200, precision="fp64", iters=60),
        # A mid-size design study continued from given fields (uploaded, advanced, read back), odd sizes.
        dict(name="expansion_54k_mixed_continue", kind="continue", geom="expansion", scale=0.2477, precision="mixed",
             iters=40),
        # The production steady run: 256 x 4096 bands, mixed precision, continued from given fields.
        dict(name="expansion_874k_mixed_continue", kind="continue", geom="expansion", scale=1.0, precision="mixed",
             iters=20),
        # The same mesh all in FP64 from rest: the accuracy oracle of every mixed run.
        dict(name="expansion_874k_fp64", kind="run", geom="expansion", scale=1.0, precision="fp64", iters=10),
        # Unstructured triangles with least squares and the non-orthogonal corrector.
        dict(name="bullet_486k_mixed", kind="run", geom="bullet", scale=1.0, precision="mixed", iters=10),
        # One BDF2 step of the pulsatile transient with the flexible-CG pressure solve: the largest call.
        dict(name="pulsatile_2M_mixed_fcg", kind="run", geom="pulsatile", scale=TRANSIENT, precision="mixed", iters=3,
             steps=1, fcg=30),
        # A parameter study: 32 independent pipes and expansions of uneven size in one batch.
        dict(name="batch_32_fp64", kind="run", geom="batch", n=32, mix=0, size=1.0, precision="fp64", iters=10),
        # Heat and mass transport with a reactive wall on top of the flow.
        dict(name="scalars_218k_fp64", kind="run", geom="scalars", scale=0.5, precision="fp64", iters=12),
        # The learned preconditioner on its own: inference, and the gradient a training step takes.
        dict(name="network_predict_874k", kind="predict", scale=1.0),
        dict(name="network_grad_218k", kind="grad", scale=0.5),
        # Monitoring: residuals of device arrays that another program owns.
        dict(name="residual_874k", kind="residual", scale=1.0, norm=0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges: size, odd band counts, precision and
    options drawn; no case costs more than the largest listed one."""
    kind = rng.choice(["expansion", "expansion", "pipe", "bullet", "pulsatile", "batch", "scalars", "predict", "grad",
                       "residual"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "expansion":
        scale = math.sqrt(_log(rng, 800, 900_000) / FULL)
        return dict(kind=rng.choice(["run", "continue"]), geom=kind, scale=scale, precision=prec,
                    iters=rng.randint(5, 20), scheme=rng.choice([0, 1, 2]), gradient=rng.choice([0, 1]))
    if kind == "pipe":
        n = _log(rng, 400, 60_000)
        nr = max(5, int(math.sqrt(n / rng.uniform(4.0, 8.0))))
        return dict(kind="run", geom=kind, nr=nr, nz=max(10, int(n / nr)), precision=prec, iters=rng.randint(10, 60),
                    linear=rng.choice([0, 1]))
    if kind == "bullet":
        return dict(kind="run", geom=kind, scale=math.sqrt(_log(rng, 1_200, 480_000) / 486_000), precision=prec,
                    iters=rng.randint(4, 10))
    if kind == "pulsatile":
        scale = math.sqrt(_log(rng, 3_000, 1_500_000) / FULL)
        return dict(kind="run", geom=kind, scale=scale, precision=prec, iters=rng.randint(2, 3),
                    steps=rng.randint(1, 2), fcg=rng.randint(8, 15), learned=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind="run", geom=kind, n=rng.randint(3, 32), mix=rng.randint(1, 1000),
                    size=_log(rng, 0.05, 0.8), precision=prec, iters=rng.randint(5, 10))
    if kind == "scalars":
        return dict(kind="run", geom=kind, scale=math.sqrt(_log(rng, 800, 220_000) / FULL), precision="fp64",
                    iters=rng.randint(5, 12))
    hi = {"predict": 860_000, "grad": 210_000, "residual": 1_900_000}[kind]
    c = dict(kind=kind, scale=math.sqrt(_log(rng, 900, hi) / FULL))
    if kind == "residual":
        c["norm"] = rng.choice([0, 1, 2])
    return c


# ------------------------------------------------------------------ meshes
@functools.lru_cache(maxsize=6)
def _blocks_mesh(key):
    kind, a, b = key
    if kind == "pipe":
        return abi.multiblock(cases.pipe(nr=a, nz=b).blocks)
    return abi.multiblock(cases.expansion(scale=a).blocks)


@functools.lru_cache(maxsize=2)
def _batch_members(n, mix, size):
    members = batch.random_cases(n=n, seed=mix, scale=size)
    return members, [abi.multiblock(c.blocks) for c in members]


def _pinned(n, dtype=torch.float64):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


def _settings(c, case):
    s = case.settings
    s.update(maxIter=c["iters"], resTol=[1e-30, 1e-30, 1e-30])
    if c.get("scheme") is not None:
        s["convectionScheme"] = c["scheme"]
    if c.get("gradient") is not None:
        s["gradientScheme"] = c["gradient"]
    if c.get("linear") is not None:
        s["linearType"] = c["linear"]
    if c.get("fcg"):
        s["mgMaxIter"] = c["fcg"]
    return s


def _flow_case(c, seed):
    """(Case, mesh, batch offsets): the flow of `seed` on the case's mesh; the
    throat Reynolds number (inlet velocity) differs from seed to seed."""
    rng = np.random.default_rng(seed)
    re = 500.0 * rng.uniform(0.8, 1.2)
    geom = c["geom"]
    if geom == "pipe":
        case = cases.pipe(nr=c["nr"], nz=c["nz"], U0=0.05 * re / 500.0)
        return case, _blocks_mesh(("pipe", c["nr"], c["nz"])), None
    if geom == "bullet":
        case = cases.bullet(scale=c["scale"], re=0.4 * re, seed=seed)  # the jitter of the vertices too
        return case, case.mesh, None
    if geom == "pulsatile":
        case = cases.pulsatile_expansion(scale=c["scale"], dt=1e-4, steps=c["steps"])
        u = case.groups[0].bcs[cases.U]
        case.groups[0].bcs[cases.U] = (u[0], u[1] * re / 500.0) + tuple(u[2:])
        return case, _blocks_mesh(("expansion", c["scale"], 0)), None
    if geom == "batch":
        members, meshes = _batch_members(c["n"], c["mix"], c["size"])
        groups = []
        for m in members:
            f = rng.uniform(0.8, 1.2)
            gs = []
            for g in m.groups:
                bcs = {k: (v[0], v[1] * f) if k == cases.U else v for k, v in g.bcs.items()}
                gs.append(cases.Group(g.id, g.btype, bcs, g.total_length))
            groups.append(gs)
        mesh, start, bcs = batch.pack_union(meshes, groups)
        case = cases.Case("batch", [], [], dict(members[0].settings), mesh=mesh)
        return (case, bcs), mesh, start
    case = cases.expansion(scale=c["scale"], re=re)
    if geom == "scalars":
        case = cases.with_scalars(case, wall_c=cases.michaelis_menten(1e-3, 0.2), wall_layers=[(1e-6, 1e-4)], D=1e-6,
                                  t_in=300.0 + 10.0 * rng.uniform(0.5, 1.5), c_in=rng.uniform(0.8, 1.2))
    return case, _blocks_mesh(("expansion", c["scale"], 0)), None


def _initial_fields(mesh, settings, seed):
    """A start a user brings along: the developed profile of each section with
    a few per cent of smooth disturbance, its pressure drop, and the face mass
    fluxes of the undisturbed profile."""
    rng = np.random.default_rng(seed + 77)
    rho, mu = settings["rho"], settings["mu"]
    r_in, r_out, l_in, total = 0.002, 0.006, 0.04, 0.16
    ubar = 500.0 * rng.uniform(0.8, 1.2) * mu / (rho * 2.0 * r_in)

    def profile(z, r):
        R = np.where(z < l_in, r_in, r_out)
        return 2.0 * ubar * (r_in / R) ** 2 * (1.0 - np.minimum(r / R, 1.0) ** 2)

    z, r = mesh["cellCenterZ"], mesh["cellCenterR"]
    wave = np.zeros(len(z))
    for _ in range(3):
        k, m, ph = rng.uniform(1, 12), rng.uniform(1, 4), rng.uniform(0, 2 * np.pi)
        wave += 0.01 * np.sin(2 * np.pi * k * z / total + ph) * np.cos(np.pi * m * r / r_out)
    u = profile(z, r) * (1.0 + wave)
    v = 0.01 * ubar * wave
    g1, g2 = (8.0 * mu * ubar * (r_in / R) ** 2 / R ** 2 for R in (r_in, r_out))
    p = np.where(z < l_in, g2 * (total - l_in) + g1 * (l_in - z), g2 * (total - z)) * (1.0 + wave)
    uf = profile(mesh["faceCenterZ"], mesh["faceCenterR"])
    md = rho * uf * mesh["faceNormalZ"] * mesh["faceArea"]
    out = {}
    for k, a in (("u", u), ("v", v), ("p", p), ("mDot", md)):
        out[k] = _pinned(len(a))
        out[k][:] = a
    return out


# ----------------------------------------------------------------- network
@functools.lru_cache(maxsize=4)
def _graph(scale):
    """The mesh and, per level, (cells, neighbour pairs, map to the next level)
    of the hierarchy the network lives on."""
    mesh = _blocks_mesh(("expansion", scale, 0))
    n, r, col, slot = _level0(mesh)
    levels = []
    cells = abi.mg_levels_host(mesh)
    for lv in range(len(cells)):
        if lv + 1 == len(cells):
            levels.append((n, r, col, None))
            break
        c2c, _, start, nb = abi.mg_level_maps_host(mesh, lv)
        levels.append((n, r, col, c2c))
        n = len(start) - 1
        r = np.repeat(np.arange(n), np.diff(start))
        keep = (nb >= 0) & (nb != r)
        r, col = r[keep], nb[keep]
    return mesh, levels


def _level0(mesh):
    start, ids = mesh["cellFaceStart"], mesh["cellFaceIDs"]
    own, nb = mesh["faceOwner"], mesh["faceNeighbor"]
    n = int(mesh["nCells"])
    row = np.repeat(np.arange(n), np.diff(start))
    other = np.where(own[ids] == row, nb[ids], own[ids])
    keep = other >= 0
    return n, row[keep], other[keep], np.nonzero(keep)[0]


CHANNELS = (16, 32, 64, 128)


def _net_layers(depth):
    """Layers in forward order, (weight group, input width, output width, level),
    and the groups' offsets in the flat parameter vector."""
    ch = [CHANNELS[min(lv, 3)] for lv in range(depth)]
    groups, total, order = {}, 0, []

    def layer(key, k, co, lv):
        nonlocal total
        if key not in groups:
            groups[key] = (total, k, co)
            total += k * co + co
        order.append((key, k, co, lv))

    layer("in", 2, ch[0], 0)
    layer("enc0", 2 * ch[0], ch[0], 0)
    for lv in range(1, depth):
        layer("down%d" % min(lv, 4), ch[lv - 1], ch[lv], lv)
        layer("enc%d" % min(lv, 3), 2 * ch[lv], ch[lv], lv)
    layer("mid%d" % min(depth - 1, 3), 2 * ch[-1], ch[-1], depth - 1)
    for lv in range(depth - 2, -1, -1):
        layer("up%d" % min(lv, 3), ch[lv + 1], ch[lv], lv)
        layer("dec%d" % min(lv, 3), 2 * ch[lv], ch[lv], lv)
    layer("out", ch[0], 1, 0)
    return groups, total, order


def _weights(depth, seed):
    """Weights as after some training: the spread of a fan-in initialisation,
    small biases."""
    groups, total, _ = _net_layers(depth)
    rng = np.random.default_rng(seed + 5)
    p = np.zeros(total, np.float32)
    for key, (o, k, co) in groups.items():
        a = math.sqrt((3.0 if key == "out" else 6.0) / k)
        p[o:o + k * co] = rng.uniform(-a, a, k * co)
        p[o + k * co:o + k * co + co] = rng.uniform(-0.05, 0.05, co)
    return p


def _pressure_system(mesh, seed):
    """A p'-like system on the mesh in FP32: (right-hand side, its solution,
    diagonal, boundary deficit, off-diagonals per slot)."""
    rng = np.random.default_rng(seed + 11)
    n, row, col, slot = _level0(mesh)
    w = rng.uniform(0.5, 2.0, mesh["nFaces"])
    af = np.zeros(len(mesh["cellFaceIDs"]))
    af[slot] = -w[mesh["cellFaceIDs"][slot]]
    off = np.bincount(row, weights=-af[slot], minlength=n)
    ac = off + rng.uniform(0.01, 0.1, n)
    z, r = mesh["cellCenterZ"] / 0.16, mesh["cellCenterR"] / 0.006
    t = np.zeros(n)
    for _ in range(6):
        t += rng.standard_normal() * np.sin(rng.uniform(1, 20) * z + rng.uniform(0, 6)) * np.cos(rng.uniform(0, 6) * r)
    t += 0.01 * rng.standard_normal(n)
    af, ac, t = (x.astype(np.float32) for x in (af, ac, t))
    b = (ac.astype(np.float64) * t + np.bincount(row, weights=af[slot].astype(np.float64) * t[col], minlength=n))
    return b.astype(np.float32), t, ac, ((ac - off) / ac).astype(np.float32), af


# ---------------------------------------------------------------- the passes
def prepare(case, seed):
    kind = case["kind"]
    if kind == "residual":
        return _prepare_residual(case, seed)
    if kind in ("predict", "grad"):
        flow = cases.expansion(scale=case["scale"], max_iter=1)
        mesh, levels = _graph(case["scale"])
        s = abi.Solver(mesh, flow.bc_fields(), flow.settings)
        s.learned_init(abi.NET_BF16_WEIGHTS, seed=0)
        s.learned_set_params(_weights(len(levels), seed))
        b, t, ac, d, af = _pressure_system(mesh, seed)
        if kind == "predict":
            return dict(kind=kind, solver=s, args=(b, ac, d))
        s.learned_harvest(0, 1)
        s.learned_add_sample(b, t, ac, d, af)
        return dict(kind=kind, solver=s)
    flow, mesh, start = _flow_case(case, seed)
    bcs = None
    if isinstance(flow, tuple):
        flow, bcs = flow
    settings = _settings(case, flow)
    fcg = dict(pressure_solver=abi.PSOLVE_FCG, pressure_tol=1e-2, prolong_scale=2.0) if case.get("fcg") else {}
    s = abi.Solver(mesh, flow.bc_fields() if bcs is None else bcs, settings,
                   precision=abi.PREC_MIXED if case["precision"] == "mixed" else abi.PREC_FP64, **fcg)
    if start is not None:
        s.set_batch(start)
    if case.get("learned"):
        s.learned_init(abi.NET_BF16_WEIGHTS, seed=seed % 1000 + 1)
        s.learned_enable(abi.LEARNED_ALWAYS)
    names = ("u", "v", "p", "mDot") + (("T", "C") if case["geom"] == "scalars" else ())
    state = dict(kind=kind, solver=s,
                 out={k: _pinned(mesh["nFaces"] if k == "mDot" else mesh["nCells"]) for k in names})
    if kind == "continue":
        state["start"] = _initial_fields(mesh, settings, seed)
    return state


def run(state):
    kind = state["kind"]
    if kind == "residual":
        return _run_residual(state)
    s = state["solver"]
    if kind == "predict":
        return s.learned_predict(*state["args"])
    if kind == "grad":
        loss, grad = s.learned_grad(0)
        return dict(loss=np.float32(loss), grad=grad)
    if kind == "continue":
        for k, a in state["start"].items():
            s.set(k, a)
    r = s.solve(cont=kind == "continue")
    out = {k: s.get(k, out=a) for k, a in state["out"].items()}
    out["residual"] = np.array(r["residual"])
    out["iterations"] = r["iterations"]
    return out


def _prepare_residual(case, seed):
    """The momentum systems, fields and mass fluxes of a flow solver, held by
    the caller as torch tensors."""
    mesh = _blocks_mesh(("expansion", case["scale"], 0))
    n, f, slots = int(mesh["nCells"]), int(mesh["nFaces"]), len(mesh["cellFaceIDs"])
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def rand(m, lo, hi):
        return lo + (hi - lo) * torch.rand(m, dtype=torch.float64, device="cuda", generator=gen)

    dev = {k: torch.from_numpy(np.ascontiguousarray(mesh[k])).cuda()
           for k in ("cellFaceStart", "cellFaceIDs", "faceOwner", "faceNeighbor")}
    ids = dev["cellFaceIDs"].long()
    af = torch.where(dev["faceNeighbor"][ids] >= 0, rand(slots, -2e-6, -1e-7), torch.zeros((), dtype=torch.float64,
                                                                                           device="cuda"))
    ac = -af.reshape(n, -1).sum(1) / 0.7
    dev.update(AF=af, ACu=ac * rand(n, 1.0, 1.1), ACv=ac * rand(n, 1.1, 1.2), bu=rand(n, -1e-6, 1e-6),
               bv=rand(n, -1e-7, 1e-7), u=rand(n, -0.1, 1.0), v=rand(n, -0.05, 0.05), mDot=rand(f, -1e-6, 1e-6))
    out = {k: torch.empty(n, dtype=torch.float64, device="cuda") for k in ("resU", "resV", "resC")}
    out["sums"] = torch.empty(5, dtype=torch.float64, device="cuda")
    return dict(kind="residual", sizes=(n, f, slots), dev=dev, norm=case["norm"], out=out)


def _run_residual(st):
    dev, out = st["dev"], st["out"]
    err = ctypes.create_string_buffer(256)
    code = abi.lib().axisim_residual_static(
        *st["sizes"], *(dev[k].data_ptr() for k in ("cellFaceStart", "cellFaceIDs", "faceOwner", "faceNeighbor", "AF",
                                                    "ACu", "ACv", "bu", "bv", "u", "v", "mDot")),
        st["norm"], st["norm"], *(out[k].data_ptr() for k in ("resU", "resV", "resC", "sums")),
        torch.cuda.current_stream().cuda_stream, err, len(err))
    if code:
        raise RuntimeError(err.value.decode())
    return out


# ------------------------------------------------------------ what it takes
def work(case):
    kind = case["kind"]
    if kind == "residual":
        n, f = _sizes(case)
        return dict(bytes=4 * (n + 1) + 16 * n + 8 * f + 32 * n + 8 * (6 * n + f) + 24 * n + 40,
                    flops=n * (4 * 5 + 12))
    if kind in ("predict", "grad"):
        n = _sizes(case)[0]
        cells, depth = [n], 1
        while cells[-1] > 64:
            cells.append(max(1, cells[-1] // 4))
        _, total, order = _net_layers(len(cells))
        flops = sum(2 * cells[lv] * k * co for _, k, co, lv in order)
        graph = sum(4 * (4 + 1) * m for m in cells)
        if kind == "predict":
            return dict(bytes=16 * n + graph + 4 * total, flops=flops)
        return dict(bytes=16 * n + 16 * n + graph + 8 * total, flops=3 * flops)
    n, f = _sizes(case)
    w = 3 if case["geom"] == "bullet" else 4
    # per iteration: connectivity and geometry, the fields read and written
    # once, the momentum sweeps' and V-cycles' arithmetic on every cell
    its = case["iters"] * case.get("steps", 1)
    cycles = case.get("fcg") or 3
    byts = 8 * f + 8 * 8 * f + 4 * w * n + 8 * 6 * n + 2 * 8 * (3 * n + f)
    flops = n * (20 * 2 * (2 * w + 3) + cycles * 4 / 3 * 3 * (2 * w + 3) + 60 * w)
    if case["geom"] == "scalars":
        byts += 4 * 8 * n
        flops += n * (20 * 2 * (2 * w + 3) + 40 * w)
    return dict(bytes=float(its * byts), flops=float(its * flops))


def _sizes(case):
    """(cells, faces) of the case's mesh, by its band counts."""
    geom = case.get("geom", "expansion")
    if geom == "pipe":
        n, edge = case["nr"] * case["nz"], case["nr"] + case["nz"]
    elif geom == "bullet":
        n, edge = int(486_000 * case["scale"] ** 2), 0
        return n, n * 3 // 2
    elif geom == "batch":
        members = batch.random_cases(n=case["n"], seed=case["mix"], scale=case["size"])
        n, edge = sum(cases.cell_count(c) for c in members), 0
    else:
        n, edge = cases.cell_count(cases.expansion(scale=case["scale"])), int(4400 * case["scale"])
    return n, 2 * n + edge


# ------------------------------------------------------------ in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "residual":
        return _exact_residual(case, seed)
    if kind in ("predict", "grad"):
        return _exact_network(case, seed)
    return None  # a SIMPLE run rests on the whole method (aggregation order, sweeps): FP64 runs are their own oracle


def _exact_residual(case, seed):
    st = _prepare_residual(case, seed)
    n, f, slots = st["sizes"]
    d = st["dev"]
    ids = d["cellFaceIDs"].long().reshape(n, -1)
    own, nb = d["faceOwner"].long(), d["faceNeighbor"].long()
    me = torch.arange(n, device="cuda")
    out = {k: d["AC" + k] * d[k] for k in ("u", "v")}
    scale = {k: out[k].clone() for k in out}
    imb = torch.zeros(n, dtype=torch.float64, device="cuda")
    for j in range(ids.shape[1]):
        face = ids[:, j]
        mine = own[face] == me
        other = torch.where(mine, nb[face], own[face])
        inner = nb[face] >= 0
        for k in ("u", "v"):
            out[k] = out[k] + torch.where(inner, d["AF"].reshape(n, -1)[:, j] * d[k][other.clamp(min=0)], 0.0)
        imb = imb + torch.where(mine, d["mDot"][face], -d["mDot"][face])
    ru, rv = (d["b" + k] - out[k] for k in ("u", "v"))
    ru, rv = ru.abs(), rv.abs()
    stat = (lambda x: x.sum(), lambda x: (x * x).sum(), lambda x: x.max())[case["norm"]]
    sums = torch.stack([stat(ru), scale["u"].abs().sum(), stat(rv), scale["v"].abs().sum(), imb.abs().sum()])
    return dict(resU=ru, resV=rv, resC=imb, sums=sums)


def _exact_network(case, seed):
    """The network and its loss in 64 bits on the rounded weights (BF16
    weights are what the option computes with)."""
    mesh, levels = _graph(case["scale"])
    b, t, ac, d, af = _pressure_system(mesh, seed)
    dev = torch.device("cuda")
    p = torch.from_numpy(_weights(len(levels), seed)).to(dev).bfloat16().double().requires_grad_(case["kind"] == "grad")
    groups, _, _ = _net_layers(len(levels))

    def as_dev(x):
        return torch.from_numpy(np.ascontiguousarray(x).astype(np.int64)).to(dev)

    lv = []
    for n, r, c, c2c in levels:
        r, c = as_dev(r), as_dev(c)
        deg = torch.bincount(r, minlength=n).double().clamp(min=1)
        lv.append((n, r, c, deg, None if c2c is None else as_dev(c2c)))

    def dense(key, x):
        o, k, co = groups[key]
        return x @ p[o:o + k * co].reshape(k, co) + p[o + k * co:o + k * co + co]

    def mp(key, x, level):
        n, r, c, deg, _ = lv[level]
        mean = torch.zeros_like(x).index_add(0, r, x[c]) / deg[:, None]
        return torch.relu(dense(key, torch.cat([x, mean], 1)))

    b64, t64, ac64, d64 = (torch.from_numpy(x).to(dev).double() for x in (b, t, ac, d))
    q = b64 / ac64
    sigma = q.square().mean().sqrt()
    enc = [mp("enc0", torch.relu(dense("in", torch.stack([q / sigma, d64], 1))), 0)]
    for level in range(1, len(lv)):
        c2c, n = lv[level - 1][4], lv[level][0]
        cnt = torch.bincount(c2c, minlength=n).double().clamp(min=1)
        x = enc[-1]
        x = torch.zeros(n, x.shape[1], dtype=x.dtype, device=dev).index_add(0, c2c, x) / cnt[:, None]
        enc.append(mp("enc%d" % min(level, 3), torch.relu(dense("down%d" % min(level, 4), x)), level))
    x = mp("mid%d" % min(len(lv) - 1, 3), enc[-1], len(lv) - 1)
    for level in range(len(lv) - 2, -1, -1):
        x = torch.relu(dense("up%d" % min(level, 3), x[lv[level][4]]) + enc[level])
        x = mp("dec%d" % min(level, 3), x, level)
    y = dense("out", x)[:, 0]
    if case["kind"] == "predict":
        return (sigma * y).detach()
    n, r, c, slot = _level0(mesh)
    a = torch.from_numpy(af[slot]).to(dev).double()
    Ay = ac64 * y + torch.zeros_like(y).index_add(0, as_dev(r), a * y[as_dev(c)])
    loss = 1.0 - (y @ b64) ** 2 / ((y @ Ay) * (b64 @ t64))
    loss.backward()
    return dict(loss=loss.detach(), grad=p.grad)
