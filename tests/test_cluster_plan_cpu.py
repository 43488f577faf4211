"""The plan of the deep multigrid levels' cluster launch, built on the host without
a device: what each CTA of the kernel would read, on hierarchies whose coarsest
level is as large as a batch's merged one.
"""
import functools

import numpy as np
import pytest

import axisim.abi as abi
from axisim import batch, cases

OP_COARSEST = 5  # the coarsest level's sweeps, one row a thread
ROWS = ("rows", "row0", "live", "cells", "wide", "slot0", "slots", "nb", "so", "halo", "c2c", "ms", "ml", "value64",
        "value32")


def level_of(plan, cta, i):
    """A level's entry in the table of a CTA's packed topology."""
    t = plan["blob"][cta].view(np.int32)
    return dict(zip(ROWS, (int(v) for v in t[i * len(ROWS):(i + 1) * len(ROWS)])))


@functools.lru_cache(maxsize=None)
def _pipe(nr, nz):
    return abi.multiblock(cases.pipe(nr=nr, nz=nz, max_iter=1).blocks)


def pack(members):
    """A batch of `members`, (cases, radial cells, axial cells) each."""
    sizes = [(nr, nz) for n, nr, nz in members for _ in range(n)]
    groups = cases.pipe(nr=8, nz=40, max_iter=1).groups
    return batch.pack_union([_pipe(*s) for s in sizes], [groups] * len(sizes))[:2]


# rows of the merged deepest level -> the batch
BATCHES = {512: [(16, 8, 64)], 513: [(15, 8, 64), (1, 16, 32)], 768: [(24, 40, 200)], 1024: [(32, 8, 64)],
           1056: [(32, 16, 32)]}


@pytest.mark.parametrize("coarse", [1, 2, 30])
@pytest.mark.parametrize("rows", list(BATCHES))
def test_a_row_of_the_coarsest_level_has_a_thread(rows, coarse):
    mesh, start = pack(BATCHES[rows])
    cells, _ = abi.mg_batch_levels_host(mesh, start)
    assert cells[-1] == rows
    plan = abi.vcycle_cluster_host(mesh, start, coarse=coarse)
    assert plan["first"] + plan["count"] == len(cells)
    for op, level, *_ in plan["steps"]:
        n = int(cells[plan["first"] + level])
        assert op != OP_COARSEST or n <= plan["threads"], (n, plan["threads"])


def joint(sizes):
    """Independent cases in one mesh, without their ranges: they share one hierarchy, whose
    coarse cells have no neighbour once a case is down to one cell."""
    groups = cases.pipe(nr=8, nz=40, max_iter=1).groups
    return batch.pack_union([_pipe(*s) for s in sizes], [groups] * len(sizes))


# cases of 50 to 400 cells: whole 32-cell slices of isolated cells on the deeper levels
SMALL = [(5 + i % 4, 10 + 2 * (i % 20)) for i in range(100)]
# the same, ordered by size, so that the isolated cells lie together
SORTED = sorted(SMALL, key=lambda s: s[0] * s[1])


@pytest.mark.parametrize("make", [lambda: joint(SMALL), lambda: joint(SORTED), lambda: joint(SORTED[:33]),
                                  lambda: joint([(2, 4)] * 40 + [(40, 200)]), lambda: pack(BATCHES[513]),
                                  lambda: pack(BATCHES[1056]), lambda: (cases.bullet(scale=0.2, max_iter=1).mesh, None)],
                         ids=["small", "sorted", "few", "mixed", "batch513", "batch1056", "triangles"])
def test_every_reference_lies_in_its_array(make):
    mesh, start = make()[:2]
    is_batch = start is not None and len(start) - 1 in (16, 32)
    cells = abi.mg_batch_levels_host(mesh, start)[0] if is_batch else abi.mg_levels_host(mesh)
    plan = abi.vcycle_cluster_host(mesh, start if is_batch else None)
    if plan is None:
        return
    size = plan["blob"].shape[1]
    seen = [0] * plan["count"]
    for cta in range(plan["ctas"]):
        blob = plan["blob"][cta]
        for i in range(plan["count"]):
            level, r = plan["first"] + i, level_of(plan, cta, i)
            if r["rows"] == 0:
                continue
            seen[i] += r["rows"]
            take = lambda at, n, t: blob[at:at + n * np.dtype(t).itemsize].view(t)  # noqa: E731
            nb, halo = take(r["nb"], r["slots"], np.uint16), take(r["halo"], r["live"] - r["rows"], np.int32)
            assert r["nb"] + 2 * r["slots"] <= size and r["live"] < r["cells"]
            assert halo.size == 0 or (0 <= halo.min() and halo.max() < cells[level])
            n = np.arange(r["rows"])
            if r["wide"]:
                so = take(r["so"], (r["rows"] + 31) // 32, np.uint32)
                base, groups = (so & 0xFFFFFF)[n >> 5].astype(int) + (n & 31), (so >> 24)[n >> 5].astype(int)
            else:
                base, groups = (n & ~31) * 8 + (n & 31), np.ones(r["rows"], int)
            ends = base + 32 * (8 * groups - 1)
            assert groups.min() >= 1 and ends.max() < r["slots"], (cta, level)
            refs = np.concatenate([nb[(base + 32 * j)[8 * groups > j]] for j in range(8 * groups.max())])
            assert refs.max() < r["cells"]
            pad = (refs >= r["live"]) & (refs != r["cells"] - 1)
            assert not pad.any()
            if not is_batch:  # the neighbours themselves
                _, _, fs, fn = abi.mg_level_maps_host(mesh, level - 1)
                ids = np.concatenate([r["row0"] + np.arange(r["rows"]), halo])
                for k in range(r["rows"]):
                    mine = nb[base[k] + 32 * np.arange(8 * groups[k])]
                    want = fn[fs[r["row0"] + k]:fs[r["row0"] + k + 1]]
                    np.testing.assert_array_equal(ids[mine[mine < r["live"]]], want[want >= 0])
            if i + 1 < plan["count"]:
                c2c = take(r["c2c"], r["live"], np.int32)
                assert 0 <= c2c.min() and c2c.max() < cells[level + 1]
            if i > 0:
                ms = take(r["ms"], r["live"] + 1, np.int32)
                assert np.all(np.diff(ms) >= 0)
                ml = take(r["ml"], int(ms[-1]), np.int32)
                assert 0 <= ml.min() and ml.max() < cells[level - 1]
            for value, width in ((r["value64"], 8), (r["value32"], 4)):
                assert value % 16 == 0 and value + width * (4 * r["cells"] + r["slots"]) <= 220 * 1024
    assert seen == [int(c) for c in cells[plan["first"]:]]
