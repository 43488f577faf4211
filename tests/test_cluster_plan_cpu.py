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
