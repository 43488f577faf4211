"""axisim_residual_static after calls that overlapped in time, and after calls that
could not wait for their kernel (needs a B200): overlapping calls may give wrong
sums, but a later call on its own gives the right ones, its own status and no
count of another call's bad indices.
"""
import ctypes as C
import threading

import numpy as np
import pytest

from axisim import cases
import axisim.abi as abi

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

KEYS = ("cellFaceStart", "cellFaceIDs", "faceOwner", "faceNeighbor", "AF", "ACu", "ACv", "bu", "bv", "u", "v", "mDot")


class _Call:
    """One mesh's arrays and its own outputs and stream."""

    def __init__(self, nr, nz):
        m = abi.multiblock(cases.pipe(nr=nr, nz=nz).blocks)
        self.n, self.f, self.s = int(m["nCells"]), int(m["nFaces"]), len(m["cellFaceIDs"])
        rng = np.random.default_rng(self.n)
        d = {k: rng.standard_normal(self.n) for k in ("ACu", "ACv", "bu", "bv", "u", "v")}
        d.update(AF=rng.standard_normal(self.s), mDot=rng.standard_normal(self.f))
        d.update({k: np.ascontiguousarray(m[k]) for k in KEYS[:4]})
        self.dev = {k: torch.from_numpy(a).cuda() for k, a in d.items()}
        self.out = {k: torch.zeros(self.n, dtype=torch.float64, device="cuda") for k in ("resU", "resV", "resC")}
        self.out["sums"] = torch.zeros(5, dtype=torch.float64, device="cuda")
        self.stream = torch.cuda.Stream()

    def __call__(self, ids=None):
        err = C.create_string_buffer(256)
        dev = dict(self.dev, **({} if ids is None else {"cellFaceIDs": ids}))
        st = abi.lib().axisim_residual_static(
            self.n, self.f, self.s, *(dev[k].data_ptr() for k in KEYS), 0, 0,
            *(self.out[k].data_ptr() for k in ("resU", "resV", "resC", "sums")), self.stream.cuda_stream, err, len(err))
        return st, err.value.decode()

    def alone(self):
        self.out["sums"].fill_(float("nan"))
        torch.cuda.synchronize()
        st, msg = self()
        assert st == abi.OK, msg
        return self.out["sums"].cpu().numpy()


SIZES = [(15, 17), (64, 100), (256, 700), (300, 1000)]


def test_a_call_after_overlapping_ones_is_right():
    calls = [_Call(*s) for s in SIZES]
    torch.cuda.synchronize()
    want = [c.alone() for c in calls]
    bad = calls[1].dev["cellFaceIDs"].clone()
    bad[::7] = calls[1].f  # out of range: skipped, counted, reported to that call alone
    torch.cuda.synchronize()
    for _ in range(3):
        def work(i):
            for _ in range(150):
                calls[i](bad if i == 1 else None)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for c, w in zip(calls, want):
            for _ in range(3):
                np.testing.assert_array_equal(c.alone(), w)


def test_a_call_after_ones_that_could_not_wait_is_right():
    calls = [_Call(*s) for s in SIZES]
    torch.cuda.synchronize()
    want = [c.alone() for c in calls]
    x = torch.zeros(8, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    # a thread whose other stream is being captured may launch but not wait; its wait ends the capture
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=side):
            x.add_(1)
            for c in calls * 4:
                st, msg = c()
                assert st == abi.E_CUDA and "captur" in msg, (st, msg)
    torch.cuda.synchronize()
    for c, w in zip(calls, want):
        for _ in range(3):
            np.testing.assert_array_equal(c.alone(), w)
