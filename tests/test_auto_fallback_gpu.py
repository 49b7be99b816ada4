"""GTOMRLN_PATH_AUTO where the row-segment kernels' plan cannot be had: the
first call with a grid under stream capture, and a device without room for the
plan's scratch.  The direct kernels, which need neither, do the work."""
import numpy as np
import pytest
import torch

import gtom_b200 as G
from gtom_b200 import _lib
from oracle import oracle as O
from tests.helpers import rel_l2
from tests.synthdata import random_angles

pytestmark = pytest.mark.gpu

# sizes at which AUTO takes the segment kernels: projection, insertion in
# FP32 sums, insertion in fixed point
CASES = [("project", 128, 4500), ("insert", 160, 400), ("insert", 192, 300), ("shifted", 128, 450)]


class _Call:
    def __init__(self, op, n, batch):
        gen = torch.Generator(device="cuda").manual_seed(n + batch)
        rng = np.random.default_rng(n)
        V, e = (2 * n if op == "project" else 2 * n + 1), O.elements_fft(n)
        self.op, self.n, self.batch, self.V = op, n, batch, V
        self.mats = torch.from_numpy(G.matrices_from_angles(random_angles(rng, batch), 2.0)).cuda().reshape(-1)
        nv = (V // 2 + 1) * V * V
        slices = torch.randn(batch * e, dtype=torch.complex64, device="cuda", generator=gen)
        volume = torch.randn(nv, dtype=torch.complex64, device="cuda", generator=gen)
        self.ft, self.out = (slices, volume) if op != "project" else (volume, slices)
        self.shifts = torch.zeros(3 * batch, device="cuda")
        self.ones = torch.ones(batch, device="cuda")
        self.w = torch.zeros(nv, device="cuda")

    def run(self):
        n, V, b = self.n, self.V, self.batch
        if self.op == "project":
            G.d_rlnProject(self.ft, (V, V, V), self.out, (n, n, 1), n // 2, self.mats, b)
        elif self.op == "insert":
            G.d_rlnBackproject(self.out, self.w, (V, V, V), self.ft, None, (n, n, 1), n // 2, self.mats, None,
                               (1, 0, 0, 1), 0.0, False, False, b)
        else:
            G.d_rlnBackprojectShifted(self.out, self.w, (V, V, V), self.ft, None, (n, n, 1), n // 2, self.mats,
                                      self.shifts, self.ones, b)

    def direct(self):
        ops = ("project",) if self.op == "project" else ("backproject",)
        for o in ops:
            G.set_path(o, "direct")
        try:
            self.clear()
            self.run()
        finally:
            for o in ops:
                G.set_path(o, "auto")
        return self.out.clone(), self.w.clone()

    def clear(self):
        self.out.zero_()
        self.w.zero_()

    def same(self, want):
        if self.op == "project":
            return torch.equal(self.out, want[0])
        # FP32 sums in another order
        return (rel_l2(self.out.cpu().numpy(), want[0].cpu().numpy()) <= 1e-6 and
                rel_l2(self.w.cpu().numpy(), want[1].cpu().numpy()) <= 1e-6)


@pytest.mark.parametrize("op,n,batch", CASES)
def test_first_call_can_be_captured(gtom_lib, cuda, op, n, batch):
    c = _Call(op, n, batch)
    want = c.direct()
    torch.cuda.synchronize()
    _lib.call("gtomrln_release_caches")  # no grid is known
    c.clear()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c.run()
    c.clear()
    graph.replay()
    torch.cuda.synchronize()
    assert c.same(want)


@pytest.mark.parametrize("op,n,batch", CASES)
def test_without_room_for_the_plan(gtom_lib, cuda, op, n, batch):
    c = _Call(op, n, batch)
    want = c.direct()
    c.clear()
    torch.cuda.synchronize()
    _lib.call("gtomrln_release_caches")
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(max(0, free - (40 << 20)), dtype=torch.uint8, device="cuda")
    try:
        c.run()
        torch.cuda.synchronize()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert c.same(want)
