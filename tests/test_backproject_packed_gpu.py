"""The direct backprojector through its packed scratch (one 16-byte reduction
per target) against the same slices inserted in calls too small for it, which
reduce into the volumes themselves, and against the oracle's FP32 port.  The
forms differ only in the order of the FP32 sums: 1e-6 (the bar of the
segment path's two accumulations), and the port's 1e-5."""
import numpy as np
import pytest
import torch

import gtom_b200 as G
from oracle import oracle as O
from tests.helpers import rel_l2
from tests.synthdata import random_angles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,decentered,square,volumes", [(16, 4000, False, False, 1), (33, 1100, False, False, 1),
                                                               (32, 1300, True, False, 1), (32, 1300, False, True, 1),
                                                               (24, 2500, False, False, 3)])
def test_packed_equals_plain(gtom_lib, cuda, n, batch, decentered, square, volumes):
    rng = np.random.default_rng(n + batch)
    V = 2 * n if decentered else 2 * n + 1
    e, nvox = O.elements_fft(n), (V // 2 + 1) * V * V
    ang = random_angles(rng, batch)
    iv = None if volumes == 1 else rng.integers(-1, volumes, batch).astype(np.int32)  # -1: skipped
    ft = torch.from_numpy((rng.normal(size=(batch, e)) + 1j * rng.normal(size=(batch, e))).astype(np.complex64)).cuda()
    w = torch.from_numpy(rng.uniform(0.1, 1.0, (batch, e)).astype(np.float32)).cuda()
    out = []
    for parts in (1, 8):
        vf = torch.ones(volumes * nvox, dtype=torch.complex64, device="cuda")
        vw = torch.ones(volumes * nvox, device="cuda")
        for a in np.array_split(np.arange(batch), parts):
            s = slice(int(a[0]), int(a[-1]) + 1)
            G.d_rlnBackproject(vf, vw, (V, V, V), ft[s].reshape(-1), w[s].reshape(-1), (n, n, 1), n // 2,
                               ang[s].reshape(-1), None if iv is None else iv[s], (1.01, 0.0, 0.0, 0.99), 0.0, 2.0,
                               decentered, square, len(a))
        out.append((vf.cpu().numpy(), vw.cpu().numpy()))
    for a, b in zip(*out):
        assert rel_l2(a, b) <= 1e-6
        assert np.array_equal(a == 1, b == 1)  # voxels that receive nothing are left alone


def test_packed_matches_the_port(gtom_lib, cuda):
    rng = np.random.default_rng(5)
    n, batch, V = 32, 1500, 65
    e, nvox = O.elements_fft(n), (V // 2 + 1) * V * V
    mats = O.matrices_f64(random_angles(rng, batch), 2.0).astype(np.float32)
    ft = (rng.normal(size=(batch, e)) + 1j * rng.normal(size=(batch, e))).astype(np.complex64)
    vf = torch.zeros(nvox, dtype=torch.complex64, device="cuda")
    vw = torch.zeros(nvox, device="cuda")
    G.d_rlnBackproject(vf, vw, (V, V, V), torch.from_numpy(ft).cuda().reshape(-1), None, (n, n, 1), n // 2,
                       torch.from_numpy(mats).cuda().reshape(-1), None, (1, 0, 0, 1), 0.0, False, False, batch)
    of, ow = np.zeros(nvox, np.complex64), np.zeros(nvox, np.float32)
    O.backproject(of, ow, V, ft, None, n, n // 2, mats, decentered=False, fp32=True)
    assert rel_l2(vf.cpu().numpy(), of) <= 1e-5 and rel_l2(vw.cpu().numpy(), ow) <= 1e-5


def test_overlapping_calls_lose_nothing(gtom_lib, cuda):
    """Forty packed insertions on two streams into one pair of volumes: each
    voxel holds all of them.  An addition lost to the other stream would miss
    one call's share (a fortieth) of its voxel; the order of forty FP32 sums
    makes 40 * 2^-24."""
    rng = np.random.default_rng(8)
    n, batch, V, calls = 32, 1300, 65, 20
    e, nvox = O.elements_fft(n), (V // 2 + 1) * V * V
    mats = torch.from_numpy(G.matrices_from_angles(random_angles(rng, batch), 2.0)).cuda().reshape(-1)
    ft = torch.ones(batch * e, dtype=torch.complex64, device="cuda")

    def insert(vf, vw):
        G.d_rlnBackproject(vf, vw, (V, V, V), ft, None, (n, n, 1), n // 2, mats, None, (1, 0, 0, 1), 0.0, False, False,
                           batch)

    new = lambda: (torch.zeros(nvox, dtype=torch.complex64, device="cuda"), torch.zeros(nvox, device="cuda"))
    one, both = new(), new()
    insert(*one)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(calls):
        for s in streams:
            with torch.cuda.stream(s):
                insert(*both)
    torch.cuda.synchronize()
    want = 2 * calls * one[1].double()
    assert ((both[1].double() - want).abs() <= 1e-5 * want).all()
    assert rel_l2(both[0].cpu().numpy(), (2 * calls * one[0]).cpu().numpy()) <= 1e-5
