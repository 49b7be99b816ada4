"""What an insertion must keep whichever kernel takes it: a value that is not
finite reaches the map, and calls that overlap on two streams lose nothing."""
import numpy as np
import pytest
import torch

import gtom_b200 as G
from oracle import oracle as O
from tests.synthdata import random_angles

pytestmark = pytest.mark.gpu


def _insert(path, V, n, mats, ft, w, ivol=None, volumes=1, batch=None):
    nv = (V // 2 + 1) * V * V * volumes
    vf = torch.zeros(nv, dtype=torch.complex64, device="cuda")
    vw = torch.zeros(nv, device="cuda")
    G.set_path("backproject", path)
    try:
        G.d_rlnBackproject(vf, vw, (V, V, V), ft.reshape(-1), None if w is None else w.reshape(-1), (n, n, 1), n // 2,
                           mats, ivol, (1, 0, 0, 1), 0.0, False, False, ft.shape[0])
    finally:
        G.set_path("backproject", "auto")
    return vf, vw


def _mats(rng, batch):
    return torch.from_numpy(G.matrices_from_angles(random_angles(rng, batch), 2.0)).cuda().reshape(-1)


@pytest.mark.parametrize("n", [64, 128, 256])
@pytest.mark.parametrize("where", ["real", "imaginary", "weight"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_not_finite_pixel_reaches_the_map(gtom_lib, cuda, n, where, value):
    """One pixel in the whole batch, which the magnitude sample of the
    fixed-point sums all but surely misses: the voxels it touches are not
    finite, the same ones as by the direct kernel's FP32 reductions."""
    rng = np.random.default_rng(n)
    batch, e, V = 400, O.elements_fft(n), 2 * n + 1
    mats = _mats(rng, batch)
    gen = torch.Generator(device="cuda").manual_seed(n)
    ft = torch.randn(batch, e, dtype=torch.complex64, device="cuda", generator=gen)
    w = torch.rand(batch, e, device="cuda", generator=gen) + 0.5
    at = (n // 5) * (n // 2 + 1) + n // 7  # row v = n/5, column u = n/7
    if where == "weight":
        w[211, at] = value
    else:
        torch.view_as_real(ft)[211, at, 0 if where == "real" else 1] = value
    bad = []
    for path in ("segment", "direct"):
        vf, vw = _insert(path, V, n, mats, ft, w)
        bad.append(torch.stack([~torch.isfinite(vf.real), ~torch.isfinite(vf.imag), ~torch.isfinite(vw)]))
    assert bad[1].any() and torch.equal(bad[0], bad[1])


@pytest.mark.parametrize("path", ["brick", "segment", "segment_fp32"])
@pytest.mark.parametrize("decentered", [False, True])
def test_overlapping_calls_lose_nothing(gtom_lib, cuda, path, decentered):
    """Twenty insertions on two streams into one pair of volumes: an addition
    lost to the other stream would miss a twentieth of its voxel."""
    rng = np.random.default_rng(8)
    n, batch, calls = 32, 300, 10
    V = 2 * n if decentered else 2 * n + 1
    nv = (V // 2 + 1) * V * V
    mats = _mats(rng, batch)
    ft = torch.ones(batch * O.elements_fft(n), dtype=torch.complex64, device="cuda")

    def insert(vf, vw):
        G.d_rlnBackproject(vf, vw, (V, V, V), ft, None, (n, n, 1), n // 2, mats, None, (1, 0, 0, 1), 0.0, decentered,
                           False, batch)

    new = lambda: (torch.zeros(nv, dtype=torch.complex64, device="cuda"), torch.zeros(nv, device="cuda"))
    one, both = new(), new()
    G.set_path("backproject", path)
    try:
        insert(*one)
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        for _ in range(calls):
            for s in streams:
                with torch.cuda.stream(s):
                    insert(*both)
        torch.cuda.synchronize()
    finally:
        G.set_path("backproject", "auto")
    want = 2 * calls * one[1].double()
    assert ((both[1].double() - want).abs() <= 1e-4 * want).all()
