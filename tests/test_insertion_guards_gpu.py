"""What an insertion must keep whichever kernel GTOMRLN_PATH_AUTO takes: a
value that is not finite reaches the map, calls that overlap on two streams
lose nothing, sums of small weights beside large ones stay FP32 sums below the
sizes of the fixed-point path, and a call with volume indices on the device
does not wait for the stream there."""
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


@pytest.mark.parametrize("n,batch", [(64, 2500), (128, 450), (160, 300), (180, 200), (256, 150)])
def test_auto_sums_small_weights_in_fp32(gtom_lib, cuda, n, batch):
    """Weights of 1 but for a ring of 1e-5 (the neighbourhood of a CTF zero):
    every sum inside the ring, far from its rims, agrees with the direct
    kernel's.  Both add N positive FP32 terms, N below 64 there, in some
    order: (N - 1) 2^-24 each, 8e-6 together."""
    rng = np.random.default_rng(n + batch)
    e, V = O.elements_fft(n), 2 * n + 1
    y, x = np.meshgrid(np.fft.fftfreq(n) * n, np.arange(n // 2 + 1), indexing="ij")
    r = np.sqrt(x * x + y * y).reshape(-1)
    r0 = 0.3 * n
    w = torch.from_numpy(np.where(np.abs(r - r0) < 4, 1e-5, 1.0).astype(np.float32)).cuda().repeat(batch, 1)
    ft = torch.randn(batch, e, dtype=torch.complex64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    mats = _mats(rng, batch)
    got, want = (_insert(p, V, n, mats, ft, w)[1].double().cpu().numpy() for p in ("auto", "direct"))
    z, yy, xx = np.meshgrid(np.arange(V) - n, np.arange(V) - n, np.arange(V // 2 + 1), indexing="ij", sparse=True)
    ring = (np.abs(np.sqrt(xx * xx + yy * yy + z * z) - 2 * r0) < 5).reshape(-1)
    sel = ring & (want > 0)
    assert sel.sum() > 1000
    assert want[sel].max() <= 64 * 1e-5
    assert (np.abs(got - want)[sel] / want[sel]).max() <= 8e-6


@pytest.mark.parametrize("n,batch", [(100, 3333), (128, 500), (160, 250)])
def test_device_indices_do_not_wait(gtom_lib, cuda, n, batch):
    rng = np.random.default_rng(3)
    V = 2 * n + 1
    mats = _mats(rng, batch)
    ft = torch.ones(batch, O.elements_fft(n), dtype=torch.complex64, device="cuda")
    iv = torch.from_numpy(rng.integers(0, 2, batch).astype(np.int32)).cuda()
    _insert("auto", V, n, mats, ft, None, iv, 2)  # caches and modules in place
    nv = (V // 2 + 1) * V * V * 2
    vf, vw = torch.zeros(nv, dtype=torch.complex64, device="cuda"), torch.zeros(nv, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(400_000_000)  # ~0.2 s of the stream
    done = torch.cuda.Event()
    done.record()
    G.d_rlnBackproject(vf, vw, (V, V, V), ft.reshape(-1), None, (n, n, 1), n // 2, mats, iv, (1, 0, 0, 1), 0.0, False,
                       False, batch)
    waited = done.query()
    torch.cuda.synchronize()
    assert not waited
