"""The gridding iteration on grids without compiled transforms
(gtom_b200/csrc/gridgen.cu: the same passes as gridsym.cu with run-time
lengths) against the cuFFT path and the FP64 oracle: radices 2 to 16 with the
primes up to 13, odd half lengths, tiles of 16 columns and rows with a
remainder, the smallest grid.  The bars are
tests/test_gridsym_gpu.py's: the paths differ only in how the FP32
transforms round."""
import numpy as np
import pytest
import torch

import gtom_b200 as G
from gtom_b200 import _lib
from gtom_b200 import batch as GB
from oracle import oracle as O
from tests.helpers import rel_l2
from tests.test_gridsym_gpu import _dev, _inputs, _on

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ori,pad", [(8, 2), (20, 2), (24, 3), (25, 2), (26, 2), (33, 2), (49, 2), (65, 2), (80, 2),
                                     (110, 2), (143, 2), (160, 2)])
def test_maps_match_cufft(gtom_lib, cuda, ori, pad):
    data, w, D = _inputs(ori, pad)
    d_data, d_w = _dev(data), _dev(w)
    maps = {}
    for path in ("direct", "symmetric"):
        out = torch.full((ori ** 3,), float("nan"), device="cuda")
        _on(path, lambda: G.d_ReconstructGridding(d_data, d_w, out, (ori,) * 3, (D,) * 3, pad, 0, 0, 10))
        maps[path] = out.cpu().numpy()
    assert rel_l2(maps["symmetric"], maps["direct"]) <= 1e-5


@pytest.mark.parametrize("grid", [160, 288, 320, 384, 576, 768])
def test_compiled_lengths_match_cufft(gtom_lib, cuda, grid):
    """gridsym.cu's lengths of 12, 40 and 48 elements a thread."""
    ori, D = grid // 2, grid + 1
    gen = torch.Generator(device="cuda").manual_seed(grid)
    w = torch.rand(D, D, D // 2 + 1, device="cuda", generator=gen) + 0.5
    data = torch.randn(D, D, D // 2 + 1, dtype=torch.complex64, device="cuda", generator=gen)
    w[:, :, 0] = 0.5 * (w[:, :, 0] + w[:, :, 0].flip(0, 1))
    data[:, :, 0] = 0.5 * (data[:, :, 0] + data[:, :, 0].flip(0, 1).conj())
    maps = {}
    for path in ("direct", "symmetric"):
        out = torch.full((ori ** 3,), float("nan"), device="cuda")
        _on(path, lambda: G.d_ReconstructGridding(data.reshape(-1), w.reshape(-1), out, (ori,) * 3, (D,) * 3, 2, 0, 0, 3))
        maps[path] = out.cpu().numpy()
    assert rel_l2(maps["symmetric"], maps["direct"]) <= 1e-5


@pytest.mark.parametrize("ori,iterations", [(8, 3), (20, 10), (33, 2), (39, 2), (45, 0)])
def test_maps_match_oracle(gtom_lib, cuda, ori, iterations):
    data, w, D = _inputs(ori, seed=2, hermitian=False)
    out = torch.zeros(ori ** 3, device="cuda")
    G.d_ReconstructGridding(_dev(data), _dev(w), out, (ori,) * 3, (D,) * 3, 2, 0, 0, iterations)
    ref = O.reconstruct_gridding(data, w, ori, (D, D, D), 2, iterations=iterations)
    assert rel_l2(out.cpu().numpy().reshape(ori, ori, ori), ref) <= 1e-4


@pytest.mark.parametrize("momentum", [0.0, 0.9])
def test_weights_change_and_distance_match_cufft(gtom_lib, cuda, momentum):
    """The update with and without momentum, its convergence sums and the
    distance to reference weights, at a grid of 5 and 11."""
    ori = 55
    _, w, D = _inputs(ori, seed=4)
    d_w = _dev(w)
    ref = _on("direct", lambda: G.gridding_weights(d_w, (D,) * 3, ori, 2, 40, 0.0))[0]
    got = {p: _on(p, lambda: G.gridding_weights(d_w, (D,) * 3, ori, 2, 4, 1e-12, momentum, ref_fnw=ref,
                                                return_distance=True)) for p in ("direct", "symmetric")}
    a, b = got["symmetric"], got["direct"]
    assert rel_l2(a[0].cpu().numpy(), b[0].cpu().numpy()) <= 5e-6
    assert a[2] == b[2] and a[3] == pytest.approx(b[3], rel=1e-4) and a[5] == pytest.approx(b[5], rel=1e-4)


def test_batch_matches_single_calls(gtom_lib, cuda):
    """Stacks of volumes (blockIdx.y) of two such boxes in one handle."""
    rng = np.random.default_rng(9)
    subs = []
    for box in (40, 44, 40):
        e = (box // 2 + 1) * box
        ang = rng.uniform(-3, 3, (6, 3)).astype(np.float32)
        mats = torch.from_numpy(G.matrices_from_angles(ang, 2.0)).cuda().reshape(-1)
        ft = torch.from_numpy((rng.normal(size=6 * e) + 1j * rng.normal(size=6 * e)).astype(np.complex64)).cuda()
        w = torch.from_numpy(rng.uniform(0.5, 1.5, 6 * e).astype(np.float32)).cuda()
        subs.append(GB.Subvolume(box, ft, w, mats, torch.zeros(box ** 3, device="cuda")))
    rec = GB.BatchReconstructor(subs, 2, 3)
    rec.run()
    torch.cuda.synchronize()
    got = [s.out.clone() for s in subs]
    rec.close()
    GB.reconstruct_separately(subs, 2, 3)
    torch.cuda.synchronize()
    for g, s in zip(got, subs):
        assert rel_l2(g.cpu().numpy(), s.out.cpu().numpy()) <= 1e-4


@pytest.mark.parametrize("iterations", [0, 3])
@pytest.mark.parametrize("ori", [20, 32])
@pytest.mark.parametrize("at", ["corner", "column", "nyquist", "inside"])
def test_data_that_are_not_finite_spread(gtom_lib, cuda, ori, at, iterations):
    """Zero times a NaN is not zero: the map is NaN on every path, also for
    data outside the sphere, whose columns the symmetric passes leave out, and
    also where no iteration lies between the start and the final map."""
    data, w, D = _inputs(ori)
    data = data.reshape(D, D, D // 2 + 1).copy()
    c = D // 2
    data[{"corner": (1, 1, 0), "column": (c, 1, D // 2 - 1), "nyquist": (c, c, D // 2),
          "inside": (c, c + 2, 1)}[at]] = complex(np.nan, np.nan)
    for path in ("direct", "symmetric"):
        out = torch.zeros(ori ** 3, device="cuda")
        _on(path, lambda: G.d_ReconstructGridding(_dev(data.reshape(-1)), _dev(w), out, (ori,) * 3, (D,) * 3, 2, 0, 0,
                                                  iterations))
        assert not torch.isfinite(out).any()


@pytest.mark.parametrize("ori", [44, 160])
def test_captured_call_before_the_tables(gtom_lib, cuda, ori):
    """A captured call with cuFFT's plans at hand, on a grid the symmetric path
    has not seen: its twiddle table cannot be made there, so the plans do the
    work."""
    data, w, D = _inputs(ori)
    d_data, d_w, out = _dev(data), _dev(w), torch.zeros(ori ** 3, device="cuda")
    run = lambda: G.d_ReconstructGridding(d_data, d_w, out, (ori,) * 3, (D,) * 3, 2, 0, 0, 3)
    torch.cuda.synchronize()
    _lib.call("gtomrln_release_caches")
    _on("direct", run)
    want = out.clone()
    out.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    graph.replay()
    torch.cuda.synchronize()
    assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) <= 1e-6
