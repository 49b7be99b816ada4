"""The segment projector's records, dealt by rows and pixels, against the
direct kernel, bit for bit, at the sizes where the dealing can go wrong: fewer
records than a chunk, one row, a disk inside one brick, non-finite third
columns (which the records leave out)."""
import numpy as np
import pytest
import torch

import gtom_b200 as G
from tests.synthdata import random_angles

pytestmark = pytest.mark.gpu


def _volume(rng, P):
    n = (P // 2 + 1) * P * P
    return torch.from_numpy((rng.normal(size=n) + 1j * rng.normal(size=n)).astype(np.complex64)).cuda()


def _project(vol, P, n, rmax, mats, path):
    out = torch.full((mats.shape[0] * (n // 2 + 1) * n,), float("nan"), dtype=torch.complex64, device="cuda")
    G.set_path("project", path)
    try:
        G.d_rlnProject(vol, (P, P, P), out, (n, n, 1), rmax, torch.from_numpy(mats).cuda().reshape(-1), mats.shape[0])
        torch.cuda.synchronize()
    finally:
        G.set_path("project", "auto")
    return out.cpu().numpy()


@pytest.mark.parametrize("n,P,rmax,batch", [(16, 32, 8, 1), (16, 32, 0, 3), (16, 32, 1, 9), (64, 128, 32, 7),
                                            (40, 60, 20, 33), (17, 34, 8, 100)])
def test_segment_dealing(gtom_lib, cuda, n, P, rmax, batch):
    rng = np.random.default_rng(n + batch)
    mats = G.matrices_from_angles(random_angles(rng, batch), P / n)
    vol = _volume(rng, P)
    np.testing.assert_array_equal(_project(vol, P, n, rmax, mats, "segment"),
                                  _project(vol, P, n, rmax, mats, "direct"))


def test_segment_not_finite_third_column(gtom_lib, cuda):
    rng = np.random.default_rng(3)
    mats = G.matrices_from_angles(random_angles(rng, 12), 2.0)
    mats[2, 6], mats[5, 8] = np.inf, np.nan
    vol = _volume(rng, 64)
    a, b = _project(vol, 64, 32, 16, mats, "segment"), _project(vol, 64, 32, 16, mats, "direct")
    np.testing.assert_array_equal(a, b)
    assert np.isfinite(a[:2 * 17 * 32]).all()
