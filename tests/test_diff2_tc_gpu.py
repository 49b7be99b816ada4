"""The dense squared differences on the tensor cores (diff2_tc.cu) at the
edges of their tiles (128 references x 64 shifts, 16 elements a stage, four
stages an accumulator set, a range of elements per CTA), against float64.

Bound: FP32 operands carry 2^-24 each, the dropped lo lo products 2^-22 of
random sign, sums are combined in FP32 with a few 2^-24 per term of the
chain: 2e-6 of each output where nothing cancels (half of the operands' power
at least; closer matches take the direct kernel), and for the
cross-correlation 2e-6 of the operands' power."""
import numpy as np
import pytest
import torch

from gtom_b200.estep import d_rlnSquaredDifferences

pytestmark = pytest.mark.gpu


def _case(n, npart, nrefs, nshifts, seed=0, dev="cuda"):
    g = torch.Generator(device="cpu")
    g.manual_seed(seed + n)
    e = (n // 2 + 1) * n
    c = lambda k: torch.view_as_complex(torch.randn((k, e, 2), generator=g))
    part, refs = c(npart), c(nrefs)
    ph = torch.rand((nshifts, e), generator=g) * 6.2831853
    shifts = torch.polar(torch.ones_like(ph), ph)
    ctf = torch.rand((npart, e), generator=g) * 2 - 1
    w = torch.rand(e, generator=g) + 0.1
    return [t.contiguous() for t in (part, refs, shifts, ctf, w)]


def _expect(part, refs, shifts, ctf, w, cc):
    out = []
    for p in range(part.shape[0]):
        a = refs.to(torch.complex128) * (ctf[p].double() if ctf is not None else 1.0)
        b = part[p].to(torch.complex128) * shifts.to(torch.complex128)
        if cc:
            out.append(-(a @ b.conj().T).real / (a.abs() ** 2).sum(1).sqrt()[:, None])
        else:
            ww = w.double() if w is not None else torch.ones(a.shape[1], dtype=torch.float64)
            aw, bw = a * ww.sqrt(), b * ww.sqrt()
            out.append(0.5 * ((aw.abs() ** 2).sum(1)[:, None] + (bw.abs() ** 2).sum(1)[None]
                              - 2 * (aw @ bw.conj().T).real))
    return torch.stack(out).numpy()


def _run(part, refs, shifts, ctf, w, n, cc):
    d = lambda t: None if t is None else t.cuda()
    out = torch.full((part.shape[0] * refs.shape[0] * shifts.shape[0],), float("nan"), device="cuda")
    d_rlnSquaredDifferences(d(part), d(w), d(ctf), (n, n, 1), part.shape[0], d(shifts), shifts.shape[0], d(refs),
                            refs.shape[0], 4, out, cc)
    return out.cpu().numpy().reshape(part.shape[0], refs.shape[0], shifts.shape[0])


# 45: an odd element count (rows not 16-byte aligned), 31: 496 elements, the
# direct kernel's side of the line; 32: 544 elements
@pytest.mark.parametrize("n,npart,nrefs,nshifts", [(31, 1, 5, 3), (32, 1, 1, 1), (32, 2, 128, 64), (45, 3, 129, 65),
                                                   (64, 2, 127, 9), (96, 1, 300, 130), (128, 2, 40, 49)])
@pytest.mark.parametrize("cc", [False, True])
def test_tiles(gtom_lib, cuda, n, npart, nrefs, nshifts, cc):
    part, refs, shifts, ctf, w = _case(n, npart, nrefs, nshifts)
    got, want = _run(part, refs, shifts, ctf, w, n, cc), _expect(part, refs, shifts, ctf, w, cc)
    if cc:
        power = np.sqrt((part.abs().double() ** 2).sum(1).numpy())[:, None, None]
        assert np.abs(got - want).max() <= 2e-6 * power.max()
    else:
        assert (np.abs(got - want) / want).max() <= 2e-6


def test_without_ctf_and_weights(gtom_lib, cuda):
    part, refs, shifts, _, _ = _case(48, 1, 70, 20)
    got, want = _run(part, refs, shifts, None, None, 48, False), _expect(part, refs, shifts, None, None, False)
    assert (np.abs(got - want) / want).max() <= 2e-6


def test_not_finite_values_and_matches(gtom_lib, cuda):
    """An infinite reference value and a particle that equals a reference:
    their tiles are the direct kernel's, the others stay as they are."""
    part, refs, shifts, ctf, w = _case(64, 2, 200, 70)
    shifts[5] = 1.0
    part[1] = ctf[1] * refs[150]
    refs[3, 7] = complex(float("inf"), 0.0)
    got, want = _run(part, refs, shifts, ctf, w, 64, False), _expect(part, refs, shifts, ctf, w, False)
    assert np.all(np.isinf(got[:, 3]) & (got[:, 3] > 0))
    assert 0 <= got[1, 150, 5] <= 1e-9 * np.median(want[1, 10])
    want[1, 150, 5] = got[1, 150, 5]
    rows = np.arange(200) != 3
    assert (np.abs(got - want)[:, rows] / np.maximum(want[:, rows], 1e-30)).max() <= 5e-6


# 8320 x 80 and 33024 x 80: enough tiles that a CTA sums all elements itself
@pytest.mark.parametrize("n,npart", [(32, 1), (48, 1), (128, 80), (256, 80)])
@pytest.mark.parametrize("ratio", [0.97, 0.7, 0.55, 0.45, 0.27])
@pytest.mark.parametrize("cc", [False, True])
def test_no_less_precise_than_the_direct_kernel(gtom_lib, cuda, n, npart, ratio, cc):
    """Particles that match the references in part (squared differences of
    `ratio` times half of the operands' power): the rms error against 64 bits
    stays below the direct kernel's, which a captured call takes, or is the
    same where the tile is close enough to be the direct kernel's."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    e, nrefs, nshifts, rho = (n // 2 + 1) * n, 256, 8, 1 - ratio
    c = lambda k: torch.randn(k, e, dtype=torch.complex64, device="cuda", generator=gen)
    part = c(1)
    ctf = torch.rand(1, e, device="cuda", generator=gen) * 0.5 + 0.5
    w = torch.rand(e, device="cuda", generator=gen) + 0.1
    turn = torch.rand(1, e, device="cuda", generator=gen) * 6.2831853
    shifts = torch.polar(torch.ones(nshifts, e, device="cuda"), turn + torch.linspace(0, 0.1, nshifts, device="cuda")[:, None])
    refs = (rho * part * shifts[0] + (1 - rho ** 2) ** 0.5 * c(nrefs)) / ctf
    parts, ctfs = part.repeat(npart, 1), ctf.repeat(npart, 1)

    def run(out):
        d_rlnSquaredDifferences(parts, w, ctfs, (n, n, 1), npart, shifts, nshifts, refs, nrefs, 4, out, cc)

    got, direct = (torch.full((npart, nrefs, nshifts), float("nan"), device="cuda") for _ in range(2))
    run(got)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(direct)
    graph.replay()
    torch.cuda.synchronize()
    a, b = refs.to(torch.complex128) * ctf[0].double(), part[0].to(torch.complex128) * shifts.to(torch.complex128)
    if cc:
        want, scale = -(a @ b.conj().T).real / (a.abs() ** 2).sum(1).sqrt()[:, None], (b.abs() ** 2).sum(1).sqrt()[None]
    else:
        aw, bw = a * w.double().sqrt(), b * w.double().sqrt()
        want = 0.5 * ((aw.abs() ** 2).sum(1)[:, None] + (bw.abs() ** 2).sum(1)[None]) - (aw @ bw.conj().T).real
        scale = want
    err = [((x[-1].double() - want) / scale) for x in (got, direct)]
    rms = [float(x.pow(2).mean().sqrt()) for x in err]
    assert rms[0] <= rms[1]
    assert float(err[0].abs().max()) <= (2e-6 if npart == 1 or ratio >= 0.5 or cc else 2e-5)
