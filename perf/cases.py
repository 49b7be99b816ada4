"""The work that the speed of this library is judged by.

Each case is one call (or the one call and what a caller has to do around it)
of a public entry point, at sizes between the smallest and the largest that
the repository's configurations, tests and benchmark use: boxes of 32 to 256
voxels at padding 2, batches of one hundred to ten thousand slices, ten
gridding iterations, uneven sub-tomogram batches, particle preprocessing and
the E-step's squared differences.  `draw` gives further cases of the same
ranges, odd and ragged sizes among them.

Inputs are made with torch and numpy from the seed alone: band-limited
particles with a falling spectrum, orientations uniform on SO(3) or around a
preferred view, CTF-weighted images of low signal-to-noise ratio.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gtom_b200 as G
from gtom_b200 import batch as GB
from gtom_b200 import ctf as GC
from gtom_b200 import estep as GE

PAD = 2
DEV = "cuda"
BOXES = (32, 48, 64, 96, 128)  # sub-tomogram boxes of the uneven batches


# ------------------------------------------------------------------- cases --
def listed() -> list[dict]:
    return [
        # initial-model scale: a thousand small projections of one reference,
        # matrices on the device (latency and L2 gathers)
        dict(name="project_small", op="project", box=64, slices=1000, angles=False, shifted=False),
        # an alignment step at a box that no tuning knows: host angles, the
        # phase shift and global weight of every particle applied
        dict(name="project_shifted_ragged", op="project", box=180, slices=2345, angles=True, shifted=True),
        # single-particle refinement: ten thousand projections at 256
        dict(name="project_large", op="project", box=256, slices=10000, angles=False, shifted=False),
        # the small configuration's insertion: unit weights
        dict(name="backproject_small", op="backproject", box=64, slices=1000, angles=False, ctf=False, volumes=1,
             general=False),
        # two half-maps at an odd box by host angles and volume indices, with
        # anisotropic magnification and Ewald curvature
        dict(name="backproject_general_ragged", op="backproject", box=100, slices=3333, angles=True, ctf=True,
             volumes=2, general=True),
        # single-particle refinement: ten thousand CTF-weighted insertions at 256
        dict(name="backproject_large", op="backproject", box=256, slices=10000, angles=False, ctf=True, volumes=1,
             general=False),
        # gridding reconstruction with the default ten iterations: the small
        # configuration (launches count), a usual box, and the large one
        dict(name="reconstruct_small", op="reconstruct", box=64, slices=1000, iterations=10),
        dict(name="reconstruct_mid", op="reconstruct", box=160, slices=1500, iterations=10),
        dict(name="reconstruct_large", op="reconstruct", box=256, slices=2000, iterations=10),
        # sub-tomogram averaging: tilt series of uneven boxes inserted and
        # reconstructed by one handle
        dict(name="batch_uneven", op="batch", volumes=64, tilts=41, iterations=10),
        # the step before insertion: real-space particles to CTF-weighted
        # spectra and weights
        dict(name="preprocess", op="preprocess", box=256, particles=2000),
        # the E-step's dense comparison of particles, references and shifts
        dict(name="squared_differences", op="diff2", box=128, particles=16, refs=600, shifts=49, cc=False),
    ]


def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, lo: int, hi: int) -> int:
    return 2 * int(round(_log_uniform(rng, lo, hi) / 2))


def draw(rng) -> dict:
    op = rng.choice(("project", "project", "backproject", "backproject", "reconstruct", "reconstruct", "batch",
                     "preprocess", "diff2"))
    if op == "project":
        return dict(op=op, box=_box(rng, 32, 256), slices=int(_log_uniform(rng, 100, 10000)),
                    angles=rng.random() < 0.5, shifted=rng.random() < 0.4)
    if op == "backproject":
        return dict(op=op, box=_box(rng, 32, 256), slices=int(_log_uniform(rng, 100, 10000)),
                    angles=rng.random() < 0.5, ctf=rng.random() < 0.7, volumes=rng.choice((1, 1, 2)),
                    general=rng.random() < 0.3)
    if op == "reconstruct":
        return dict(op=op, box=_box(rng, 32, 256), slices=int(_log_uniform(rng, 500, 2000)), iterations=10)
    if op == "batch":
        return dict(op=op, volumes=int(_log_uniform(rng, 8, 64)), tilts=rng.choice((31, 41, 61)), iterations=10)
    if op == "preprocess":
        return dict(op=op, box=_box(rng, 64, 256), particles=int(_log_uniform(rng, 100, 4000)))
    return dict(op=op, box=_box(rng, 48, 160), particles=int(_log_uniform(rng, 2, 32)),
                refs=int(_log_uniform(rng, 16, 600)), shifts=int(_log_uniform(rng, 9, 100)),
                cc=rng.random() < 0.3)


# ------------------------------------------------------------------ inputs --
def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _angles(seed: int, count: int) -> np.ndarray:
    """(count, 3) rot, tilt, psi in radians: half uniform on SO(3), half
    around one preferred view."""
    r = np.random.default_rng([int(seed), 11])
    tilt = np.arccos(r.uniform(-1, 1, count))
    near = r.random(count) < 0.5
    tilt[near] = np.clip(np.abs(r.normal(0.6, 0.35, int(near.sum()))), 0, np.pi)
    return np.stack([r.uniform(-np.pi, np.pi, count), tilt, r.uniform(-np.pi, np.pi, count)], 1).astype(np.float32)


def _matrices(angles: np.ndarray, scale: float, dtype) -> np.ndarray:
    """(count, 9): scale times the transposed ZYZ Euler matrix, column-major."""
    a, b, g = (angles[:, i].astype(dtype) for i in range(3))
    ca, sa, cb, sb, cg, sg = np.cos(a), np.sin(a), np.cos(b), np.sin(b), np.cos(g), np.sin(g)
    rows = [cg * cb * ca - sg * sa, cg * cb * sa + sg * ca, -cg * sb,
            -sg * cb * ca - cg * sa, -sg * cb * sa + cg * ca, sg * sb,
            sb * ca, sb * sa, cb]
    return (np.stack(rows, 1) * dtype(scale)).astype(dtype)


def _freq(n: int, dev=DEV):
    """Signed x (n/2+1) and y (n) frequencies of a half-complex n x n slice."""
    x = torch.arange(n // 2 + 1, device=dev)
    y = torch.arange(n, device=dev)
    return x, torch.where(y <= n // 2, y, y - n)


def _particle(n: int, gen) -> torch.Tensor:
    """n^3 real volume: noise with a spectrum falling like a molecule's,
    inside a soft sphere."""
    k = torch.fft.fftfreq(n, device=DEV)
    kx = torch.fft.rfftfreq(n, device=DEV)
    r2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kx[None, None, :] ** 2
    v = torch.fft.irfftn(torch.fft.rfftn(torch.randn((n, n, n), device=DEV, generator=gen))
                         * torch.exp(-20.0 * r2) / (0.02 + r2.sqrt()), s=(n, n, n))
    c = torch.arange(n, device=DEV, dtype=torch.float32) - n // 2
    rr = (c[:, None, None] ** 2 + c[None, :, None] ** 2 + c[None, None, :] ** 2).sqrt()
    return v * torch.sigmoid((0.4 * n - rr) / 1.5)


def _padded_ft(vol: torch.Tensor) -> torch.Tensor:
    """Decentred half-complex transform of the volume in its padded box."""
    n = vol.shape[0]
    P = PAD * n
    big = torch.zeros((P, P, P), device=DEV)
    o = P // 2 - n // 2
    big[o:o + n, o:o + n, o:o + n] = vol
    return torch.fft.rfftn(torch.fft.ifftshift(big)).to(torch.complex64).reshape(-1).contiguous()


def _ctf_values(n: int, count: int, seed: int) -> torch.Tensor:
    """(count, n (n/2+1)) CTFs: 300 kV, Cs 2.7 mm, 1 A/pixel, defocus 0.5-3 um."""
    r = np.random.default_rng([int(seed), 12])
    x, y = _freq(n)
    r2 = ((x[None, :] ** 2 + y[:, None] ** 2).float() / n ** 2).reshape(1, -1)
    lam = 12.2643247 / math.sqrt(3e5 * (1 + 3e5 * 0.978466e-6))
    df = torch.from_numpy(r.uniform(5e3, 3e4, (count, 1)).astype(np.float32)).to(DEV)
    return torch.sin(math.pi * lam * df * r2 - math.pi / 2 * 2.7e7 * lam ** 3 * r2 * r2 + 0.07)


def _images(n: int, count: int, gen) -> torch.Tensor:
    """count noisy particle images: a soft blob of random place and size in
    unit noise."""
    c = torch.arange(n, device=DEV, dtype=torch.float32)
    p = n / 2 + (torch.rand((count, 2), device=DEV, generator=gen) - 0.5) * n / 4
    s = n * (0.05 + 0.1 * torch.rand((count, 1, 1), device=DEV, generator=gen))
    d2 = (c[None, :, None] - p[:, 0, None, None]) ** 2 + (c[None, None, :] - p[:, 1, None, None]) ** 2
    img = torch.randn((count, n, n), device=DEV, generator=gen)
    return img.add_(torch.exp(d2.mul_(-0.5).div_(s * s)), alpha=0.5)


def _slices(case: dict, seed: int):
    """Slices to insert, (count, e) complex64, and their weights or None."""
    n, count, gen = case["box"], case["slices"], _gen(seed)
    e = n * (n // 2 + 1)
    ft = torch.empty((count, e), dtype=torch.complex64, device=DEV)
    w = torch.empty((count, e), device=DEV) if case["ctf"] else None
    for a in range(0, count, 1000):
        b = min(count, a + 1000)
        ft[a:b] = torch.fft.rfft2(_images(n, b - a, gen)).reshape(b - a, e)
        if w is not None:
            c = _ctf_values(n, b - a, seed + a)
            ft[a:b] *= c
            w[a:b] = c * c
    return ft, w


def _geometry(case: dict, seed: int):
    """Magnification (columns of the 2 x 2 matrix) and Ewald radius (pixels)."""
    if not case["general"]:
        return (1.0, 0.0, 0.0, 1.0), 0.0
    r = np.random.default_rng([int(seed), 13])
    m = [1 + r.uniform(-0.01, 0.01), r.uniform(-0.004, 0.004), r.uniform(-0.004, 0.004), 1 + r.uniform(-0.01, 0.01)]
    return tuple(float(np.float32(v)) for v in m), float(case["box"] * 100)


def _ivolume(case: dict, seed: int):
    if case["volumes"] == 1:
        return None
    return np.random.default_rng([int(seed), 14]).integers(0, case["volumes"], case["slices"]).astype(np.int32)


def _insert(vol, wts, D, ft, w, mats, n, mag=(1, 0, 0, 1), curve=0.0, ivol=None, half=True):
    """Trilinear insertion in 64 bits into centred accumulators (complex as
    two float64 columns) with plain torch: the weights rounded to binary16,
    neighbours with x < 0 mirrored, the x = 0 plane completed."""
    x, y = _freq(n)
    x, y = torch.meshgrid(x, y, indexing="xy")
    x, y = x.reshape(-1), y.reshape(-1)
    keep = ~((x == 0) & (y < 0))
    qx = mag[0] * x.double() + mag[2] * y.double()
    qy = mag[1] * x.double() + mag[3] * y.double()
    qz = curve * (x * x + y * y).double()
    keep &= torch.floor(qx * qx + qy * qy + qz * qz) < (n // 2) ** 2
    at = keep.nonzero().reshape(-1)
    q = torch.stack([qx[at], qy[at], qz[at]], 1)
    rl = D // 2 + 1
    flat = vol.view(-1)
    step = max(1, (3 << 20) // max(1, at.numel()))
    for a in range(0, mats.shape[0], step):
        m = mats[a:a + step].double().reshape(-1, 3, 3)  # columns first
        pos = torch.einsum("pc,bcr->bpr", q, m).reshape(-1, 3)
        v = torch.view_as_real(ft[a:a + step][:, at].reshape(-1)).double()
        pw = w[a:a + step][:, at].reshape(-1).double() if w is not None else torch.ones_like(v[:, 0])
        off = 0
        if ivol is not None:
            off = (ivol[a:a + step].long() * (rl * D * D)).repeat_interleave(at.numel())
        b0 = torch.floor(pos + torch.tensor([1e-5, 0, 0], device=DEV, dtype=torch.float64))
        f = pos - b0
        b0 = b0.long()
        g = (1 - f, f)

        def rnd(t):
            return t.half().double() if half else t

        for i in range(8):
            dx, dy, dz = i & 1, (i >> 1) & 1, i >> 2
            wt = rnd(g[dx][:, 0] * rnd(g[dy][:, 1] * g[dz][:, 2]))
            nx, ny, nz = b0[:, 0] + dx, b0[:, 1] + dy, b0[:, 2] + dz
            sgn = torch.where(nx < 0, -1, 1)
            for again in (False, True):
                s = sgn if not again else -torch.ones_like(sgn)
                tx, ty, tz = nx * s if not again else torch.zeros_like(nx), ny * s + D // 2, nz * s + D // 2
                ww = wt if not again else wt * ((nx == 0) & ((ny != 0) | (nz != 0))).double()
                # the clamps of the insertion (a negative coordinate counts as large)
                tx = torch.where((tx < 0) | (tx > D // 2), D // 2, tx)
                ty = torch.where((ty < 0) | (ty > D - 1), D - 1, ty)
                tz = torch.where((tz < 0) | (tz > D - 1), D - 1, tz)
                o = (tz * D + ty) * rl + tx + off
                sel = slice(None)
                if again:
                    sel = ww.nonzero().reshape(-1)
                    if sel.numel() == 0:
                        continue
                os, wws, ss = o[sel], ww[sel], s[sel]
                flat.index_add_(0, 2 * os, wws * v[sel, 0])
                flat.index_add_(0, 2 * os + 1, wws * v[sel, 1] * ss)
                wts.index_add_(0, os, wws * pw[sel])


def _accumulators(case: dict, seed: int):
    """Centred accumulators of an insertion of `slices` CTF-weighted slices."""
    n = case["box"]
    D = n * PAD + 1
    nv = (D // 2 + 1) * D * D
    vol = torch.zeros((nv, 2), dtype=torch.float64, device=DEV)
    wts = torch.zeros(nv, dtype=torch.float64, device=DEV)
    ft, w = _slices(dict(case, ctf=True), seed)
    mats = torch.from_numpy(_matrices(_angles(seed, case["slices"]), float(PAD), np.float32)).to(DEV)
    _insert(vol, wts, D, ft, w, mats, n, half=False)
    return torch.view_as_complex(vol.float().contiguous()), wts.float()


def _batch_boxes(case: dict) -> list[int]:
    """Boxes drawn uniformly, the same ones for every seed of a case."""
    r = np.random.default_rng([case["volumes"], 15])
    return [int(n) for n in r.choice(BOXES, case["volumes"])]


def _tilt_series(case: dict, seed: int) -> list[dict]:
    tilts = np.deg2rad(np.linspace(-60, 60, case["tilts"]))
    out = []
    for i, n in enumerate(_batch_boxes(case)):
        E = _matrices(_angles(seed + 7 * i + 1, 1), 1.0, np.float64)[0].reshape(3, 3)
        mats = np.empty((case["tilts"], 9), np.float32)
        for k, t in enumerate(tilts):
            c, s = math.cos(t), math.sin(t)
            mats[k] = (PAD * (np.array([[c, 0, -s], [0, 1, 0], [s, 0, c]]) @ E)).reshape(-1)
        ft, w = _slices(dict(box=n, slices=case["tilts"], ctf=True), seed + 1000 + i)
        out.append(dict(box=n, ft=ft, w=w, mats=torch.from_numpy(mats).to(DEV)))
    return out


def _ctf_params(case: dict, seed: int) -> np.ndarray:
    r = np.random.default_rng([int(seed), 16])
    b = case["particles"]
    p = np.zeros((b, 14), np.float32)
    p[:, 0], p[:, 3], p[:, 4], p[:, 8], p[:, 12] = 1e-10, 2.7e-3, 3e5, 0.07, 1.0
    p[:, 5] = -r.uniform(0.5e-6, 3e-6, b)
    p[:, 6] = r.uniform(0, np.pi, b)
    p[:, 7] = r.uniform(0, 0.1e-6, b)
    return p


def _estep(case: dict, seed: int) -> dict:
    """Particles, references, CTFs, shift phases and inverse noise spectra of
    whitened single-particle data."""
    n, gen = case["box"], _gen(seed)
    e = n * (n // 2 + 1)
    x, y = _freq(n)
    r2 = (x[None, :] ** 2 + y[:, None] ** 2).float().reshape(-1) / n ** 2
    amp = torch.exp(-10 * r2) / (0.05 + r2.sqrt())

    def cplx(count):
        return torch.view_as_complex(torch.randn((count, e, 2), device=DEV, generator=gen))

    refs = cplx(case["refs"]) * amp
    ctf = _ctf_values(n, case["particles"], seed).contiguous()
    sigma = 2.0 + 2.0 * torch.exp(-30 * r2)
    r = np.random.default_rng([int(seed), 17])
    pick = torch.from_numpy(r.integers(0, case["refs"], case["particles"])).to(DEV)
    part = refs[pick] * ctf + cplx(case["particles"]) * sigma
    sh = torch.from_numpy(r.uniform(-5, 5, (case["shifts"], 2)).astype(np.float32)).to(DEV)
    xx, yy = torch.meshgrid(x, y, indexing="xy")
    ph = -2 * math.pi / n * (sh[:, :1] * xx.reshape(1, -1) + sh[:, 1:] * yy.reshape(1, -1))
    return dict(refs=refs.contiguous(), ctf=ctf, part=part.contiguous(),
                shifts=torch.polar(torch.ones_like(ph), ph).contiguous(),
                minvsigma2=(0.5 / (sigma * sigma)).contiguous())


# ------------------------------------------------------------- the measured --
def prepare(case: dict, seed: int) -> dict:
    st = dict(case=case)
    op = case["op"]
    if op in ("project", "backproject"):
        n, count = case["box"], case["slices"]
        ang = _angles(seed, count)
        st["angles"] = ang.reshape(-1)
        st["mats"] = torch.from_numpy(_matrices(ang, float(PAD), np.float32)).to(DEV).reshape(-1)
        e = n * (n // 2 + 1)
    if op == "project":
        st["vol"] = _padded_ft(_particle(n, _gen(seed)))
        st["out"] = torch.empty(count * e, dtype=torch.complex64, device=DEV)
        if case["shifted"]:
            r = np.random.default_rng([int(seed), 18])
            st["shifts"] = r.uniform(-4, 4, (count, 3)).astype(np.float32)
            st["gw"] = r.uniform(0.5, 1.5, count).astype(np.float32)
            st["d_shifts"] = torch.from_numpy(st["shifts"] * np.float32(2 * np.pi / n)).to(DEV).reshape(-1)
            st["d_gw"] = torch.from_numpy(st["gw"]).to(DEV)
    elif op == "backproject":
        ft, w = _slices(case, seed)
        st["ft"], st["w"] = ft.reshape(-1), None if w is None else w.reshape(-1)
        D = n * PAD + 1
        nv = (D // 2 + 1) * D * D * case["volumes"]
        st["vf"] = torch.empty(nv, dtype=torch.complex64, device=DEV)
        st["vw"] = torch.empty(nv, device=DEV)
        st["mag"], st["ewald"] = _geometry(case, seed)
        st["ivol"] = _ivolume(case, seed)
        st["d_ivol"] = None if st["ivol"] is None else torch.from_numpy(st["ivol"]).to(DEV)
    elif op == "reconstruct":
        st["data"], st["weight"] = _accumulators(case, seed)
        st["out"] = torch.empty(case["box"] ** 3, device=DEV)
    elif op == "batch":
        st["subs"] = [GB.Subvolume(s["box"], s["ft"].reshape(-1), s["w"].reshape(-1), s["mats"].reshape(-1),
                                   torch.empty(s["box"] ** 3, device=DEV)) for s in _tilt_series(case, seed)]
        st["handle"] = GB.BatchReconstructor(st["subs"], PAD, case["iterations"])
    elif op == "preprocess":
        st["images"] = _images(case["box"], case["particles"], _gen(seed))
        st["params"] = GC.ctf_params(_ctf_params(case, seed))
    else:
        st.update(_estep(case, seed))
        st["out"] = torch.empty(case["particles"] * case["refs"] * case["shifts"], device=DEV)
    return st


def run(st: dict):
    case = st["case"]
    op = case["op"]
    if op == "project":
        n, count = case["box"], case["slices"]
        P = n * PAD
        if case["shifted"]:
            if case["angles"]:
                G.d_rlnProjectShifted(st["vol"], (P, P, P), st["out"], (n, n, 1), st["angles"], st["shifts"], st["gw"],
                                      float(PAD), count)
            else:
                G.d_rlnProjectShifted(st["vol"], (P, P, P), st["out"], (n, n, 1), n // 2, st["mats"], st["d_shifts"],
                                      st["d_gw"], count)
        elif case["angles"]:
            G.d_rlnProject(st["vol"], (P, P, P), st["out"], (n, n, 1), st["angles"], float(PAD), count)
        else:
            G.d_rlnProject(st["vol"], (P, P, P), st["out"], (n, n, 1), n // 2, st["mats"], count)
        return st["out"]
    if op == "backproject":
        n, count = case["box"], case["slices"]
        D = n * PAD + 1
        st["vf"].zero_()
        st["vw"].zero_()
        if case["angles"]:
            G.d_rlnBackproject(st["vf"], st["vw"], (D, D, D), st["ft"], st["w"], (n, n, 1), n // 2, st["angles"],
                               st["ivol"], st["mag"], st["ewald"], float(PAD), False, False, count)
        else:
            G.d_rlnBackproject(st["vf"], st["vw"], (D, D, D), st["ft"], st["w"], (n, n, 1), n // 2, st["mats"],
                               st["d_ivol"], st["mag"], st["ewald"] * PAD, False, False, count)
        return st["vf"], st["vw"]
    if op == "reconstruct":
        n = case["box"]
        D = n * PAD + 1
        G.d_ReconstructGridding(st["data"], st["weight"], st["out"], (n, n, n), (D, D, D), PAD, 0, 0,
                                case["iterations"])
        return st["out"]
    if op == "batch":
        st["handle"].run()
        return [s.out for s in st["subs"]]
    if op == "preprocess":
        return GC.preprocess_particles(st["images"], st["params"])
    n = case["box"]
    GE.d_rlnSquaredDifferences(st["part"], st["minvsigma2"], st["ctf"], (n, n, 1), case["particles"], st["shifts"],
                               case["shifts"], st["refs"], case["refs"], 8, st["out"], case["cc"])
    return st["out"]


# ---------------------------------------------------- what a case requires --
def _disk(n: int) -> float:
    """Samples of a slice inside rmax = n/2."""
    return math.pi * n * n / 8


def _gridding_flops(n: int, iterations: int) -> float:
    P = n * PAD
    return (2 * iterations + 1) * 2.5 * P ** 3 * math.log2(P ** 3) + iterations * 4 * P ** 3


def work(case: dict) -> dict:
    op = case["op"]
    if op == "project":
        n, s = case["box"], case["slices"]
        e = n * (n // 2 + 1)
        samples = _disk(n) * s
        # the sphere of the half volume that the samples touch, at most once
        vol = 8 * min(2 / 3 * math.pi * n ** 3, 8 * samples)
        return dict(bytes=vol + 8 * e * s + 36 * s, flops=samples * 60)
    if op == "backproject":
        n, s = case["box"], case["slices"]
        D = n * PAD + 1
        samples = _disk(n) * s
        return dict(bytes=samples * (12 if case["ctf"] else 8) + 12 * (D // 2 + 1) * D * D * case["volumes"] + 36 * s,
                    flops=samples * 90)
    if op == "reconstruct":
        n = case["box"]
        D = n * PAD + 1
        return dict(bytes=12 * (D // 2 + 1) * D * D + 4 * n ** 3, flops=_gridding_flops(n, case["iterations"]))
    if op == "batch":
        b = f = 0.0
        for n in _batch_boxes(case):
            b += _disk(n) * case["tilts"] * 12 + 4 * n ** 3
            f += _gridding_flops(n, case["iterations"]) + _disk(n) * case["tilts"] * 90
        return dict(bytes=b, flops=f)
    if op == "preprocess":
        n, p = case["box"], case["particles"]
        return dict(bytes=p * (4 * n * n + 12 * n * (n // 2 + 1)),
                    flops=p * (2.5 * n * n * math.log2(n * n) + 30 * n * (n // 2 + 1)))
    n = case["box"]
    e = n * (n // 2 + 1)
    p, r, s = case["particles"], case["refs"], case["shifts"]
    return dict(bytes=e * (12 * p + 8 * (r + s) + 4) + 4 * p * r * s, flops=8.0 * e * p * r * s)


def tolerance(case: dict):
    """About four times what two correct implementations at the same
    precision show against each other (or against 64 bits)."""
    op = case["op"]
    if op == "project":
        # FP32 positions of up to 256 voxels, the phase's fast sine on top
        return dict(rel=4e-6, max=1e-3)
    if op == "backproject":
        # binary16 weights: an ulp of a position can move a weight by 2^-11
        return dict(rel=2e-5, max=1e-2)
    if op == "reconstruct":
        return dict(rel=1e-5, max=1e-3)
    if op == "batch":
        # few tilts leave voxels whose weights nearly vanish: ten iterations
        # amplify the rounding of the sums there
        return dict(rel=1e-4, max=1e-2)
    if op == "preprocess":
        # the CTF's phase of up to hundreds of radians in FP32, fast sine
        return dict(rel=8e-5, max=1e-2)
    return dict(rel=5e-6, max=1e-4)


# ------------------------------------------------------------------- exact --
def _exact_project(case: dict, seed: int):
    n, count = case["box"], case["slices"]
    P, e = n * PAD, n * (n // 2 + 1)
    vol = _padded_ft(_particle(n, _gen(seed)))
    ang = _angles(seed, count)
    if case["angles"]:
        mats = torch.from_numpy(_matrices(ang, float(PAD), np.float64)).to(DEV)
    else:
        mats = torch.from_numpy(_matrices(ang, float(PAD), np.float32)).to(DEV).double()
    x, y = _freq(n)
    x, y = torch.meshgrid(x, y, indexing="xy")
    x, y = x.reshape(-1), y.reshape(-1)
    at = (x * x + y * y <= (n // 2) ** 2).nonzero().reshape(-1)
    q = torch.stack([x[at], y[at]], 1).double()
    if case["shifted"]:
        r = np.random.default_rng([int(seed), 18])
        sh = torch.from_numpy(r.uniform(-4, 4, (count, 3)).astype(np.float32)).to(DEV).double() * (2 * math.pi / n)
        gw = torch.from_numpy(r.uniform(0.5, 1.5, count).astype(np.float32)).to(DEV).double()
    out = torch.zeros((count, e), dtype=torch.complex64, device=DEV)
    rl, last = P // 2 + 1, vol.numel() - 1
    step = max(1, (3 << 20) // at.numel())
    for a in range(0, count, step):
        m = mats[a:a + step].reshape(-1, 3, 3)[:, :2]
        pos = torch.einsum("pc,bcr->bpr", q, m).reshape(-1, 3)
        flip = pos[:, 0] < -1e-5
        pos = torch.where(flip[:, None], -pos, pos)
        b0 = torch.floor(pos + torch.tensor([1e-5, 0, 0], device=DEV, dtype=torch.float64))
        f = pos - b0
        b0 = b0.long()
        v = torch.zeros(pos.shape[0], dtype=torch.complex128, device=DEV)
        for i in range(8):
            d = (i & 1, (i >> 1) & 1, i >> 2)
            w = torch.ones_like(f[:, 0])
            for k in range(3):
                w = w * (f[:, k] if d[k] else 1 - f[:, k])
            iy, iz = (b0[:, 1] + d[1]) % P, (b0[:, 2] + d[2]) % P
            o = (iz * P + iy) * rl + b0[:, 0] + d[0]
            v += w * vol[o.clamp(0, last)].to(torch.complex128)
        v = torch.where(flip, v.conj(), v).reshape(-1, at.numel())
        if case["shifted"]:
            ph = -(sh[a:a + step, :1] * q[None, :, 0] + sh[a:a + step, 1:2] * q[None, :, 1])
            v = v * torch.polar(gw[a:a + step, None].expand_as(ph), ph)
        out[a:a + step, at] = v.to(torch.complex64)
    return out.reshape(-1)


def _exact_backproject(case: dict, seed: int):
    n = case["box"]
    D = n * PAD + 1
    nv = (D // 2 + 1) * D * D * case["volumes"]
    ft, w = _slices(case, seed)
    mats = _matrices(_angles(seed, case["slices"]), float(PAD), np.float64 if case["angles"] else np.float32)
    mag, ewald = _geometry(case, seed)
    iv = _ivolume(case, seed)
    vol = torch.zeros((nv, 2), dtype=torch.float64, device=DEV)
    wts = torch.zeros(nv, dtype=torch.float64, device=DEV)
    _insert(vol, wts, D, ft, w, torch.from_numpy(mats).to(DEV), n, mag, 1 / (2 * ewald * PAD) if ewald else 0.0,
            None if iv is None else torch.from_numpy(iv).to(DEV))
    return torch.view_as_complex(vol), wts


def _kaiser_bessel_table(radius: float, alpha: float, count: int = 10000) -> np.ndarray:
    """The Fourier transform of the blob (order 0) at i 0.5 / count, over its
    value at 0: proportional to I_{3/2}(s) / s^{3/2}, s^2 = alpha^2 - (2 pi a w)^2
    (J_{3/2} beyond)."""
    t = 2 * np.pi * radius * np.arange(count) * 0.5 / count
    s = np.sqrt(np.abs(alpha * alpha - t * t))
    with np.errstate(all="ignore"):
        inside = (np.cosh(s) - np.sinh(s) / s) / (s * s)
        outside = (np.sin(s) / s - np.cos(s)) / (s * s)
    v = np.where(t > alpha, outside, inside)
    return v / v[0]


def _decentred(src: torch.Tensor, P: int, D: int) -> torch.Tensor:
    """The centred D box on the decentred P grid, inside the sphere P/2."""
    k = torch.arange(P, device=DEV)
    k = torch.where(k < P // 2 + 1, k, k - P)
    i = (k + D // 2).clamp(0, D - 1)
    x = torch.arange(P // 2 + 1, device=DEV)
    r2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + x[None, None, :] ** 2
    v = src.reshape(D, D, D // 2 + 1)[i[:, None, None], i[None, :, None], x[None, None, :]]
    return v * (r2 < P * P // 4), r2


def _exact_gridding(data: torch.Tensor, weight: torch.Tensor, n: int, iterations: int) -> torch.Tensor:
    """The gridding reconstruction in 64 bits with torch's transforms."""
    P, D = n * PAD, n * PAD + 1
    table = torch.from_numpy(_kaiser_bessel_table(1.9 * PAD, 15.0)).to(DEV)
    k = torch.arange(P, device=DEV)
    k = torch.where(k < P // 2, k, k - P).double()
    r = (k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2).sqrt() * (20000.0 / P)
    blob = table[(r + 1e-9).long().clamp(max=9999)]
    fw, r2 = _decentred(weight.double(), P, D)
    fn = (r2 < (n // 2 * PAD) ** 2).double()
    for _ in range(iterations):
        c = torch.fft.irfftn((fw * fn).to(torch.complex128), s=(P, P, P)).mul_(blob)
        fn = (fn / torch.fft.rfftn(c).real.clamp(min=1e-4)).clamp(max=1e20)
        del c
    d, _ = _decentred(data.to(torch.complex128), P, D)
    z = torch.arange(P, device=DEV)
    x = torch.arange(P // 2 + 1, device=DEV)
    sign = 1 - 2 * ((z[:, None, None] + z[None, :, None] + x[None, None, :]) & 1)
    v = torch.fft.irfftn(d * fn * sign, s=(P, P, P), norm="forward")
    o = P // 2 - n // 2
    v = v[o:o + n, o:o + n, o:o + n]
    c = torch.arange(n, device=DEV, dtype=torch.float64) - n // 2
    s = torch.sinc((c[:, None, None] ** 2 + c[None, :, None] ** 2 + c[None, None, :] ** 2).sqrt() / P)
    return (v / (s * s) / (PAD ** 3 * n)).reshape(-1)


def _exact_batch(case: dict, seed: int):
    out = []
    for s in _tilt_series(case, seed):
        n = s["box"]
        D = n * PAD + 1
        nv = (D // 2 + 1) * D * D
        vol = torch.zeros((nv, 2), dtype=torch.float64, device=DEV)
        wts = torch.zeros(nv, dtype=torch.float64, device=DEV)
        _insert(vol, wts, D, s["ft"], s["w"], s["mats"], n)
        out.append(_exact_gridding(torch.view_as_complex(vol), wts, n, case["iterations"]))
    return out


def _exact_preprocess(case: dict, seed: int):
    n, b = case["box"], case["particles"]
    img = _images(n, b, _gen(seed))
    p = torch.from_numpy(_ctf_params(case, seed)).to(DEV).double()
    x, y = _freq(n)
    xx, yy = torch.meshgrid(x, y, indexing="xy")
    r2 = (xx * xx + yy * yy).double()[None] / n ** 2
    ang = torch.atan2(yy.double(), xx.double())[None]
    sign = (1 - 2 * ((xx + yy) & 1))[None]
    ft = torch.empty((b, n, n // 2 + 1), dtype=torch.complex128, device=DEV)
    w = torch.empty((b, n, n // 2 + 1), dtype=torch.float64, device=DEV)
    for a in range(0, b, 200):
        q = p[a:a + 200, :, None, None]
        lam = 12.2643247 / torch.sqrt(q[:, 4] * (1 + q[:, 4] * 0.978466e-6))
        k2 = r2 / (q[:, 0] * 1e10) ** 2
        df = q[:, 5] * 1e10 + q[:, 7] * 0.5e10 * torch.cos(2 * (ang - q[:, 6]))
        g = math.pi * lam * df * k2 + math.pi / 2 * q[:, 3] * 1e10 * lam ** 3 * k2 * k2 - q[:, 13] \
            - torch.atan(q[:, 8] / torch.sqrt(1 - q[:, 8] ** 2))
        c = -torch.sin(g) * q[:, 12]
        ft[a:a + 200] = torch.fft.rfft2(img[a:a + 200].double()) * (c * sign)
        w[a:a + 200] = c * c
    return ft.reshape(-1), w.reshape(-1)


def _exact_diff2(case: dict, seed: int):
    s = {k: v.to(torch.complex128 if v.is_complex() else torch.float64) for k, v in _estep(case, seed).items()}
    sw = s["minvsigma2"].sqrt()
    out = torch.empty((case["particles"], case["refs"], case["shifts"]), dtype=torch.float64, device=DEV)
    for p in range(case["particles"]):
        a = s["refs"] * s["ctf"][p]
        b = s["part"][p] * s["shifts"]
        if case["cc"]:
            out[p] = -(a @ b.conj().T).real / (a.abs() ** 2).sum(1).sqrt()[:, None]
        else:
            a, b = a * sw, b * sw
            out[p] = 0.5 * ((a.abs() ** 2).sum(1)[:, None] + (b.abs() ** 2).sum(1)[None] - 2 * (a @ b.conj().T).real)
    return out.reshape(-1)


def exact(case: dict, seed: int):
    op = case["op"]
    if op == "project":
        return _exact_project(case, seed)
    if op == "backproject":
        return _exact_backproject(case, seed)
    if op == "reconstruct":
        return _exact_gridding(*_accumulators(case, seed), case["box"], case["iterations"])
    if op == "batch":
        return _exact_batch(case, seed)
    if op == "preprocess":
        return _exact_preprocess(case, seed)
    return _exact_diff2(case, seed)
