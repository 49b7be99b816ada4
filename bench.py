#!/usr/bin/env python
"""Benchmark: RELION-style project + backproject throughput at 256^3.

Workload (single-particle scale): a 256^3 FP32 volume of 2,000 Gaussian
blobs, padding 2 (decentred complex64 half volume 257 x 512 x 512), and a
pool of 256 x 256 particles with orientations from a 3-lobe von Mises-Fisher
mixture (kappa 5-40) plus 30 % uniform, a CTF each (300 kV, Cs 2.7 mm,
1 A/px, defocus 0.5-3 um, astigmatism <= 0.1 um) and white noise at SNR
0.05.  All data are synthetic (seeded) and generated on the GPU before the
timed region.

One step = one batch of B particles through the hot path: d_rlnProject of
the B reference slices (h_angles/matrix overload, rmax 128) and
d_rlnBackproject of the B CTF-weighted particles and their CTF^2 weights
into the centred 257 x 513 x 513 accumulators.  `value` is slices per second
(one slice = one projection + one insertion) over the whole job.  After the
timed steps the 10-iteration gridding reconstruction of the accumulated
volume (P = 512) is timed once and reported under "gridding", with the
reconstructions to a relative change of 1e-4 from the reference's start and
update, with momentum, and from the learned warm start ("to_1e-4",
"warm_vs_plain_1e-4"), the same to within 1e-4 (weighted relative L2) of the
converged weights ("to_converged_1e-4", "warm_vs_plain_converged"), and the
learned-warm-start workload at 128^3 on two held-out orientation
distributions ("warm_start_128").

`e2e` is the metric through the public API with host buffers (CTF-weighted
spectra and weights in, projections out); `e2e_from_particles` the same from
real-space particle images and CTF parameters, with the library's particle
preprocessing on the GPU (N = 1).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--batch B]
    python bench.py --impl reference ...   # the reference's CPU path (port)
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

BOX = 256
PAD = 2
SEED = 1002


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--batch", type=int, default=10000, help="particles per step")
    ap.add_argument("--pool", type=int, default=40000, help="distinct particles resident on the GPU")
    ap.add_argument("--e2e-batch", type=int, default=2000)
    ap.add_argument("--path", default="auto", choices=["auto", "direct", "brick", "segment"],
                    help="implementation of the projector and backprojector (gtomrln_set_path)")
    ap.add_argument("--sweep", action="store_true",
                    help="instead of the bench: run the autotuner over brick edge x threads x pairs per "
                         "item for both operators on one step's workload and print the tables")
    ap.add_argument("--no-gridding", action="store_true")
    ap.add_argument("--no-extras", action="store_true",
                    help="skip gridding, e2e, CPU baseline and L2 probes (profiling runs)")
    ap.add_argument("--cpu-sample", type=int, default=10240,
                    help="slices timed on the host cores (about 10 s of work on 16 threads)")
    ap.add_argument("--subtomos", type=int, default=512,
                    help="sub-tomograms of the batched uneven-box workload (0 skips it)")
    ap.add_argument("--config5", action="store_true",
                    help="instead of the bench: the large combined configuration (400^3, padding 2, "
                         "2 half-maps x 4 classes) end to end on one GPU")
    ap.add_argument("--gridding-profile", type=int, default=-1, metavar="ITERATIONS",
                    help="instead of the bench: one gridding reconstruction of synthetic accumulators "
                         "(256^3 at padding 2, P = 512) with this many iterations after one warm-up "
                         "run, for profilers (prints its time)")
    ap.add_argument("--c5-particles", type=int, default=1000000)
    ap.add_argument("--c5-chunk", type=int, default=20000)
    return ap.parse_args()


# ------------------------------------------------------------------ helpers --
def counts(n: int, rmax: int):
    """Per-slice element count, samples inside rmax for the projector (<=)
    and for the backprojector (<, x = 0 & y < 0 skipped)."""
    x = np.arange(n // 2 + 1)
    y = np.arange(n)
    y = np.where(y <= n // 2, y, y - n)
    r2 = x[None, :] ** 2 + y[:, None] ** 2
    e = (n // 2 + 1) * n
    sp = int((r2 <= rmax * rmax).sum())
    sb = int(((r2 < rmax * rmax) & ~((x[None, :] == 0) & (y[:, None] < 0))).sum())
    return e, sp, sb


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def nvml_init() -> bool:
    """Initialises NVML once, before any timed work (its start-up must not
    fall into a timed region)."""
    try:
        import pynvml
        pynvml.nvmlInit()
        return True
    except Exception:
        return False


class ClockSampler:
    """Samples SM clock and throttle reasons during the timed region.

    The sampling thread starts before the warm-up (start()) so that NVML's
    first queries, which can stall the GPU for milliseconds to hundreds of
    milliseconds, fall outside the timed region; samples are kept only
    while recording (between begin() and end(), around the timed steps)."""

    def __init__(self, index: int, period: float = 0.02):
        self.index, self.period = index, period
        self.samples, self.reasons, self.max_mhz = [], set(), None
        self._stop = threading.Event()
        self._recording = threading.Event()
        self._t = None

    def start(self) -> "ClockSampler":
        try:
            import pynvml
            nvml_init()
            h = pynvml.nvmlDeviceGetHandleByIndex(self.index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(h, pynvml.NVML_CLOCK_SM)
            names = {
                "hw_slowdown": getattr(pynvml, "nvmlClocksEventReasonHwSlowdown", 0x8),
                "hw_thermal_slowdown": getattr(pynvml, "nvmlClocksEventReasonHwThermalSlowdown", 0x40),
                "sw_thermal_slowdown": getattr(pynvml, "nvmlClocksEventReasonSwThermalSlowdown", 0x20),
                "sw_power_cap": getattr(pynvml, "nvmlClocksEventReasonSwPowerCap", 0x4),
                "hw_power_brake": getattr(pynvml, "nvmlClocksEventReasonHwPowerBrakeSlowdown", 0x80),
            }

            def run():
                while not self._stop.is_set():
                    try:
                        mhz = pynvml.nvmlDeviceGetClockInfo(h, pynvml.NVML_CLOCK_SM)
                        r = pynvml.nvmlDeviceGetCurrentClocksEventReasons(h)
                        if self._recording.is_set():
                            self.samples.append(mhz)
                            for k, bit in names.items():
                                if r & bit:
                                    self.reasons.add(k)
                    except Exception:
                        pass
                    self._stop.wait(self.period)

            self._t = threading.Thread(target=run, daemon=True)
            self._t.start()
        except Exception:
            self._t = None
        return self

    def begin(self) -> None:
        self._recording.set()

    def end(self) -> None:
        self._recording.clear()

    def stop(self) -> None:
        self._recording.clear()
        self._stop.set()
        if self._t:
            self._t.join(timeout=2)

    def summary(self):
        return {"sm_mhz": statistics.median(self.samples) if self.samples else None,
                "sm_max_mhz": self.max_mhz, "reasons": sorted(self.reasons),
                "samples": len(self.samples)}


# ----------------------------------------------------------------- workload --
def synth_module():
    """The seeded input generator (gtom_b200/synth.py: torch and numpy only)
    loaded as a standalone module, so that the reference arm produces the
    same inputs without importing the library's package."""
    import importlib.util
    spec = importlib.util.spec_from_file_location("gtom_synth_standalone", ROOT / "gtom_b200" / "synth.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def bench_config(n, B, pool, P, D, world):
    """The workload description both arms print (identical, so that the two
    lines describe the same configuration)."""
    return {"workload": "single-particle 256^3, padding 2: project + CTF-weighted backproject",
            "box": n, "padding": PAD, "batch_per_step": B, "pool": pool,
            "volume": f"{P // 2 + 1}x{P}x{P} c64 decentred",
            "accumulators": f"{D // 2 + 1}x{D}x{D} c64 + f32 centred",
            "l2_flush": "inputs larger than L2 (per-step data 3.96 GB)", "parallelism": f"dp{world}"}


def make_workload(args, device, seed, impl="ours"):
    """The bench's inputs on the GPU: the padded volume, a pool of particle
    orientations (the reference's host matrix expression, bit for bit the
    same in both arms), and CTF-weighted noisy particles with their CTF^2
    weights.  The particles are projections of the volume, made by this
    library (impl "ours") or by the reference's own projector (impl
    "reference"), which agree bit for bit."""
    import torch
    if impl == "ours":
        import gtom_b200 as G
        from gtom_b200 import synth

        def mats_of(ang):
            return G.matrices_from_angles(ang, float(PAD))

        def project(volft, proj, m, c):
            G.d_rlnProject(volft, (P, P, P), proj, (n, n, 1), rmax, m, c)
    else:
        from oracle import refcuda
        synth = synth_module()
        ref = refcuda.lib()

        def mats_of(ang):
            return refcuda.matrices(ang, float(PAD))

        def project(volft, proj, m, c):
            refcuda.check(ref.ref_project(volft.data_ptr(), P, proj.data_ptr(), n, 2, rmax, m.data_ptr(), c),
                          "reference d_rlnProject")

    n, P = BOX, BOX * PAD
    D = P + 1
    rmax = n // 2
    e, sp, sb = counts(n, rmax)
    rng = np.random.default_rng(seed)
    vol = synth.blob_volume(n, 2000, seed, device)
    ft = synth.padded_half_ft(vol, PAD).reshape(-1)
    del vol
    # 64 spare zeros past the volume: the reference projector's x1 = P/2+1
    # read can touch one element past the end (src/Relion/Project.cu:155)
    vbuf = torch.zeros(ft.numel() + 64, dtype=torch.complex64, device=device)
    vbuf[:ft.numel()] = ft
    volft = vbuf[:ft.numel()]
    del ft
    N = args.pool
    ang = synth.vmf_mixture_angles(rng, N)
    mats = torch.from_numpy(mats_of(ang)).to(device)
    data = torch.empty((N, e), dtype=torch.complex64, device=device)
    wts = torch.empty((N, e), dtype=torch.float32, device=device)
    disk = synth.in_disk_mask(n, rmax, device).reshape(-1)
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    chunk = 2000
    proj = torch.empty((chunk, e), dtype=torch.complex64, device=device)
    for c0 in range(0, N, chunk):
        c = min(chunk, N - c0)
        project(volft, proj, mats[c0:c0 + c].reshape(-1), c)
        df = torch.from_numpy(rng.uniform(0.5, 3.0, c).astype(np.float32)).to(device)
        da = torch.from_numpy(rng.uniform(0.0, 0.1, c).astype(np.float32)).to(device)
        aa = torch.from_numpy(rng.uniform(0.0, np.pi, c).astype(np.float32)).to(device)
        ctf = synth.ctf_half(n, df, da, aa).reshape(c, e)
        sig = proj[:c] * ctf
        pw = (sig.abs() ** 2 * disk).sum(1, keepdim=True) / disk.sum()
        sd = torch.sqrt(pw / 0.05 / 2)
        noise = torch.complex(torch.randn((c, e), device=device, generator=gen),
                              torch.randn((c, e), device=device, generator=gen)) * sd
        data[c0:c0 + c] = (sig + noise) * ctf
        wts[c0:c0 + c] = ctf * ctf
    del proj
    torch.cuda.synchronize()
    return dict(n=n, P=P, D=D, rmax=rmax, e=e, sp=sp, sb=sb, volft=volft, angles=ang, mats=mats,
                data=data, wts=wts, N=N)


# --------------------------------------------------------------------- ours --
def run_ours(args):
    import torch
    import torch.distributed as dist
    import gtom_b200 as G
    from gtom_b200.shard import Accumulators

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=120), device_id=dev)

    G.set_path("project", args.path)
    G.set_path("backproject", args.path)
    B = args.batch
    if args.pool % B:
        args.pool = (args.pool // B + 1) * B
    ws = make_workload(args, dev, SEED + 17 * rank)
    n, P, D, rmax, e = ws["n"], ws["P"], ws["D"], ws["rmax"], ws["e"]
    nvol = (D // 2 + 1) * D * D
    acc = Accumulators(nvol, dev)  # data and weights in one buffer: one all-reduce
    acc_ft, acc_w = acc.data, acc.weights
    proj = torch.empty(B * e, dtype=torch.complex64, device=dev)
    stream = torch.cuda.current_stream()
    ev = []

    def step(i, timed):
        s = (i * B) % ws["N"]
        m = ws["mats"][s:s + B].reshape(-1)
        if timed:
            a, b, c = (torch.cuda.Event(enable_timing=True) for _ in range(3))
            a.record(stream)
        G.d_rlnProject(ws["volft"], (P, P, P), proj, (n, n, 1), rmax, m, B)
        if timed:
            b.record(stream)
        G.d_rlnBackproject(acc_ft, acc_w, (D, D, D), ws["data"][s:s + B].reshape(-1),
                           ws["wts"][s:s + B].reshape(-1), (n, n, 1), rmax, m, None, (1, 0, 0, 1), 0.0,
                           False, False, B)
        if timed:
            c.record(stream)
            ev.append((a, b, c))

    clocks = ClockSampler(local).start()
    for i in range(args.warmup):
        step(i, False)
    acc.zero_()
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    clocks.begin()
    torch.cuda.synchronize()
    start.record(stream)
    for k in range(args.steps):
        step(args.warmup + k, True)
    acc.all_reduce()  # the one exchange: sum the partial volumes of all ranks
    end.record(stream)
    torch.cuda.synchronize()
    clocks.stop()
    if world > 1:
        dist.barrier()
    ms = start.elapsed_time(end)
    t_proj = sum(a.elapsed_time(b) for a, b, _ in ev)
    t_bp = sum(b.elapsed_time(c) for _, b, c in ev)
    if world > 1:
        t = torch.tensor([ms, t_proj, t_bp], device=dev, dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms, t_proj, t_bp = t.tolist()
    slices = world * args.steps * B
    value = slices / (ms / 1e3)

    # roofline of the two kernels
    hbm_peak, peak_kind = measured_peaks()
    probe = {} if args.no_extras else l2_probe()
    # projector: compulsory DRAM bytes per launch = the output slices written
    # once plus the volume read once (the brick kernels stage each brick in
    # shared memory, so the reference's eight 8-byte gathers per sample never
    # reach DRAM); the gather count is reported beside it
    proj_bytes = B * e * 8 + ws["volft"].numel() * 8
    gather_bytes = B * (ws["sp"] * 72 + (e - ws["sp"]) * 8)
    proj_ms = t_proj / args.steps
    proj_gbs = proj_bytes / (proj_ms * 1e-3) / 1e9
    bp_reds = B * ws["sb"] * 24
    bp_ms = t_bp / args.steps
    bp_rate = bp_reds / (bp_ms * 1e-3) / 1e9
    traffic = ncu_traffic()
    roof_proj = {"kernel": "project", "bound": "hbm", "achieved": round(proj_gbs, 1), "peak": hbm_peak,
                 "unit": "GB/s", "frac": round(proj_gbs / hbm_peak, 4),
                 "traffic": None if traffic.get("project_per_slice") is None
                 else int(traffic["project_per_slice"] * B),
                 "traffic_source": "not measured in this run: ncu dram__bytes_read.sum + dram__bytes_write.sum "
                                   "per slice from profiles/ncu_traffic.json, times the batch",
                 "algorithmic_bytes": proj_bytes,
                 "algorithmic_bytes_are": "compulsory: output slices + the volume once",
                 "ms_per_launch": round(proj_ms, 4), "peak_of": peak_kind,
                 "gather_bytes": gather_bytes,
                 "gather_gbs": round(gather_bytes / (proj_ms * 1e-3) / 1e9, 1),
                 "l2_gather_peak_gbs": probe.get("l2_gather_gbs")}
    # The segment backprojector privatises every reduction in shared memory
    # and accumulates most work items in fixed point (int32 shared atomics),
    # the rest with FP32 ones: its ceiling is the int32 shared-memory atomic
    # rate, with the FP32 one and the L2 reduction rate (the direct kernel's
    # ceiling) beside it.
    i32_peak = probe.get("smem_i32_atomic_gadds")
    smem_peak = probe.get("smem_f32_atomic_gadds")
    l2_peak = probe.get("l2_red_v2_gadds") or probe.get("l2_red_gadds")
    roof_bp = {"kernel": "backproject", "bound": "smem_atomic", "achieved": round(bp_rate, 2),
               "peak": i32_peak, "unit": "G reductions/s",
               "frac": None if not i32_peak else round(bp_rate / i32_peak, 4),
               "traffic": None if traffic.get("backproject_per_slice") is None
               else int(traffic["backproject_per_slice"] * B),
               "traffic_source": "not measured in this run: ncu dram__bytes_read.sum + dram__bytes_write.sum "
                                 "per slice from profiles/ncu_traffic.json, times the batch",
               "algorithmic_reductions": bp_reds, "ms_per_launch": round(bp_ms, 4),
               "peak_of": "measured int32 shared-memory atomic rate (probe, same run)",
               "fp32_smem_atomic_peak": smem_peak,
               "frac_of_fp32_smem_atomic": None if not smem_peak else round(bp_rate / smem_peak, 4),
               "l2_red_peak": l2_peak,
               "frac_of_l2_red": None if not l2_peak else round(bp_rate / l2_peak, 4)}
    # the same kernel against HBM: its measured DRAM traffic per launch over
    # its launch time, for readers comparing against the copy bandwidth (the
    # kernel is not HBM-bound; this says how far it is from being so)
    if roof_bp["traffic"]:
        dram_gbs = roof_bp["traffic"] / (bp_ms * 1e-3) / 1e9
        roof_bp["dram_gbs"] = round(dram_gbs, 1)
        roof_bp["dram_frac_of_hbm"] = round(dram_gbs / hbm_peak, 4)
    dominant = roof_proj if t_proj >= t_bp else roof_bp

    out = {"metric": "project+backproject slices/s @256^3", "value": round(value, 1),
           "unit": "slices/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
           "ms_per_step": round(ms / args.steps, 3), "higher_is_better": True, "scaling": "weak",
           "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded blob volume, vMF+uniform "
           "orientations, CTF, SNR 0.05 noise)",
           "config": bench_config(n, B, ws["N"], P, D, world),
           # per step with the default (row-segment) path: the projector launches
           # 6 kernels (plan: pairs with the zero fill, scan, fill, items; the
           # segment kernel; the direct fallback over its list) and the
           # backprojector 6 (plan x4, segment kernel, direct fallback); the
           # binned path adds a zero fill to the projector's; the direct path
           # launches one kernel per operator; summed over the ranks
           "gpu_launches": world * {"brick": 13, "direct": 2}.get(args.path, 12) * args.steps,
           "roofline": dominant, "rooflines": [roof_proj, roof_bp],
           "kernel_ms_per_step": {"project": round(proj_ms, 4), "backproject": round(bp_ms, 4)},
           "peaks": probe, "clocks": clocks.summary()}

    # The one-GPU measurements (gridding, the next operators, the batched
    # reconstructions, the CPU baseline) run at N = 1 only; with N ranks every
    # rank takes the same collective steps: the end-to-end leg on all ranks
    # between barriers, the slowest rank's time, a barrier before teardown.
    single = world == 1
    if single and not (args.no_gridding or args.no_extras):
        out["gridding"] = time_gridding(G, torch, acc_ft, acc_w, n, D, dev)
    if single and not args.no_extras:
        out["extensions"] = time_extensions(args, G, torch, ws, acc_ft, acc_w, dev, hbm_peak, probe)
    if single and not args.no_extras and args.subtomos > 0:
        out["batched_uneven"] = time_batched(args, torch, dev)
    if single and not args.no_extras:
        out["small_config"] = small_config_ours(G, torch, dev)
    if not args.no_extras:
        if world > 1:
            dist.barrier()
        e2e = run_e2e(args, G, torch, ws, dev)
        if world > 1:
            t = torch.tensor([e2e["ms_per_step"]], device=dev, dtype=torch.float64)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms_e2e = float(t.item())
            e2e.update({"value": round(world * e2e["batch_per_step"] / (ms_e2e * 1e-3), 1),
                        "ms_per_step": round(ms_e2e, 3),
                        "h2d_bytes_per_step": world * e2e["h2d_bytes_per_step"],
                        "d2h_bytes_per_step": world * e2e["d2h_bytes_per_step"],
                        "per_rank": "each rank copies batch_per_step particles; bytes are whole-job, "
                                    "time the slowest rank's"})
        out["e2e"] = e2e
        if single:
            out["e2e_from_particles"] = run_e2e_particles(args, G, torch, ws, dev)
            out["cpu_baseline"] = cpu_baseline(args, ws)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    if rank == 0:
        print(json.dumps(out), flush=True)


def small_config_ours(G, torch, dev):
    """Config 1 in full through this library: 64^3 blobs, padding 2, 1 000
    uniform slices projected, inserted with unit CTF and weights, then the
    10-iteration gridding reconstruction; device time per stage (CUDA
    events, best of 5 after a warm-up)."""
    from gtom_b200 import synth
    n, vbuf, nv_in, mats = small_config_inputs(dev, synth, lambda a: G.matrices_from_angles(a, float(PAD)))
    P, D, rmax, B = n * PAD, n * PAD + 1, n // 2, mats.shape[0]
    volft = vbuf[:nv_in]
    e = (n // 2 + 1) * n
    nvol = (D // 2 + 1) * D * D
    proj = torch.empty(B * e, dtype=torch.complex64, device=dev)
    acc_ft = torch.zeros(nvol, dtype=torch.complex64, device=dev)
    acc_w = torch.zeros(nvol, dtype=torch.float32, device=dev)
    rec = torch.empty(n ** 3, dtype=torch.float32, device=dev)
    m = mats.reshape(-1)
    best = None
    for rep in range(6):
        acc_ft.zero_()
        acc_w.zero_()
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
        ev[0].record()
        G.d_rlnProject(volft, (P, P, P), proj, (n, n, 1), rmax, m, B)
        ev[1].record()
        G.d_rlnBackproject(acc_ft, acc_w, (D, D, D), proj, None, (n, n, 1), rmax, m, None, (1, 0, 0, 1), 0.0,
                           False, False, B)
        ev[2].record()
        G.d_ReconstructGridding(acc_ft, acc_w, rec, (n,) * 3, (D,) * 3, PAD, 0, 0, 10)
        ev[3].record()
        torch.cuda.synchronize()
        cur = [ev[i].elapsed_time(ev[i + 1]) for i in range(3)]
        if rep > 0 and (best is None or sum(cur) < sum(best)):
            best = cur
    return {"workload": "64^3 blobs, padding 2, 1 000 uniform slices: project, backproject (unit CTF and "
                        "weights), 10-iteration gridding",
            "ms": {"project": round(best[0], 4), "backproject": round(best[1], 4), "gridding": round(best[2], 4),
                   "total": round(sum(best), 4)}}


def symmetric_grid(P):
    """Whether the default gridding path on grid P is the symmetric one: even,
    16 .. 768, no prime factor above 13, or 800 (GTOMRLN_PATH_SYMMETRIC)."""
    rest = P
    for p in (2, 3, 5, 7, 11, 13):
        while rest % p == 0:
            rest //= p
    return P == 800 or (P % 2 == 0 and 16 <= P <= 768 and rest == 1)


def time_gridding(G, torch, acc_ft, acc_w, n, D, dev):
    out = torch.empty(n ** 3, dtype=torch.float32, device=dev)
    G.d_ReconstructGridding(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, PAD, 0, 0, 1)  # plans, pool
    torch.cuda.synchronize()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    G.d_ReconstructGridding(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, PAD, 0, 0, 10)
    b.record()
    torch.cuda.synchronize()
    ms10 = a.elapsed_time(b)
    a.record()
    G.d_ReconstructGridding(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, PAD, 0, 0, 1)
    b.record()
    torch.cuda.synchronize()
    ms1 = a.elapsed_time(b)
    P = n * PAD
    nc, nr = (P // 2 + 1) * P * P, P ** 3
    compulsory = 12 * nc + 8 * nr
    # the default path on this grid: four passes over the (P/2+1) x P x
    # (P/2+1) complex work array W (16 B per element each) plus Fw in and Fnw
    # in and out (12 B per spectrum element) per iteration
    # inside the sphere: columns x < P/2, and on the sides that face the
    # spectrum only those inside its circle
    nw, circle = (P // 2 + 1) * P * (P // 2), math.pi / 4
    sym_bytes = int((4 + 4 * circle) * 8 * nw + 12 * (2 / 3) * math.pi * (P // 2) ** 3)
    per_it = (ms10 - ms1) / 9
    res = {"ms_10_iterations": round(ms10, 3), "ms_per_iteration": round(per_it, 4), "P": P,
           "path": "symmetric (four passes over the Hermitian half along z)" if symmetric_grid(P) else "cufft",
           "compulsory_bytes_per_iteration": compulsory, "path_bytes_per_iteration": sym_bytes,
           "path_gbs": round(sym_bytes / (per_it * 1e-3) / 1e9, 1), "to_1e-4": {}}
    hbm, hbm_kind = measured_peaks()
    res["path_frac_of_hbm"] = round(sym_bytes / (per_it * 1e-3) / 1e9 / hbm, 4)
    res["hbm_peak"] = {"gbs": hbm, "of": hbm_kind}
    # the cuFFT path (GTOMRLN_PATH_DIRECT) on the same accumulators, for scale
    G.set_path("gridding", "direct")
    try:
        G.d_ReconstructGridding(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, PAD, 0, 0, 1)
        torch.cuda.synchronize()
        a.record()
        G.d_ReconstructGridding(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, PAD, 0, 0, 10)
        b.record()
        torch.cuda.synchronize()
        res["ms_10_iterations_cufft"] = round(a.elapsed_time(b), 3)
    finally:
        G.set_path("gridding", "auto")
    # to a relative change of 1e-4: the reference's update from its sphere-mask
    # start, the momentum update, and both from the learned start (the
    # network trained at 128^3; its inputs are scale- and radius-normalised)
    from gtom_b200 import warmstart as WS
    p128 = WS.load_params(128, dev)
    modes = [("plain", 0.0, None), ("momentum", 0.9, None)]
    if p128 is not None:
        modes += [("plain+mlp", 0.0, p128), ("momentum+mlp", 0.9, p128)]
    for name, mom, prm in modes:
        # two untimed iterations first: the mode's buffers (the momentum
        # extrapolation, the network's scratch) come from the pool once
        G.reconstruct_gridding_warm(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, prm, PAD, 2, 0.0, mom)
        torch.cuda.synchronize()
        a.record()
        it, ch, used = G.reconstruct_gridding_warm(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, prm, PAD, 1000,
                                                   1e-4, mom)
        b.record()
        torch.cuda.synchronize()
        res["to_1e-4"][name] = {"iterations": it, "final_change": ch, "ms": round(a.elapsed_time(b), 3),
                                "warm_used": used}
    t = res["to_1e-4"]
    best = "momentum+mlp" if "momentum+mlp" in t else "momentum"
    res["warm_vs_plain_1e-4"] = {"mode": best, "speedup": round(t["plain"]["ms"] / t[best]["ms"], 3)}
    # to within 1e-4 (weighted relative L2) of the converged weights: the
    # iterations each mode needs (the library's distance to weights
    # converged with momentum to a change of 1e-6), then the whole
    # reconstruction timed for exactly that many iterations (no convergence
    # test inside, so no per-iteration synchronisation)
    ref, _, _, _, _ = G.gridding_weights(acc_w, (D,) * 3, n, PAD, 5000, 1e-6, 0.9)
    conv = {}
    for name, mom, prm in modes:
        if name == "plain+mlp":
            continue
        _, _, k, _, _, dist = G.gridding_weights(acc_w, (D,) * 3, n, PAD, 8000, 0.0, mom, mlp_params=prm,
                                                 ref_fnw=ref, ref_tolerance=1e-4, return_distance=True)
        entry = {"iterations": k, "distance": dist, "reached": bool(dist <= 1e-4)}
        if entry["reached"]:
            torch.cuda.synchronize()
            a.record()
            G.reconstruct_gridding_warm(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, prm, PAD, k, 0.0, mom)
            b.record()
            torch.cuda.synchronize()
            entry["ms"] = round(a.elapsed_time(b), 3)
        conv[name] = entry
    del ref
    res["to_converged_1e-4"] = conv
    if conv["plain"].get("ms") and conv.get(best, {}).get("ms"):
        res["warm_vs_plain_converged"] = {"mode": best,
                                          "speedup": round(conv["plain"]["ms"] / conv[best]["ms"], 3)}
    if p128 is not None:  # the 128^3 learned-warm-start workload: two held-out distributions
        rng = np.random.default_rng(1004)
        dists = [WS.random_distribution(rng) for _ in range(360)][300:302]
        volft = synth_volft(128, dev)
        res["warm_start_128"] = WS.summarise(WS.evaluate(p128, 128, dists, PAD, volft=volft))
    return res


def time_extensions(args, G, torch, ws, acc_ft, acc_w, dev, hbm_peak, probe):
    """The next operators on the same workload, CUDA events around one call
    after one untimed call: the shifted projector and backprojector (a
    per-slice phase shift and global weight; row-segment brick kernels, like
    the main pair) and the particle preprocessing (batched R2C + centring
    phase + CTF and CTF^2)."""
    from gtom_b200.ctf import preprocess_particles
    n, P, D, rmax, e = ws["n"], ws["P"], ws["D"], ws["rmax"], ws["e"]
    B = min(args.batch, ws["N"])
    rng = np.random.default_rng(7)
    m = ws["mats"][:B].reshape(-1)
    shifts = torch.from_numpy((rng.uniform(-5, 5, (B, 3)) * 2 * np.pi / n).astype(np.float32)).to(dev).reshape(-1)
    gw = torch.from_numpy(rng.uniform(0.5, 1.5, B).astype(np.float32)).to(dev)
    proj = torch.empty(B * e, dtype=torch.complex64, device=dev)

    def timed(fn):
        fn()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b)

    res = {}
    ms = timed(lambda: G.d_rlnProjectShifted(ws["volft"], (P, P, P), proj, (n, n, 1), rmax, m, shifts, gw, B))
    byt = B * e * 8 + ws["volft"].numel() * 8  # compulsory: output slices + the volume once
    res["project_shifted"] = {"slices_per_s": round(B / (ms * 1e-3), 1), "ms": round(ms, 3),
                              "compulsory_gbs": round(byt / (ms * 1e-3) / 1e9, 1),
                              "frac_of_hbm": round(byt / (ms * 1e-3) / 1e9 / hbm_peak, 4)}
    ms = timed(lambda: G.d_rlnBackprojectShifted(acc_ft, acc_w, (D, D, D), ws["data"][:B].reshape(-1),
                                                 ws["wts"][:B].reshape(-1), (n, n, 1), rmax, m, shifts, gw, B))
    reds = B * ws["sp"] * 24
    l2 = probe.get("l2_red_v2_gadds")
    sm = probe.get("smem_f32_atomic_gadds")
    res["backproject_shifted"] = {"slices_per_s": round(B / (ms * 1e-3), 1), "ms": round(ms, 3),
                                  "g_reductions_per_s": round(reds / (ms * 1e-3) / 1e9, 1),
                                  "frac_of_smem_atomic": None if not sm else round(reds / (ms * 1e-3) / 1e9 / sm, 4),
                                  "frac_of_l2_red_v2": None if not l2 else round(reds / (ms * 1e-3) / 1e9 / l2, 4)}
    # the general insertion (Backproject.cu:57-63, 145-152, 183-189): a 1.2 %
    # anisotropic magnification, the Ewald curvature of 300 kV electrons at
    # 1 A/pixel (sphere radius n / 0.0197 pixels, supersampled by 2) and two
    # target volumes (half-maps) chosen per particle, against the plain
    # insertion of the same particles into one volume
    iv = torch.from_numpy(rng.integers(0, 2, B).astype(np.int32)).to(dev)
    nvox = (D // 2 + 1) * D * D
    g_ft = torch.zeros(2 * nvox, dtype=torch.complex64, device=dev)
    g_w = torch.zeros(2 * nvox, dtype=torch.float32, device=dev)
    data, wts = ws["data"][:B].reshape(-1), ws["wts"][:B].reshape(-1)
    ms_plain = timed(lambda: G.d_rlnBackproject(acc_ft, acc_w, (D, D, D), data, wts, (n, n, 1), rmax, m, None,
                                                (1, 0, 0, 1), 0.0, False, False, B))
    ms_gen = timed(lambda: G.d_rlnBackproject(g_ft, g_w, (D, D, D), data, wts, (n, n, 1), rmax, m, iv,
                                              (1.012, 0.004, -0.006, 0.993), 2.0 * n / 0.0197, False, False, B))
    res["backproject_general"] = {"slices_per_s": round(B / (ms_gen * 1e-3), 1), "ms": round(ms_gen, 3),
                                  "plain_ms": round(ms_plain, 3), "ratio_to_plain": round(ms_gen / ms_plain, 3),
                                  "geometry": "magnification (1.012, 0.004, -0.006, 0.993), Ewald radius "
                                              f"{2.0 * n / 0.0197:.0f} px, 2 volumes by d_ivolume"}
    del g_ft, g_w
    imgs = torch.randn((B, n, n), device=dev)
    params = [dict(defocus=-float(d) * 1e-6) for d in rng.uniform(0.5, 3.0, B)]
    from gtom_b200.ctf import ctf_params
    arr = ctf_params(params)
    ms = timed(lambda: preprocess_particles(imgs, arr))
    byt = B * (n * n * 4 + e * 12)
    res["preprocess_particles"] = {"particles_per_s": round(B / (ms * 1e-3), 1), "ms": round(ms, 3),
                                   "compulsory_gbs": round(byt / (ms * 1e-3) / 1e9, 1),
                                   "frac_of_hbm": round(byt / (ms * 1e-3) / 1e9 / hbm_peak, 4)}
    del imgs, proj
    res.update(time_next_rows(G, torch, ws, dev, hbm_peak, probe))
    return res


def time_next_rows(G, torch, ws, dev, hbm_peak, probe):
    """The remaining operators beside the path, one timed call each after one
    untimed call: the 3D->3D projector (64 rotations of a 128^3 box from the
    bench's 512^3 padded volume), the dense squared differences of the
    E-step (64 particles x 256 references x 128 shifts at 128^2, groups of
    8 x 8) and the tomographic gather insertion (41 tilts of 128^2 into a
    128^3 volume)."""
    from gtom_b200.estep import d_rlnSquaredDifferences
    from gtom_b200 import synth
    rng = np.random.default_rng(11)

    def timed(fn):
        fn()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b)

    out = {}
    # 3D -> 3D projection: rotated copies of the volume's 128^3 central region
    P, n3, nb = ws["P"], 128, 64
    r3 = n3 // 2
    e3 = (n3 // 2 + 1) * n3 * n3
    x = np.arange(n3 // 2 + 1)[None, None, :]
    yz = np.where(np.arange(n3) <= n3 // 2, np.arange(n3), np.arange(n3) - n3)
    samples = int(((x ** 2 + yz[None, :, None] ** 2 + yz[:, None, None] ** 2) <= r3 * r3).sum())
    mats = torch.from_numpy(G.matrices_from_angles(synth.vmf_mixture_angles(rng, nb), float(P // n3))).to(dev)
    proj3 = torch.empty(nb * e3, dtype=torch.complex64, device=dev)
    ms = timed(lambda: G.d_rlnProject(ws["volft"], (P, P, P), proj3, (n3, n3, n3), r3, mats.reshape(-1), nb))
    byt = nb * (samples * 72 + (e3 - samples) * 8)
    out["project_3d"] = {"volumes_per_s": round(nb / (ms * 1e-3), 1), "ms": round(ms, 3), "box": n3,
                         "algorithmic_gbs": round(byt / (ms * 1e-3) / 1e9, 1),
                         "frac_of_hbm": round(byt / (ms * 1e-3) / 1e9 / hbm_peak, 4)}
    del proj3
    # E-step squared differences, dense layout [particle][reference][shift]
    n2, npart, nref, nsh, tile = 128, 64, 256, 128, 8
    e2 = (n2 // 2 + 1) * n2
    cplx = lambda *sh: torch.complex(torch.randn(sh, device=dev), torch.randn(sh, device=dev))
    part, shf, refs = cplx(npart, e2), cplx(nsh, e2), cplx(nref, e2)
    wv = torch.rand(e2, device=dev) + 0.1
    ctf = torch.rand(npart, e2, device=dev) * 2 - 1
    d2 = torch.empty(npart * nref * nsh, device=dev)
    ms = timed(lambda: d_rlnSquaredDifferences(part, wv, ctf, (n2, n2, 1), npart, shf, nsh, refs, nref, tile, d2))
    flops = 8.0 * npart * nref * nsh * e2  # per (particle, reference, shift, element)
    fp32 = probe.get("fp32_fma_tflops")
    out["squared_differences"] = {"comparisons_per_s": round(npart * nref * nsh / (ms * 1e-3), 1),
                                  "ms": round(ms, 3), "tflops": round(flops / (ms * 1e-3) / 1e12, 2),
                                  "flops_per_element": 8,
                                  "frac_of_fp32": None if not fp32 else round(flops / (ms * 1e-3) / 1e12 / fp32, 4)}
    del part, shf, refs, ctf, d2
    # tomographic gather insertion
    nt, nv = 41, 128
    et = (nv // 2 + 1) * nv
    tm = torch.from_numpy(synth.tilt_matrices(np.zeros(3, np.float32), np.linspace(-60, 60, nt), 1.0)).to(dev)
    tp = cplx(nt, et)
    tw = torch.rand(nt, et, device=dev)
    tv = torch.zeros((nv // 2 + 1) * nv * nv, dtype=torch.complex64, device=dev)
    ms = timed(lambda: G.d_BackprojectTomo(tv, (nv, nv, nv), tp.reshape(-1), tw.reshape(-1), (nv, nv, 1), nv // 2,
                                           tm.reshape(-1), nt))
    vox = int(((x ** 2 + yz[None, :, None] ** 2 + yz[:, None, None] ** 2) < (nv // 2) ** 2).sum())  # nv == n3
    out["backproject_tomo"] = {"tilt_series_per_s": round(1 / (ms * 1e-3), 2), "ms": round(ms, 3), "box": nv,
                               "tilts": nt, "voxel_slice_pairs_per_s": round(vox * nt / (ms * 1e-3), 1)}
    return out


def time_batched(args, torch, dev):
    """The batched uneven-box workload: sub-tomograms of box 32-128 with 41
    tilts each (synth.tilt_series_batch), reconstructed (insertion + 10
    gridding iterations) as one graph-captured batch after the autotuner has
    chosen the insertion launch shape, against one d_rlnBackproject +
    d_ReconstructGridding pair per sub-tomogram through this library and,
    on a sample, through the reference's CUDA code."""
    from gtom_b200 import synth
    from gtom_b200.batch import BatchReconstructor, Subvolume, autotune, reconstruct_separately
    t0 = time.perf_counter()
    raw = synth.tilt_series_batch(args.subtomos, 1003, dev)
    subs = [Subvolume(r["box"], r["projft"], r["projweights"], r["matrices"], r["out"]) for r in raw]
    torch.cuda.synchronize()
    gen_s = time.perf_counter() - t0
    ref = [Subvolume(x.box, x.projft, x.projweights, x.matrices, torch.empty_like(x.out)) for x in subs]
    scratch = {}

    def timed(fn, reps=3):
        fn()
        torch.cuda.synchronize()
        ts = []
        for _ in range(reps):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            fn()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return statistics.median(ts)

    sep_ms = timed(lambda: reconstruct_separately(ref, PAD, 10, scratch))
    rec = BatchReconstructor(subs, PAD, 10)
    tune = autotune(rec, threads=(128, 256, 512), slices=(1, 4), blocks=(4, 8), reps=2)
    graph_ms = timed(lambda: rec.run(use_graph=True), reps=5)
    direct_ms = timed(lambda: rec.run(use_graph=False), reps=3)
    worst = max(float(torch.linalg.norm(a.out - b.out) / torch.linalg.norm(b.out)) for a, b in zip(subs, ref))
    res = {"subtomograms": len(subs), "boxes": sorted({x.box for x in subs}), "tilts": 41,
           "slices": int(sum(x.nslices for x in subs)), "generate_s": round(gen_s, 1),
           "separate_calls_ms": round(sep_ms, 2), "batched_graph_ms": round(graph_ms, 2),
           "batched_no_graph_ms": round(direct_ms, 2), "speedup_vs_separate": round(sep_ms / graph_ms, 2),
           "autotune_best": {"threads": tune["best"][0], "slices_per_item": tune["best"][1],
                             "ctas_per_sm": tune["best"][2], "ms": round(tune["ms"], 2)},
           "max_rel_l2_vs_separate": worst}
    res["reference_separate"] = reference_separate(subs[:64], dev, len(subs))
    rec.close()
    return res


def reference_separate(subs, dev, total):
    """The reference's d_rlnBackproject + d_ReconstructGridding (rebuilt from
    its sources into oracle/_ref/, each call synchronising as the reference
    does) per sub-tomogram on a sample, scaled to the whole batch."""
    import ctypes as C
    import torch
    from oracle import oracle as O
    if not O.REF_PATH.exists():
        return None
    ref = C.CDLL(str(O.REF_PATH))
    p, i, f, d = C.c_void_p, C.c_int, C.c_float, C.c_double
    ref.ref_backproject.argtypes = [p, p, i, p, p, i, i, i, p, p, f, f, f, f, f, i, i, i]
    ref.ref_reconstruct_gridding.argtypes = [p, p, p, i, i, i, i, d, i, d]
    out = torch.empty(128 ** 3, dtype=torch.float32, device=dev)
    t0 = time.perf_counter()
    for s in subs:
        D = s.box * PAD + 1
        nvol = (D // 2 + 1) * D * D
        acc_ft = torch.zeros(nvol + 64, dtype=torch.complex64, device=dev)
        acc_w = torch.zeros(nvol + 64, dtype=torch.float32, device=dev)
        rc = ref.ref_backproject(acc_ft.data_ptr(), acc_w.data_ptr(), D, s.projft.data_ptr(),
                                 s.projweights.data_ptr(), s.box, 2, s.box // 2, s.matrices.data_ptr(), None,
                                 1, 0, 0, 1, 0.0, 0, 0, s.nslices)
        rc = rc or ref.ref_reconstruct_gridding(acc_ft.data_ptr(), acc_w.data_ptr(), out.data_ptr(), s.box, D,
                                                PAD, 10, 1.9, 0, 15.0)
        if rc:
            return {"error": f"reference CUDA returned {rc}"}
    torch.cuda.synchronize()
    ms = (time.perf_counter() - t0) * 1e3
    return {"sample": len(subs), "sample_ms": round(ms, 1), "ms_scaled_to_batch": round(ms * total / len(subs), 1)}


def synth_volft(box, dev):
    from gtom_b200 import synth
    return synth.padded_half_ft(synth.blob_volume(box, 2000, 1004, dev), PAD).reshape(-1)


def run_e2e(args, G, torch, ws, dev):
    """The same metric through the public API with host buffers: per step the
    particle data and weights are copied from pinned host memory, the h_angles
    overloads build and upload the matrices, and the projections are read
    back to pinned host memory.  The steps are pipelined as a caller would
    run them: two device buffer sets alternate, the host->device copies of
    step k (copy stream) overlap the projection and insertion of step k-1
    (compute stream) and the read-back of step k-2 (read-back stream);
    events order each buffer's reuse."""
    Be = min(args.e2e_batch, ws["N"])
    n, P, D, rmax, e = ws["n"], ws["P"], ws["D"], ws["rmax"], ws["e"]
    h_data = ws["data"][:Be].cpu().pin_memory()
    h_wts = ws["wts"][:Be].cpu().pin_memory()
    h_proj = [torch.empty((Be, e), dtype=torch.complex64).pin_memory() for _ in range(2)]
    ang = ws["angles"][:Be].copy()
    d_data = [torch.empty((Be, e), dtype=torch.complex64, device=dev) for _ in range(2)]
    d_wts = [torch.empty((Be, e), dtype=torch.float32, device=dev) for _ in range(2)]
    d_proj = [torch.empty((Be, e), dtype=torch.complex64, device=dev) for _ in range(2)]
    nvol = (D // 2 + 1) * D * D
    acc_ft = torch.zeros(nvol, dtype=torch.complex64, device=dev)
    acc_w = torch.zeros(nvol, dtype=torch.float32, device=dev)
    s_in, s_comp, s_out = (torch.cuda.Stream(device=dev) for _ in range(3))
    ev_in, ev_comp, ev_out = ([torch.cuda.Event() for _ in range(2)] for _ in range(3))
    for ev in ev_in + ev_comp + ev_out:
        ev.record()

    def step(k):
        b = k % 2
        s_in.wait_event(ev_comp[b])  # step k-2 no longer reads this buffer set
        with torch.cuda.stream(s_in):
            d_data[b].copy_(h_data, non_blocking=True)
            d_wts[b].copy_(h_wts, non_blocking=True)
        ev_in[b].record(s_in)
        s_comp.wait_event(ev_in[b])
        s_comp.wait_event(ev_out[b])  # step k-2's projections have been read back
        G.d_rlnProject(ws["volft"], (P, P, P), d_proj[b].reshape(-1), (n, n, 1), ang, float(PAD), Be,
                       stream=s_comp)
        G.d_rlnBackproject(acc_ft, acc_w, (D, D, D), d_data[b].reshape(-1), d_wts[b].reshape(-1), (n, n, 1),
                           rmax, ang, None, (1, 0, 0, 1), 0.0, float(PAD), False, False, Be, stream=s_comp)
        ev_comp[b].record(s_comp)
        s_out.wait_event(ev_comp[b])
        with torch.cuda.stream(s_out):
            h_proj[b].copy_(d_proj[b], non_blocking=True)
        ev_out[b].record(s_out)

    for k in range(2):
        step(k)
    torch.cuda.synchronize()
    a, z = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record(s_in)
    for k in range(args.steps):
        step(2 + k)
    done = torch.cuda.current_stream()
    for st in (s_in, s_comp, s_out):
        done.wait_stream(st)
    z.record(done)
    torch.cuda.synchronize()
    ms = a.elapsed_time(z)
    return {"value": round(args.steps * Be / (ms / 1e3), 1), "unit": "slices/s",
            "h2d_bytes_per_step": Be * e * 12, "d2h_bytes_per_step": Be * e * 8,
            "batch_per_step": Be, "ms_per_step": round(ms / args.steps, 3),
            "pipeline": "2 buffer sets; copy-in, compute and read-back streams overlap across steps"}


def run_e2e_particles(args, G, torch, ws, dev):
    """The end-to-end leg as a RELION caller runs it from real-space
    particles: per step the n x n float32 images are copied from pinned host
    memory with their CTF parameters (host arrays), the library's particle
    preprocessing makes CTF * FT and CTF^2 on the GPU, then the projection and
    insertion run as in run_e2e, and the projections are read back.  Same
    two-buffer, three-stream pipeline.  The image stack is synthesised once
    from the workload's spectra (its content does not change the timing)."""
    from gtom_b200 import ctf as CTF
    Be = min(args.e2e_batch, ws["N"])
    n, P, D, rmax, e = ws["n"], ws["P"], ws["D"], ws["rmax"], ws["e"]
    spec = ws["data"][:Be].reshape(Be, n, n // 2 + 1)
    imgs = torch.fft.fftshift(torch.fft.irfft2(spec, s=(n, n)), dim=(-2, -1)).float().contiguous()
    h_img = imgs.cpu().pin_memory()
    del imgs, spec
    rng = np.random.default_rng(SEED + 5)
    params = CTF.ctf_params([{"defocus": -rng.uniform(0.5e-6, 3e-6), "defocusdelta": rng.uniform(0, 0.1e-6),
                              "astigmatismangle": rng.uniform(0, np.pi), "Cs": 2.7e-3} for _ in range(Be)])
    h_proj = [torch.empty((Be, e), dtype=torch.complex64).pin_memory() for _ in range(2)]
    ang = ws["angles"][:Be].copy()
    d_img = [torch.empty((Be, n, n), dtype=torch.float32, device=dev) for _ in range(2)]
    d_proj = [torch.empty((Be, e), dtype=torch.complex64, device=dev) for _ in range(2)]
    nvol = (D // 2 + 1) * D * D
    acc_ft = torch.zeros(nvol, dtype=torch.complex64, device=dev)
    acc_w = torch.zeros(nvol, dtype=torch.float32, device=dev)
    s_in, s_comp, s_out = (torch.cuda.Stream(device=dev) for _ in range(3))
    ev_in, ev_comp, ev_out = ([torch.cuda.Event() for _ in range(2)] for _ in range(3))
    for ev in ev_in + ev_comp + ev_out:
        ev.record()

    def step(k):
        b = k % 2
        s_in.wait_event(ev_comp[b])  # step k-2 no longer reads this buffer set
        with torch.cuda.stream(s_in):
            d_img[b].copy_(h_img, non_blocking=True)
        ev_in[b].record(s_in)
        s_comp.wait_event(ev_in[b])
        s_comp.wait_event(ev_out[b])  # step k-2's projections have been read back
        with torch.cuda.stream(s_comp):
            pf, pw = CTF.preprocess_particles(d_img[b], params, stream=s_comp)
        G.d_rlnProject(ws["volft"], (P, P, P), d_proj[b].reshape(-1), (n, n, 1), ang, float(PAD), Be,
                       stream=s_comp)
        G.d_rlnBackproject(acc_ft, acc_w, (D, D, D), pf, pw, (n, n, 1), rmax, ang, None, (1, 0, 0, 1), 0.0,
                           float(PAD), False, False, Be, stream=s_comp)
        ev_comp[b].record(s_comp)
        s_out.wait_event(ev_comp[b])
        with torch.cuda.stream(s_out):
            h_proj[b].copy_(d_proj[b], non_blocking=True)
        ev_out[b].record(s_out)

    for k in range(2):
        step(k)
    torch.cuda.synchronize()
    a, z = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record(s_in)
    for k in range(args.steps):
        step(2 + k)
    done = torch.cuda.current_stream()
    for st in (s_in, s_comp, s_out):
        done.wait_stream(st)
    z.record(done)
    torch.cuda.synchronize()
    ms = a.elapsed_time(z)
    return {"value": round(args.steps * Be / (ms / 1e3), 1), "unit": "slices/s",
            "h2d_bytes_per_step": Be * n * n * 4 + Be * 14 * 4, "d2h_bytes_per_step": Be * e * 8,
            "batch_per_step": Be, "ms_per_step": round(ms / args.steps, 3),
            "pipeline": "real-space particles and CTF parameters in; preprocessing (R2C, centring, CTF, "
                        "CTF^2), projection and insertion on the GPU; projections out"}


# ------------------------------------------------------------- CPU baseline --
def cpu_sample_inputs(ws, count):
    """Host copies of the volume and the first `count` particles."""
    vol = ws["volft"].cpu().numpy()
    data = ws["data"][:count].cpu().numpy()
    wts = ws["wts"][:count].cpu().numpy()
    mats = ws["mats"][:count].cpu().numpy()
    return vol, data, wts, mats


def time_cpu_port(vol, data, wts, mats, n, P, D, rmax, threads=None):
    from oracle import oracle as O
    if threads:
        O.set_threads(threads)
    count = mats.shape[0]
    t0 = time.perf_counter()
    O.project(vol, P, n, rmax, mats, fp32=True)
    t1 = time.perf_counter()
    nv = (D // 2 + 1) * D * D
    vf, vw = np.zeros(nv, np.complex64), np.zeros(nv, np.float32)
    O.backproject(vf, vw, D, data, wts, n, rmax, mats, decentered=False, fp32=True)
    t2 = time.perf_counter()
    return count / (t2 - t0), t1 - t0, t2 - t1


def cpu_baseline(args, ws):
    from oracle import oracle as O
    count = min(args.cpu_sample, ws["N"])
    vol, data, wts, mats = cpu_sample_inputs(ws, count)
    rate, tp, tb = time_cpu_port(vol, data, wts, mats, ws["n"], ws["P"], ws["D"], ws["rmax"])
    return {"value": round(rate, 2), "unit": "slices/s", "cores": O.num_threads(), "kind": "port",
            "sample": f"{count} slices of the 256^3 workload (project {tp:.2f} s + backproject {tb:.2f} s), "
                      "OpenMP FP32 restatement of the reference kernels"}


# ---------------------------------------------------------------- reference --
def run_reference(args):
    """The reference arm: the reference's kernels on this box, on the same
    workload as the GPU arm (same seeded inputs, same batch per step, same
    config).  The reference ships no CPU implementation of this path
    (RELION's liblion is not vendored), so `value` is the OpenMP FP32
    restatement of its projector and backprojector kernels on all host
    cores; the reference's own CUDA kernels, rebuilt from its sources, are
    timed beside it (`reference_cuda`), with its gridding reconstruction and
    the small configuration (64^3, 1 000 slices) in full.  Nothing of the
    library under test is loaded: the inputs come from the same seeded
    generator, the particles from the reference's own projector."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import torch
    from oracle import oracle as O
    dev = torch.device("cuda", int(os.environ.get("LOCAL_RANK", "0")))
    torch.cuda.set_device(dev)
    B = args.batch
    a2 = argparse.Namespace(**vars(args))
    if a2.pool % B:
        a2.pool = (a2.pool // B + 1) * B
    ws = make_workload(a2, dev, SEED, impl="reference")
    n, P, D, rmax, N = ws["n"], ws["P"], ws["D"], ws["rmax"], ws["N"]
    vol = ws["volft"].cpu().numpy()

    def batch_of(i, count):
        s0 = (i * B) % N
        return (ws["data"][s0:s0 + count].cpu().numpy(), ws["wts"][s0:s0 + count].cpu().numpy(),
                ws["mats"][s0:s0 + count].cpu().numpy())

    warm = min(B, 500)
    for i in range(args.warmup):  # untimed: page-in and thread start-up on a 500-slice sample
        time_cpu_port(vol, *batch_of(i, warm), n, P, D, rmax)
    el = 0.0
    for k in range(args.steps):  # each step: the full batch, host copies outside the timing
        d, w, m = batch_of(args.warmup + k, B)
        t = time.perf_counter()
        time_cpu_port(vol, d, w, m, n, P, D, rmax)
        el += time.perf_counter() - t
    value = args.steps * B / el
    out = {"impl": "reference", "metric": "project+backproject slices/s @256^3", "value": round(value, 2),
           "unit": "slices/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
           "ms_per_step": round(el / args.steps * 1e3, 3), "higher_is_better": True, "scaling": "weak",
           "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded blob volume, vMF+uniform "
           "orientations, CTF, SNR 0.05 noise)",
           "config": bench_config(n, B, N, P, D, world),
           "cpu_baseline": {"value": round(value, 2), "unit": "slices/s", "cores": O.num_threads(),
                            "kind": "port",
                            "sample": f"{B} slices per step (the whole batch; warm-up steps on {warm}); the "
                                      "reference ships no CPU path for this (liblion is not vendored), so "
                                      "the OpenMP FP32 restatement of its kernels runs"},
           "e2e": {"value": round(value, 2), "unit": "slices/s", "h2d_bytes_per_step": 0,
                   "d2h_bytes_per_step": 0}}
    rc = reference_cuda(args, ws, dev)
    if rc is not None:
        out["reference_cuda"] = rc
        out["small_config"] = small_config_reference(dev)
    print(json.dumps(out), flush=True)


def reference_cuda(args, ws, dev):
    """Times the reference's own CUDA kernels (rebuilt from its sources for
    sm_100a into oracle/_ref/) on the same workload: d_rlnProject and
    d_rlnBackproject of one batch, then d_ReconstructGridding (10
    iterations, P = 512) of the accumulated volume."""
    import torch
    from oracle import refcuda
    if not refcuda.available():
        return None
    ref = refcuda.lib()
    n, P, D, rmax, e = ws["n"], ws["P"], ws["D"], ws["rmax"], ws["e"]
    B = min(args.batch, ws["N"])
    proj = torch.empty(B * e, dtype=torch.complex64, device=dev)
    nvol = (D // 2 + 1) * D * D
    acc_ft = torch.zeros(nvol, dtype=torch.complex64, device=dev)
    acc_w = torch.zeros(nvol, dtype=torch.float32, device=dev)
    m = ws["mats"][:B].contiguous()
    t = []
    for rep in range(3):
        acc_ft.zero_()
        acc_w.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        refcuda.check(ref.ref_project(ws["volft"].data_ptr(), P, proj.data_ptr(), n, 2, rmax, m.data_ptr(), B),
                      "reference d_rlnProject")
        t1 = time.perf_counter()
        refcuda.check(ref.ref_backproject(acc_ft.data_ptr(), acc_w.data_ptr(), D, ws["data"].data_ptr(),
                                          ws["wts"].data_ptr(), n, 2, rmax, m.data_ptr(), None, 1, 0, 0, 1, 0.0,
                                          0, 0, B), "reference d_rlnBackproject")
        t2 = time.perf_counter()
        t.append((t1 - t0, t2 - t1))
    tp = min(x[0] for x in t)
    tb = min(x[1] for x in t)
    rec = torch.empty(n ** 3, dtype=torch.float32, device=dev)
    tg = []
    for rep in range(2):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        refcuda.check(ref.ref_reconstruct_gridding(acc_ft.data_ptr(), acc_w.data_ptr(), rec.data_ptr(), n, D, PAD,
                                                   10, 1.9, 0, 15.0), "reference d_ReconstructGridding")
        tg.append(time.perf_counter() - t0)
    return {"value": round(B / (tp + tb), 1), "unit": "slices/s", "batch": B,
            "project_ms": round(tp * 1e3, 3), "backproject_ms": round(tb * 1e3, 3),
            "gridding_10it_ms": round(min(tg) * 1e3, 3),
            "how": "reference d_rlnProject / d_rlnBackproject (matrix overloads) and d_ReconstructGridding "
                   "(10 iterations, P = 512, its own cuFFT plans per call) rebuilt from source for sm_100a "
                   "with its own flags; each call synchronises (as the reference does); best of 3 / 2"}


SMALL_BOX = 64


def small_config_inputs(dev, synth, mats_of):
    """The small plain configuration: a 64^3 volume of 200 Gaussian blobs
    (sigma U(1.5, 4) voxels, amplitude U(0.2, 1), centres within radius 28),
    padding 2, 1 000 slices at uniform SO(3) orientations."""
    import torch
    n = SMALL_BOX
    rng = np.random.default_rng(1001)
    vol = synth.blob_volume(n, 200, 1001, dev, radius_frac=28.0 / n)
    ft = synth.padded_half_ft(vol, PAD).reshape(-1)
    vbuf = torch.zeros(ft.numel() + 64, dtype=torch.complex64, device=dev)
    vbuf[:ft.numel()] = ft
    ang = synth.vmf_mixture_angles(rng, 1000, uniform_frac=1.0)
    mats = torch.from_numpy(mats_of(ang)).to(dev)
    return n, vbuf, ft.numel(), mats


def small_config_reference(dev):
    """Config 1 in full through the reference: its CUDA kernels (project,
    backproject with unit CTF and weights, 10-iteration gridding) and the CPU
    port (projector and backprojector restated, gridding in the FP64 numpy
    restatement) on the host cores."""
    import torch
    from oracle import oracle as O
    from oracle import refcuda
    ref = refcuda.lib()
    n, vbuf, nv_in, mats = small_config_inputs(dev, synth_module(), lambda a: refcuda.matrices(a, float(PAD)))
    P, D, rmax, B = n * PAD, n * PAD + 1, n // 2, mats.shape[0]
    e = (n // 2 + 1) * n
    nvol = (D // 2 + 1) * D * D
    proj = torch.empty(B * e, dtype=torch.complex64, device=dev)
    acc_ft = torch.zeros(nvol, dtype=torch.complex64, device=dev)
    acc_w = torch.zeros(nvol, dtype=torch.float32, device=dev)
    rec = torch.empty(n ** 3, dtype=torch.float32, device=dev)
    best = None
    for rep in range(3):
        acc_ft.zero_()
        acc_w.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        refcuda.check(ref.ref_project(vbuf.data_ptr(), P, proj.data_ptr(), n, 2, rmax, mats.data_ptr(), B), "project")
        t1 = time.perf_counter()
        refcuda.check(ref.ref_backproject(acc_ft.data_ptr(), acc_w.data_ptr(), D, proj.data_ptr(), None, n, 2, rmax,
                                          mats.data_ptr(), None, 1, 0, 0, 1, 0.0, 0, 0, B), "backproject")
        t2 = time.perf_counter()
        refcuda.check(ref.ref_reconstruct_gridding(acc_ft.data_ptr(), acc_w.data_ptr(), rec.data_ptr(), n, D, PAD,
                                                   10, 1.9, 0, 15.0), "gridding")
        t3 = time.perf_counter()
        cur = (t1 - t0, t2 - t1, t3 - t2)
        best = cur if best is None or sum(cur) < sum(best) else best
    vol = vbuf[:nv_in].cpu().numpy()
    m = mats.cpu().numpy()
    t0 = time.perf_counter()
    p = O.project(vol, P, n, rmax, m, fp32=True)
    t1 = time.perf_counter()
    vf, vw = np.zeros(nvol, np.complex64), np.zeros(nvol, np.float32)
    O.backproject(vf, vw, D, p, None, n, rmax, m, decentered=False, fp32=True)
    t2 = time.perf_counter()
    O.reconstruct_gridding(vf.reshape(D, D, D // 2 + 1), vw.reshape(D, D, D // 2 + 1), n, (D, D, D), PAD)
    t3 = time.perf_counter()
    return {"workload": "64^3 blobs, padding 2, 1 000 uniform slices: project, backproject (unit CTF and "
                        "weights), 10-iteration gridding",
            "reference_cuda_ms": {"project": round(best[0] * 1e3, 3), "backproject": round(best[1] * 1e3, 3),
                                  "gridding": round(best[2] * 1e3, 3), "total": round(sum(best) * 1e3, 3)},
            "cpu_port_ms": {"project": round((t1 - t0) * 1e3, 1), "backproject": round((t2 - t1) * 1e3, 1),
                            "gridding_fp64_numpy": round((t3 - t2) * 1e3, 1), "total": round((t3 - t0) * 1e3, 1),
                            "cores": O.num_threads()}}


PROBE_SRC = ROOT / "bench_probe" / "l2_probe.cu"
PROBE_LIB = ROOT / "bench_probe" / "libbench_probe.so"


def build_probe() -> Path:
    """Compiles the roofline microbenchmarks (bench_probe/l2_probe.cu, bench
    only: the product library neither contains nor loads them) for sm_100a
    when the library is missing or older than its source."""
    import subprocess
    if not PROBE_LIB.exists() or PROBE_LIB.stat().st_mtime < PROBE_SRC.stat().st_mtime:
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        nvcc = str(Path(cuda) / "bin" / "nvcc") if (Path(cuda) / "bin" / "nvcc").exists() else "nvcc"
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
                        "-Xcompiler", "-fPIC", "-shared", "-o", str(PROBE_LIB), str(PROBE_SRC)], check=True)
    return PROBE_LIB


def l2_probe():
    import ctypes as C
    try:
        path = build_probe()
    except Exception:
        return {}
    L = C.CDLL(str(path))
    L.gtomrln_probe_l2_red.restype = C.c_double
    L.gtomrln_probe_l2_red.argtypes = [C.c_int] * 5
    L.gtomrln_probe_l2_gather.restype = C.c_double
    L.gtomrln_probe_l2_gather.argtypes = [C.c_int] * 4
    out = {}
    for vec, key in ((1, "l2_red_gadds"), (2, "l2_red_v2_gadds"), (4, "l2_red_v4_gadds")):
        v = L.gtomrln_probe_l2_red(vec, 26, 148 * 8, 256, 256)
        out[key] = round(v / 1e9, 2) if v > 0 else None
    g = L.gtomrln_probe_l2_gather(26, 148 * 8, 256, 256)
    out["l2_gather_gbs"] = round(g / 1e9, 1) if g > 0 else None
    L.gtomrln_probe_smem_update.restype = C.c_double
    L.gtomrln_probe_smem_update.argtypes = [C.c_int] * 4
    for mode, key in ((0, "smem_f32_atomic_gadds"), (1, "smem_i32_atomic_gadds")):
        v = L.gtomrln_probe_smem_update(mode, 148 * 4, 256, 4096)
        out[key] = round(v / 1e9, 1) if v > 0 else None
    L.gtomrln_probe_fp32_fma.restype = C.c_double
    L.gtomrln_probe_fp32_fma.argtypes = [C.c_int] * 3
    v = L.gtomrln_probe_fp32_fma(148 * 8, 256, 8192)
    out["fp32_fma_tflops"] = round(v / 1e12, 2) if v > 0 else None
    L.gtomrln_probe_fp32x2_fma.restype = C.c_double
    L.gtomrln_probe_fp32x2_fma.argtypes = [C.c_int] * 3
    v = L.gtomrln_probe_fp32x2_fma(148 * 8, 256, 8192)
    out["fp32x2_fma_tflops"] = round(v / 1e12, 2) if v > 0 else None
    out["how"] = ("L2: random addresses in a 64 MiB L2-resident buffer, 148*8 blocks x 256 threads; "
                  "shared memory: random words of a 48 KB array, 148*4 blocks x 256 threads; "
                  "FP32: 8 independent FMA chains per thread, 148*8 blocks x 256 threads")
    return out


def ncu_traffic():
    p = ROOT / "profiles" / "ncu_traffic.json"
    if p.exists():
        try:
            return json.loads(p.read_text())
        except Exception:
            return {}
    return {}


def run_sweep(args):
    """The autotuner's tables for both operators on one step of the bench's
    workload (gtom_b200.autotune.tune: median of 3 timed calls per shape)."""
    import torch
    import gtom_b200 as G
    from gtom_b200 import autotune
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    G.set_path("project", args.path)
    G.set_path("backproject", args.path)
    a2 = argparse.Namespace(**vars(args))
    a2.pool = args.batch
    ws = make_workload(a2, dev, SEED)
    n, P, D, rmax, e, B = ws["n"], ws["P"], ws["D"], ws["rmax"], ws["e"], args.batch
    nvol = (D // 2 + 1) * D * D
    acc_ft = torch.zeros(nvol, dtype=torch.complex64, device=dev)
    acc_w = torch.zeros(nvol, dtype=torch.float32, device=dev)
    proj = torch.empty(B * e, dtype=torch.complex64, device=dev)
    m = ws["mats"][:B].reshape(-1)

    def run_p():
        G.d_rlnProject(ws["volft"], (P, P, P), proj, (n, n, 1), rmax, m, B)

    def run_b():
        G.d_rlnBackproject(acc_ft, acc_w, (D, D, D), ws["data"][:B].reshape(-1), ws["wts"][:B].reshape(-1),
                           (n, n, 1), rmax, m, None, (1, 0, 0, 1), 0.0, False, False, B)

    out = {}
    for op, fn in (("project", run_p), ("backproject", run_b)):
        cands = autotune.candidates(op, threads=(512, 768, 1024), chunks=(1024, 4096, 16384))
        res = autotune.tune(op, fn, cands, reps=3, path="brick" if args.path == "brick" else "segment")
        out[op] = {"best": res["best"], "ms": round(res["ms"], 3),
                   "table": [(e_, t_, c_, round(ms, 3)) for e_, t_, c_, ms in sorted(res["table"], key=lambda r: r[3])]}
        G.set_brick_tuning(op)  # back to the compiled-in default for the next operator's timing
    print(json.dumps({"sweep": out, "path": args.path, "batch": B, "box": n, "padding": PAD}), flush=True)


def run_config5(args):
    """The large combined configuration on one B200: a 400^3 FP32 blob
    volume per class (2 000 Gaussians each), padding 2 (complex64
    401 x 800 x 800 per class), and 1 000 000 400 x 400 particles split into
    2 half-maps x 4 classes of 40 / 30 / 20 / 10 %, with CTFs and noise as
    in the single-particle workload (SNR 0.05).  The particles are generated
    on the GPU in chunks (projected from their class, CTF, noise; 965 GB in
    all, never resident at once) and every chunk is inserted into the eight
    centred 801^3 accumulators with one backprojection call whose d_ivolume
    selects the volume (2 class + half) per particle, the row-segment kernel
    with one work item per (volume, brick).  Then each of the eight volumes
    is reconstructed with the gridding correction from the learned warm
    start and the momentum update to a relative change of 1e-4 (P = 800,
    the symmetric-spectrum iteration with radix-5 transforms).  Reported: insertion slices/s (device time of the
    insertion calls alone), generation time, per-volume gridding time and
    iterations, the 10-iteration plain gridding at P = 800 for scale, and
    the device memory in use at its peak against the GPU's total."""
    import torch
    import gtom_b200 as G
    from gtom_b200 import synth
    from gtom_b200 import warmstart as WS
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    n, P, D = 400, 800, 801
    rmax, e = n // 2, (n // 2 + 1) * n
    nvox = (D // 2 + 1) * D * D
    fracs = np.array([0.4, 0.3, 0.2, 0.1])
    total, chunk = args.c5_particles, args.c5_chunk
    rng = np.random.default_rng(1005)
    peak = [0]

    def note_memory():
        free, tot = torch.cuda.mem_get_info()
        peak[0] = max(peak[0], tot - free)
        return tot

    t0 = time.perf_counter()
    vols = []
    for c in range(4):
        v = synth.blob_volume(n, 2000, 2000 + c, dev)
        vols.append(synth.padded_half_ft(v, PAD).reshape(-1))
        del v
        torch.cuda.empty_cache()
    torch.cuda.synchronize()
    t_vols = time.perf_counter() - t0
    acc_ft = torch.zeros(8 * nvox, dtype=torch.complex64, device=dev)
    acc_w = torch.zeros(8 * nvox, dtype=torch.float32, device=dev)
    proj = torch.empty((chunk, e), dtype=torch.complex64, device=dev)
    disk = synth.in_disk_mask(n, rmax, dev).reshape(-1)
    gen = torch.Generator(device=dev)
    gen.manual_seed(1005)
    ev = []
    per_volume = np.zeros(8, np.int64)
    t0 = time.perf_counter()
    for c0 in range(0, total, chunk):
        cnt = min(chunk, total - c0)
        counts = rng.multinomial(cnt, fracs)
        cls = np.repeat(np.arange(4), counts)
        ivol = (2 * cls + rng.integers(0, 2, cnt)).astype(np.int32)
        np.add.at(per_volume, ivol, 1)
        mats = torch.from_numpy(G.matrices_from_angles(synth.vmf_mixture_angles(rng, cnt), float(PAD))).to(dev)
        s0 = 0
        for c in range(4):
            k = int(counts[c])
            if k:
                G.d_rlnProject(vols[c], (P, P, P), proj[s0:s0 + k].reshape(-1), (n, n, 1), rmax,
                               mats[s0:s0 + k].reshape(-1), k)
            s0 += k
        df = torch.from_numpy(rng.uniform(0.5, 3.0, cnt).astype(np.float32)).to(dev)
        da = torch.from_numpy(rng.uniform(0.0, 0.1, cnt).astype(np.float32)).to(dev)
        aa = torch.from_numpy(rng.uniform(0.0, np.pi, cnt).astype(np.float32)).to(dev)
        ctf = synth.ctf_half(n, df, da, aa).reshape(cnt, e)
        sig = proj[:cnt] * ctf
        pw = (sig.abs() ** 2 * disk).sum(1, keepdim=True) / disk.sum()
        sd = torch.sqrt(pw / 0.05 / 2)
        data = (sig + torch.complex(torch.randn((cnt, e), device=dev, generator=gen),
                                    torch.randn((cnt, e), device=dev, generator=gen)) * sd) * ctf
        wts = ctf * ctf
        del sig
        d_iv = torch.from_numpy(ivol).to(dev)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        G.d_rlnBackproject(acc_ft, acc_w, (D, D, D), data.reshape(-1), wts.reshape(-1), (n, n, 1), rmax,
                           mats.reshape(-1), d_iv, (1, 0, 0, 1), 0.0, False, False, cnt)
        b.record()
        ev.append((a, b))
        if c0 == 0:
            torch.cuda.synchronize()
            note_memory()
        del data, wts, ctf
    torch.cuda.synchronize()
    t_all = time.perf_counter() - t0
    ins_ms = sum(a.elapsed_time(b) for a, b in ev)
    note_memory()
    del proj, vols
    torch.cuda.empty_cache()
    p128 = WS.load_params(128, dev)
    out = torch.empty(n ** 3, dtype=torch.float32, device=dev)
    # one untimed short run first: the final transform's plan, the tables and
    # the pool's buffers are made once per grid
    G.reconstruct_gridding_warm(acc_ft[:nvox], acc_w[:nvox], out, (n,) * 3, (D,) * 3, p128, PAD, 2, 0.0, 0.9)
    torch.cuda.synchronize()
    grid = []
    for v in range(8):
        sl = slice(v * nvox, (v + 1) * nvox)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        it, ch, used = G.reconstruct_gridding_warm(acc_ft[sl], acc_w[sl], out, (n,) * 3, (D,) * 3, p128, PAD, 1000,
                                                   1e-4, 0.9)
        b.record()
        torch.cuda.synchronize()
        note_memory()
        grid.append({"volume": v, "class": v // 2, "half": v % 2, "particles": int(per_volume[v]),
                     "iterations": it, "final_change": ch, "learned_start_kept": used,
                     "ms": round(a.elapsed_time(b), 2)})
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    G.d_ReconstructGridding(acc_ft[:nvox], acc_w[:nvox], out, (n,) * 3, (D,) * 3, PAD, 0, 0, 10)
    b.record()
    torch.cuda.synchronize()
    tot = note_memory()
    print(json.dumps({
        "config": "large combined: 400^3 blob volume per class, padding 2, 1 000 000 particles of 400^2 in 2 "
                  "half-maps x 4 classes (40/30/20/10 %), CTF, SNR 0.05; one insertion call per chunk into 8 "
                  "volumes by d_ivolume; learned warm start + momentum gridding per volume to change 1e-4",
        "particles": total, "chunk": chunk,
        "insert_slices_per_s": round(total / (ins_ms * 1e-3), 1), "insert_ms": round(ins_ms, 1),
        "generate_and_insert_s": round(t_all, 1), "class_volumes_s": round(t_vols, 1),
        "gridding": grid, "gridding_total_ms": round(sum(g["ms"] for g in grid), 1),
        "gridding_10it_plain_ms": round(a.elapsed_time(b), 2),
        "peak_device_memory_gb": round(peak[0] / 1e9, 2), "device_memory_gb": round(tot / 1e9, 2),
        "accumulators_gb": round(8 * nvox * 12 / 1e9, 2)}), flush=True)


def run_gridding_profile(iterations):
    """One d_ReconstructGridding of smooth synthetic accumulators (a radial
    weight profile with 20 % noise, Hermitian on x = 0, and random data
    under it) at the bench's box, after one warm-up run: the launch sequence
    a profiler captures for the gridding kernels."""
    import torch
    import gtom_b200 as G
    dev = torch.device("cuda:0")
    n, D = BOX, BOX * PAD + 1
    g = torch.Generator(device=dev)
    g.manual_seed(512)
    z = torch.arange(D, device=dev, dtype=torch.float32) - D // 2
    x = torch.arange(D // 2 + 1, device=dev, dtype=torch.float32)
    r = torch.sqrt(z[:, None, None] ** 2 + z[None, :, None] ** 2 + x[None, None, :] ** 2)
    w = torch.where(r < n * PAD / 2, 1.0 + 30.0 * torch.exp(-r / (n / 3)), torch.zeros_like(r))
    w = w * (0.8 + 0.4 * torch.rand(w.shape, device=dev, generator=g))
    w[:, :, 0] = 0.5 * (w[:, :, 0] + torch.flip(w[:, :, 0], (0, 1)))
    data = torch.complex(torch.randn(w.shape, device=dev, generator=g),
                         torch.randn(w.shape, device=dev, generator=g)) * (w * torch.exp(-r / n))
    data[:, :, 0] = 0.5 * (data[:, :, 0] + torch.flip(data[:, :, 0], (0, 1)).conj())
    del r
    acc_w, acc_ft = w.reshape(-1).contiguous(), data.reshape(-1).contiguous()
    del w, data
    out = torch.zeros(n ** 3, device=dev)
    G.d_ReconstructGridding(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, PAD, 0, 0, iterations)
    torch.cuda.synchronize()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    G.d_ReconstructGridding(acc_ft, acc_w, out, (n,) * 3, (D,) * 3, PAD, 0, 0, iterations)
    b.record()
    torch.cuda.synchronize()
    print(json.dumps({"gridding_profile": {"P": n * PAD, "iterations": iterations,
                                           "ms": round(a.elapsed_time(b), 3),
                                           "finite": bool(torch.isfinite(out).all().item())}}))


def main():
    args = parse_args()
    if args.sweep:
        run_sweep(args)
        return
    if args.config5:
        run_config5(args)
        return
    if args.gridding_profile >= 0:
        run_gridding_profile(args.gridding_profile)
        return
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
