#!/usr/bin/env python
"""Benchmark: fused BCLP iterations/s at 256^3 x 360 angles with absorption.

One step = one BCLP iteration (vamtoolbox/optimizer/BCLP.py:277-534) on the
3-D parallel-beam absorbing target (seeded union of ellipsoids / cylinders in
a radius-120 vial, 256^3 float32, 360 angles over [0, 360), radial
absorption mask with e^-1 transmission across the container): reference-parity
backprojection, fused dose pass, forward projection, clamped update, all on
the device, replayed from one CUDA graph.  With N GPUs every rank owns a
256-slice z-slab of a 256 x 256 x 256N target (weak scaling); slices are
independent in both projectors, so the only exchange is an all-reduce of the
9 loss / norm sums per iteration.

Reported beside the headline:
  e2e         the same iteration driven with host buffers: every step's g comes from
              pinned host memory (copied while the previous step computes) and the
              step's loss sums go back to pinned host memory;
  plain       the reference's numpy loop calling the projector per step with host
              arrays (engine="host"), the plain per-call GPU path;
  fwd_adj     forward + reference-parity backprojection pairs per second;
  roofline    of the dominant kernel of the step (the projector with the larger share of the
              measured kernel time), HBM bytes it must move, and the bytes it loads on chip;
  cpu_baseline the reference's algorithm (oracle/vamoracle.c, OpenMP) on a bounded
              z-slab sample on this host's cores, extrapolated to the full volume.
`--impl reference` prints the CPU reference arm's line instead.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "BCLP iter/s & fwd+adj proj/s, 256³×360 ang: fused vs plain GPU, relL2≤1e-4"
UNIT = "iter/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--size", type=int, default=256)
    ap.add_argument("--angles", type=int, default=360)
    ap.add_argument("--plain-steps", type=int, default=2)
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-autotune", action="store_true")
    ap.add_argument("--no-multi", action="store_true", help="skip the 16-target batched BCLP measurement")
    ap.add_argument("--no-ray", action="store_true", help="skip the ray-tracer BCLP measurement")
    ap.add_argument("--no-configs", action="store_true", help="skip the 2-D CAL / OSMO / grayscale BCLP legs")
    ap.add_argument("--no-algebraic", action="store_true", help="skip the propagation-matrix / SpMV leg")
    ap.add_argument("--no-formats", action="store_true", help="skip the projector-frame / fan-beam rebin leg")
    ap.add_argument("--no-vec", action="store_true", help="skip the vector-geometry (inclined rays) projector leg")
    ap.add_argument("--ray-size", type=int, default=128)
    ap.add_argument("--e2e-iters", type=int, default=40, help="iterations of the timed optimize() call (e2e)")
    ap.add_argument("--dist-backend", default="nccl", choices=["nccl", "gloo"],
                    help="process-group backend of a multi-rank run (gloo: host collectives, e.g. to run the "
                         "multi-rank control flow with several ranks on one device)")
    return ap.parse_args()


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


# ---------------------------------------------------------------------------
# workload
# ---------------------------------------------------------------------------
PIXEL_CM = 0.002          # 500 voxels / cm


def build_problem(n, n_angles, seed):
    from vamtoolbox_b200 import geometry, synthetic

    target = synthetic.ellipsoids_3d(n, seed=seed, radius=120.0 * n / 256)
    angles = np.linspace(0, 360, n_angles, endpoint=False)
    R = n / 2 * PIXEL_CM                       # container radius = grid radius
    alpha = 1.0 / (2 * R)                      # e^-1 transmission across the diameter
    tg = geometry.TargetGeometry(target=target)
    pg = geometry.ProjectionGeometry(angles, "parallel", CUDA=True, projector_pixel_size=PIXEL_CM,
                                     absorption_coeff=alpha, container_radius=R)
    pg.calcAbsorptionMask(tg)
    return tg, pg


def workload_name(n, n_angles):
    """The workload string both bench arms print."""
    return f"BCLP iteration, parallel beam, {n}^3 x {n_angles} angles, radial absorption mask e^-1"


def bclp_options(n_iter):
    from vamtoolbox_b200.optimize import Options

    return Options(method="BCLP", n_iter=n_iter, p=2, q=1, eps=0.1, learning_rate=1e-5, filter="ram-lak")


def strip_pixels(n, angles, bins=2):
    """Image pixels that the forward's strips of ``bins`` detector bins touch, per lattice sample: the distinct
    taps of a strip over its samples (each is loaded once), averaged over a few of the angles."""
    c0 = n // 2
    j, k = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    total = samples = 0
    for th in np.deg2rad(angles[:: max(len(angles) // 16, 1)]):
        row = np.cos(th) * (k - c0) - np.sin(th) * (j - c0) + c0
        col = np.sin(th) * (k - c0) + np.cos(th) * (j - c0) + c0
        r0, q0 = np.floor(row).astype(np.int64), np.floor(col).astype(np.int64)
        keys = []
        for t in range(4):
            r, q = r0 + (t >> 1), q0 + (t & 1)
            ok = (r >= 0) & (r < n) & (q >= 0) & (q < n)
            keys.append((((j // bins) * n + r) * n + q)[ok])
        total += np.unique(np.concatenate(keys)).size
        samples += n * n
    return total / samples


def block_rows(n, angles, inside):
    """Detector rows that a 2 x 2 pixel block's interpolation reads per angle (each loaded once by the block-table
    kernel), summed over the blocks that have a pixel inside the clip circle, averaged over a few of the angles."""
    m = n + n % 2
    x, y = np.meshgrid(np.arange(m) - n // 2, n // 2 - np.arange(m))
    use = np.zeros((m, m), bool)
    use[:n, :n] = inside
    quads = lambda v: v.reshape(m // 2, 2, m // 2, 2).transpose(0, 2, 1, 3).reshape(-1, 4)
    total = count = 0
    for th in np.deg2rad(angles[:: max(len(angles) // 16, 1)]):
        b = quads(np.floor(x * np.cos(th) - y * np.sin(th)).astype(np.int64))
        u = quads(use)
        rows = np.sort(np.concatenate([np.where(u, b, 1 << 40), np.where(u, b + 1, 1 << 40)], axis=1), axis=1)
        new = np.concatenate([np.ones((len(rows), 1), bool), np.diff(rows, axis=1) > 0], axis=1)
        total += int((new & (rows < 1 << 40)).sum())
        count += 1
    return total / count


def count_angle_pairs(angles):
    """Pairs (a, a + 180 deg) the forward kernel samples from one lattice (same rule as the plan)."""
    used = np.zeros(len(angles), bool)
    pairs = 0
    for i in range(len(angles)):
        if used[i]:
            continue
        used[i] = True
        for k in range(i + 1, len(angles)):
            if used[k]:
                continue
            d = np.fmod(angles[k] - angles[i] - 180.0, 360.0)
            d = d + 360.0 if d < 0 else d
            if d < 1e-9 or 360.0 - d < 1e-9:
                used[k] = True
                pairs += 1
                break
    return pairs


# ---------------------------------------------------------------------------
# clocks
# ---------------------------------------------------------------------------
class ClockSampler:
    """SM clock and clock-event reasons sampled every 10 ms from a host thread (NVML, read only),
    started before the timed region; falls back to ``nvidia-smi -lms 100``."""

    _REASONS = {"hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40,
                "sw_power_cap": 0x4}

    def __init__(self, index):
        self.rows, self.proc, self.thread = [], None, None
        self._stop = threading.Event()
        try:
            import pynvml

            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = self._handle(pynvml, index)
            self.thread = threading.Thread(target=self._loop, daemon=True)
            self.thread.start()
            t0 = time.perf_counter()
            while not self.rows and time.perf_counter() - t0 < 1.0:
                time.sleep(0.002)
            return
        except Exception:
            self.thread = None
        self.path = Path(tempfile.mkstemp(suffix=".csv")[1])
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={index}", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                                          "-lms", "100"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    @staticmethod
    def _handle(pynvml, index):
        import torch

        try:
            pr = torch.cuda.get_device_properties(index)
            bus = f"{pr.pci_domain_id:08X}:{pr.pci_bus_id:02X}:{pr.pci_device_id:02X}.0"
            return pynvml.nvmlDeviceGetHandleByPciBusId(bus)
        except Exception:
            vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
            ids = [v for v in vis.split(",") if v.strip().isdigit()]
            return pynvml.nvmlDeviceGetHandleByIndex(int(ids[index]) if index < len(ids) else index)

    def _loop(self):
        nv, h = self.nv, self.h
        get_reasons = getattr(nv, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
            nv.nvmlDeviceGetCurrentClocksThrottleReasons
        mx = nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM)
        while not self._stop.is_set():
            try:
                self.rows.append((nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM), mx, int(get_reasons(h))))
            except Exception:
                break
            time.sleep(0.01)

    def stop(self):
        if self.thread is not None:
            self._stop.set()
            self.thread.join(timeout=2)
            rows = list(self.rows)
            if not rows:
                return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"], "source": "nvml"}
            reasons = sorted({k for r in rows for k, bit in self._REASONS.items() if r[2] & bit})
            return {"sm_mhz": statistics.median(r[0] for r in rows), "sm_max_mhz": max(r[1] for r in rows),
                    "reasons": reasons, "samples": len(rows), "source": "nvml, 10 ms"}
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        rows = []
        for line in self.path.read_text().splitlines():
            p = [x.strip() for x in line.split(",")]
            if len(p) >= 9:
                rows.append(p)
        self.path.unlink(missing_ok=True)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows), "source": "nvidia-smi, 100 ms"}


# ---------------------------------------------------------------------------
# CPU reference algorithm (oracle): timed baseline and parity at the timed size
# ---------------------------------------------------------------------------
def rel_l2(a, b):
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def rel_err(a, b):
    return float(abs(float(a) - float(b)) / max(abs(float(b)), 1e-300))


def cpu_bclp_sample(tg, pg, g0, opts, n_slices, steps=1):
    """Time `steps` BCLP iterations of the reference's algorithm on n_slices z-slices."""
    from oracle import oracle as O

    rm = opts.response_model
    f_T = np.asarray(tg.array[:, :, :n_slices], dtype=np.float64)
    g = np.asarray(g0[:, :, :n_slices], dtype=np.float64).copy()
    mask = np.asarray(pg.absorption_mask)[:, :, 0]
    ang = np.asarray(pg.angles, dtype=np.float64)
    absn = ("mask", mask)
    t0 = time.perf_counter()
    for _ in range(steps):
        dose = O.parallel_backward_ref(g, ang, absorption=absn)
        mapped = rm.map(dose)
        e = mapped - f_T
        eb = np.abs(e) - opts.eps
        v = eb > 0
        loss = np.sum(v * opts.weight * np.abs(eb) ** opts.p) ** (opts.q / opts.p)
        operand = v * opts.weight * np.abs(eb) ** (opts.p - 1) * np.sign(e) * rm.dmapdf(dose)
        fwd = O.parallel_forward(operand, ang, absorption=absn)
        grad = (opts.q * loss ** ((opts.q - opts.p) / opts.q)) * fwd if loss != 0 else fwd
        g = np.clip(g - opts.learning_rate * grad, opts.blb, opts.bub)
    return (time.perf_counter() - t0) / steps


def device_bclp_step(it):
    """One eager BCLP iteration of the device engine from its current g; returns host float64 copies of
    the input g and of every product of the step (dose, mapped dose, forward of the operand, the 9 loss /
    norm sums, updated g)."""
    import torch

    g_in = it.g.double().cpu().numpy()
    it.step()
    torch.cuda.synchronize(it.device)
    h = lambda t: t.double().cpu().numpy()
    return {"g": g_in, "dose": h(it.dose), "mapped": h(it.mapped), "fwd": h(it.grad), "stats": h(it.stats),
            "g_new": h(it.g)}


def bclp_parity(dev_out, ref):
    """relL2 of the device iteration's products against the float64 oracle's, same input g."""
    st, rs = dev_out["stats"], ref["stats"]
    return {"dose": rel_l2(dev_out["dose"], ref["dose"]), "mapped_dose": rel_l2(dev_out["mapped"], ref["mapped"]),
            "forward_of_operand": rel_l2(dev_out["fwd"], ref["fwd"]), "g_new": rel_l2(dev_out["g_new"], ref["g_new"]),
            "loss_sum": rel_err(st[0], rs[0]), "l1_norm": rel_err(st[3], rs[3]), "linf_norm": rel_err(st[7], rs[7])}


def oracle_bclp_iteration(tg, pg, opts, g):
    """The float64 oracle's BCLP iteration (whole volume, all angles) from sinogram g, and its time."""
    from oracle import iterations as OI

    rm = opts.response_model
    tables = (rm.interp_f_0, rm.interp_map_0, rm.interp_dmapdf_0)
    mask = np.atleast_3d(np.asarray(pg.absorption_mask))[:, :, 0] if pg.absorption_mask is not None else None
    t0 = time.perf_counter()
    ref = OI.bclp_iteration(g, np.asarray(tg.array, np.float64), np.asarray(pg.angles, np.float64), mask, tables,
                            opts.eps, opts.weight, opts.p, opts.q, opts.learning_rate, opts.blb, opts.bub)
    return ref, time.perf_counter() - t0


def cpu_baseline_and_parity(it, tg, pg, opts):
    """One full BCLP iteration of the reference's algorithm (float64 C oracle, OpenMP on all host
    threads) from the device engine's current sinogram: its time is the CPU baseline (no extrapolation:
    every z-slice and angle), its products are the parity reference for the device iteration run from
    the same sinogram."""
    from oracle import oracle as O

    dev_out = device_bclp_step(it)
    ref, t = oracle_bclp_iteration(tg, pg, opts, dev_out["g"])
    cores = O.num_threads()
    n = tg.array.shape
    cpu = {"value": 1.0 / t, "unit": UNIT, "cores": cores, "kind": "port",
           "sample": f"1 BCLP iteration over the whole {n[0]}x{n[1]}x{n[2]} volume x {pg.n_angles} angles "
                     f"(float64 C oracle, OpenMP {cores} threads), {t:.2f} s measured, not extrapolated"}
    par = {"reference": "float64 oracle (restated reference projectors + numpy BCLP body), same input g",
           "workload": f"one BCLP iteration, {n[0]}^3 x {pg.n_angles} angles, radial absorption mask, whole volume",
           "relL2": bclp_parity(dev_out, ref), "tolerance": {"projector products": 1e-5, "optimizer state": 1e-4}}
    return cpu, par


# ---------------------------------------------------------------------------
# our arm
# ---------------------------------------------------------------------------
def multi_target_problems(seed=5, n_iter=25):
    """16 targets of uneven size: 8 2-D slices from {128, 256, 384, 512}^2 and 8 volumes from
    {64, 96, 128, 160}^3, angle counts from {180, 360, 720}, per-target absorption between 0 and
    e^-1 transmission across the container, binary or 3-level grayscale, BCLP options per target."""
    from vamtoolbox_b200 import geometry, synthetic
    from vamtoolbox_b200.optimize import Options

    rng = np.random.default_rng(seed)
    probs, desc = [], []
    for k in range(16):
        two_d = k < 8
        n = int(rng.choice([128, 256, 384, 512] if two_d else [64, 96, 128, 160]))
        na = int(rng.choice([180, 360, 720]))
        R = n / 2 * PIXEL_CM
        alpha = float(rng.uniform(0.0, 1.0 / (2 * R)))
        gray = bool(rng.uniform() < 0.5)
        if two_d:
            t = synthetic.ellipses_2d(n, seed=100 + k, radius=0.45 * n)
        else:
            t = synthetic.ellipsoids_3d(n, seed=100 + k, radius=0.45 * n)
        if gray:  # 3-level grayscale: the binary target with an inner shell at one half
            t = np.where(t > 0, np.where(np.roll(t, 3, axis=0) > 0, 1.0, 0.5), 0.0)
        tg = geometry.TargetGeometry(target=t)
        pg = geometry.ProjectionGeometry(np.linspace(0, 360, na, endpoint=False), "parallel", CUDA=True,
                                         projector_pixel_size=PIXEL_CM, absorption_coeff=alpha,
                                         container_radius=R)
        pg.calcAbsorptionMask(tg)
        opts = Options(method="BCLP", n_iter=n_iter, p=2, q=1, eps=0.1, learning_rate=1e-5)
        probs.append((tg, pg, opts))
        desc.append(f"{n}^{2 if two_d else 3}x{na}{'g' if gray else 'b'}")
    return probs, desc


def run_multi_target(dev, n_iter=25, parity=True):
    """Aggregate BCLP iter/s of 16 uneven targets, four ways, each a captured graph replayed n_iter
    times after 3 warm-up replays: all targets per iteration in two persistent work-queue batches
    (vam_batch_submit; all backprojections, then all forwards), the same with the targets in two halves
    half an iteration apart (each batch mixes one half's backprojections with the other's forwards),
    every target's chain on its own stream in one graph, and each target's own graph replayed on its
    own, one target after another."""
    import torch

    from vamtoolbox_b200.fused import graph_kernel_nodes
    from vamtoolbox_b200.optimizer.multi import MultiTargetBCLP

    probs, desc = multi_target_problems(n_iter=n_iter)
    multi = MultiTargetBCLP(probs, schedule="persistent")
    for s_ in multi.solvers:
        s_.P.plan.autotune(use_cache=False, ops=("forward", "backward"))
    st = torch.cuda.current_stream(dev)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def timed(replays):
        for r in replays:
            for _ in range(3):
                r()
        torch.cuda.synchronize(dev)
        e0.record(st)
        for r in replays:
            for _ in range(n_iter):
                r()
        e1.record(st)
        torch.cuda.synchronize(dev)
        return e0.elapsed_time(e1)

    out = {"targets": desc, "iterations_each": n_iter,
           "metric": "aggregate BCLP iterations/s over 16 uneven targets (target-iterations per second)"}
    total = len(probs) * n_iter
    launches = {}
    for sched in ("persistent", "streams", "phased"):
        multi.schedule = sched
        g = multi.capture()
        launches[sched] = graph_kernel_nodes(g)
        t = timed([g.replay])
        del g
        out[f"{sched}_iter_s"] = round(total / (t / 1e3), 2)
        out[f"{sched}_ms_per_iteration_of_all"] = round(t / n_iter, 4)
    graphs = [it.capture() for it in multi.its]
    launches["one_at_a_time"] = sum(graph_kernel_nodes(gr) or 0 for gr in graphs)
    t_seq = timed([gr.replay for gr in graphs])
    del graphs
    out["one_at_a_time_iter_s"] = round(total / (t_seq / 1e3), 2)
    for sched in ("persistent", "streams", "phased"):
        out[f"speedup_{sched}"] = round(out[f"{sched}_iter_s"] / out["one_at_a_time_iter_s"], 3)
    out["launches_per_iteration"] = launches
    if parity:
        out["parity"] = multi_target_parity(multi, probs, desc)
    return out


def multi_target_parity(multi, probs, desc, n_check=2):
    """Every schedule's sinograms after n_check captured iterations from one saved start against each
    target's own graph replayed alone (bit for bit), and one iteration of the largest slice and of the
    smallest volume against the float64 oracle from the same sinogram (whole target, all angles)."""
    import torch

    saved = [it.g.clone() for it in multi.its]
    got = {}
    for sched in ("persistent", "streams", "phased"):
        multi.schedule = sched
        multi.reset(saved)
        g = multi.capture()
        for _ in range(n_check):
            g.replay()
        torch.cuda.synchronize(multi.device)
        del g
        got[sched] = [it.g.clone() for it in multi.its]
    multi.reset(saved)
    graphs = [it.capture() for it in multi.its]
    for gr in graphs:
        for _ in range(n_check):
            gr.replay()
    torch.cuda.synchronize(multi.device)
    del graphs
    alone = [it.g.clone() for it in multi.its]
    out = {"bitwise_equal_to_one_at_a_time": {s: all(torch.equal(a, b) for a, b in zip(v, alone))
                                              for s, v in got.items()},
           "iterations_compared": n_check}
    cost = [float(np.asarray(tg.array).size) * pg.n_angles for tg, pg, _ in probs]
    two_d = [k for k, d in enumerate(desc) if "^2x" in d]
    three_d = [k for k, d in enumerate(desc) if "^3x" in d]
    picks = [max(two_d, key=lambda k: cost[k]), min(three_d, key=lambda k: cost[k])]
    for k in picks:
        tg, pg, opts = probs[k]
        dev_out = device_bclp_step(multi.its[k])
        ref, t = oracle_bclp_iteration(tg, pg, opts, dev_out["g"])
        out[desc[k]] = {"oracle_s": round(t, 2), "relL2": bclp_parity(dev_out, ref)}
    out["reference"] = "float64 oracle, one BCLP iteration from the same g, whole target"
    return out


def ray_problem(n, n_angles, seed=0):
    """Ray-tracer workload: n^3 graded-index medium n = 1.50 + 0.02 (r/R)^2 + a smooth perturbation
    (central-difference gradient), smooth attenuation with e^-1 transmission across the grid, physical
    path length + forward symplectic Euler at h = voxel / 2, parallel rays (n detector x n_angles x n z),
    a seeded random-ellipsoid target."""
    import torch

    from vamtoolbox_b200 import geometry, medium, synthetic

    tg = geometry.TargetGeometry(target=synthetic.ellipsoids_3d(n, seed=seed, radius=0.45 * n))
    cv = tg.constructCoordVec()
    a0 = 1.0 / (n * (cv[0][1] - cv[0][0]))
    nx = synthetic.graded_index(cv, seed=seed)
    ax = synthetic.smooth_attenuation(cv, a0, seed=seed)
    im = medium.IndexModel(cv, type="interpolation", form="freeform", n_x=torch.as_tensor(nx))
    am = medium.AttenuationModel(cv, type="interpolation", form="freeform", alpha_x=torch.as_tensor(ax))
    pg = geometry.ProjectionGeometry(np.linspace(0, 360, n_angles, endpoint=False), "ray_trace", CUDA=True,
                                     index_model=im, attenuation_model=am, absorption_model=am,
                                     ray_trace_method="eikonal", eikonal_parametrization="physical_path_length",
                                     ray_trace_ode_solver="forward_symplectic_euler", ray_trace_ray_config="parallel",
                                     inclination_angle=0.0, ray_density=1)
    return tg, pg, cv, nx, ax


def ray_cpu_sample(cv, nx, ax, n_angles, budget_s=6.0):
    """The float64 C oracle of the reference's tracer (integrate + deposit, all host threads) on a
    few angles' rays, extrapolated to all angles (every angle traces the same number of rays)."""
    from oracle import oracle as O

    xv, yv, zv = cv
    h = (xv[1] - xv[0]) / 2
    kw = dict(step_size=h, max_num_step=3 * xv.size, n_kind=1, n_grid=nx, a_kind=3, a_grid=ax, absorb=ax)
    grid = dict(xv=xv, yv=yv, zv=zv)
    rng = np.random.default_rng(0)
    f = rng.uniform(0, 1, (xv.size, yv.size, zv.size))
    k = 1
    while True:
        ang = np.linspace(0, 360, n_angles, endpoint=False)[:k]
        x0, v0, _ = O.setup_rays_parallel(xv, yv, zv, ang)
        t0 = time.perf_counter()
        g, _ = O.ray_trace("integrate", grid, x0, v0, 1.0, f=f, **kw)
        O.ray_trace("deposit", grid, x0, v0, 1.0, g=rng.uniform(0, 1, g.shape), **kw)
        t = time.perf_counter() - t0
        if t > budget_s / 4 or k >= n_angles:
            break
        k = min(n_angles, k * 4)
    per_iter = t * n_angles / k
    return {"value": round(1.0 / per_iter, 6), "unit": "iter/s", "cores": O.num_threads(), "kind": "port",
            "sample": f"{k} of {n_angles} angles ({x0.shape[0]} rays), integrate + deposit in the float64 C "
                      f"oracle, extrapolated over angles ({t:.2f} s measured)"}


def run_ray_bclp(dev, n=128, n_angles=360, steps=5, warmup=2, cpu=True):
    """BCLP iterations/s through the ray tracer (deposit -> fused dose pass -> integrate -> update, one
    captured graph), with the kernels' own times and the CPU oracle beside it."""
    import torch

    from vamtoolbox_b200.fused import graph_kernel_nodes
    from vamtoolbox_b200.optimize import Options
    from vamtoolbox_b200.optimizer.BCLP import BCLPNorm

    tg, pg, cv, nx, ax = ray_problem(n, n_angles)
    opts = Options(method="BCLP", n_iter=steps + warmup + 2, p=2, q=1, eps=0.1, learning_rate=1e-5)
    bclp = BCLPNorm(tg, pg, opts)
    it = bclp.device_iteration()
    g = it.capture()
    st = torch.cuda.current_stream(dev)
    for _ in range(warmup):
        g.replay()
    torch.cuda.synchronize(dev)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(st)
    for _ in range(steps):
        g.replay()
    e1.record(st)
    torch.cuda.synchronize(dev)
    ms = e0.elapsed_time(e1) / steps
    launches = graph_kernel_nodes(g)
    del g
    kt = {}
    for name, fn in (("deposit", lambda: it.back(it.g, it.dose)), ("integrate", lambda: it.fwd(it.operand, it.grad))):
        fn()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(st)
        fn()
        b.record(st)
        torch.cuda.synchronize(dev)
        kt[name] = round(a.elapsed_time(b), 3)
    plan = bclp.P.plan
    rays = int(plan.num_rays)
    cap = int(plan.max_num_step) if hasattr(plan, "max_num_step") else 3 * n
    cache = None
    if getattr(plan, "has_trajectories", False):
        # the same kernels tracing every call (the cache dropped), and the one-time trace that fills it
        active_cached = int(plan.active_at_cap())
        plan.drop_trajectories()
        traced = {}
        for name, fn in (("deposit", lambda: it.back(it.g, it.dose)), ("integrate", lambda: it.fwd(it.operand, it.grad))):
            fn()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(st)
            fn()
            b.record(st)
            torch.cuda.synchronize(dev)
            traced[name] = round(a.elapsed_time(b), 3)
        torch.cuda.synchronize(dev)
        t0 = time.perf_counter()
        plan.prepare_trajectories()
        torch.cuda.synchronize(dev)
        cache = {"bytes": int(plan.trajectory_bytes(plan.cached_rays)), "rays_cached": int(plan.cached_rays),
                 "prepare_ms": round((time.perf_counter() - t0) * 1e3, 2),
                 "kernel_ms_traced": traced, "rays_active_at_cap_cached": active_cached,
                 "what": "ray paths traced once per medium (position and attenuance per step, 16 B per ray-step); "
                         "integrate / deposit stream them (integrate bit-identical, deposit equal up to atomic "
                         "order)"}
    out = {"workload": f"BCLP iteration through the ray tracer, {n}^3 graded-index medium, {n_angles} angles, "
                       f"{rays} rays, step cap {cap}",
           "bclp_iter_s": round(1000.0 / ms, 3), "ms_per_iteration": round(ms, 3), "kernel_ms": kt,
           "ray_steps_per_s": round(rays * cap / (kt["integrate"] * 1e-3), 1),
           "rays_active_at_cap": int(plan.active_at_cap()), "launches_per_iteration": launches,
           "trajectory_cache": cache}
    if cpu:
        try:
            out["cpu_baseline"] = ray_cpu_sample(cv, nx, ax, n_angles)
        except Exception as exc:
            out["cpu_baseline"] = {"error": f"{type(exc).__name__}: {exc}"}
        try:
            out["parity"] = ray_chunk_parity(plan, cv, nx, ax, np.linspace(0, 360, n_angles, endpoint=False))
        except Exception as exc:
            out["parity"] = {"error": f"{type(exc).__name__}: {exc}"}
    return out


def ray_chunk_parity(plan, cv, nx, ax, angles, first=0, count=16, seed=11):
    """Integrate and deposit at the full workload size against the float64 oracle tracer on one block of
    `count` angles: the device traces every ray (integrate of a seeded field; deposit of seeded energies
    on the block's rays, zero elsewhere), the oracle traces the block's rays."""
    import torch

    from oracle import iterations as OI

    n0, na, nz = plan.sino_shape
    rng = np.random.default_rng(seed)
    f = rng.uniform(0.0, 1.0, plan.grid_shape)
    g_rows = rng.uniform(0.0, 1.0, (n0, count, nz)).astype(np.float32)
    g_all = np.zeros((n0, na, nz), np.float32)
    g_all[:, first:first + count] = g_rows
    dev = plan.device
    integral = plan.integrate(torch.as_tensor(f, dtype=torch.float32, device=dev)).reshape(n0, na, nz)
    dose = plan.deposit(torch.as_tensor(g_all, device=dev))
    torch.cuda.synchronize(dev)
    t0 = time.perf_counter()
    ri, rd, act = OI.ray_chunk(cv, nx, ax, angles, first, count, f, g_rows, plan.step_size, plan.max_num_step)
    t = time.perf_counter() - t0
    return {"reference": "float64 oracle tracer (float32 ray state, as the reference), one block of angles",
            "sample": f"angles {first}..{first + count - 1} of {na} ({n0 * count * nz} rays), step cap "
                      f"{plan.max_num_step}", "oracle_s": round(t, 2),
            "relL2": {"integrate": rel_l2(integral[:, first:first + count].double().cpu().numpy(), ri),
                      "deposit": rel_l2(dose.double().cpu().numpy(), rd)},
            "tolerance": 1e-4, "oracle_rays_active_at_cap": int(act)}


def time_optimize_e2e(n, n_angles, n_iter=40, seed=1000):
    """The headline workload through the public call a user makes: optimize(target_geo, proj_geo,
    Options(method="BCLP", n_iter)) on numpy inputs, returning numpy outputs (sinogram, dose, loss log).
    One untimed call warms the plan, cuFFT and allocator caches; the second call is timed on the wall
    clock between two device synchronisations (projector plan, absorption mask upload, device set-up of
    g0, the captured iterations and the float64 downloads all inside)."""
    import torch

    from vamtoolbox_b200 import optimize as vopt

    out = None
    for _ in range(2):
        tg, pg = build_problem(n, n_angles, seed=seed)
        opts = bclp_options(n_iter)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        sino, recon, loss = vopt.optimize(tg, pg, opts)
        torch.cuda.synchronize()
        t = time.perf_counter() - t0
        assert isinstance(sino.array, np.ndarray) and isinstance(recon.array, np.ndarray)
        out = {"call_s": t, "device_ms_per_iteration": getattr(opts, "device_iteration_ms", None),
               "h2d": int(np.asarray(tg.array).size * 8), "d2h": int(sino.array.nbytes + recon.array.nbytes),
               "finite": bool(np.isfinite(sino.array).all() and np.isfinite(recon.array).all())}
        del sino, recon, loss  # a caller done with one result before the next call
    out["n_iter"] = n_iter
    return out


def e2e_line(opt, replay, device_value):
    """The contract's e2e object: the whole optimize() call (iterations per second of the call, set-up
    and transfers included) when it was measured, else the graph replay with per-step host copies."""
    if not opt or "call_s" not in opt:
        line = dict(replay)
        if opt:
            line["optimize"] = opt
        return line
    n = opt["n_iter"]
    return {"value": round(n / opt["call_s"], 4), "unit": UNIT, "h2d_bytes_per_step": opt["h2d"] / n,
            "d2h_bytes_per_step": opt["d2h"] / n,
            "path": f"vamtoolbox_b200.optimize.optimize(target_geo, proj_geo, Options(method='BCLP', n_iter={n})): "
                    "numpy float64 target in; numpy float64 sinogram, dose and loss log out; one call timed whole",
            "n_iter": n, "call_s": round(opt["call_s"], 5),
            "device_ms_per_iteration": round(opt["device_ms_per_iteration"], 4) if opt["device_ms_per_iteration"] else None,
            "fraction_of_device_loop": round(n / opt["call_s"] / device_value, 4), "outputs_finite": opt["finite"],
            "graph_replay": replay}


def _time_optimize(make, n_iter):
    """The public optimize() call: its wall-clock seconds (synchronised, setup and host copies included)
    and the device engine's own per-iteration time (CUDA events around its iteration loop)."""
    import torch

    from vamtoolbox_b200 import optimize as vopt

    best = None
    for _ in range(2):  # the first call warms caches and allocators
        tg, pg, opts = make(n_iter)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        vopt.optimize(tg, pg, opts)
        torch.cuda.synchronize()
        best = (time.perf_counter() - t0, getattr(opts, "device_iteration_ms", None))
    t, ms = best
    return {"n_iter": n_iter, "optimize_call_s": round(t, 4), "device_ms_per_iteration": round(ms, 4) if ms else None,
            "iter_s": round(1000.0 / ms, 3) if ms else None}


def config_cal_2d(n_iter):
    """2-D CAL: a 256^2 ellipse target zero-padded to 363^2 (the 363-bin detector), 360 angles, lr 0.4,
    d_h 0.5."""
    from vamtoolbox_b200 import geometry, synthetic
    from vamtoolbox_b200.optimize import Options

    t = synthetic.ellipses_2d(256, seed=1)
    t = np.pad(t, ((53, 54), (53, 54)))
    tg = geometry.TargetGeometry(target=t)
    pg = geometry.ProjectionGeometry(np.linspace(0, 360, 360, endpoint=False), "parallel", CUDA=True)
    return tg, pg, Options(method="CAL", n_iter=n_iter, learning_rate=0.4, d_h=0.5)


def config_osmo(n_iter):
    """OSMO at 256^3 x 360 angles with e^-1 radial absorption."""
    from vamtoolbox_b200.optimize import Options

    tg, pg = build_problem(256, 360, seed=2)
    return tg, pg, Options(method="OSMO", n_iter=n_iter)


def config_gray_bclp(n_iter, p=2, n=192, n_angles=720):
    """Grayscale BCLP: 192^3 smoothed-noise 3-level target with a ramp, 720 angles, generalised-logistic
    response table (M 0.6, B 12), eps 0.05, weights 1 inside / 0.5 outside, Lp norm p, q 1."""
    from vamtoolbox_b200 import geometry, response, synthetic
    from vamtoolbox_b200.optimize import Options

    t = synthetic.grayscale_3d(n, seed=3)
    tg = geometry.TargetGeometry(target=t)
    pg = geometry.ProjectionGeometry(np.linspace(0, 360, n_angles, endpoint=False), "parallel", CUDA=True)
    rm = response.ResponseModel(type="interpolation", form="gen_log_fun", M=0.6, B=12)
    w = np.where(t > 0, 1.0, 0.5)
    return tg, pg, Options(method="BCLP", n_iter=n_iter, response_model=rm, eps=0.05, weight=w, p=p, q=1,
                           learning_rate=1e-3)


def cal_parity(tg, pg, opts):
    """One CAL iteration of the device engine against the float64 oracle's from the same state."""
    import torch

    from oracle import iterations as OI
    from vamtoolbox_b200.optimizer.CAL import CALDevice
    from vamtoolbox_b200.projectorconstructor import projectorconstructor

    c = CALDevice(tg, pg, opts, projectorconstructor(tg, pg))
    x0, b0 = c.x.double().cpu().numpy(), c.b.double().cpu().numpy()
    c.step(1)
    torch.cuda.synchronize()
    xd = c.x.double().cpu().numpy()
    xd = xd / xd.max()
    t0 = time.perf_counter()
    xr, br, ver = OI.cal_step(x0, b0, np.atleast_3d(tg.array), np.atleast_3d(tg.gel_inds),
                              np.atleast_3d(tg.void_inds), np.asarray(pg.angles, np.float64), opts.d_h,
                              opts.sigmoid, opts.learning_rate)
    n = np.sum(tg.gel_inds) + np.sum(tg.void_inds)
    return {"reference": "float64 oracle, one CAL iteration from the device state", "oracle_s": round(time.perf_counter() - t0, 2),
            "relL2": {"sinogram": rel_l2(c.b.double().cpu().numpy(), br), "reconstruction": rel_l2(xd, xr)},
            "ver": float(c.ver.item()), "ver_oracle": float(ver),
            "ver_voxels_apart": float(abs(float(c.ver.item()) - ver) * n)}


def osmo_parity(tg, pg, opts):
    """The first OSMO half step (void voxels) of the device engine against the float64 oracle's from the
    same model and reconstruction, whole volume."""
    import torch

    from oracle import iterations as OI
    from vamtoolbox_b200.optimizer.OSMO import OSMODevice
    from vamtoolbox_b200.projectorconstructor import projectorconstructor

    it = OSMODevice(tg, pg, opts, projectorconstructor(tg, pg))
    x0, xm0 = it.x.double().cpu().numpy(), it.xm.double().cpu().numpy()
    it.half(False)
    torch.cuda.synchronize()
    mask = np.asarray(pg.absorption_mask)[:, :, 0] if pg.absorption_mask is not None else None
    t0 = time.perf_counter()
    xr, br, xmr = OI.osmo_half(x0, xm0, tg.gel_inds, tg.void_inds, False, opts.d_l,
                               np.asarray(pg.angles, np.float64), mask, opts.inhibition)
    return {"reference": "float64 oracle, one OSMO half step from the device state, whole volume",
            "oracle_s": round(time.perf_counter() - t0, 2),
            "relL2": {"model": rel_l2(it.xm.double().cpu().numpy(), xmr), "sinogram": rel_l2(it.b.double().cpu().numpy(), br),
                      "reconstruction": rel_l2(it.x.double().cpu().numpy(), xr)}}


def gray_bclp_parity(tg, pg, opts):
    """One grayscale BCLP iteration (response table, weights) of the device engine against the float64
    oracle's from the same sinogram, whole volume."""
    from vamtoolbox_b200.optimizer.BCLP import BCLPNorm

    dev_out = device_bclp_step(BCLPNorm(tg, pg, opts).device_iteration())
    ref, t = oracle_bclp_iteration(tg, pg, opts, dev_out["g"])
    return {"reference": "float64 oracle, one BCLP iteration from the same g, whole volume", "oracle_s": round(t, 2),
            "relL2": bclp_parity(dev_out, ref)}


def run_configs(parity=True):
    """The reference's other headline workloads, each through optimize(target, proj, Options(...)) on
    the device engine: 2-D CAL 256^2 padded to a 363-bin detector with 360 angles; OSMO 256^3 with e^-1
    absorption and 360 angles; grayscale BCLP 192^3 with 720 angles and a generalised-logistic response.
    With parity, each also runs one iteration from the same state on the device and in the float64
    oracle and reports the relL2 of the products."""
    out = {}
    for key, make, n_iter, desc, par in (
            ("cal_2d_256_363x360", config_cal_2d, 20, "2-D CAL, 256^2 target padded to 363^2, 360 angles, lr 0.4, d_h 0.5",
             cal_parity),
            ("osmo_256cube_360_absorbing", config_osmo, 30, "OSMO, 256^3, 360 angles, e^-1 radial absorption", osmo_parity),
            ("bclp_gray_192cube_720", config_gray_bclp, 40, "grayscale BCLP, 192^3, 720 angles, response M 0.6 B 12, eps 0.05, "
                                              "weights 1 / 0.5, p 2, q 1", gray_bclp_parity)):
        try:
            r = _time_optimize(make, n_iter)
            r["workload"] = desc
            out[key] = r
        except Exception as exc:  # report, never fail the headline number on it
            out[key] = {"error": f"{type(exc).__name__}: {exc}"}
            continue
        if parity:
            try:
                r["parity"] = par(*make(n_iter))
            except Exception as exc:  # report, never fail the headline number on it
                r["parity"] = {"error": f"{type(exc).__name__}: {exc}"}
    out["unit"] = "iter/s of the device engine's iteration loop; optimize_call_s is the whole call"
    return out


def run_algebraic(dev, n=128, n_angles=360, reps=5):
    """Algebraic propagation: the ray tracer's propagation matrix of one n^2 slice (n_angles angles) built
    on the device, then applied z-tiled to an n^2 x n volume forward and backward (CSR kernel); beside it
    the reference's CPU path for the same product (a SciPy CSR matrix times the tiled block)."""
    import scipy.sparse
    import torch

    from vamtoolbox_b200 import geometry, medium, synthetic
    from vamtoolbox_b200.projector.pyTorchAlgebraicPropagation import PyTorchAlgebraicPropagator
    from vamtoolbox_b200.projector.pyTorchRayTrace import PyTorchRayTracingPropagator

    tg2 = geometry.TargetGeometry(target=np.zeros((n, n)))
    cv = tg2.constructCoordVec()
    a0 = 1.0 / (n * (cv[0][1] - cv[0][0]))
    im = medium.IndexModel(cv, type="interpolation", form="freeform",
                           n_x=torch.as_tensor(synthetic.graded_index(cv, seed=0)))
    am = medium.AttenuationModel(cv, type="interpolation", form="freeform",
                                 alpha_x=torch.as_tensor(synthetic.smooth_attenuation(cv, a0)))
    pg = geometry.ProjectionGeometry(np.linspace(0, 360, n_angles, endpoint=False), "ray_trace", CUDA=True,
                                     index_model=im, attenuation_model=am, absorption_model=am,
                                     eikonal_parametrization="physical_path_length",
                                     ray_trace_ode_solver="forward_symplectic_euler", ray_trace_ray_config="parallel")
    P = PyTorchRayTracingPropagator(tg2, pg)
    torch.cuda.synchronize(dev)
    t0 = time.perf_counter()
    P.output_torch_tensor = True
    M = P.buildPropagationMatrix()
    torch.cuda.synchronize(dev)
    t_build = time.perf_counter() - t0
    tg3 = geometry.TargetGeometry(target=np.zeros((n, n, n)))
    A = PyTorchAlgebraicPropagator(tg3, None, output_torch_tensor=True, matrix=M)
    x = torch.rand(n * n * n, device=dev)
    b = torch.rand(A.n_row_eff, device=dev)
    st = torch.cuda.current_stream(dev)

    def tim(fn):
        fn()
        torch.cuda.synchronize(dev)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        for _ in range(reps):
            fn()
        e1.record(st)
        torch.cuda.synchronize(dev)
        return e0.elapsed_time(e1) / reps

    t_f, t_b = tim(lambda: A.forward(x)), tim(lambda: A.backward(b))
    nnz = int(M._nnz())
    # compulsory bytes of one product: the matrix once (4 B value + 4 B column + row pointers), x and y
    fwd_bytes = nnz * 8 + (A.n_row_internal + 1) * 8 + 4 * (A.n_col_eff + A.n_row_eff)
    peaks = {}
    try:
        peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
    except Exception:
        pass
    hbm = peaks.get("hbm_gbs") or 6650.0
    idx = M.indices().cpu().numpy()
    S = scipy.sparse.csr_matrix((M.values().cpu().numpy(), (idx[0], idx[1])), shape=tuple(M.shape))
    X = np.random.default_rng(0).uniform(size=(S.shape[1], n)).astype(np.float32)
    t0 = time.perf_counter()
    S @ X
    t_cpu = time.perf_counter() - t0
    bclp = algebraic_bclp(S, n, n_angles)
    return {"workload": f"propagation matrix of one {n}^2 slice x {n_angles} angles, z-tiled over {n} layers",
            "bclp": bclp,
            "nnz": nnz, "matrix_build_s": round(t_build, 4), "forward_ms": round(t_f, 4), "backward_ms": round(t_b, 4),
            "fwd_adj_per_s": round(1000.0 / (t_f + t_b), 3),
            "roofline_forward": {"bound": "hbm", "achieved": round(fwd_bytes / (t_f * 1e-3) / 1e9, 1), "peak": hbm,
                                 "unit": "GB/s", "frac": round(fwd_bytes / (t_f * 1e-3) / 1e9 / hbm, 4),
                                 "algorithmic_bytes": fwd_bytes},
            "cpu_baseline": {"value": round(1000.0 / (t_cpu * 1e3), 4), "unit": "forward products/s",
                             "cores": 1, "kind": "reference",
                             "sample": "the same CSR matrix times the tiled block in SciPy (the reference's CPU "
                                       "algebraic propagation), one product"}}


def algebraic_bclp(S, n, n_angles, n_iter=20, host_iter=2):
    """BCLP through the algebraic propagator (the matrix saved as .npz and named by an algebraic
    projection geometry, as the reference's example does) on an n^3 ellipsoid target: iterations/s of the
    fused device engine (CSR products captured with the dose pass and update) and of the reference's host
    loop (a product and a host round trip per projection), each timed as one optimize() call."""
    import os
    import tempfile

    import scipy.sparse

    from vamtoolbox_b200 import geometry, synthetic
    from vamtoolbox_b200.optimize import Options, optimize

    out = {"workload": f"BCLP, {n}^3 target, {n_angles} angles, algebraic propagator (z-tiled matrix)"}
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "P.npz")
        scipy.sparse.save_npz(path, S)
        for engine, k in (("device", n_iter), ("host", host_iter)):
            tg = geometry.TargetGeometry(target=synthetic.ellipsoids_3d(n, seed=7, radius=0.45 * n))
            pg = geometry.ProjectionGeometry(np.linspace(0, 360, n_angles, endpoint=False), "algebraic", CUDA=False,
                                             loading_path_for_matrix=path)
            opts = Options(method="BCLP", n_iter=k, p=2, q=1, eps=0.1, learning_rate=1e-5, filter=None, engine=engine)
            t0 = time.perf_counter()
            optimize(tg, pg, opts)
            out[f"{engine}_call_s"] = round(time.perf_counter() - t0, 3)
            out[f"{engine}_iterations"] = k
            if engine == "device" and getattr(opts, "device_iteration_ms", None):
                out["device_iter_s"] = round(1000.0 / opts.device_iteration_ms, 2)
    out["host_iter_s_upper_bound"] = round(host_iter / out["host_call_s"], 3)
    return out


def run_formats(dev, n=256, n_angles=360, screen=(1920, 1080), reps=5, cpu=True):
    """Output formats: the n x n_angles x n float64 sinogram of the headline configuration converted to
    n_angles projector frames of screen[0] x screen[1] (99.5th-percentile normalisation, the DLP
    workflow's settings), and rebinned for a fan-beam projector (vial 300 px wide).  Device time with
    the sinogram resident, the frame kernel alone against the HBM roofline, end to end from a host
    array to host images, and the oracle's numpy port of the reference's CPU code beside it."""
    import torch

    from vamtoolbox_b200 import _lib, geometry
    from vamtoolbox_b200 import imagesequence as ims

    rng = np.random.default_rng(3)
    sino = (rng.random((n, n_angles, n)) ** 3 * 40.0)
    sino[: n // 10] = 0.0
    cfg = ims.ImageConfig(screen, normalization_percentile=99.5, invert_u=True)
    st = torch.cuda.current_stream(dev)
    t_dev = torch.from_numpy(sino).to(dev)

    def tim(fn, k=reps):
        fn()
        torch.cuda.synchronize(dev)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        for _ in range(k):
            fn()
        e1.record(st)
        torch.cuda.synchronize(dev)
        return e0.elapsed_time(e1) / k

    t_pipeline = tim(lambda: ims.device_frames(t_dev, cfg))
    frames = ims.device_frames(t_dev, cfg)
    # the percentile select and the frame call alone (blank fill + window gather), through the C ABI
    P = ims._prepare(t_dev, cfg)
    k0, k1, gamma = ims.percentile_ranks(t_dev.numel(), cfg.normalization_percentile, np.dtype(np.float64))
    pair = torch.empty(2, dtype=torch.float64, device=dev)
    wb = _lib.load().vam_select_workspace_bytes()
    work = torch.empty(wb, dtype=torch.uint8, device=dev)
    sel = lambda: _lib.call("vam_select_pair", _lib.ptr(t_dev), _lib.DTYPE_F64, t_dev.numel(), k0, k1,
                            _lib.ptr(pair), _lib.ptr(work), wb, _lib.stream_ptr())
    t_select = tim(sel)
    col, row = ims.placement_tables(cfg, n, n, n, n, True, False)
    prm = P.prm
    prm.n_u, prm.n_v = screen
    prm.box_v0, prm.box_v1, prm.box_u0, prm.box_u1 = ims.table_box(col, row)
    col_d, row_d = torch.from_numpy(col).to(dev), torch.from_numpy(row).to(dev)
    prm.src_col_dev, prm.src_row_dev = col_d.data_ptr(), row_d.data_ptr()
    kern = lambda: _lib.call("vam_imageseq_frames", _lib.ptr(t_dev), _lib.DTYPE_F64, n, n_angles, n,
                             ctypes.byref(prm), _lib.ptr(frames), _lib.stream_ptr())
    t_frames = tim(kern)
    frame_bytes = frames.numel() + t_dev.numel() * 8 + 4 * (screen[0] + screen[1])
    # end to end through ImageSeq: host float64 array in, host images out (page-locked, reused by
    # torch's host caching allocator once a sequence is released)
    ims.ImageSeq(cfg, sino)
    torch.cuda.synchronize(dev)
    t0 = time.perf_counter()
    for _ in range(3):
        seq = ims.ImageSeq(cfg, sino)
        del seq
    torch.cuda.synchronize(dev)
    t_e2e = (time.perf_counter() - t0) / 3
    # fan-beam rebinning of the same sinogram
    pg = geometry.ProjectionGeometry(np.linspace(0, 360, n_angles, endpoint=False))

    def rebin():
        return geometry.rebinFanBeam(geometry.Sinogram(t_dev, pg), 300, screen, 1.5, 1.7)

    t_rebin = tim(rebin, 3)
    peaks = {}
    try:
        peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
    except Exception:
        pass
    hbm = peaks.get("hbm_gbs") or 6650.0
    out = {"workload": f"{n}x{n_angles}x{n} float64 sinogram -> {n_angles} frames {screen[0]}x{screen[1]} uint8, "
                       "99.5th-percentile normalisation; fan-beam rebin to a 300 px vial",
           "frames_per_s_device": round(n_angles / (t_pipeline * 1e-3), 1),
           "pipeline_ms": round(t_pipeline, 4), "select_ms": round(t_select, 4), "frame_kernel_ms": round(t_frames, 4),
           "e2e": {"value": round(n_angles / t_e2e, 1), "unit": "frames/s", "h2d_bytes_per_step": int(sino.nbytes),
                   "d2h_bytes_per_step": int(frames.numel()),
                   "path": "ImageSeq(cfg, numpy sinogram).images"},
           "roofline_frames": {"bound": "hbm", "achieved": round(frame_bytes / (t_frames * 1e-3) / 1e9, 1),
                               "peak": hbm, "unit": "GB/s",
                               "frac": round(frame_bytes / (t_frames * 1e-3) / 1e9 / hbm, 4),
                               "algorithmic_bytes": int(frame_bytes)},
           "rebin_ms": round(t_rebin, 4)}
    if cpu:
        from oracle import formats as ofmt

        t0 = time.perf_counter()
        ofmt.image_frames(sino, ofmt.config(screen[0], screen[1], normalization_percentile=99.5, invert_u=True))
        t_cpu = time.perf_counter() - t0
        nz_s = 16
        t0 = time.perf_counter()
        ofmt.rebin_fan(sino[:, :, :nz_s], pg.angles, 300, screen, 1.5, 1.7)
        t_cpu_rebin = (time.perf_counter() - t0) * n / nz_s
        out["cpu_baseline"] = {"value": round(n_angles / t_cpu, 2), "unit": "frames/s", "cores": 1, "kind": "port",
                               "sample": "the whole sequence through the oracle's numpy port of ImageSeq "
                                         "(percentile, quantise, insert)",
                               "rebin_ms": round(t_cpu_rebin * 1e3, 1),
                               "rebin_sample": f"{nz_s} of {n} z slices through the numpy port of rebinFanBeam, "
                                               "scaled to all slices"}
    return out


def run_vec_geometry(dev, n=256, n_angles=360, incline=15.0, reps=5, cpu=True):
    """Vector-geometry (ASTRA-model) parallel projector, the reference's CUDA path: forward and
    backprojection of an n^3 volume at n_angles angles with vertical rays (slice-exact kernels) and
    rays inclined by `incline` degrees (laminography); the oracle's float64 numpy model beside it on
    a sample of angles."""
    import torch

    from vamtoolbox_b200.projector.Projector3DParallelCUDA import VecPlan, genVectorsAstra, parallel3d_vectors

    ang = np.linspace(0, 360, n_angles, endpoint=False)
    st = torch.cuda.current_stream(dev)
    g = torch.Generator(device=dev).manual_seed(0)
    x = torch.rand((n, n, n), device=dev, generator=g)
    b = torch.rand((n, n_angles, n), device=dev, generator=g)

    def tim(fn):
        fn()
        torch.cuda.synchronize(dev)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        for _ in range(reps):
            fn()
        e1.record(st)
        torch.cuda.synchronize(dev)
        return e0.elapsed_time(e1) / reps

    out = {"workload": f"{n}^3 volume, {n_angles} angles, detector {n} x {n}"}
    for name, vec in (("vertical", parallel3d_vectors(np.deg2rad(ang))), (f"inclined_{incline:g}deg",
                                                                       genVectorsAstra(ang, incline))):
        p = VecPlan(n, n, n, vec, n, n, dev)
        ob, ox = torch.empty_like(b), torch.empty_like(x)
        t_f = tim(lambda: p.forward(x, ob))
        t_b = tim(lambda: p.backward(b, ox))
        taps = 2 if p.info()["flat_forward"] else 4
        out[name] = {"forward_ms": round(t_f, 4), "backward_ms": round(t_b, 4),
                     "fwd_bwd_per_s": round(1000.0 / (t_f + t_b), 2),
                     "forward_taps_GBs": round(4.0 * taps * n * n_angles * n * n / (t_f * 1e-3) / 1e9, 1),
                     "hbm_bytes_per_call": 4 * (n ** 3 + n * n_angles * n)}
        del p
    # 2-D line model (ASTRA "line" projector of the reference's 2-D CUDA class): 512^2 image, 720 angles
    from vamtoolbox_b200.projector.Projector2DParallelCUDA import Line2DPlan

    n2, a2 = 512, 720
    ang2 = np.linspace(0, 180, a2, endpoint=False)
    lp = Line2DPlan(n2, n2, ang2, n2, dev)
    img = torch.rand((n2, n2), device=dev, generator=g)
    s2 = torch.rand((n2, a2), device=dev, generator=g)
    t_lf = tim(lambda: lp.forward(img))
    t_lb = tim(lambda: lp.backward(s2))
    out["line_2d"] = {"workload": f"{n2}^2 image, {a2} angles, {n2} bins", "forward_ms": round(t_lf, 4),
                      "backward_ms": round(t_lb, 4)}
    if cpu:
        from oracle import vecgeom as OV

        t0 = time.perf_counter()
        OV.line2d_forward(img.cpu().double().numpy(), ang2[:1], n2)
        out["line_2d"]["cpu_forward_s"] = round((time.perf_counter() - t0) * a2, 1)
        out["line_2d"]["cpu_sample"] = "1 of 720 angles through the oracle's ray-clipping numpy model, scaled"
    if cpu:
        from oracle import vecgeom as OV

        k = 2
        vol = x.cpu().double().numpy()
        vec = genVectorsAstra(ang[:k], incline)
        t0 = time.perf_counter()
        OV.forward(vol, vec, n, n)
        t_cpu = (time.perf_counter() - t0) * n_angles / k
        out["cpu_baseline"] = {"value": round(1.0 / t_cpu, 5), "unit": "forward projections/s", "cores": 1,
                               "kind": "port", "sample": f"{k} of {n_angles} inclined angles through the oracle's "
                                                         "float64 numpy model, scaled to all angles",
                               "forward_s": round(t_cpu, 2)}
    return out


def run_ours(args):
    import torch

    ws_, rank, local = dist_env()
    local = local % max(torch.cuda.device_count(), 1)  # one rank per device; ranks share devices only if asked
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    dist = None
    if ws_ > 1:
        import datetime

        import torch.distributed as dist

        if args.dist_backend == "nccl":
            dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120), device_id=dev)
        else:
            dist.init_process_group("gloo", timeout=datetime.timedelta(seconds=120))
    from vamtoolbox_b200 import _lib
    from vamtoolbox_b200.optimizer.BCLP import BCLPNorm

    _lib.load()
    n, na = args.size, args.angles
    tg, pg = build_problem(n, na, seed=1000 + rank)
    n_iter = args.warmup + args.steps + 4
    opts = bclp_options(n_iter)
    bclp = BCLPNorm(tg, pg, opts)
    # launch shapes timed once on this device before any timed region (no cache: every run measures)
    tuning = None if args.no_autotune else bclp.P.plan.autotune(use_cache=False)

    reduce_stats = None
    if dist is not None:
        def reduce_stats(stats):
            dist.all_reduce(stats[:7], op=dist.ReduceOp.SUM)
            dist.all_reduce(stats[7:], op=dist.ReduceOp.MAX)

    it = bclp.device_iteration(reduce_stats=reduce_stats)
    st = torch.cuda.current_stream(dev)

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize(dev)

    # ---- fused iteration: graph when single GPU, eager stream-ordered otherwise
    from vamtoolbox_b200.fused import graph_kernel_nodes

    if dist is None:
        graph = it.capture()
        run_step = graph.replay
        launches_per_step = graph_kernel_nodes(graph)
    else:
        graph = None
        run_step = it.step
        probe = bclp.device_iteration().capture()  # same kernels without the all-reduce, never replayed
        launches_per_step = graph_kernel_nodes(probe)
        del probe
    for _ in range(args.warmup):
        run_step()
    barrier()
    clocks = ClockSampler(local)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    torch.cuda.nvtx.range_push("timed")  # lets a profiler restrict its launch list to these steps
    e0.record(st)
    for _ in range(args.steps):
        run_step()
    e1.record(st)
    torch.cuda.nvtx.range_pop()
    barrier()
    clk = clocks.stop()
    ms = e0.elapsed_time(e1) / args.steps
    ms_max = ms
    if dist is not None:
        t = torch.tensor([ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms_max = float(t.item())
    value = ws_ * 1000.0 / ms_max

    # ---- per-kernel timing over an eager pass (same kernels, events on the stream)
    plan = bclp.P.plan
    kt = {"forward": [], "backward_ref": [], "dose_pass+update": []}
    for _ in range(args.steps):
        a, b_, c, d = (torch.cuda.Event(enable_timing=True) for _ in range(4))
        a.record(st)
        it.back(it.g, it.dose)
        b_.record(st)
        it.ws.bclp_dose_pass(it.dose, it.fT, it.prm, it.mapped, it.operand, it.stats)
        c.record(st)
        it.fwd(it.operand, it.grad)
        d.record(st)
        torch.cuda.synchronize(dev)
        kt["backward_ref"].append(a.elapsed_time(b_))
        kt["dose_pass+update"].append(b_.elapsed_time(c))
        kt["forward"].append(c.elapsed_time(d))
    kmean = {k: float(np.mean(v)) for k, v in kt.items()}

    # ---- fwd + adj projection pairs / s
    e2, e3 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e2.record(st)
    for _ in range(args.steps):
        plan.forward(it.operand, it.grad)
        plan.backward_ref(it.g, it.dose)
    e3.record(st)
    torch.cuda.synchronize(dev)
    fwd_adj = 1000.0 / (e2.elapsed_time(e3) / args.steps)
    e2.record(st)
    for _ in range(args.steps):
        plan.forward(it.operand, it.grad)
        plan.adjoint(it.g, it.dose)
    e3.record(st)
    torch.cuda.synchronize(dev)
    fwd_matched = 1000.0 / (e2.elapsed_time(e3) / args.steps)

    # ---- end to end with host buffers (pinned), every step: the step's input sinogram in from the
    # host, the step's result (the 9 loss / norm sums of the iteration) back to the host.  The copy
    # engine brings step k+1's input into a device staging buffer while step k computes (double
    # buffered); each step starts with a device-to-device move of its staged input into the
    # iteration's g.  Every step's input crosses PCIe inside the timed region.
    g_host = it.g.detach().cpu().pin_memory()
    s_out = torch.empty(9, dtype=torch.float32).pin_memory()
    cs = torch.cuda.Stream(dev)
    staging = [torch.empty_like(it.g) for _ in range(2)]
    copied = [torch.cuda.Event() for _ in range(2)]
    consumed = [torch.cuda.Event() for _ in range(2)]

    def stage(k, after=None):
        b = k % 2
        if after is not None:
            cs.wait_event(after)
        cs.wait_event(consumed[b])
        with torch.cuda.stream(cs):
            staging[b].copy_(g_host, non_blocking=True)
            copied[b].record(cs)

    def e2e_steps(n):
        start = torch.cuda.Event()
        start.record(st)
        stage(0, after=start)
        for k in range(n):
            st.wait_event(copied[k % 2])
            it.g.copy_(staging[k % 2])
            consumed[k % 2].record(st)
            if k + 1 < n:
                stage(k + 1)
            run_step()
            s_out.copy_(it.stats, non_blocking=True)

    e2e_steps(2)
    barrier()
    e2.record(st)
    e2e_steps(args.steps)
    e3.record(st)
    barrier()
    e2e_ms = e2.elapsed_time(e3) / args.steps
    if dist is not None:
        t = torch.tensor([e2e_ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_ms = float(t.item())
    h2d = g_host.numel() * 4
    d2h = s_out.numel() * 4
    e2e_replay = {"value": round(1000.0 * ws_ / e2e_ms, 4), "unit": UNIT, "h2d_bytes_per_step": h2d,
                  "d2h_bytes_per_step": d2h,
                  "path": "captured iteration graph replayed per step; each step's g copied in from pinned host "
                          "memory (double-buffered on a copy stream) and its 9 loss / norm sums copied out"}

    # ---- end to end through the public drop-in call: optimize() with numpy in and numpy out
    e2e_opt = None
    if ws_ == 1:
        try:
            e2e_opt = time_optimize_e2e(n, na, n_iter=args.e2e_iters)
        except Exception as exc:  # report, never fail the headline number on it
            e2e_opt = {"error": f"{type(exc).__name__}: {exc}"}

    # ---- plain per-call GPU path (reference numpy loop, host arrays)
    plain = None
    if rank == 0 and args.plain_steps > 0:
        from vamtoolbox_b200.optimize import Options

        o2 = Options(method="BCLP", n_iter=args.plain_steps, p=2, q=1, eps=0.1, learning_rate=1e-5, engine="host")
        b2 = BCLPNorm.__new__(BCLPNorm)
        b2.__dict__.update(bclp.__dict__)
        b2.logs = type(bclp.logs)(o2)
        b2.logs.startTiming()
        b2.exit_param = None
        t0 = time.perf_counter()
        b2.gradientDescentHost()
        torch.cuda.synchronize(dev)
        plain = args.plain_steps / (time.perf_counter() - t0 - 0.0)

    # ---- roofline of the dominant kernel: the projector with the larger share of the step
    peaks = {}
    try:
        peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
    except Exception:
        pass
    hbm_peak = peaks.get("hbm_gbs")
    peak_src = "measured" if hbm_peak else "fallback"
    hbm_peak = hbm_peak or 6650.0
    ny = nx = n
    vol_bytes = ny * nx * n * 4
    sino_bytes = ny * na * n * 4
    dom = "backward_ref" if kmean["backward_ref"] > kmean["forward"] else "forward"
    dom_ms = kmean[dom]
    achieved = (vol_bytes + sino_bytes) / (dom_ms * 1e-3) / 1e9
    if dom == "forward":
        # pixels the kernel loads: a strip of two detector bins loads each pixel it touches once, 4 B a
        # slice; angle pairs (a, a+180) share one lattice of (N+1)^2 samples (even N), unpaired angles use
        # N^2; the reference's warp reads four taps at N^2 points per angle
        pairs = count_angle_pairs(np.linspace(0, 360, na, endpoint=False))
        lattice = pairs * (n + 1 - n % 2) ** 2 + (na - 2 * pairs) * n * n
        per_sample = strip_pixels(n, np.linspace(0, 360, na, endpoint=False))
        tap_bytes, ref_tap_bytes = 4.0 * per_sample * lattice * n, 16.0 * n * n * na * n
        dom_name = "forward projector (R1)"
    else:
        # 2 detector rows x 4 B per (pixel, angle, slice) in the reference's np.interp; the block-table kernel
        # loads the distinct rows of each 2 x 2 block inside the clip circle once
        from vamtoolbox_b200.util.data import circle_inside_mask

        rows = block_rows(n, np.linspace(0, 360, na, endpoint=False), circle_inside_mask(ny, nx))
        tap_bytes, ref_tap_bytes = 4.0 * rows * na * n, 8.0 * ny * nx * na * n
        dom_name = "reference-parity backprojection (R2)"
    onchip_peak = 148 * 128 * 1.965e9 / 1e9     # L1/shared load bandwidth, nominal
    traffic = None
    tf = ROOT / "profiles" / ("forward_traffic.json" if dom == "forward" else "backward_traffic.json")
    if tf.exists():
        try:
            tr = json.loads(tf.read_text())
            traffic = tr.get("bytes_per_launch_scaled")
        except Exception:
            traffic = None

    multi = None
    if ws_ == 1 and not args.no_multi:
        try:
            multi = run_multi_target(dev)
        except Exception as exc:  # report, never fail the headline number on it
            multi = {"error": f"{type(exc).__name__}: {exc}"}

    configs = None
    if ws_ == 1 and not args.no_configs:
        configs = run_configs(parity=not args.no_cpu)

    algebraic = None
    if ws_ == 1 and not args.no_algebraic:
        try:
            algebraic = run_algebraic(dev)
        except Exception as exc:  # report, never fail the headline number on it
            algebraic = {"error": f"{type(exc).__name__}: {exc}"}

    fmt = None
    if ws_ == 1 and not args.no_formats:
        try:
            fmt = run_formats(dev, cpu=not args.no_cpu)
        except Exception as exc:  # report, never fail the headline number on it
            fmt = {"error": f"{type(exc).__name__}: {exc}"}

    vecg = None
    if ws_ == 1 and not args.no_vec:
        try:
            vecg = run_vec_geometry(dev, cpu=not args.no_cpu)
        except Exception as exc:  # report, never fail the headline number on it
            vecg = {"error": f"{type(exc).__name__}: {exc}"}

    ray = None
    if ws_ == 1 and not args.no_ray:
        try:
            ray = run_ray_bclp(dev, n=args.ray_size, cpu=not args.no_cpu)
        except Exception as exc:  # report, never fail the headline number on it
            ray = {"error": f"{type(exc).__name__}: {exc}"}

    cpu, parity = None, None
    if ws_ == 1 and not args.no_cpu:  # the CPU baseline (and the parity pass beside it) at N = 1 only
        try:
            # a fresh iteration state (g = g0) with no cross-rank hook: only rank 0 runs it
            cpu, parity = cpu_baseline_and_parity(bclp.device_iteration(), tg, pg, opts)
        except Exception as exc:  # report, never fail the GPU number on it
            cpu = {"value": None, "unit": UNIT, "error": f"{type(exc).__name__}: {exc}"}

    if rank == 0:
        line = {
            "metric": METRIC, "value": round(value, 4), "unit": UNIT, "n_gpus": ws_, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": round(ms_max, 4), "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded ellipsoid/cylinder target, "
            "shapes of the 256^3 x 360 absorbing OSMO/BCLP configuration)",
            "config": {"workload": workload_name(n, na), "per_rank": f"{n}^3 z-slab of the target per GPU",
                       "global_batch": ws_, "target": [n, n, n * ws_],
                       "angles": na, "parallelism": f"z-slab x{ws_}" if ws_ > 1 else "single GPU",
                       "l2": "inputs larger than L2 (working set ~450 MB per iteration)",
                       "graph": dist is None, "launch_shapes": tuning},
            "e2e": e2e_line(e2e_opt, e2e_replay, value / ws_),
            "plain_gpu": {"value": plain, "unit": UNIT, "path": "reference numpy BCLP loop, projector per call with "
                                                                 "host arrays"},
            "fused_vs_plain": (value / ws_ / plain) if plain else None,
            "fwd_adj_proj_per_s": round(fwd_adj, 3),
            "fwd_matched_adj_proj_per_s": round(fwd_matched, 3),
            "kernel_ms": {k: round(v, 4) for k, v in kmean.items()},
            "gpu_launches": (launches_per_step * args.steps) if launches_per_step is not None else None,
            "gpu_launches_source": "kernel nodes of the captured iteration graph x timed steps",
            "multi_target": multi,
            "ray_tracer": ray,
            "algebraic": algebraic,
            "output_formats": fmt,
            "vector_geometry": vecg,
            "configs": configs,
            "roofline": {"bound": "hbm", "achieved": round(achieved, 2), "peak": hbm_peak, "unit": "GB/s",
                         "frac": round(achieved / hbm_peak, 5), "traffic": traffic, "peak_source": peak_src,
                         "kernel": dom_name, "kernel_ms": round(dom_ms, 4),
                         "onchip": {"gathered_tap_bytes": tap_bytes, "reference_tap_bytes": ref_tap_bytes,
                                    "achieved_GBs": round(tap_bytes / (dom_ms * 1e-3) / 1e9, 1),
                                    "nominal_peak_GBs": round(onchip_peak, 1),
                                    "frac": round(tap_bytes / (dom_ms * 1e-3) / 1e9 / onchip_peak, 4)}},
            "cpu_baseline": cpu,
            "parity": parity,
            "clocks": clk,
        }
        print(json.dumps(line), flush=True)
    del graph
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()


def run_reference(args):
    ws_, rank, _ = dist_env()
    if rank != 0:
        return
    from oracle import oracle as O

    n, na = args.size, args.angles
    tg, pg = build_problem(n, na, seed=1000)
    opts = bclp_options(4)
    # initial sinogram as the reference builds it: forward of map_inv(target), filter, scale (CPU oracle, sample)
    n_s = 1
    f0 = opts.response_model.map_inv(tg.array[:, :, :n_s])
    absn = ("mask", np.asarray(pg.absorption_mask)[:, :, 0])
    from vamtoolbox_b200.util.data import filterSinogram

    g_s = filterSinogram(O.parallel_forward(f0, pg.angles, absorption=absn), "ram-lak") * np.pi / (2 * na)
    g_s = np.clip(g_s, 0, None)
    t1 = cpu_bclp_sample(tg, pg, g_s, opts, n_s)
    n_slice = int(max(1, min(n, args.cpu_seconds / max(t1, 1e-6))))
    f0 = opts.response_model.map_inv(tg.array[:, :, :n_slice])
    g_s = np.clip(filterSinogram(O.parallel_forward(f0, pg.angles, absorption=absn), "ram-lak") * np.pi / (2 * na), 0,
                  None)
    for _ in range(max(0, min(args.warmup, 1))):
        cpu_bclp_sample(tg, pg, g_s, opts, n_slice)
    ts = [cpu_bclp_sample(tg, pg, g_s, opts, n_slice) for _ in range(max(1, min(args.steps, 3)))]
    per = float(np.mean(ts)) * n / n_slice
    value = 1.0 / per
    cores = O.num_threads()
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws_, "steps": len(ts), "warmup": args.warmup,
            "ms_per_step": per * 1e3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic", "impl": "reference",
            "config": {"workload": workload_name(n, na), "per_rank": f"{n}^3 z-slab of the target per GPU",
                       "global_batch": ws_, "target": [n, n, n * ws_], "angles": na},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": f"{n_slice} of {n} z-slices per step, float64 C restatement of the reference's "
                                       f"projectors + numpy BCLP body, extrapolated over z"},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
