#!/usr/bin/env python
"""Throughput of the PCISPH particle step on one B200 (or N independent replicas).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--workload wave_breaker|dam_break_pcisph|dam_break_sph|batched|waterfall]
                    [--warm compare|zero|mlp] [--emit every-step|reference] [--dry-run]

Metric: PCISPH particle-updates/s at <= 1 % density error. One step is one full
PhysicSolver::update of the workload (grid build, neighbour lists, density,
non-pressure forces, the predict-correct loop to eta = 1 % with 3..50 iterations,
integration, collisions); a particle-update is one particle advanced one step.

Default workload: the ~1M-particle wave breaker (108x68x135 = 991,440 particles,
2x1x1 walls, two box obstacles and a sphere obstacle, dt 0.0004), seeded synthetic
input generated by liquidsimulation_b200.scenes. With --warm compare (the default)
the plain PCISPH solver (zero initial pressure, the reference's semantics) gives `value`;
the learned warm start (an MLP trained on the plain solver's converged steps during the
untimed lead-in) and LSP_WARM_AUTO are timed beside it over the same window.

`same_state` compares the two methods on equal inputs, at the configured dt 0.0008 and at
0.0004: along the learned trajectory every 10th state is copied into a plain solver and both
take one step from it; `learned_vs_plain_same_state` is the ratio of their qualifying
particle-updates/s (sampled steps that met eta, per device time; null when the plain steps
met eta on no sample), `device_time_ratio` the plain over the learned device time per step.
`long_window` runs both arms afresh for --long-steps steps and counts the steps that met eta:
the reference's zero-start PCISPH runs away in the wave breaker's deep column there while the
warm-started run stays converged (a comparison of two trajectories, not of equal inputs).

`value` times K device-resident steps with CUDA events on the solver's stream.
`e2e` times K steps through the C ABI with host buffers: each step uploads the
caller-order state from pinned host memory (lsp_write_state), steps, and reads the
state back (lsp_read_state). `e2e_readback` times the drop-in's own pattern beside it: the
state stays on the device and each step reads the positions and velocities back
(lsp_read_particles), nothing uploaded. Both replay the K steps `value` timed, from their
start state (restored untimed), so all three time the same steps. The roofline block comes from per-launch events of
the timed steps: every kernel class (`roofline.passes`) with its algorithmic bytes, device
time and fraction of the measured HBM peak; the dominant class heads the block, with ncu's
DRAM bytes for it where a capture exists (profiles/ncu_figures.json).

Multi-GPU: the path does not shard (one scene per GPU, replicas only); each rank
advances its own seeded scene and value sums all ranks' particle-updates over the
slowest rank's device time. Without torchrun, --gpus N starts its N ranks itself.

--impl reference times the reference's own sequential CPU solver (oracle/_ref, the
unmodified LiquidPhysics sources compiled here) on the box's host cores: one
independent sub-scene per thread, each a bounded sample of the workload (same lattice
spacing and parameters, smaller block) after the same lead-in. Sub-scenes need fewer
iterations per step than the full scene, so both lines carry iterations_mean and
particle_iterations_per_s; the reference line adds the restatement under the GPU arm's
iteration rule (min 3) as port_same_iteration_rule.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import math
import os
import statistics
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "PCISPH particle-updates/s at <=1% density error, learned vs plain, 1 B200"
UNIT = "particle-updates/s"
L2_BYTES = 126 * 1024 * 1024

# Algorithmic DRAM bytes per particle of each kernel class: every per-particle input read
# once and every output written once, neighbour re-reads served on chip. Neighbour-list
# bytes are not algorithmic and show up only in the measured traffic. grid_scan counts per
# cell (GRID_SCAN_BYTES_PER_CELL), the loop per particle-iteration plus its integration.
ALGO_BYTES = {
    "grid_keys": 16 + 4 + 4,         # read x|id; write cell key, slot in cell
    "grid_scatter": 4 + 4 + 4 + 8,   # read key, slot, caller id; write (index, id)
    "grid_gather": 8 + 4 + 64 + 64 + 4 + 4,   # read (index, id), key, 64 B state; write state, slot_of_id, key
    "neighbors": 16 + 4 + 4 + 4,     # read x; write count, rho, p (the list itself is not algorithmic)
    "density": 24,                   # read x; write rho, p
    "nonpressure": 52,               # read x, v, rho; write F
    "sph_pressure": 56,              # all forces of SPH: read x, p / rho^2, v, rho; write F
    "pci_predict": 84,               # read x, v, v_half, F, F_p, rho (write x*, v_half*)
    "pci_density": 28,               # read x*, p; write rho*, p
    "pci_force": 44,                 # read x*, p/rho*^2, rho; write F_p
    "integrate_collide": 116,
    "pci_loop": 156,                 # predict + density + force per iteration (+ integrate_collide once)
    "warm_start": 40,
}
GRID_SCAN_BYTES_PER_CELL = 12        # read the histogram, write the cell table, clear the histogram
GRID_HISTORY_BYTES = 32              # warm-start pressure history moved by grid_gather when kept
# ncu figures of the kernels (DRAM bytes, issue and DRAM activity of one capture each), kept
# beside their summaries; the roofline block scales them to this run's launches.
NCU_FIGURES = os.path.join(ROOT, "profiles", "ncu_figures.json")


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--workload", default="wave_breaker",
                    choices=["wave_breaker", "dam_break_pcisph", "dam_break_sph", "batched", "waterfall"])
    ap.add_argument("--warm", choices=["compare", "zero", "mlp"], default="compare",
                    help="compare: time plain and learned arms, value = plain")
    ap.add_argument("--loop", choices=["persistent", "host"], default="persistent")
    ap.add_argument("--train-steps", type=int, default=100,
                    help="untimed plain steps before timing; the learned arm trains on the converged ones")
    ap.add_argument("--train-iters", type=int, default=8, help="Adam steps per training step")
    ap.add_argument("--dt", type=float, default=None, help="override the workload's time step")
    ap.add_argument("--long-steps", type=int, default=200,
                    help="steps of the long learned-vs-plain window after the timed phase (0 = off)")
    ap.add_argument("--same-steps", type=int, default=200,
                    help="learned steps of the same-state comparison (0 = off)")
    ap.add_argument("--same-every", type=int, default=10,
                    help="same-state comparison: every k-th learned step is also stepped by plain PCISPH")
    ap.add_argument("--same-dts", default="0.0008,0.0004",
                    help="time steps of the same-state comparison (wave breaker: 0.0008 is the configured one)")
    ap.add_argument("--wf-particles", type=int, default=4_000_000,
                    help="waterfall: particles emitted before the timed steps")
    ap.add_argument("--emit", choices=["every-step", "reference"], default="every-step",
                    help="waterfall: a sheet before every step (as specified) or at the reference's cadence "
                         "(one lattice spacing of travel between sheets)")
    ap.add_argument("--dry-run", action="store_true",
                    help="replica plumbing without a GPU: each rank steps a small CPU oracle sample of the "
                         "workload, ranks meet over gloo; checks the multi-process path, not a benchmark")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-seconds", type=float, default=20.0)
    return ap.parse_args()


def make_scene(workload, seed_offset=0):
    from liquidsimulation_b200 import scenes
    if workload == "wave_breaker":
        return scenes.wave_breaker(seed=3 + seed_offset)
    if workload == "dam_break_pcisph":
        return scenes.dam_break_pcisph(seed=2 + seed_offset)
    return scenes.dam_break_sph(seed=1 + seed_offset)


def workload_label(args, scene=None, head="plain"):
    """The workload name and particle count a bench line carries in `config` (the same for
    our arm and the reference arm)."""
    from liquidsimulation_b200 import abi, scenes
    if args.workload == "batched":
        scs = scenes.batched_dam_breaks(seed=4)
        return f"batched_dam_breaks x{len(scs)} ({head} PCISPH, one graph per step)", int(sum(sc.n for sc in scs))
    if args.workload == "waterfall":
        cadence = ("one sheet appended per step" if args.emit == "every-step"
                   else "one sheet per lattice spacing of travel, the reference's cadence")
        return f"waterfall grown to ~{args.wf_particles} particles (plain PCISPH, {cadence})", int(args.wf_particles)
    sc = scene or make_scene(args.workload)
    solver = "PCISPH" if sc.params.solver == abi.LSP_SOLVER_PCISPH else "SPH"
    return f"{sc.name} ({args.workload}, {head} {solver}, {args.loop} loop)", int(sc.n)


def sample_scene(workload, target_n):
    """A bounded CPU sample of the workload: same spacing, parameters and walls, smaller block.
    For the batch, the batch's scene whose size is closest to target_n."""
    from liquidsimulation_b200 import scenes
    if workload == "batched":
        return min(scenes.batched_dam_breaks(seed=4), key=lambda sc: abs(sc.n - target_n))
    if workload == "waterfall":
        # The emitter's first sheets (2,000 particles each) in the waterfall box.
        sc = scenes.waterfall(seed=5)
        sheets = [scenes.waterfall_sheet(k, seed=5) for k in range(max(1, target_n // 2000))]
        sc.positions = np.concatenate([x for x, _ in sheets])
        sc.velocities = np.concatenate([v for _, v in sheets])
        return sc
    full = make_scene(workload)
    s = full.spacing
    if workload == "wave_breaker":
        frac = (target_n / full.n) ** (1.0 / 3.0)
        block = (0.8 * frac, 0.5 * frac, 1.0 * frac)
        sc = scenes.wave_breaker(seed=3, s=s, block=block)
    elif workload == "dam_break_pcisph":
        frac = (target_n / full.n) ** (1.0 / 3.0)
        counts = tuple(max(2, int(c * frac)) for c in (64, 102, 64))
        sc = scenes.dam_break_pcisph(seed=2, counts=counts, s=s)
    else:
        sc = full
    return sc


CPU_SAMPLE_PARTICLES = 12000


def lead_steps(args):
    """Untimed steps before the timed phase (the SPH dam break's reference solver goes
    non-finite at step 47, so its lead-in is capped at 20)."""
    return min(args.train_steps, 20) if args.workload == "dam_break_sph" else args.train_steps


def line_config(args, world):
    """The `config` of a bench line, built from the command's arguments alone, so that our arm
    and the reference arm print the same dict for the same workload. It names the one way the
    reference arm's work differs: the reference CPU solver runs bounded sub-scenes of the
    workload, which need fewer PCISPH iterations per step than the full scene, so both lines
    also report their mean iterations and particle-iterations/s."""
    from liquidsimulation_b200 import scenes
    label, n = workload_label(args)
    cfg = {"workload": label, "particles": n, "particles_total": n * world}
    if args.workload == "batched":
        scs = scenes.batched_dam_breaks(seed=4)
        cfg.update(scenes=len(scs), scene_sizes=[int(sc.n) for sc in scs], dt=args.dt or scs[0].dt,
                   eta=scs[0].params.pci_eta, untimed_steps_before=min(args.train_steps, 50) + 1,
                   l2=f"inputs larger than L2 (~{n / 1e6:.2f}M particles, ~450 MiB working set), no flush")
    elif args.workload == "waterfall":
        sc = scenes.waterfall(seed=5)
        cfg.update(dt=sc.dt, eta=sc.params.pci_eta, emitted_per_step=2000,
                   l2=f"inputs larger than L2 ({n / 1e6:.0f}M particles), no flush")
    else:
        sc = make_scene(args.workload)
        working_set = n * (64 * 2 + 16 * 5 + 4 * 8) + n * 4 * 36
        cfg.update(dt=args.dt or sc.dt, eta=sc.params.pci_eta, min_iterations=sc.params.pci_min_iterations,
                   max_iterations=sc.params.pci_max_iterations, untimed_steps_before=lead_steps(args),
                   l2=f"inputs larger than L2: working set ~{working_set / 2**20:.0f} MiB > 126 MiB, no flush")
    cfg["parallelism"] = f"replicas x{world}" if world > 1 else "single GPU"
    cfg["reference_arm"] = (
        f"the reference's CPU solver (oracle/_ref) on one independent ~{CPU_SAMPLE_PARTICLES}-particle sub-scene "
        f"per host thread (same spacing, parameters and walls, smaller block), after the same "
        f"{cfg.get('untimed_steps_before', 0)}-step lead-in; a sub-scene needs fewer PCISPH iterations per step "
        f"than the full scene, so both lines report iterations_mean and particle_iterations_per_s")
    return cfg


# ------------------------------------------------------------------ distributed helpers

class Dist:
    """One process per GPU (torchrun). The path does not shard: ranks run independent replica
    scenes and meet only for the barrier around the timed region and the max-over-ranks of
    the device time (no collective on the data path). backend: "nccl" on GPUs, "gloo" on CPU."""

    def __init__(self, gpus=1, backend="nccl"):
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local = int(os.environ.get("LOCAL_RANK", "0"))
        self.backend = backend
        self.pg = None
        if self.world > 1:
            import torch
            import torch.distributed as dist
            from datetime import timedelta
            kw = {}
            if backend == "nccl":
                torch.cuda.set_device(self.local)
                kw["device_id"] = torch.device("cuda", self.local)
            dist.init_process_group(backend, timeout=timedelta(seconds=120), **kw)
            self.pg = dist

    def _tensor(self, v):
        import torch
        return torch.tensor([v], dtype=torch.float64, device="cuda" if self.backend == "nccl" else "cpu")

    def barrier(self):
        if self.pg:
            t = self._tensor(0.0)
            self.pg.all_reduce(t)
            if self.backend == "nccl":
                import torch
                torch.cuda.synchronize()

    def max(self, v: float) -> float:
        if not self.pg:
            return v
        t = self._tensor(v)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def sum(self, v: float) -> float:
        if not self.pg:
            return v
        t = self._tensor(v)
        self.pg.all_reduce(t)
        return float(t.item())

    def close(self):
        if self.pg:
            self.pg.destroy_process_group()


# ------------------------------------------------------------------ clocks

class ClockSampler:
    """Samples the SM clock, its maximum, power and the throttle reasons through NVML
    (read-only queries) every millisecond while the timed region runs, so that even a 30 ms
    region yields a couple of dozen samples (nvidia-smi's 200 ms floor would give none)."""

    REASONS = (("hw_slowdown", "nvmlClocksEventReasonHwSlowdown"),
               ("hw_thermal_slowdown", "nvmlClocksEventReasonHwThermalSlowdown"),
               ("sw_thermal_slowdown", "nvmlClocksEventReasonSwThermalSlowdown"),
               ("sw_power_cap", "nvmlClocksEventReasonSwPowerCap"),
               ("hw_power_brake_slowdown", "nvmlClocksEventReasonHwPowerBrakeSlowdown"))

    def __init__(self, index, period_s=0.001):
        self.index = index
        self.period = period_s
        self.samples = []
        self.stop_evt = threading.Event()
        self.thread = None
        self.source = "nvml"
        self.power = None

    def _handle(self, nv):
        try:
            import torch
            pr = torch.cuda.get_device_properties(self.index)
            bus = f"{pr.pci_domain_id:08x}:{pr.pci_bus_id:02x}:{pr.pci_device_id:02x}.0"
            return nv.nvmlDeviceGetHandleByPciBusId(bus)
        except Exception:
            return nv.nvmlDeviceGetHandleByIndex(self.index)

    def _loop(self, nv, h, mx):
        while not self.stop_evt.is_set():
            try:
                sm = nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)
                rs = nv.nvmlDeviceGetCurrentClocksEventReasons(h)
                self.samples.append((sm, mx, rs, self.power))
            except Exception:
                pass
            self.ready.set()
            self.stop_evt.wait(self.period)

    def start(self):
        """Returns once the sampling thread has taken its first sample, so the timed region
        that follows is covered from its first step. The maximum clock is fixed and power is
        slow to read: both are queried once here, before the thread starts."""
        try:
            import pynvml as nv
            nv.nvmlInit()
            h = self._handle(nv)
            self.nv = nv
        except Exception:
            self.source = "unavailable"
            return
        try:
            mx = nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM)
            self.power = nv.nvmlDeviceGetPowerUsage(h) / 1000.0
        except Exception:
            mx, self.power = None, None
        self.ready = threading.Event()
        self.thread = threading.Thread(target=self._loop, args=(nv, h, mx), daemon=True)
        self.thread.start()
        self.ready.wait(timeout=2.0)

    def stop(self):
        if self.thread is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvml unavailable"], "samples": 0}
        self.stop_evt.set()
        self.thread.join(timeout=5)
        try:
            self.nv.nvmlShutdown()
        except Exception:
            pass
        sm = [x[0] for x in self.samples]
        bits = [(nm, getattr(self.nv, attr)) for nm, attr in self.REASONS]
        reasons = sorted({nm for x in self.samples for nm, bit in bits if x[2] & bit})
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": self.samples[0][1] if sm else None,
                "sm_min_mhz": min(sm) if sm else None,
                "power_w_at_start": round(self.power, 1) if self.power is not None else None,
                "reasons": reasons, "samples": len(sm), "source": f"NVML every {self.period * 1e3:.0f} ms"}


# ------------------------------------------------------------------ our arm

def prepare_arm(args, dist, learned, auto=False):
    """Builds the workload and advances it to its timed phase: --train-steps plain steps,
    during which the learned arm's network trains online on the plain pressures. The
    learned arm then starts every step from the network's guess (LSP_WARM_MLP); with auto,
    from the zero start until a step needs more than half the iteration cap (default switch
    point) or misses eta, and from the guess after that (LSP_WARM_AUTO)."""
    from liquidsimulation_b200 import abi
    from liquidsimulation_b200.solver import from_scene
    scene = make_scene(args.workload, seed_offset=dist.rank)
    if args.dt:
        scene.dt = args.dt
    scene.params.loop_mode = abi.LSP_LOOP_HOST if args.loop == "host" else abi.LSP_LOOP_PERSISTENT
    solver = from_scene(scene, device=dist.local)
    train = {"steps": args.train_steps, "loss": None, "plain_iterations_mean": None}
    its = []
    if learned:
        solver.mlp_record(True)
        solver.mlp_set_loss_asymmetry(4.0)
    trained = 0
    for t in range(args.train_steps):
        st = solver.update(scene.dt)
        its.append(st.iterations)
        # Targets are plain-PCISPH pressures of steps that met eta; the network never
        # trains on its own warm-started outputs (that feedback loop diverges).
        if learned and st.converged:
            train["loss"] = solver.mlp_train(iterations=args.train_iters, batch=65536, lr=2e-3, seed=t)
            trained += 1
    train["trained_on_steps"] = trained
    if learned:
        solver.mlp_record(False)
        solver.set_warm_start(abi.LSP_WARM_AUTO if auto else abi.LSP_WARM_MLP)
    if its:
        train["plain_iterations_mean"] = float(np.mean(its))
    return scene, solver, train


def time_arm(args, dist, scene, solver, clocks=None, profiler_range=False, snapshot=False):
    """W warm-up steps, then exactly K steps timed with CUDA events on the solver's stream.
    The library's per-launch profile (an event pair around every launch, on the same stream)
    runs during the timed steps, so the kernel-class times behind the roofline are those of
    the timed steps; its cost is inside the timed value (about 0.9 % of a wave-breaker step,
    measured against the same steps unprofiled). With snapshot, the caller-order state at the
    start and at the end of the timed steps is read (outside the timed region) and returned
    as start_state / end_state, so the end-to-end arms can replay the same steps and check
    that they arrive at the same bits."""
    from liquidsimulation_b200 import abi
    lib, h = solver._lib, solver._h
    for _ in range(args.warmup):
        solver.update(scene.dt)
    start_state = solver.read_state() if snapshot else None
    dist.barrier()
    solver.synchronize()
    l0 = ctypes.c_int64()
    lib.lsp_launch_count(h, ctypes.byref(l0))
    abi.check(lib, lib.lsp_profile(h, 1))
    if profiler_range:
        # Marks the timed steps for a profiler started with capture off (ncu
        # --profile-from-start off); no effect otherwise.
        import torch
        torch.cuda.profiler.start()
    if clocks:
        clocks.start()
    abi.check(lib, lib.lsp_timer_mark(h, 0))
    stats = [solver.update(scene.dt) for _ in range(args.steps)]
    abi.check(lib, lib.lsp_timer_mark(h, 1))
    ms = ctypes.c_float()
    abi.check(lib, lib.lsp_timer_elapsed(h, 0, 1, ctypes.byref(ms)))
    solver.synchronize()
    if profiler_range:
        torch.cuda.profiler.stop()
    clock_info = clocks.stop() if clocks else None
    end_state = solver.read_state() if snapshot else None
    prof_ms = (ctypes.c_double * 16)()
    prof_n = (ctypes.c_int64 * 16)()
    abi.check(lib, lib.lsp_profile_read(h, prof_ms, prof_n, 16))
    abi.check(lib, lib.lsp_profile(h, 0))
    profile = {abi.PROF_NAMES[k]: {"ms": prof_ms[k], "launches": prof_n[k]}
               for k in range(len(abi.PROF_NAMES)) if prof_n[k] > 0}
    l1 = ctypes.c_int64()
    lib.lsp_launch_count(h, ctypes.byref(l1))
    dist.barrier()
    t_max = dist.max(ms.value)
    updates = dist.sum(float(scene.n) * args.steps)
    eta = scene.params.pci_eta
    return {
        "value": updates / (t_max / 1e3), "ms_per_step": t_max / args.steps, "updates": updates,
        "iterations": {"mean": float(np.mean([s.iterations for s in stats])),
                       "min": int(min(s.iterations for s in stats)), "max": int(max(s.iterations for s in stats))},
        "max_density_error_ratio": float(max(s.max_density_error_ratio for s in stats)),
        "qualifying_steps": sum(1 for s in stats if s.converged and s.max_density_error_ratio <= eta + 1e-12),
        "warm_start_kept": sum(1 for s in stats if s.warm_start_used),
        "launches": int(l1.value - l0.value), "clocks": clock_info, "profile": profile, "stats": stats,
        "start_state": start_state, "end_state": end_state,
    }


def load_ncu_figures():
    try:
        with open(NCU_FIGURES) as fh:
            return json.load(fh)
    except (OSError, ValueError):
        return {}


def profile_arm(args, scene, timed, cells=None):
    """Roofline of every kernel class from the per-launch events of the timed steps: its
    algorithmic bytes per step over its device time, against the measured HBM peak; the
    dominant class heads the block. Where an ncu capture of the kernel exists its DRAM bytes
    (scaled to this run's particles and iterations) and issue activity are reported beside."""
    pstats = timed["stats"]
    n = scene.n
    classes = timed["profile"]
    total = sum(v["ms"] for v in classes.values()) or 1.0
    try:
        peak, src = float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["hbm_gbs"]), "measured"
    except Exception:
        peak, src = 6650.0, "fallback"
    ncu = load_ncu_figures()
    its = sum(s.iterations for s in pstats) / max(1, len(pstats))
    loop_integrates = "pci_loop" in classes and "integrate_collide" not in classes
    history = scene.params.warm_start != 0

    def algo_per_launch(name, launches_per_step):
        if name == "pci_loop":
            b = (ALGO_BYTES["pci_loop"] * its + (ALGO_BYTES["integrate_collide"] if loop_integrates else 0)) * n
        elif name == "grid_scan":
            b = GRID_SCAN_BYTES_PER_CELL * (cells or 0)
        elif name == "grid_gather":
            b = (ALGO_BYTES[name] + (GRID_HISTORY_BYTES if history else 0)) * n
        else:
            b = ALGO_BYTES.get(name, 0) * n
        return b / max(1.0, launches_per_step)

    passes = {}
    for name, v in classes.items():
        launches_per_step = v["launches"] / args.steps
        ms_step = v["ms"] / args.steps
        algo_step = algo_per_launch(name, 1.0) if name not in ("pci_predict", "pci_density", "pci_force") \
            else ALGO_BYTES[name] * n * its
        gbs = algo_step / (ms_step / 1e3) / 1e9 if ms_step > 0 else None
        e = {"ms_per_step": round(ms_step, 4), "launches_per_step": round(launches_per_step, 2),
             "algorithmic_bytes_per_step": int(algo_step), "achieved_gbs": round(gbs, 1) if gbs else None,
             "frac": round(gbs / peak, 4) if gbs else None, "share": round(v["ms"] / total, 3)}
        f = ncu.get(name)
        if f:
            e["ncu"] = {k: f[k] for k in ("kernel", "issue_active", "dram_frac", "dram_bytes_per_unit", "unit",
                                          "capture") if k in f}
        passes[name] = e
    top_name, top_v = max(classes.items(), key=lambda kv: kv[1]["ms"])
    avg_ms = top_v["ms"] / top_v["launches"]
    algo = algo_per_launch(top_name, top_v["launches"] / args.steps) if top_name != "pci_loop" \
        else algo_per_launch("pci_loop", 1.0)
    achieved = algo / (avg_ms / 1e3) / 1e9
    traffic, traffic_src, issue = None, None, None
    f = ncu.get(top_name)
    if f and f.get("dram_bytes_per_unit"):
        units = n * its if f.get("unit") == "particle-iteration" else n
        traffic = int(f["dram_bytes_per_unit"] * units + (f.get("dram_bytes_per_particle_extra", 0) * n))
        traffic_src = (f"ncu dram__bytes_read.sum + dram__bytes_write.sum of {f['kernel']} ({f['capture']}), "
                       f"per {f['unit']}, scaled to this launch")
        issue = {"issue_active_frac": f.get("issue_active"), "dram_frac": f.get("dram_frac"),
                 "source": f"ncu of {f['kernel']} ({f['capture']})"}
    return {"bound": "hbm", "kernel": top_name, "achieved": round(achieved, 1), "peak": peak,
            "peak_source": src, "unit": "GB/s", "frac": round(achieved / peak, 4),
            "algorithmic_bytes_per_launch": int(algo), "avg_launch_ms": round(avg_ms, 5), "traffic": traffic,
            "traffic_source": traffic_src, "binding_limit": issue,
            "share_of_step": round(top_v["ms"] / total, 3), "passes": passes}


def e2e_arm(args, dist, scene, solver, expect=None):
    """K steps through the C ABI with pinned host buffers: upload state, step, read state.
    expect: the caller-order state the same K steps reached in the timed arm; the final host
    buffers are compared with it bit for bit (replay_bit_identical)."""
    from liquidsimulation_b200 import abi
    lib, h, n = solver._lib, solver._h, scene.n
    nbytes = n * 4
    bufs = []
    for size in (3 * nbytes, 3 * nbytes, 3 * nbytes, 3 * nbytes, nbytes):
        ptr = ctypes.c_void_p()
        abi.check(lib, lib.lsp_host_alloc(size, ctypes.byref(ptr)))
        bufs.append(ptr)
    fp = ctypes.POINTER(ctypes.c_float)
    x, v, hv, ov = (ctypes.cast(b, fp) for b in bufs[:4])
    first = ctypes.cast(bufs[4], ctypes.POINTER(ctypes.c_int32))
    abi.check(lib, lib.lsp_read_state(h, x, v, hv, ov, first, n))
    st = abi.LspStepStats()
    dist.barrier()
    solver.synchronize()
    abi.check(lib, lib.lsp_timer_mark(h, 2))
    for _ in range(args.steps):
        abi.check(lib, lib.lsp_write_state(h, x, v, hv, ov, first, n))
        abi.check(lib, lib.lsp_step(h, ctypes.c_float(scene.dt), ctypes.byref(st)))
        abi.check(lib, lib.lsp_read_state(h, x, v, hv, ov, first, n))
    abi.check(lib, lib.lsp_timer_mark(h, 3))
    ems = ctypes.c_float()
    abi.check(lib, lib.lsp_timer_elapsed(h, 2, 3, ctypes.byref(ems)))
    e_max = dist.max(ems.value)
    same = None
    if expect is not None:
        got = [np.ctypeslib.as_array(q, shape=(n * 3,)) for q in (x, v, hv, ov)]
        got.append(np.ctypeslib.as_array(first, shape=(n,)))
        same = all(np.array_equal(np.ascontiguousarray(e).reshape(-1).view(np.uint32), g.view(np.uint32))
                   for e, g in zip(expect, got))
    for b in bufs:
        lib.lsp_host_free(b)
    return {"value": dist.sum(float(n) * args.steps) / (e_max / 1e3), "unit": UNIT,
            "h2d_bytes_per_step": int(n * (4 * 12 + 4)), "d2h_bytes_per_step": int(n * (4 * 12 + 4)),
            "steps": "the timed steps of value, replayed from their start state",
            "replay_bit_identical": same}


def readback_arm(args, dist, scene, solver):
    """K steps through the C ABI as the drop-in of the reference's solver runs them (the
    CUDA branch of SPHSolver::update): the state stays on the device, each step reads the
    positions and velocities back in caller order into pinned host buffers (what the
    application draws), and nothing is uploaded."""
    from liquidsimulation_b200 import abi
    lib, h, n = solver._lib, solver._h, scene.n
    bufs = []
    for _ in range(2):
        ptr = ctypes.c_void_p()
        abi.check(lib, lib.lsp_host_alloc(3 * n * 4, ctypes.byref(ptr)))
        bufs.append(ptr)
    fp = ctypes.POINTER(ctypes.c_float)
    x, v = (ctypes.cast(b, fp) for b in bufs)
    st = abi.LspStepStats()
    dist.barrier()
    solver.synchronize()
    abi.check(lib, lib.lsp_timer_mark(h, 6))
    for _ in range(args.steps):
        abi.check(lib, lib.lsp_step(h, ctypes.c_float(scene.dt), ctypes.byref(st)))
        abi.check(lib, lib.lsp_read_particles(h, x, v, n))
    abi.check(lib, lib.lsp_timer_mark(h, 7))
    ems = ctypes.c_float()
    abi.check(lib, lib.lsp_timer_elapsed(h, 6, 7, ctypes.byref(ems)))
    e_max = dist.max(ems.value)
    for b in bufs:
        lib.lsp_host_free(b)
    return {"value": dist.sum(float(n) * args.steps) / (e_max / 1e3), "unit": UNIT,
            "h2d_bytes_per_step": 0, "d2h_bytes_per_step": int(n * 24),
            "pattern": "state resident on the device; x and v read back each step (the drop-in's update)"}


def long_window(args, dist: Dist, learned: bool, auto: bool = False):
    """A fresh arm run for --long-steps steps after the same lead-in: per-step iterations and
    errors, and the throughput of the steps that met eta (qualifying particle-updates over the
    device time of the whole window). A step that fails (the reference's zero-pressure PCISPH
    can run away in a deep column) ends the window and is reported. The plain arm's window
    includes its neighbour-list regrowths, whose host-side allocation time varies from run
    to run on a shared node; the window's clocks are sampled and reported."""
    from liquidsimulation_b200 import abi
    scene, solver, train = prepare_arm(args, dist, learned=learned, auto=auto)
    lib, h = solver._lib, solver._h
    eta = scene.params.pci_eta
    its, errs, qual, failed, tried = [], [], 0, None, []
    clocks = ClockSampler(dist.local, period_s=0.01)
    clocks.start()
    abi.check(lib, lib.lsp_timer_mark(h, 4))
    for k in range(args.long_steps):
        try:
            st = solver.update(scene.dt)
        except abi.LspError as e:
            failed = {"step": k, "error": str(e)}
            break
        its.append(st.iterations)
        errs.append(st.max_density_error_ratio)
        tried.append(st.warm_start_tried)
        qual += 1 if (st.converged and st.max_density_error_ratio <= eta + 1e-12) else 0
    abi.check(lib, lib.lsp_timer_mark(h, 5))
    ms = ctypes.c_float()
    abi.check(lib, lib.lsp_timer_elapsed(h, 4, 5, ctypes.byref(ms)))
    clock_info = clocks.stop()
    solver.close()
    t = dist.max(ms.value) / 1e3
    out = {"steps_run": len(its), "qualifying_steps": qual,
           "iterations_mean": float(np.mean(its)) if its else None, "iterations_max": int(max(its)) if its else None,
           "max_density_error_ratio": float(max(errs)) if errs else None,
           "qualifying_updates_per_s": dist.sum(float(scene.n) * qual) / t if t > 0 else None,
           "all_updates_per_s": dist.sum(float(scene.n) * len(its)) / t if t > 0 else None,
           "failed": failed, "clocks": clock_info, "guess_tried_steps": int(sum(tried)),
           "first_guess_step": (args.train_steps + tried.index(1)) if 1 in tried else None}
    if learned:
        out["warm_training"] = train
    return out


def same_state(args, dist: Dist, dt: float):
    """Learned vs plain PCISPH from identical states, at time step dt.

    One learned trajectory: plain steps while they meet eta (at most --train-steps), the
    network training on each; then the learned warm start (LSP_WARM_MLP) for --same-steps
    steps. Every --same-every-th of those steps starts from a state that is first copied
    into a plain solver (lsp_write_state, caller order), which then takes one step of its
    own: both solvers step from the same positions and velocities, so their iteration counts
    and device times compare the two methods on equal inputs, not on two trajectories that
    have drifted apart. Each sampled step is timed with CUDA events on its solver's stream."""
    from liquidsimulation_b200 import abi
    from liquidsimulation_b200.solver import from_scene
    scene = make_scene(args.workload, seed_offset=dist.rank)
    scene.dt = dt
    eta = scene.params.pci_eta
    learned = from_scene(scene, device=dist.local)
    learned.mlp_record(True)
    learned.mlp_set_loss_asymmetry(4.0)
    lead, trained, failed = 0, 0, None
    for t in range(args.train_steps):
        st = learned.update(dt)
        lead += 1
        if not (st.converged and st.max_density_error_ratio <= eta + 1e-12):
            break   # the zero start stopped meeting eta: the warm start takes over from here
        learned.mlp_train(iterations=args.train_iters, batch=65536, lr=2e-3, seed=t)
        trained += 1
    learned.mlp_record(False)
    learned.set_warm_start(abi.LSP_WARM_MLP)
    plain = from_scene(scene, device=dist.local)

    def timed_step(s):
        lib, h = s._lib, s._h
        abi.check(lib, lib.lsp_timer_mark(h, 8))
        st = s.update(dt)
        abi.check(lib, lib.lsp_timer_mark(h, 9))
        ms = ctypes.c_float()
        abi.check(lib, lib.lsp_timer_elapsed(h, 8, 9, ctypes.byref(ms)))
        return st, ms.value

    rows = []
    for k in range(args.same_steps):
        sample = k % args.same_every == 0
        try:
            if sample:
                plain.write_state(*learned.read_state())
                sp, mp = timed_step(plain)
            sl, ml = timed_step(learned)
        except abi.LspError as e:
            failed = {"step": lead + k, "error": str(e)}
            break
        if sample:
            rows.append((sp.iterations, sl.iterations, mp, ml,
                         int(sp.converged and sp.max_density_error_ratio <= eta + 1e-12),
                         int(sl.converged and sl.max_density_error_ratio <= eta + 1e-12), sl.warm_start_used))
    plain.close()
    learned.close()
    out = {"dt": dt, "plain_lead_steps": lead, "trained_on_steps": trained, "samples": len(rows),
           "every": args.same_every, "failed": failed}
    if rows:
        r = np.array(rows, np.float64)
        pm, lm = float(r[:, 2].mean()), float(r[:, 3].mean())
        out.update({
            "window": f"steps {lead}..{lead + args.same_steps} of the learned trajectory",
            "plain": {"iterations_mean": float(r[:, 0].mean()), "ms_per_step": pm, "qualifying": int(r[:, 4].sum())},
            "learned": {"iterations_mean": float(r[:, 1].mean()), "ms_per_step": lm,
                        "qualifying": int(r[:, 5].sum()), "guess_kept": int(r[:, 6].sum())},
            "iterations_saved_frac": float(1.0 - r[:, 1].sum() / r[:, 0].sum()),
            # Plain over learned device time per step, whether or not the steps met eta.
            "device_time_ratio": pm / lm if lm > 0 else None})
        ratio = qualifying_ratio(r[:, 4].sum(), r[:, 2].sum(), r[:, 5].sum(), r[:, 3].sum())
        out.update({"learned_vs_plain_same_state": ratio, "target": 1.5,
                    "target_met": bool(ratio is not None and ratio >= 1.5)})
    return out


def qualifying_ratio(plain_qualifying, plain_ms, learned_qualifying, learned_ms):
    """The metric's learned-over-plain ratio on equal inputs: qualifying particle-updates/s,
    the steps that met eta per device time (both arms step the same particles). None when
    the plain arm met eta on no step (the ratio is then undefined) or no time was taken."""
    if plain_qualifying <= 0 or plain_ms <= 0 or learned_ms <= 0:
        return None
    return float((learned_qualifying / learned_ms) / (plain_qualifying / plain_ms))


def run_ours(args, dist: Dist):
    import torch
    torch.cuda.set_device(dist.local)
    if args.workload == "dam_break_sph":
        # Plain SPH has no pressure loop to warm-start, and the reference's own solver goes
        # non-finite at step 47 of this scene (k = 3 is too soft for dt = 0.002): the plain
        # arm alone, after a short lead-in.
        args.warm, args.long_steps, args.train_steps = "zero", 0, lead_steps(args)
    arms = {}
    plain = None
    if args.warm in ("compare", "zero"):
        scene, solver, train = prepare_arm(args, dist, learned=False)
        plain = time_arm(args, dist, scene, solver, ClockSampler(dist.local), profiler_range=True,
                         snapshot=not args.no_e2e)
        plain["train"] = train
        arms["plain"] = (scene, solver, plain)
    if args.warm in ("compare", "mlp"):
        scene, solver, train = prepare_arm(args, dist, learned=True)
        learned = time_arm(args, dist, scene, solver, ClockSampler(dist.local), profiler_range=args.warm == "mlp",
                           snapshot=not args.no_e2e and args.warm == "mlp")
        learned["train"] = train
        arms["learned"] = (scene, solver, learned)
    if args.warm == "compare":
        scene, solver, train = prepare_arm(args, dist, learned=True, auto=True)
        arms["auto"] = (scene, solver, time_arm(args, dist, scene, solver, ClockSampler(dist.local)))
    head = "plain" if "plain" in arms else "learned"
    scene, solver, main = arms[head]
    roofline = profile_arm(args, scene, main, cells=solver.grid_cells())
    # Both end-to-end arms replay the timed steps from their start state (restored before each,
    # untimed), so they time the same work per step as `value`; later steps of the wave
    # breaker need more iterations.
    e2e = readback = None
    if not args.no_e2e:
        solver.write_state(*main["start_state"])
        e2e = e2e_arm(args, dist, scene, solver, expect=main["end_state"])
        solver.write_state(*main["start_state"])
        readback = readback_arm(args, dist, scene, solver)
    result = {
        "metric": METRIC, "value": main["value"], "unit": UNIT, "n_gpus": dist.world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": main["ms_per_step"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded lattice scenes)",
        "config": line_config(args, dist.world),
        "iterations": main["iterations"],
        "iterations_mean": main["iterations"]["mean"],
        "particle_iterations_per_s": main["value"] * main["iterations"]["mean"],
        "max_density_error_ratio": main["max_density_error_ratio"],
        "qualifying_steps": main["qualifying_steps"],
        "warm_start_kept": main["warm_start_kept"],
        "roofline": roofline,
        "e2e": e2e,
        "e2e_readback": readback,
        "gpu_launches": main["launches"],
        "clocks": main["clocks"],
    }
    if "learned" in arms and head == "plain":
        lrn = arms["learned"][2]
        result["learned"] = {k: lrn[k] for k in ("value", "ms_per_step", "iterations", "max_density_error_ratio",
                                                  "qualifying_steps", "warm_start_kept", "launches")}
        result["learned_vs_plain"] = lrn["value"] / main["value"]
        result["training"] = lrn["train"]
    if "auto" in arms and head == "plain":
        aut = arms["auto"][2]
        result["auto"] = {k: aut[k] for k in ("value", "ms_per_step", "iterations", "max_density_error_ratio",
                                              "qualifying_steps", "warm_start_kept", "launches")}
        result["auto"]["guess_tried_steps"] = sum(1 for s in aut["stats"] if s.warm_start_tried)
        result["auto_vs_plain"] = aut["value"] / main["value"]
    for _, solver, _ in arms.values():
        solver.close()
    if args.same_steps > 0 and args.warm == "compare":
        ss = [same_state(args, dist, float(d)) for d in args.same_dts.split(",") if d.strip()]
        result["same_state"] = ss
        # The learned part's headline: particle-updates/s of the learned step over the plain
        # step from the same states, at each time step.
        result["learned_vs_plain_same_state"] = {f"dt={x['dt']:g}": x.get("learned_vs_plain_same_state")
                                                 for x in ss}
    if args.long_steps > 0 and args.warm == "compare":
        lw = {"plain": long_window(args, dist, learned=False), "learned": long_window(args, dist, learned=True),
              "auto": long_window(args, dist, learned=True, auto=True),
              "window": f"steps {args.train_steps}..{args.train_steps + args.long_steps} of fresh runs "
                        f"(same lead-in; learned and auto trained on the converged lead-in steps)"}
        qp, ql = lw["plain"]["qualifying_updates_per_s"], lw["learned"]["qualifying_updates_per_s"]
        qa = lw["auto"]["qualifying_updates_per_s"]
        lw["learned_vs_plain_qualifying"] = (ql / qp) if qp else None
        lw["auto_vs_plain_qualifying"] = (qa / qp) if qp else None
        result["long_window"] = lw
    return result


def batched_arm(args, dist: Dist, learned: bool, auto: bool = False):
    """One arm of the batched workload: 64 independent PCISPH dam breaks (2,000-64,000
    particles each, log-uniform) in one batch, one CUDA graph per step with one persistent
    kernel for every scene's PCISPH loop, launch shape chosen by the batch's autotuner. The
    learned arm records features and trains its network on the plain steps of the lead-in
    (only steps where every scene converged), then warm-starts (auto: LSP_WARM_AUTO, each scene
    switching to the guess after its own step above half the iteration cap or above eta)."""
    from liquidsimulation_b200 import abi, scenes
    from liquidsimulation_b200.solver import batch_from_scenes
    scs = scenes.batched_dam_breaks(seed=4 + dist.rank)
    dt = args.dt or scs[0].dt
    b = batch_from_scenes(scs, device=dist.local)
    lib, h = b._lib, b._h
    n = b.total
    lead = min(args.train_steps, 50)
    trained = 0
    loss = None
    if learned:
        b.mlp_record(True)
        b.mlp_set_loss_asymmetry(4.0)
    for t in range(lead):
        st = b.update(dt)
        if learned and all(x.converged for x in st):
            loss = b.mlp_train(iterations=args.train_iters, batch=65536, lr=2e-3, seed=t)
            trained += 1
    if learned:
        b.mlp_record(False)
        b.set_warm_start(abi.LSP_WARM_AUTO if auto else abi.LSP_WARM_MLP)
    tuning, _ = b.autotune(dt, repeats=3)
    for _ in range(args.warmup):
        b.update(dt)
    # The end-to-end arm below replays the timed steps from this state.
    start_state = b.read_state() if not args.no_e2e and not learned else None
    dist.barrier()
    l0 = b.launch_count()
    clocks = ClockSampler(dist.local)
    clocks.start()
    abi.check(lib, lib.lsp_batch_timer_mark(h, 0))
    stats = [b.update(dt) for _ in range(args.steps)]
    abi.check(lib, lib.lsp_batch_timer_mark(h, 1))
    ms = ctypes.c_float()
    abi.check(lib, lib.lsp_batch_timer_elapsed(h, 0, 1, ctypes.byref(ms)))
    clock_info = clocks.stop()
    launches = b.launch_count() - l0
    dist.barrier()
    t_max = dist.max(ms.value)
    updates = dist.sum(float(n) * args.steps)
    flat = [st for step in stats for st in step]
    counts = np.array([sc.n for sc in scs], np.float64)
    its = np.array([[st.iterations for st in step] for step in stats], np.float64)
    k_mean = float((its * counts).sum() / (counts.sum() * len(stats)))
    eta = scs[0].params.pci_eta
    arm = {"value": updates / (t_max / 1e3), "ms_per_step": t_max / args.steps, "updates": updates,
           "iterations": {"mean_particle_weighted": k_mean, "min": int(its.min()), "max": int(its.max())},
           "max_density_error_ratio": float(max(st.max_density_error_ratio for st in flat)),
           "qualifying_scene_steps": sum(1 for st in flat if st.converged and st.max_density_error_ratio <= eta + 1e-12),
           "scene_steps": len(flat), "warm_start_kept": sum(st.warm_start_used for st in flat),
           "launches": int(launches), "clocks": clock_info, "k_mean": k_mean,
           "autotune": {"threads": tuning.threads, "loop_blocks": tuning.loop_blocks,
                        "candidates": [{"threads": tuning.cand_threads[i], "loop_blocks": tuning.cand_loop_blocks[i],
                                        "ms": round(tuning.cand_ms[i], 4)} for i in range(tuning.candidates)]},
           "launch": b.get_launch(), "lead": lead,
           "train": {"trained_on_steps": trained, "loss": loss} if learned else None}
    e2e = None
    if not args.no_e2e and not learned:
        b.write_state(*start_state)
        bufs = []
        for size in (12 * n, 12 * n, 12 * n, 12 * n, 4 * n):
            ptr = ctypes.c_void_p()
            abi.check(lib, lib.lsp_host_alloc(size, ctypes.byref(ptr)))
            bufs.append(ptr)
        fp = ctypes.POINTER(ctypes.c_float)
        x, v, hv, ov = (ctypes.cast(q, fp) for q in bufs[:4])
        first = ctypes.cast(bufs[4], ctypes.POINTER(ctypes.c_int32))
        abi.check(lib, lib.lsp_batch_read_state(h, x, v, hv, ov, first, n))
        st = (abi.LspStepStats * len(scs))()
        dist.barrier()
        abi.check(lib, lib.lsp_batch_timer_mark(h, 2))
        for _ in range(args.steps):
            abi.check(lib, lib.lsp_batch_write_state(h, x, v, hv, ov, first, n))
            abi.check(lib, lib.lsp_batch_step(h, ctypes.c_float(dt), st))
            abi.check(lib, lib.lsp_batch_read_state(h, x, v, hv, ov, first, n))
        abi.check(lib, lib.lsp_batch_timer_mark(h, 3))
        ems = ctypes.c_float()
        abi.check(lib, lib.lsp_batch_timer_elapsed(h, 2, 3, ctypes.byref(ems)))
        e_max = dist.max(ems.value)
        for q in bufs:
            lib.lsp_host_free(q)
        e2e = {"value": dist.sum(float(n) * args.steps) / (e_max / 1e3), "unit": UNIT,
               "h2d_bytes_per_step": int(n * 52), "d2h_bytes_per_step": int(n * 52)}
    arm["e2e"] = e2e
    b.close()
    return scs, dt, arm


def run_batched(args, dist: Dist):
    import torch
    torch.cuda.set_device(dist.local)
    arms = {}
    if args.warm in ("compare", "zero"):
        scs, dt, arms["plain"] = batched_arm(args, dist, learned=False)
    if args.warm in ("compare", "mlp"):
        scs, dt, arms["learned"] = batched_arm(args, dist, learned=True)
    if args.warm == "compare":
        scs, dt, arms["auto"] = batched_arm(args, dist, learned=True, auto=True)
    head = "plain" if "plain" in arms else "learned"
    main = arms[head]
    n = sum(sc.n for sc in scs)
    # Whole-step roofline (the graph runs every pass back to back): algorithmic bytes of all
    # passes per particle-update over the device time of a step.
    per_update = sum(ALGO_BYTES[k] for k in ("grid_keys", "grid_scatter", "grid_gather", "neighbors",
                                             "nonpressure", "integrate_collide")) \
        + ALGO_BYTES["pci_loop"] * main["k_mean"]
    try:
        peak, src = float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["hbm_gbs"]), "measured"
    except Exception:
        peak, src = 6650.0, "fallback"
    step_s = main["ms_per_step"] / 1e3
    achieved = per_update * n / step_s / 1e9
    result = {
        "metric": METRIC, "value": main["value"], "unit": UNIT, "n_gpus": dist.world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": main["ms_per_step"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded lattice scenes)",
        "config": line_config(args, dist.world),
        "launch": main["launch"], "autotune": main["autotune"],
        "iterations": main["iterations"],
        "iterations_mean": main["k_mean"],
        "particle_iterations_per_s": main["value"] * main["k_mean"],
        "max_density_error_ratio": main["max_density_error_ratio"],
        "qualifying_scene_steps": main["qualifying_scene_steps"], "scene_steps": main["scene_steps"],
        "roofline": {"bound": "hbm", "kernel": "whole batched step (graph)", "achieved": round(achieved, 1),
                     "peak": peak, "peak_source": src, "unit": "GB/s", "frac": round(achieved / peak, 4),
                     "algorithmic_bytes_per_launch": int(per_update * n), "avg_launch_ms": round(step_s * 1e3, 5),
                     "traffic": None},
        "e2e": main["e2e"],
        "gpu_launches": main["launches"],
        "clocks": main["clocks"],
    }
    if "learned" in arms and head == "plain":
        lrn = arms["learned"]
        result["learned"] = {k: lrn[k] for k in ("value", "ms_per_step", "iterations", "max_density_error_ratio",
                                                  "qualifying_scene_steps", "warm_start_kept", "launches", "train")}
        result["learned_vs_plain"] = lrn["value"] / main["value"]
    if "auto" in arms and head == "plain":
        aut = arms["auto"]
        result["auto"] = {k: aut[k] for k in ("value", "ms_per_step", "iterations", "max_density_error_ratio",
                                               "qualifying_scene_steps", "warm_start_kept", "launches")}
        result["auto_vs_plain"] = aut["value"] / main["value"]
    return result


WATERFALL_SPEED = 1.5    # m/s, the emitted sheet's velocity along +x


def waterfall_arm(args, dist: Dist, learned: bool):
    """One arm of the waterfall: grows the scene to --wf-particles by appending 40 x 50
    sheets (spacing 0.008 m, 1.5 m/s along +x), then times K more steps with the emitter
    running. --emit every-step appends a sheet before every step, as the workload specifies;
    --emit reference appends one when the time accumulated since the last sheet reaches one
    lattice spacing of travel, spacing / speed, and then restarts the count, as the
    reference's waterfall scenario does (WaterfallScenario.cpp:55-74: 1.6 r / inflow speed).
    The learned arm runs OnlineWarmStart: plain training steps for the first 50 steps and then
    every 500th step, the network's guess on the others, the zero start as fallback."""
    from liquidsimulation_b200 import abi, scenes
    from liquidsimulation_b200.solver import from_scene, OnlineWarmStart
    sc = scenes.waterfall(seed=5 + dist.rank)
    s = from_scene(sc, device=dist.local)
    lib, h = s._lib, s._h
    policy = OnlineWarmStart(s, every=500, lead=50, iterations=args.train_iters) if learned else None
    interval = np.float32(np.float32(sc.spacing) / np.float32(WATERFALL_SPEED))
    acc = np.float32(0.0)
    sheet = 0

    def emit():
        nonlocal acc, sheet
        if args.emit == "reference":
            acc = np.float32(acc + np.float32(sc.dt))
            if acc < interval:
                return 0
            acc = np.float32(0.0)
        x, v = scenes.waterfall_sheet(sheet, seed=5 + dist.rank)
        s.add_particles(x, v)
        sheet += 1
        return x.shape[0]

    def step():
        return policy.update(sc.dt) if policy else s.update(sc.dt)

    steps_before = 0
    while s.get_particle_count() < args.wf_particles:
        emit()
        if s.get_particle_count():
            step()
        steps_before += 1
    for _ in range(args.warmup):
        emit()
        step()
    n0 = s.get_particle_count()
    dist.barrier()
    l0 = ctypes.c_int64()
    lib.lsp_launch_count(h, ctypes.byref(l0))
    clocks = ClockSampler(dist.local)
    clocks.start()
    abi.check(lib, lib.lsp_timer_mark(h, 0))
    stats, updates = [], 0
    for _ in range(args.steps):
        emit()
        updates += s.get_particle_count()
        stats.append(step())
    abi.check(lib, lib.lsp_timer_mark(h, 1))
    ms = ctypes.c_float()
    abi.check(lib, lib.lsp_timer_elapsed(h, 0, 1, ctypes.byref(ms)))
    clock_info = clocks.stop()
    l1 = ctypes.c_int64()
    lib.lsp_launch_count(h, ctypes.byref(l1))
    dist.barrier()
    t_max = dist.max(ms.value)
    total = dist.sum(float(updates))
    eta = sc.params.pci_eta
    out = {"value": total / (t_max / 1e3), "ms_per_step": t_max / args.steps, "particles_at_start": n0,
           "steps_before": steps_before + args.warmup, "sheets_emitted": sheet,
           "iterations": {"mean": float(np.mean([x.iterations for x in stats])),
                          "max": int(max(x.iterations for x in stats))},
           "max_density_error_ratio": float(max(x.max_density_error_ratio for x in stats)),
           "qualifying_steps": sum(1 for x in stats if x.converged and x.max_density_error_ratio <= eta + 1e-12),
           "launches": int(l1.value - l0.value), "clocks": clock_info}
    if policy:
        out["online_training"] = {"training_steps": policy.training_steps, "trained_steps": policy.trained_steps,
                                  "warm_steps": policy.warm_steps, "fallback_steps": policy.fallback_steps,
                                  "warm_kept_in_timed_steps": sum(x.warm_start_used for x in stats)}
    s.close()
    return out


def run_waterfall(args, dist: Dist):
    import torch
    torch.cuda.set_device(dist.local)
    plain = waterfall_arm(args, dist, learned=False)
    line = {
        "metric": METRIC, "value": plain["value"], "unit": UNIT, "n_gpus": dist.world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": plain["ms_per_step"], "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded emitted sheets)",
        "config": line_config(args, dist.world),
        "particles_at_start": plain["particles_at_start"], "emitted_steps_before": plain["steps_before"],
        "sheets_emitted": plain["sheets_emitted"],
        "iterations": plain["iterations"], "iterations_mean": plain["iterations"]["mean"],
        "particle_iterations_per_s": plain["value"] * plain["iterations"]["mean"],
        "max_density_error_ratio": plain["max_density_error_ratio"], "qualifying_steps": plain["qualifying_steps"],
        "roofline": None, "e2e": None, "gpu_launches": plain["launches"], "clocks": plain["clocks"],
    }
    if args.warm == "compare":
        lrn = waterfall_arm(args, dist, learned=True)
        line["learned"] = {k: lrn[k] for k in ("value", "ms_per_step", "iterations", "max_density_error_ratio",
                                              "qualifying_steps", "launches", "online_training")}
        line["learned_vs_plain"] = lrn["value"] / plain["value"]
    return line


# ------------------------------------------------------------------ CPU (reference) arm

def host_cores():
    """(threads the process may use, physical cores, CPU model) of this host."""
    threads = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
    cores, model, phys = set(), None, None
    try:
        with open("/proc/cpuinfo") as fh:
            for ln in fh:
                k, _, v = ln.partition(":")
                k, v = k.strip(), v.strip()
                if k == "model name" and model is None:
                    model = v
                elif k == "physical id":
                    phys = v
                elif k == "core id":
                    cores.add((phys, v))
    except OSError:
        pass
    return threads, (len(cores) or None), model


def cpu_reference_sample(args, steps, warmup, seconds, threads=None, kind=None, min_iterations=None):
    """Times a CPU solver on one independent sub-scene of the workload per host thread:
    kind "reference" is the reference's own sequential solver (oracle/_ref, its loop without
    a minimum iteration count), kind "port" the oracle restatement (one thread per
    sub-scene, min_iterations as given). Every sub-scene first runs the workload's untimed
    lead-in, so the timed steps come from the same phase of the flow as the GPU arm's."""
    from oracle import oracle as O
    kind = kind or ("reference" if O.ref_available() else "port")
    threads = threads or host_cores()[0]
    sc = sample_scene(args.workload, CPU_SAMPLE_PARTICLES)
    if args.dt:
        sc.dt = args.dt
    if min_iterations is not None:
        sc.params.pci_min_iterations = min_iterations
    elif kind == "reference":
        sc.params.pci_min_iterations = 1   # the reference has no minimum; its loop bound stays 50
    if args.workload == "batched":
        lead = min(args.train_steps, 50) + 1
    elif args.workload == "waterfall":
        lead = 0
    else:
        lead = lead_steps(args)
    if kind == "reference":
        def make():
            return O.RefSolver(sc)
    else:
        def make():
            return O.OracleSolver(sc)
    solvers = [make() for _ in range(threads)]
    iterations = []

    def advance(solver, k, record):
        if kind == "port":
            O.set_threads(1)   # OpenMP's thread count is per calling thread: one core per sub-scene
        for _ in range(k):
            r = solver.step(sc.dt)
            if record:
                iterations.append(r if isinstance(r, int) else r.iterations)

    def run(k, record=False):
        ts = [threading.Thread(target=advance, args=(s, k, record)) for s in solvers]
        for t in ts:
            t.start()
        for t in ts:
            t.join()

    t_lead = time.perf_counter()
    run(lead)
    t_lead = time.perf_counter() - t_lead
    run(warmup)
    step_times = []
    deadline = time.perf_counter() + seconds
    for _ in range(steps):
        t0 = time.perf_counter()
        run(1, record=True)
        step_times.append(time.perf_counter() - t0)
        if time.perf_counter() > deadline:
            break
    iterations_mean = float(np.mean(iterations)) if iterations else None
    # The reference is single-threaded: one sub-scene alone on one core, one more step.
    t0 = time.perf_counter()
    advance(solvers[0], 1, False)
    single = sc.n / (time.perf_counter() - t0)
    for s in solvers:
        s.close()
    per_step = float(np.mean(step_times))
    value = threads * sc.n / per_step
    _, phys, model = host_cores()
    return {"value": value, "unit": UNIT, "cores": threads, "kind": kind,
            "sample": f"{threads} independent {sc.n}-particle sub-scenes of {args.workload} (same spacing, "
                      f"parameters and walls), {len(step_times)} timed steps after a {lead}-step lead-in and "
                      f"{warmup} warm-up, min {sc.params.pci_min_iterations} / max "
                      f"{sc.params.pci_max_iterations} PCISPH iterations",
            "steps_timed": len(step_times), "ms_per_step": per_step * 1e3, "lead_steps": lead,
            "lead_s": round(t_lead, 2), "single_core_value": single, "physical_cores": phys, "cpu_model": model,
            "iterations_mean": iterations_mean,
            "particle_iterations_per_s": value * iterations_mean if iterations_mean else None}


def run_reference(args):
    threads, phys, model = host_cores()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    r = cpu_reference_sample(args, args.steps, args.warmup, seconds=max(30.0, args.cpu_seconds), threads=threads)
    line = {
        "metric": METRIC, "value": r["value"], "unit": UNIT, "n_gpus": 0, "steps": r["steps_timed"],
        "warmup": args.warmup, "ms_per_step": r["ms_per_step"], "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded lattice scenes)", "impl": "reference",
        "config": line_config(args, world),
        "iterations_mean": r["iterations_mean"], "particle_iterations_per_s": r["particle_iterations_per_s"],
        "cpu_baseline": {k: r[k] for k in ("value", "unit", "cores", "kind", "sample", "physical_cores",
                                           "cpu_model", "iterations_mean", "single_core_value")},
        "e2e": {"value": r["value"], "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    if args.workload not in ("dam_break_sph",):
        # The restatement with the GPU arm's iteration rule (min 3), beside the reference's own.
        sc = sample_scene(args.workload, CPU_SAMPLE_PARTICLES)
        port = cpu_reference_sample(args, min(args.steps, 5), 1, seconds=15.0, threads=threads, kind="port",
                                    min_iterations=sc.params.pci_min_iterations)
        line["port_same_iteration_rule"] = {k: port[k] for k in ("value", "cores", "kind", "sample",
                                                                  "iterations_mean", "particle_iterations_per_s")}
    return line


def spawn_ranks(args):
    """`python bench.py --gpus N` without torchrun: starts N ranks of this same command on this
    host, one per GPU (RANK = LOCAL_RANK = r, WORLD_SIZE = N, MASTER_ADDR 127.0.0.1 and a free
    port), as torchrun would, and waits for all of them. Rank 0 prints the line; the exit
    status is the worst of the ranks'."""
    import socket
    import subprocess
    with socket.socket() as sk:
        sk.bind(("127.0.0.1", 0))
        port = sk.getsockname()[1]
    procs = []
    for r in range(args.gpus):
        env = dict(os.environ, RANK=str(r), LOCAL_RANK=str(r), WORLD_SIZE=str(args.gpus),
                   MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
        procs.append(subprocess.Popen([sys.executable, os.path.abspath(__file__), *sys.argv[1:]], env=env,
                                      stdout=None if r == 0 else subprocess.DEVNULL))
    return max(p.wait() for p in procs)


def run_dry(args, dist: Dist):
    """--dry-run: the replica path on the CPU. Each rank steps its own seeded sample of the
    workload with the oracle for K steps (after W warm-up steps), times them on the host, and
    the ranks combine the counts and the slowest time exactly as the GPU run does."""
    from oracle import oracle as O
    sc = sample_scene(args.workload if args.workload != "batched" else "dam_break_pcisph", 2000)
    O.set_threads(1)
    o = O.OracleSolver(sc)
    for _ in range(args.warmup):
        o.step(sc.dt)
    dist.barrier()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        o.step(sc.dt)
    ms = (time.perf_counter() - t0) * 1e3
    o.close()
    dist.barrier()
    t_max = dist.max(ms)
    updates = dist.sum(float(sc.n) * args.steps)
    return {"metric": METRIC, "value": updates / (t_max / 1e3), "unit": UNIT, "n_gpus": dist.world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": t_max / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded lattice scenes)",
            "config": {"workload": f"dry run: {sc.n}-particle CPU oracle sample of {args.workload} per rank",
                       "parallelism": f"replicas x{dist.world}" if dist.world > 1 else "single process"},
            "dry_run": True, "particles_per_rank": sc.n}


def main():
    args = parse()
    if args.gpus > 1 and "WORLD_SIZE" not in os.environ:
        return spawn_ranks(args)
    if args.impl == "reference":
        rank = int(os.environ.get("RANK", "0"))
        if rank != 0:
            return 0
        print(json.dumps(run_reference(args)))
        return 0
    dist = Dist(args.gpus, backend="gloo" if args.dry_run else "nccl")
    try:
        if args.dry_run:
            res = run_dry(args, dist)
        elif args.workload == "batched":
            res = run_batched(args, dist)
        elif args.workload == "waterfall":
            res = run_waterfall(args, dist)
        else:
            res = run_ours(args, dist)
        if dist.rank == 0:
            if not args.no_cpu_baseline and dist.world == 1 and not args.dry_run:
                cb = res["cpu_baseline"] = cpu_reference_sample(args, 3, 1, args.cpu_seconds)
                # Per unit of PCISPH work: the CPU sample's sub-scenes need fewer iterations per
                # step than the full scene, so particle-iterations/s compares like with like.
                if cb.get("particle_iterations_per_s") and res.get("particle_iterations_per_s"):
                    res["vs_cpu_baseline"] = {
                        "particle_updates": res["value"] / cb["value"],
                        "particle_iterations": res["particle_iterations_per_s"] / cb["particle_iterations_per_s"]}
            print(json.dumps(res))
    finally:
        dist.close()
    return 0


if __name__ == "__main__":
    sys.exit(main())
