"""Benchmark of the GB300 mesh-to-SDF engine on the 0.10 mm mug workload.

Workload (one step = one full mesh-to-SDF build): the procedural mug (cup of
revolution + swept-torus handle) with ~180k triangles on an 860 x 860 x 880 lattice at
0.1 mm (650,848,000 voxels, 2.6 GB of FP32), fast path. The headline mode is exact
signs (signed crossings, exact winding number for columns through holes and for the
3 x 4096 stratified probes, the reference's 8-round lockstep eikonal); `plain` reports
the reference-compatible mode (parity signs, same eikonal) on the same lattice.

* value   -- Gvoxels/s with the triangles resident in HBM and the grid written to
             HBM (device buffers), timed with CUDA events around K steps.
* e2e     -- the same through the public API with host buffers: every step copies the
             triangles from pinned host memory and the whole grid back to pinned host
             memory inside the timed region.
* roofline-- the dominant kernel (the eikonal sweep): 8 algorithmic bytes per voxel
             per directional sweep, averaged over the sweeps of the timed steps (CUDA
             events on the engine's stream), against MEASURED_PEAKS.json hbm_gbs.
* cpu_baseline -- the CPU oracle's restatement of the reference path on this host's
             cores, on a bounded z-slab of the same workload.

`--impl reference` times that CPU restatement (all host threads) as the reference arm.
With torchrun (N > 1) every rank builds its own copy (replicas only); rank 0 prints.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT / "rhizome_v24.15_gb300"))
sys.path.insert(0, str(ROOT))

WORKLOAD = "mug_c2_860"
METRIC = "Gvoxels/s mesh-to-SDF @652M voxels, exact signs; learned+batched vs plain on GB300"
UNIT = "Gvoxels/s"
SWEEPS_PER_ROUND = 6


def _peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled while the timed region runs."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.rows = []
        self._stop = threading.Event()
        self._t = None

    def _run(self):
        while not self._stop.is_set():
            try:
                out = subprocess.run(["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.Q}",
                                      "--format=csv,noheader,nounits"], capture_output=True, text=True,
                                     timeout=5).stdout.strip()
                if out:
                    self.rows.append([c.strip() for c in out.splitlines()[0].split(",")])
            except Exception:
                pass
            self._stop.wait(0.2)

    def __enter__(self):
        self._t = threading.Thread(target=self._run, daemon=True)
        self._t.start()
        return self

    def __exit__(self, *a):
        self._stop.set()
        if self._t:
            self._t.join(timeout=10)

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"]}
        sm = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({n for r in self.rows for n, v in zip(names, r[5:9]) if v.strip().lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows)}


def max_over_ranks(dist, x: float) -> float:
    """Max of a per-rank float over all ranks (identity without a process group)."""
    if dist is None:
        return float(x)
    import torch

    t = torch.tensor([float(x)], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_gvox(world: int, voxels_per_rank: int, ms_per_step: float) -> float:
    """Whole-job throughput: every rank builds its own grid (replicas); the job's time
    is the slowest rank's."""
    return world * voxels_per_rank / (ms_per_step * 1e-3) / 1e9


def make_workload(dims=None, h=None, name=WORKLOAD):
    from gbsdf import meshgen

    tris, mn, mx, h = meshgen.workload(name, dims=dims, h=h)
    return tris, mn, mx, h


def run_learned_report(gbsdf, torch, dev, mlp):
    """Learned proposals on the two defective workloads -- the 512^3 vessel tree (holes,
    jitter, duplicated vertices) and the 1024^3 spherical-harmonic blob (1% holes) -- with
    exact-signs mode's grid as the sign truth (it equals the FP64 winding number off the
    surface). Per workload: plain (reference) mode; learned mode with no brick proposed
    (every score -inf: the plain signs through the learned pipeline); learned mode with
    the shipped network. `recall` = the share of the no-proposal run's sign errors (voxels
    more than 1e-3 voxel off the surface) that the proposals fix; `exact_decisions` = voxels
    the exact winding kernel decided (columns through holes, patch boxes, proposed bricks),
    against the lattice's voxel count; times are host wall-clock per build (device-resident
    buffers, one warm-up build first)."""
    from gbsdf import learn, meshgen

    def timed(fn):
        fn()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        r = fn()
        torch.cuda.synchronize()
        return r, (time.perf_counter() - t0) * 1e3

    rep = {}
    for name in ("vessel_c3_512", "blob_c5_1024"):
        tris, mn, mx, h = meshgen.workload(name)
        dims = mx.astype(np.int64) - mn + 1
        n = int(np.prod(dims))
        td = torch.from_numpy(tris).to(dev)
        truth = torch.empty(n, dtype=torch.float32, device=dev)
        out = torch.empty_like(truth)
        off = None

        def run(buf, **kw):
            return gbsdf.compute_mesh_sdf(td, h, mn, mx, out=buf, path=gbsdf.PATH_FAST, raise_on_error=False, **kw)[1]

        def errors():
            return int(((torch.signbit(out) != torch.signbit(truth)) & off).sum().item())

        rt, tt = timed(lambda: run(truth, mode=gbsdf.MODE_EXACT_SIGNS))
        off = truth.abs() > 1e-3 * h
        rp, tp = timed(lambda: run(out, mode=gbsdf.MODE_REFERENCE))
        plain = {"status": rp.status, "ms": tp}
        if rp.ok:
            plain["sign_errors"] = errors()
            plain["exact_decisions"] = int(rp.stats["fixup_voxels"] + rp.stats["patched_voxels"])
        low = torch.full((int(np.prod(learn.brick_grid(mn, mx))),), -1e30, dtype=torch.float32, device=dev)
        r0, t0 = timed(lambda: run(out, mode=gbsdf.MODE_LEARNED, brick_scores=low))
        e0 = errors() if r0.ok else None
        rl, tl = timed(lambda: run(out, mode=gbsdf.MODE_LEARNED, mlp_params=mlp))
        el = errors() if rl.ok else None
        decided = int(rl.stats["fixup_voxels"] + rl.stats["patched_voxels"] + rl.stats["proposed"] * 512)
        rep[name] = {
            "voxels": n, "triangles": int(len(tris)),
            "exact_signs": {"ms": tt, "exact_decisions": int(rt.stats["fixup_voxels"] + rt.stats["patched_voxels"])},
            "plain": plain,
            "learned_no_proposals": {"status": r0.status, "ms": t0, "sign_errors": e0,
                                     "escalated": int(r0.stats["escalated"])},
            "learned": {"status": rl.status, "ms": tl, "sign_errors": el, "escalated": int(rl.stats["escalated"]),
                        "proposed_bricks": int(rl.stats["proposed"]), "exact_decisions": decided,
                        "exact_decisions_saved": 1.0 - decided / n,
                        "recall": (None if not e0 or el is None else (e0 - el) / e0)},
        }
        del truth, out, td, low
        torch.cuda.empty_cache()
    return rep


_X_SCHED = {1: "sweep_x_kernel", 2: "sweep_x_tma_kernel", 3: "sweep_x_pipe_kernel", 4: "sweep_x_pipe2_kernel",
            5: "sweep_x_wide_kernel", 6: "sweep_x_pipe_kernel (narrow tiles)"}
_W_SCHED = {1: "sweep_walk_kernel", 2: "sweep_walk_pipe_kernel", 3: "sweep_walk_vec_kernel", 4: "sweep_walk_vec2_kernel",
            5: "sweep_walk_narrow_kernel"}


def _sweep_kernels(sched):
    """Kernel names of a build's last-round sweep schedule (x + 10 w)."""
    return f"{_X_SCHED.get(int(sched) % 10, '?')} (x) / {_W_SCHED.get(int(sched) // 10, '?')} (y, z)"


def run_batched(gbsdf, torch, dev, mode, steps, warmup, local, mlp):
    """The 64-mesh batched workload: one planned batch (one CUDA graph per run) against
    64 sequential single-mesh calls, device-resident triangles and outputs, timed on the
    host around whole runs (each run returns after its last kernel). Modes: the headline
    mode, plain (the reference-compatible fast path) and learned (plain signs, the
    sign-risk network's proposals re-decided exactly, and re-decided signs instead of a
    decline where plain's verify diverges). A plain mesh that declines has no output: the
    reference would rebuild it with its O(voxels x triangles) legacy kernel, which is not
    timed here."""
    from gbsdf import meshgen

    meshes = meshgen.batch_workload()
    dmeshes = [(torch.from_numpy(t).to(dev), h, mn, mx) for t, h, mn, mx in meshes]
    outs = [torch.empty(int(np.prod(mx.astype(np.int64) - mn + 1)), dtype=torch.float32, device=dev)
            for _, _, mn, mx in meshes]
    vox = sum(int(o.numel()) for o in outs)
    tris = sum(len(t) for t, _, _, _ in meshes)

    def timed(fn, slow=False):
        # the plain mode's patch boxes make some of these meshes cost seconds: fewer
        # repetitions for those passes
        w, k = (1, max(1, steps // 2)) if slow else (warmup, steps)
        for _ in range(w):
            fn()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(k):
            fn()
        torch.cuda.synchronize()
        return (time.perf_counter() - t0) / k * 1e3

    res = {"workload": f"64 meshes (mug / vessel tree / perturbed sphere), {tris} triangles, cubic lattices "
                       f"64^3-384^3, {vox} voxels, fast path, device buffers",
           "voxels": vox}
    launches = 0
    for name, m in (("batched", mode), ("batched_plain", gbsdf.MODE_REFERENCE),
                    ("batched_learned", gbsdf.MODE_LEARNED)):
        kw = {"mlp_params": mlp} if m == gbsdf.MODE_LEARNED else {}
        with gbsdf.Batch(dmeshes, outs=outs, mode=m, device=local, **kw) as b:
            st, stats = b.run()
            ms = timed(b.run, slow=(m == gbsdf.MODE_REFERENCE))
            if name == "batched":
                launches = stats[0]["kernel_launches"]
        # a mesh whose verification diverges is declined (the reference's fall-back case);
        # it still costs its full build and is counted in the throughput
        res[name] = {"value": vox / (ms * 1e-3) / 1e9, "unit": UNIT, "ms_per_step": ms,
                     "declined": sum(1 for x in st if x != 0)}
        if m == gbsdf.MODE_LEARNED:
            res[name]["escalated"] = int(sum(x["escalated"] for x in stats))
            res[name]["proposed_bricks"] = int(sum(x["proposed"] for x in stats))

    declined = []

    def sequential(m):
        declined.clear()
        for (t, h, mn, mx), o in zip(dmeshes, outs):
            _, r = gbsdf.compute_mesh_sdf(t, h, mn, mx, out=o, mode=m, path=gbsdf.PATH_FAST, device=local,
                                          raise_on_error=False, mlp_params=mlp if m == gbsdf.MODE_LEARNED else None)
            declined.append(not r.ok)

    for name, m in (("sequential", mode), ("sequential_plain", gbsdf.MODE_REFERENCE),
                    ("sequential_learned", gbsdf.MODE_LEARNED)):
        ms = timed(lambda: sequential(m), slow=(m == gbsdf.MODE_REFERENCE))
        res[name] = {"value": vox / (ms * 1e-3) / 1e9, "unit": UNIT, "ms_per_step": ms,
                     "declined": int(sum(declined))}
    res["graph_kernel_launches"] = launches
    res["learned_batched_vs_plain"] = res["batched_learned"]["value"] / res["sequential_plain"]["value"]
    return res


def run_decode(gbsdf, steps):
    """The wire-format decoders on the bench mug (179,840 triangles): binary STL (decode +
    weld), ASCII STL (tokens, numbers, weld) and OBJ text, through the public API (host
    bytes in, host arrays out, device allocation per call as in the reference), against the
    oracle's single-threaded CPU restatement of the reference's decoders. Host wall-clock
    per call, median of K."""
    from gbsdf import meshgen
    from oracle import oracle as O

    kw, _, _ = meshgen.WORKLOADS[WORKLOAD]
    kw = {k: v for k, v in kw.items() if k != "kind"}
    v, f = meshgen.mug(**kw)
    stl = meshgen.to_binary_stl(v, f)
    obj = meshgen.to_obj_text(v, f, fancy=False)
    astl = meshgen.to_ascii_stl(v, f, fancy=False)
    res = {}
    for name, data, gpu, cpu in (("binary_stl", stl, gbsdf.parse_binary_stl, O.parse_binary_stl),
                                 ("ascii_stl", astl, gbsdf.parse_ascii_stl, O.parse_ascii_stl),
                                 ("obj", obj, gbsdf.parse_obj, O.parse_obj)):
        gpu(data)  # warm-up (context, module load)
        ts = []
        for _ in range(max(3, steps)):
            t0 = time.perf_counter()
            gpu(data)
            ts.append(time.perf_counter() - t0)
        tc = []
        for _ in range(3):
            t0 = time.perf_counter()
            cpu(data)
            tc.append(time.perf_counter() - t0)
        g, c = float(np.median(ts)), float(np.median(tc))
        res[name] = {"bytes": len(data), "gpu_ms": g * 1e3, "gpu_mb_s": len(data) / g / 1e6, "cpu_ms": c * 1e3,
                     "cpu_mb_s": len(data) / c / 1e6, "cpu_threads": 1}
    return res


def run_iso(gbsdf, out_dev, dims, h, mn, steps):
    """The device-resident hand-off: marching cubes of the build's SDF read in place on the
    device (gbsdf_extract_iso_surface with a device grid, mesh left on the device), against
    the reference's route -- the grid taken to the host and uploaded again by the extractor
    (cuda_marching_cubes.cu:864-866) -- with the mesh returned to the host. Host wall-clock
    per call (both calls: count query, then emit), median of K."""
    import torch

    origin = mn.astype(np.float32) * np.float32(h)
    host = out_dev.cpu().numpy()
    res = {}
    for name, fn in (("device_grid", lambda: gbsdf.extract_iso_surface(out_dev, dims, h, origin, 0.0,
                                                                        outputs_on_device=True)),
                     ("host_grid", lambda: gbsdf.extract_iso_surface(host, dims, h, origin, 0.0))):
        fn()
        ts = []
        for _ in range(max(3, steps)):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            v, i = fn()
            torch.cuda.synchronize()
            ts.append(time.perf_counter() - t0)
        res[name] = {"ms": float(np.median(ts)) * 1e3, "vertices": int(len(v)), "triangles": int(len(i) // 3)}
    res["grid_gvox_s"] = float(np.prod(dims)) / (res["device_grid"]["ms"] * 1e-3) / 1e9
    return res


def cpu_baseline(tris, mn, mx, h, z_slab=64, threads=None):
    """The oracle's restatement of the reference path (CPU), bounded to a z-slab of
    the lattice through the middle of the mug. Returns (Gvox/s, seconds, sample desc)."""
    from oracle import oracle as O

    O.build()
    threads = threads or os.cpu_count() or 1
    zc = (int(mn[2]) + int(mx[2])) // 2
    smn = np.array([mn[0], mn[1], zc - z_slab // 2], np.int32)
    smx = np.array([mx[0], mx[1], zc - z_slab // 2 + z_slab - 1], np.int32)
    n = int(np.prod(smx.astype(np.int64) - smn + 1))
    t0 = time.perf_counter()
    status, _, _, st = O.fast_sdf(tris, h, smn, smx, fsm_mode=0, gwn_mode=0, threads=threads)
    dt = time.perf_counter() - t0
    desc = (f"reference fast path restated on CPU (oracle, {threads} threads), extrapolated from a {z_slab}-plane "
            f"z-slab ({n} voxels, {z_slab} of {int(mx[2] - mn[2] + 1)} planes of the 860x860x880 lattice, all "
            f"{len(tris)} triangles, 8 FSM rounds, 3x4096 probes; status {status}) to voxels per second")
    return n / dt / 1e9, dt, desc, threads


def run_reference_gpu(tris, mn, mx, h, runs=2):
    """The reference's own fast path (cuda_rasterizer.cu:796-1159, compiled for sm_103a with
    its own nvcc flags into oracle/_ref by oracle/build_ref.sh) on this GPU, forced at the
    bench lattice: its own timer (host clock around its allocations, triangle upload, build
    and grid download), after one untimed run. A reported figure, not the target; None when
    the library was not built."""
    from oracle import ref_gpu as R

    if not R.available():
        return None
    ms, wall, ok, st = [], [], False, {}
    for i in range(runs):
        t0 = time.perf_counter()
        ok, _, m, st, _ = R.fast_sdf(tris, h, mn, mx)
        if i > 0:
            ms.append(m)
            wall.append((time.perf_counter() - t0) * 1e3)
    n = int(np.prod(mx.astype(np.int64) - mn + 1))
    m = float(np.mean(ms))
    return {"value": n / (m * 1e-3) / 1e9, "unit": UNIT, "ms_per_step": m, "wall_ms": float(np.mean(wall)),
            "accepted": bool(ok), "stats": st,
            "what": "the reference's own CUDA fast path built for sm_103a with its own flags, host-buffer "
                    "in/out (its own timer: allocations, triangle upload, build, grid download)"}


def run_reference_arm(args, rank, world):
    if rank != 0:
        return
    tris, mn, mx, h = make_workload()
    vals = []
    desc = ""
    threads = os.cpu_count() or 1
    for i in range(args.warmup + args.steps):
        v, dt, desc, threads = cpu_baseline(tris, mn, mx, h, z_slab=args.ref_slab, threads=threads)
        if i >= args.warmup:
            vals.append((v, dt))
    value = float(np.mean([v for v, _ in vals]))
    ms = float(np.mean([dt for _, dt in vals]) * 1e3)
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic", "impl": "reference",
            "config": {"workload": f"{WORKLOAD}: procedural mug, 860x860x880 lattice at 0.1 mm, ~180k triangles",
                       "sample": f"z-slab of {args.ref_slab} planes"},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port", "sample": desc},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="engine", choices=["engine", "reference"])
    ap.add_argument("--mode", default="exact-signs", choices=["reference", "exact-signs", "exact", "learned"])
    ap.add_argument("--ref-slab", type=int, default=64)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    # profiling of a smaller lattice of the same mesh (never the reported configuration)
    ap.add_argument("--workload", default=WORKLOAD, help="a named workload of gbsdf.meshgen.WORKLOADS "
                    "(the bench's own is mug_c2_860; the others are for profiling and comparison runs)")
    ap.add_argument("--dims", default=None, help="lattice override nx,ny,nz (profiling runs)")
    ap.add_argument("--h", type=float, default=None, help="voxel size override (profiling runs)")
    ap.add_argument("--no-e2e", action="store_true", help="skip the host-buffer pass (profiling runs)")
    ap.add_argument("--no-plain", action="store_true", help="skip the plain-mode pass (profiling runs)")
    ap.add_argument("--no-batch", action="store_true", help="skip the 64-mesh batched workload")
    ap.add_argument("--sweep-schedule", type=int, default=0,
                    help="force the eikonal sweep schedules, x + 10 w (profiling runs; 0 = autotuned)")
    ap.add_argument("--batch-only", action="store_true",
                    help="only the planned 64-mesh batch in --mode, W + K runs (profiling runs)")
    args = ap.parse_args()

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch.distributed as dist_mod

        dist = dist_mod
        dist.init_process_group("gloo")

    if args.impl == "reference":
        run_reference_arm(args, rank, world)
        if dist:
            dist.barrier()
            dist.destroy_process_group()
        return

    import torch

    import gbsdf

    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    modes = {"reference": gbsdf.MODE_REFERENCE, "exact-signs": gbsdf.MODE_EXACT_SIGNS, "exact": gbsdf.MODE_EXACT,
             "learned": gbsdf.MODE_LEARNED}
    mode = modes[args.mode]
    if args.batch_only:
        from gbsdf import meshgen

        meshes = meshgen.batch_workload()
        dm = [(torch.from_numpy(t).to(dev), hh, a, b) for t, hh, a, b in meshes]
        outs = [torch.empty(int(np.prod(b.astype(np.int64) - a + 1)), dtype=torch.float32, device=dev)
                for _, _, a, b in meshes]
        vox = sum(int(o.numel()) for o in outs)
        with gbsdf.Batch(dm, outs=outs, mode=mode, device=local) as bt:
            for _ in range(args.warmup):
                bt.run()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(args.steps):
                bt.run()
            torch.cuda.synchronize()
            ms = (time.perf_counter() - t0) / args.steps * 1e3
        if rank == 0:
            print(json.dumps({"metric": "planned 64-mesh batch", "value": vox / (ms * 1e-3) / 1e9, "unit": UNIT,
                              "ms_per_step": ms, "steps": args.steps, "warmup": args.warmup, "mode": args.mode}))
        return
    dims_override = tuple(int(x) for x in args.dims.split(",")) if args.dims else None
    tris, mn, mx, h = make_workload(dims_override, args.h, args.workload)
    from gbsdf import learn

    mlp = torch.from_numpy(np.load(learn.MODEL_PATH)["params"]).to(dev)
    dims = mx.astype(np.int64) - mn + 1
    N = int(np.prod(dims))
    T = len(tris)
    tris_dev = torch.from_numpy(tris).to(dev)
    out_dev = torch.empty(N, dtype=torch.float32, device=dev)

    def step_device(m=mode):
        _, res = gbsdf.compute_mesh_sdf(tris_dev, h, mn, mx, out=out_dev, mode=m, path=gbsdf.PATH_FAST,
                                        device=local, mlp_params=mlp, sweep_schedule=args.sweep_schedule)
        return res

    def barrier():
        if dist:
            dist.barrier()
        torch.cuda.synchronize()

    for _ in range(args.warmup):
        step_device()
    barrier()
    stats = []
    with ClockSampler(local) as clk:
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.steps):
            stats.append(step_device().stats)
        e1.record()
        barrier()
    dev_ms = max_over_ranks(dist, e0.elapsed_time(e1) / args.steps)
    value = whole_job_gvox(world, N, dev_ms)

    # the plain (reference-compatible) mode on the same lattice, same protocol
    plain = None
    if args.mode != "reference" and not args.no_plain:
        for _ in range(args.warmup):
            step_device(gbsdf.MODE_REFERENCE)
        barrier()
        p0 = torch.cuda.Event(enable_timing=True)
        p1 = torch.cuda.Event(enable_timing=True)
        p0.record()
        for _ in range(args.steps):
            step_device(gbsdf.MODE_REFERENCE)
        p1.record()
        barrier()
        pms = max_over_ranks(dist, p0.elapsed_time(p1) / args.steps)
        plain = {"mode": "reference", "value": whole_job_gvox(world, N, pms), "ms_per_step": pms}

    # learned mode on the same lattice, same protocol (the shipped network)
    learned = None
    if args.mode != "learned" and not args.no_plain:
        lst = []
        for _ in range(args.warmup):
            step_device(gbsdf.MODE_LEARNED)
        barrier()
        l0 = torch.cuda.Event(enable_timing=True)
        l1 = torch.cuda.Event(enable_timing=True)
        l0.record()
        for _ in range(args.steps):
            lst.append(step_device(gbsdf.MODE_LEARNED).stats)
        l1.record()
        barrier()
        lms = max_over_ranks(dist, l0.elapsed_time(l1) / args.steps)
        learned = {"mode": "learned", "value": whole_job_gvox(world, N, lms), "ms_per_step": lms,
                   "proposed_bricks": int(lst[-1]["proposed"]), "escalated": int(lst[-1]["escalated"])}

    # ---- end to end through the public API with pinned host buffers
    e2e = e2e_ms = None
    if not args.no_e2e:
        tris_pin = torch.from_numpy(tris).pin_memory()
        out_pin = torch.empty(N, dtype=torch.float32).pin_memory()
        tris_np = tris_pin.numpy()
        out_np = out_pin.numpy()
        for _ in range(max(1, args.warmup // 2)):
            gbsdf.compute_mesh_sdf(tris_np, h, mn, mx, out=out_np, mode=mode, path=gbsdf.PATH_FAST, device=local,
                                   mlp_params=mlp)
        barrier()
        e2 = torch.cuda.Event(enable_timing=True)
        e3 = torch.cuda.Event(enable_timing=True)
        e2.record()
        for _ in range(args.steps):
            gbsdf.compute_mesh_sdf(tris_np, h, mn, mx, out=out_np, mode=mode, path=gbsdf.PATH_FAST, device=local,
                                   mlp_params=mlp)
        e3.record()
        barrier()
        e2e_ms = max_over_ranks(dist, e2.elapsed_time(e3) / args.steps)
        e2e = whole_job_gvox(world, N, e2e_ms)

    # ---- roofline of the dominant kernel (eikonal sweeps), events on the engine's stream
    s0 = stats[-1]
    rounds = [s["eikonal_rounds"] - s["extra_rounds"] for s in stats]
    eik_ms = [s["ms_eikonal"] for s in stats]
    sweep_ms = [s["ms_sweeps"] if s["ms_sweeps"] > 0 else s["ms_eikonal"] for s in stats]
    sweeps = [r * SWEEPS_PER_ROUND for r in rounds]
    per_launch_ms = float(np.mean([m / max(k, 1) for m, k in zip(sweep_ms, sweeps)]))
    stage_launch_ms = float(np.mean([m / max(k, 1) for m, k in zip(eik_ms, sweeps)]))
    alg_bytes = 8.0 * N
    achieved = alg_bytes / (per_launch_ms * 1e-3) / 1e9
    peak, peak_kind = _peaks()
    traffic = None
    prof = ROOT / "profiles" / "eikonal_sweep_traffic.json"
    if prof.exists():
        try:
            traffic = json.loads(prof.read_text()).get("bytes_per_launch_full_size")
        except Exception:
            traffic = None

    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": dev_ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": (f"{WORKLOAD}: procedural mug (cup of revolution + swept-torus handle), "
                                    if args.workload == WORKLOAD else f"{args.workload}: ") +
                                   f"{'x'.join(str(int(d)) for d in dims)} lattice at {h:g} mm, {T} triangles, "
                                   "fast path",
                       "mode": args.mode, "parallelism": "replicas" if world > 1 else "single GPU",
                       "l2": "inputs larger than L2 (2.6 GB grid per step)"},
            "e2e": None if e2e is None else {"value": e2e, "unit": UNIT, "ms_per_step": e2e_ms,
                                             "h2d_bytes_per_step": int(T * 48), "d2h_bytes_per_step": int(N * 4)},
            "roofline": {"kernel": "eikonal directional sweeps, autotuned: " + _sweep_kernels(s0["sweep_schedule"]),
                         "bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": traffic, "peak_kind": peak_kind,
                         "alg_bytes_per_launch": alg_bytes, "launch_ms": per_launch_ms,
                         "stage_frac": alg_bytes / (stage_launch_ms * 1e-3) / 1e9 / peak,
                         "note": "8 algorithmic bytes per voxel per directional sweep; achieved = those bytes "
                                 "over the mean CUDA-event time per sweep of the timed builds (events around the "
                                 "rounds of sweeps, launch gaps and round bookkeeping included); stage_frac "
                                 "charges the whole eikonal stage (padded copies, audit, clamp) to the sweeps"},
            "stages_ms": {k: round(float(np.mean([s[k] for s in stats])), 3)
                          for k in ("ms_prep", "ms_splat", "ms_parity", "ms_fixup", "ms_eikonal", "ms_sweeps",
                                    "ms_verify", "ms_apply")},
            "pipeline": {k: s0[k] for k in ("eikonal_rounds", "probes", "sites", "patch_rounds", "patched_voxels",
                                             "unknown_columns", "band_voxels", "splat_evals", "gwn_pairs",
                                             "fp64_rechecks", "sweep_schedule", "sweep_schedule_first")},
            "plain": plain,
            "learned": learned,
            "precision": {"band_err_fp64_vox": s0["band_err_fp64"], "band_err_samples": s0["band_err_samples"],
                          "what": "largest |FP32 - FP64| band-splat distance over sampled band voxels, in voxels"},
            "clocks": clk.summary(),
            "gpu_launches": int(sum(s["kernel_launches"] for s in stats))}
    if mode == gbsdf.MODE_LEARNED:
        line["pipeline"]["proposed_bricks"] = s0["proposed"]
    if rank == 0 and not args.no_batch:
        line["decode"] = run_decode(gbsdf, args.steps)
        line["iso_surface"] = run_iso(gbsdf, out_dev, dims, h, mn, args.steps)
    if not args.no_batch and mode in (gbsdf.MODE_REFERENCE, gbsdf.MODE_EXACT_SIGNS):
        line["batched"] = run_batched(gbsdf, torch, dev, mode, args.steps, args.warmup, local, mlp)
    if rank == 0 and world == 1 and not args.no_batch and args.workload == WORKLOAD:
        line["learned_report"] = run_learned_report(gbsdf, torch, dev, mlp)
    if rank == 0 and world == 1 and not args.no_cpu_baseline and args.workload == WORKLOAD:
        line["reference_gpu"] = run_reference_gpu(tris, mn, mx, h)
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        v, dt, desc, threads = cpu_baseline(tris, mn, mx, h)
        line["cpu_baseline"] = {"value": v, "unit": UNIT, "cores": threads, "kind": "port", "sample": desc,
                                "seconds": dt}
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
