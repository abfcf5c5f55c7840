#!/usr/bin/env python
"""Benchmark of the XPBD cloth substep on GB300.

Workload (default ``drape256``): a 256 x 256 cloth (65536 vertices, 130050
faces) over a static 20480-face sphere; per frame 10 substeps, each with a
cell-grid LBVH rebuild of both meshes, 30 Jacobi spring/bending iterations,
broad phase in the first iteration, vertex-triangle contact projection in every
iteration, velocity and position update.  One step = one frame.  The metric is
cloth vertex-substeps per second (vertices x substeps / time).

Timing: W untimed warm-up frames, then K timed frames; before each timed frame a
256 MiB buffer is written to flush L2 (the frame's own working set, a few MB,
is smaller than L2); each frame is bracketed by CUDA events on the solver's
stream.  ``e2e`` repeats the measurement through the public API with the
state uploaded from pinned host memory and downloaded again inside the timed
region.  ``roofline`` reports the dominant kernel (the contact-pair projection,
about half of a frame) timed with CUDA events over a graph of back-to-back
launches; ``roofline_sweep`` the same for the Jacobi sweep.  ``cpu_baseline`` times the CPU
oracle (a port of the reference algorithm, OpenMP on all host cores) on one
substep of the same scene.

``--impl reference`` times that CPU port alone as the reference arm.
Multi-GPU (torchrun): every rank runs an independent replica of the workload
(the substep has no cross-cloth exchange); the value is the sum of the
replicas' work divided by the slowest rank's time.
"""
from __future__ import annotations

import argparse
import ctypes as C
import json
import os
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

METRIC = "cloth vertex-substeps/s (256x256 self-collision drape, 10 substeps x 30 Jacobi iterations)"
UNIT = "vertex-substeps/s"


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--workload", choices=["drape256", "plain64"], default="drape256")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--eager", action="store_true", help="launch kernels one by one instead of replaying a graph")
    ap.add_argument("--no-lbvh", action="store_true", help="skip the standalone 2^20-triangle LBVH measurement")
    ap.add_argument("--no-batched", action="store_true", help="skip the 512-cloth batched measurement")
    ap.add_argument("--only-batched", action="store_true", help="run only the 512-cloth batched measurement")
    ap.add_argument("--no-learned", action="store_true", help="skip the learned warm-start measurement")
    ap.add_argument("--only-learned", action="store_true", help="run only the learned warm-start measurement")
    ap.add_argument("--only-lbvh", action="store_true",
                    help="run only the standalone 2^20-triangle LBVH measurement (no CPU baseline)")
    ap.add_argument("--only-color", action="store_true", help="run only the colouring measurement")
    ap.add_argument("--only-plain64", action="store_true", help="run only the 64x64 box-scene measurement")
    ap.add_argument("--only-gs", action="store_true",
                    help="run only the Gauss-Seidel against Jacobi comparison (drape after 3 frames)")
    ap.add_argument("--profile-case", choices=sorted(PROFILE_CASES),
                    help="run one small case of a workload for a profiler capture, print 'ok <case>' and exit "
                         "(no timing, no JSON line)")
    return ap.parse_args()


def _case_drape(pkg):
    """Two frames of the 256 x 256 drape with eager launches (every kernel of a frame)."""
    scene = pkg.scenes.drape256()
    sim = pkg.scenes.make_solver(scene, device="cuda")
    sim.bending_on = "y"
    for _ in range(2):
        sim.forward(scene.n_substeps)


def _case_soup(pkg):
    """The 2^20-triangle LBVH build and query, two repetitions."""
    lbvh_soup(pkg, reps=2, with_cpu=False)


def _batched_case_solver(pkg, n_iter):
    insts = pkg.batched_scene(512, seed=0)
    return pkg.BatchedSolver(insts, dHat=(4e-3) ** 2, stiffness_stretch=1e5, stiffness_bending=1e8,
                             g=(0.0, 0.0, -9.81), dt=1 / 60, n_iter=n_iter, padding=8e-3)


def _case_batched(pkg):
    """The 512-cloth batch: two frames of grid-wide launches, then one frame of
    persistent launches (one per substep)."""
    sim = _batched_case_solver(pkg, 20)
    for _ in range(2):
        sim.forward(10)
    sim.persistent = True
    sim.forward(10)


def _case_sweeps(pkg):
    """One sweep of each kind over the 512-cloth batch from its rest state:
    int2 exact, int2 fast, packed staged exact and fast, packed direct exact
    and fast."""
    import torch
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    sim = _batched_case_solver(pkg, 20)
    dt = 1.0 / 600.0
    ks, kb = 1e8 * dt * dt, 1e5 * dt * dt
    out = torch.empty_like(sim.y4)
    for fast in (0, 1):
        sx.sx_jacobi_sweep_mode(ptr(sim.x4), ptr(sim.x4), ptr(out), ptr(sim.fixed), ptr(sim.adj_ptr), ptr(sim.adj),
                                sim.num_verts, ks, kb, 1, 0, fast, stream_handle())
    for form in (0, 1):
        for fast in (0, 1):
            sx.sx_jacobi_sweep_packed_v(ptr(sim.x4), ptr(sim.x4), ptr(out), ptr(sim.fixed), ptr(sim.adj_ptr),
                                        ptr(sim.adj_nbr16), ptr(sim.adj_rest32), sim.num_verts, ks, kb, 1, form, fast,
                                        stream_handle())


def _case_drape_sweeps(pkg):
    """One sweep of each storage form over the 256 x 256 drape's cloth from its
    predicted state (int2, packed staged, packed direct forms), exact arithmetic."""
    import torch
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    scene = pkg.scenes.drape256()
    sim = pkg.scenes.make_solver(scene, device="cuda")
    m = sim.mesh_dy
    dt = scene.dt / scene.n_substeps
    sim.compute_y(dt)
    ks, kb = sim.stiffness_bending * dt * dt, sim.stiffness_stretch * dt * dt
    out = torch.empty_like(m.y4)
    sx.sx_jacobi_sweep_mode(ptr(m.x4), ptr(m.y4), ptr(out), ptr(m.fixed), ptr(m.adj_ptr), ptr(m.adj), m.num_verts, ks,
                            kb, 1, 7, 0, stream_handle())
    for form in range(int(sx.sx_jacobi_sweep_packed_forms())):
        sx.sx_jacobi_sweep_packed_v(ptr(m.x4), ptr(m.y4), ptr(out), ptr(m.fixed), ptr(m.adj_ptr), ptr(m.adj_nbr16),
                                    ptr(m.adj_rest32), m.num_verts, ks, kb, 1, form, 0, stream_handle())


def _case_lanes(pkg):
    """One sweep in each lanes-per-vertex variant over the 64 x 64 cloth, and
    one FP64 energy reduction of the 256 x 256 drape."""
    import torch
    from starlab_physics_gb300._lib import ptr, stream_handle, sx
    from starlab_physics_gb300.autotune import variant_forms

    scene = pkg.scenes.plain64()
    sim = pkg.scenes.make_solver(scene, device="cuda")
    m = sim.mesh_dy
    dt = scene.dt / scene.n_substeps
    sim.compute_y(dt)
    ks, kb = sim.stiffness_bending * dt * dt, sim.stiffness_stretch * dt * dt
    out = torch.empty_like(m.y4)
    for v, (lanes, _) in enumerate(variant_forms()):
        if lanes > 1:
            sx.sx_jacobi_sweep_mode(ptr(m.x4), ptr(m.y4), ptr(out), ptr(m.fixed), ptr(m.adj_ptr), ptr(m.adj),
                                    m.num_verts, ks, kb, 1, v, 0, stream_handle())
    d = pkg.scenes.make_solver(pkg.scenes.drape256(), device="cuda")
    d.system_energy()


def _case_plain64(pkg):
    """Two frames of the 64 x 64 cloth over the box with eager launches."""
    scene = pkg.scenes.plain64()
    sim = pkg.scenes.make_solver(scene, device="cuda")
    sim.bending_on = "y"
    for _ in range(2):
        sim.forward(scene.n_substeps)


def _case_color(pkg):
    """Colouring of the 256 x 256 cloth's edges (one call)."""
    _, f = pkg.grid_cloth(256)
    pkg.GraphColoring(256 * 256, pkg.mesh.edges_from_faces(f), device="cuda")


def _case_learned(pkg):
    """One batched frame with the (untrained) warm-start network: features,
    inference, warm start and the Jacobi loop."""
    sim = _batched_case_solver(pkg, 4)
    sim.warm = pkg.learned.WarmStart(sim, pkg.WarmStartMLP(seed=0))
    sim.forward(10)


def _case_widening(pkg):
    """One substep of each optional path on a 128 x 128 drape (pair records +
    velocity-level contacts and friction + edge-edge contacts; Gauss-Seidel
    sweeps; iterating to a tolerance), sewing on the 64 x 64 cloth, 65 536
    edge-edge classifications, one Adam step of the warm-start network on
    65 536 rows, the FP64 energy, and a 2^18-face LBVH under the reference's tie
    rule."""
    import numpy as np
    import torch
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    scene = pkg.scenes.drape256(n=128)
    cl = pkg.TriMesh(scene.cloth_x, scene.cloth_faces, device="cuda")
    ob = pkg.TriMesh(scene.obstacle_x, scene.obstacle_faces, device="cuda", is_static=True)
    sim = pkg.Solver(cl, ob, dHat=scene.dHat, stiffness_stretch=scene.stiffness_stretch,
                     stiffness_bending=scene.stiffness_bending, g=scene.gravity, dt=scene.dt, n_iter=2,
                     rebuild=scene.rebuild, cap=scene.cap, record_pairs=True, bending_on="y")
    sim.padding = scene.padding
    sim.enable_collision_handling = True
    sim.enable_velocity_update = True
    sim.enable_edge_edge = True
    sim.mu = 0.4
    sim.forward(1)
    sim.system_energy()
    gs = pkg.scenes.make_solver(pkg.scenes.drape256(n=128), device="cuda")
    gs.bending_on = "y"
    gs.gauss_seidel = True
    gs.n_iter = 1
    gs.forward(1)
    tol = pkg.scenes.make_solver(pkg.scenes.drape256(n=128), device="cuda")
    tol.bending_on = "y"
    tol.tol = 1e-9
    tol.n_iter = 8
    tol.forward(1)
    sew_scene = pkg.scenes.plain64(collisions=False)
    sw = pkg.scenes.make_solver(sew_scene, device="cuda")
    sw.bending_on = "y"
    sw.n_iter = 1
    sw.set_sewing_pairs(np.array([[i, 63 * 64 + i] for i in range(2, 62)], np.int32), 1e5)
    sw.forward(1)
    rng = np.random.default_rng(0)
    n = 1 << 16
    p12 = torch.from_numpy(rng.normal(0, 0.01, (n, 12)).astype(np.float32)).cuda()
    dtype = torch.empty(n, dtype=torch.int32, device="cuda")
    d = torch.empty(n, dtype=torch.float32, device="cuda")
    g12 = torch.empty((n, 12), dtype=torch.float32, device="cuda")
    sx.sx_edge_edge_classify(n, ptr(p12), 1e-4, ptr(dtype), ptr(d), ptr(g12), stream_handle())
    mlp = pkg.WarmStartMLP(seed=0)
    feat = torch.randn((n, 32), device="cuda").to(torch.bfloat16)
    target4 = 1e-4 * torch.randn((n, 4), device="cuda")
    idx = torch.arange(n, dtype=torch.int32, device="cuda")
    mlp.train_step(feat, target4, idx, n)
    nf = 1 << 18
    verts, faces, _ = pkg.scenes.triangle_soup(nf, seed=1)
    V4 = torch.zeros((verts.shape[0], 4), dtype=torch.float32, device="cuda")
    V4[:, :3] = torch.from_numpy(verts).cuda()
    F = torch.from_numpy(faces.reshape(-1)).cuda()
    fmn = torch.empty((nf, 4), dtype=torch.float32, device="cuda")
    fmx = torch.empty_like(fmn)
    box = torch.empty(6, dtype=torch.float32, device="cuda")
    sx.sx_face_aabbs(ptr(V4), ptr(F), nf, 0.0, ptr(fmn), ptr(fmx), stream_handle())
    sx.sx_scene_aabb(ptr(V4), V4.shape[0], 0.0, ptr(box), stream_handle())
    pkg.LBVH(nf, "cuda", tie=0).build(fmn, fmx, box)


PROFILE_CASES = {"drape": _case_drape, "soup": _case_soup, "batched": _case_batched, "color": _case_color,
                 "learned": _case_learned, "sweeps": _case_sweeps, "drape_sweeps": _case_drape_sweeps,
                 "lanes": _case_lanes, "widening": _case_widening, "plain64": _case_plain64}


def run_profile_case(name):
    import torch
    import __graft_entry__ as ge

    pkg = ge.load_package()
    torch.cuda.set_device(0)
    PROFILE_CASES[name](pkg)
    torch.cuda.synchronize()
    print("ok", name)


def dist_setup(n_gpus):
    import torch

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl")
    elif torch.cuda.is_available():
        torch.cuda.set_device(0)
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist

        dist.barrier()


def max_over_ranks(v, world, device="cuda"):
    if world == 1:
        return v
    import torch
    import torch.distributed as dist

    t = torch.tensor([v], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_throughput(units_per_rank, ms_this_rank, world, device="cuda"):
    """Whole-job throughput of independent replicas: every rank processes
    `units_per_rank` work units; the job takes as long as its slowest rank."""
    ms = max_over_ranks(ms_this_rank, world, device)
    return world * units_per_rank / (ms / 1e3), ms


def build_scene(name):
    import __graft_entry__ as ge

    pkg = ge.load_package()
    if name == "drape256":
        return pkg, pkg.scenes.drape256()
    return pkg, pkg.scenes.plain64()


def workload_config(scene, name, sim=None):
    return {
        "workload": f"{name}: {scene.meta.get('grid')}x{scene.meta.get('grid')} cloth, "
                    f"{len(scene.cloth_faces)} faces, obstacle {0 if scene.obstacle_faces is None else len(scene.obstacle_faces)} faces",
        "vertices": int(scene.cloth_x.shape[0]),
        "substeps_per_step": scene.n_substeps,
        "jacobi_iterations": scene.n_iter,
        "bvh_rebuild": scene.rebuild,
        "contact": "vertex-triangle (static + self), dHat=thickness^2",
        "bending_on": "y",
        "l2": "flushed before every timed step (256 MiB write); working set < L2",
    }


class ClockSampler:
    """nvidia-smi clocks/throttle sampling in the background (200 ms)."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if self.proc is None or not self.path:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                rows.append((float(parts[1]), float(parts[2]), parts[5:9]))
            except ValueError:
                continue
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = sorted(r[0] for r in rows)
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i, v in enumerate(r[2]) if v.lower() == "active"})
        return {"sm_mhz": sm[len(sm) // 2], "sm_max_mhz": rows[0][1], "reasons": reasons, "samples": len(rows)}


def measured_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return 6800.0, "fallback"


def ncu_traffic(kernel_file):
    """Per-launch DRAM bytes of the dominant kernel from its committed ncu summary."""
    p = os.path.join(ROOT, "profiles", kernel_file)
    try:
        for line in open(p):
            if line.startswith("traffic_bytes_per_launch:"):
                return float(line.split(":", 1)[1].split()[0])
    except OSError:
        pass
    return None


def _oracle_solver(pkg, scene, nthreads):
    from oracle import pyoracle as po
    from starlab_physics_gb300 import mesh as M

    cl = M.TriMesh(scene.cloth_x, scene.cloth_faces, device="cpu")
    ob = M.TriMesh(scene.obstacle_x, scene.obstacle_faces, device="cpu") if scene.obstacle_x is not None else None
    if len(scene.pinned):
        cl.fixed[scene.pinned] = 0.0
    return po.OracleSolver(pkg.scenes.oracle_inputs(cl), pkg.scenes.oracle_inputs(ob) if ob else None, dt=scene.dt,
                           g=scene.gravity, k_stretch_stiffness=scene.stiffness_stretch,
                           k_bend_stiffness=scene.stiffness_bending, dHat=scene.dHat, damping=scene.damping,
                           padding=scene.padding, n_iter=scene.n_iter, collisions=scene.collisions,
                           rebuild=scene.rebuild, cap=scene.cap, nthreads=nthreads, bending_on="y",
                           contact_cull=True)


def cpu_baseline(pkg, scene, x0, v0, gpu_x_after, frame):
    """The oracle port on all host cores, on the state the GPU arm times (the
    snapshot before frame `frame`): the whole frame (its 10 substeps) timed, and
    its end state compared with the GPU's frame from the same snapshot; then one
    substep on one core."""
    import numpy as np

    cores = os.cpu_count() or 1
    orc = _oracle_solver(pkg, scene, cores)
    orc.x4[:] = x0
    orc.v4[:] = v0
    dt_sub = scene.dt / scene.n_substeps
    t0 = time.perf_counter()
    for _ in range(scene.n_substeps):
        orc.substep(dt_sub)
    el = time.perf_counter() - t0
    d = np.abs(orc.x4[:, :3].astype(np.float64) - gpu_x_after[:, :3])
    p = scene.cloth_x.astype(np.float64)
    diag = float(np.linalg.norm(p.max(0) - p.min(0)))
    V = scene.cloth_x.shape[0]
    n = scene.n_substeps
    orc1 = _oracle_solver(pkg, scene, 1)
    orc1.x4[:] = x0
    orc1.v4[:] = v0
    t0 = time.perf_counter()
    orc1.substep(dt_sub)
    el1 = time.perf_counter() - t0
    return {"value": V * n / el, "unit": UNIT, "cores": cores, "kind": "port",
            "sample": f"frame {frame} of the scene ({n} substeps) from the GPU arm's snapshot on the CPU oracle "
                      f"(OpenMP, {cores} threads), {el:.2f} s",
            "max_abs_dx_vs_gpu": float(d.max()), "max_abs_dx_over_diagonal": float(d.max()) / diag,
            "bit_exact_vs_gpu": bool(d.max() == 0.0),
            "one_core": {"value": V / el1, "unit": UNIT, "cores": 1,
                         "sample": f"1 substep of the same frame, 1 thread, {el1:.2f} s"}}


def plain64_timing(pkg, warm_frames=20, frames=20, with_cpu=True):
    """Configuration 0: the 64 x 64 cloth over the box (10 substeps x 20
    iterations), one CUDA graph per frame, sweep and contact launch
    configurations autotuned; after `warm_frames` frames (the cloth reaches the
    box at about frame 18), `frames` consecutive frames timed with CUDA events
    (the working set is L2-resident).  The CPU leg runs the oracle over the same
    frames from the same state on all host cores and compares end states."""
    import numpy as np
    import torch

    scene = pkg.scenes.plain64()
    sim = pkg.scenes.make_solver(scene, device="cuda")
    sim.bending_on = "y"
    sim.use_graph = True
    S = scene.n_substeps
    sim.forward(S)
    variant, _ = sim.autotune(S)
    pp_variant, _ = sim.autotune_contacts(S)
    for _ in range(warm_frames - 1):
        sim.forward(S)
    torch.cuda.synchronize()
    x0 = sim.mesh_dy.x4.cpu().numpy().copy()
    v0 = sim.mesh_dy.v4.cpu().numpy().copy()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(frames):
        sim.forward(S)
    b.record()
    torch.cuda.synchronize()
    ms = a.elapsed_time(b)
    V = sim.mesh_dy.num_verts
    from starlab_physics_gb300.autotune import variant_forms, variants

    out = {"workload": f"plain64: 64x64 cloth over a 12-face box, {S} substeps x {scene.n_iter} iterations, "
                       f"frames {warm_frames + 1}-{warm_frames + frames}",
           "value": V * S * frames / (ms / 1e3), "unit": UNIT, "ms_per_frame": ms / frames,
           "sweep_config": {"entries_per_load_batch": variants()[variant][0] if variant < len(variants()) else None,
                            "lanes_per_vertex": variant_forms()[variant][0] if variant < len(variants()) else 1,
                            "packed": bool(sim.packed_sweep)},
           "pairs_project_variant": pp_variant, "status_flags": sim.status_flags()}
    if with_cpu:
        cores = os.cpu_count() or 1
        orc = _oracle_solver(pkg, scene, cores)
        orc.x4[:] = x0
        orc.v4[:] = v0
        dt_sub = scene.dt / S
        t0 = time.perf_counter()
        for _ in range(frames * S):
            orc.substep(dt_sub)
        el = time.perf_counter() - t0
        d = np.abs(orc.x4[:, :3].astype(np.float64) - sim.mesh_dy.x4.cpu().numpy()[:, :3])
        out["cpu_baseline"] = {"value": V * S * frames / el, "unit": UNIT, "cores": cores, "kind": "port",
                               "sample": f"the same {frames} frames from the same state on the CPU oracle "
                                         f"(OpenMP, {cores} threads), {el:.2f} s",
                               "max_abs_dx_vs_gpu": float(d.max()), "bit_exact_vs_gpu": bool(d.max() == 0.0)}
    return out


def lbvh_soup(pkg, reps=10, with_cpu=True):
    """Standalone broad phase on 2^20 random triangles: build ms (scene box,
    Morton codes, 32-bit key/index radix sort, Karras hierarchy, refit) and query
    ms for 2^20 vertex boxes with padding 2e-3, each the mean of `reps` runs
    timed with CUDA events (L2 flushed before each)."""
    import numpy as np
    import torch

    n = 1 << 20
    verts, faces, queries = pkg.scenes.triangle_soup(n, seed=0)
    V4 = torch.zeros((verts.shape[0], 4), dtype=torch.float32, device="cuda")
    V4[:, :3] = torch.from_numpy(verts).cuda()
    Q4 = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    Q4[:, :3] = torch.from_numpy(queries).cuda()
    F = torch.from_numpy(faces.reshape(-1)).cuda()
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    fmn = torch.empty((n, 4), dtype=torch.float32, device="cuda")
    fmx = torch.empty_like(fmn)
    box = torch.empty(6, dtype=torch.float32, device="cuda")
    sx.sx_face_aabbs(ptr(V4), ptr(F), n, 0.0, ptr(fmn), ptr(fmx), stream_handle())
    bvh = pkg.LBVH(n, "cuda", tie=1)
    cap = 32
    cand = torch.empty((n, cap), dtype=torch.int32, device="cuda")
    num = torch.empty(n, dtype=torch.int32, device="cuda")
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream()

    def build():
        sx.sx_scene_aabb(ptr(V4), V4.shape[0], 0.0, ptr(box), stream_handle())
        bvh.build(fmn, fmx, box)

    build()
    bvh.query(Q4, 2e-3, cap, cand, num)
    torch.cuda.synchronize()
    tb, tq = [], []
    for _ in range(reps):
        flush.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        build()
        b.record(stream)
        flush.zero_()
        c, d = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        c.record(stream)
        bvh.query(Q4, 2e-3, cap, cand, num)
        d.record(stream)
        torch.cuda.synchronize()
        tb.append(a.elapsed_time(b))
        tq.append(c.elapsed_time(d))
    # the same build under the reference's rule for equal codes (lbvh_cell.py:256-264), whose hierarchy can be
    # malformed where codes repeat, so its refit is the one-thread-per-leaf climb
    bvh0 = pkg.LBVH(n, "cuda", tie=0)

    def build0():
        sx.sx_scene_aabb(ptr(V4), V4.shape[0], 0.0, ptr(box), stream_handle())
        bvh0.build(fmn, fmx, box)

    build0()
    torch.cuda.synchronize()
    t0s = []
    for _ in range(reps):
        flush.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        build0()
        b.record(stream)
        torch.cuda.synchronize()
        t0s.append(a.elapsed_time(b))
    codes = bvh0.codes.cpu().numpy()
    out = {"workload": "2^20-triangle soup, 2^20 queries, padding 2e-3", "build_ms": round(sum(tb) / reps, 4),
           "query_ms": round(sum(tq) / reps, 4), "candidates": int(num.sum().item()),
           "sort_bytes_per_build": n * 64, "tie_rule": "equal codes ordered by index (always a valid tree)",
           "build_ms_reference_tie_rule": round(sum(t0s) / reps, 4),
           "repeated_codes": int(n - np.unique(codes).size)}
    if with_cpu:
        from oracle import pyoracle as po

        vv = np.zeros((verts.shape[0], 4), np.float32)
        vv[:, :3] = verts
        mn, mx = po.face_aabbs(vv, faces, 0.0)
        t0 = time.perf_counter()
        fb = po.FaceBVH(mn, mx, po.scene_aabb(vv, 0.0), tie=1)
        t1 = time.perf_counter()
        ok = bool(np.array_equal(bvh.sorted_ids.cpu().numpy(), fb.sorted_ids)
                  and np.array_equal(bvh.child_a.cpu().numpy(), fb.child_a))
        fb0 = po.FaceBVH(mn, mx, po.scene_aabb(vv, 0.0), tie=0)
        out["matches_oracle_reference_tie_rule"] = bool(
            np.array_equal(bvh0.sorted_ids.cpu().numpy(), fb0.sorted_ids)
            and np.array_equal(bvh0.child_a.cpu().numpy(), fb0.child_a)
            and np.array_equal(bvh0.child_b.cpu().numpy(), fb0.child_b))
        out["cpu_baseline_build_ms"] = round(1e3 * (t1 - t0), 1)
        out["cpu_baseline_kind"] = "port (serial oracle)"
        out["matches_oracle"] = ok
    return out


def batched512(pkg, steps=5, warmup=2, world=1, rank=0):
    """Batched workload: 512 independent cloths (grid side uniform in [16,128],
    about 3.2M vertices) each over its own box, 10 substeps x 20 Jacobi
    iterations, obstacle contacts; one CUDA graph per frame.  Also times the
    Jacobi sweep over all instances, whose working set (~314 MB algorithmic per
    sweep) exceeds L2, against the HBM peak."""
    import torch
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    insts = pkg.batched_scene(512, seed=0)
    if world > 1:  # independent instances: each rank takes a balanced share, nothing is exchanged
        insts = [insts[i] for i in pkg.shard_instances(insts, rank, world)]
    sim = pkg.BatchedSolver(insts, dHat=(4e-3) ** 2, stiffness_stretch=1e5, stiffness_bending=1e8,
                            g=(0.0, 0.0, -9.81), dt=1.0 / 60.0, n_iter=20, padding=8e-3)
    sim.use_graph = True
    V, S = sim.num_verts, 10
    stream = torch.cuda.current_stream()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    sim.forward(S)
    variant, _ = sim.autotune()
    for _ in range(warmup - 1):
        sim.forward(S)
    torch.cuda.synchronize()
    x0, v0 = sim.x4.clone(), sim.v4.clone()
    tot = 0.0
    for _ in range(steps):
        sim.x4.copy_(x0)
        sim.v4.copy_(v0)
        flush.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        sim.forward(S)
        b.record(stream)
        torch.cuda.synchronize()
        tot += a.elapsed_time(b)
    # the sweep alone over every instance (exact and fast arithmetic)
    dt = 1.0 / 600.0
    ks, kb = 1e8 * dt * dt, 1e5 * dt * dt
    n_con = sim.adj.shape[0] // 2
    alg = 12 * n_con + 28 * V
    peak, kind = measured_peak()

    def sweep_roofline(fast, packed=None, form=None):
        """One sweep over every instance, timed alone (L2 flushed before each
        launch, mean of 20): the int2 sweep in the tuned variant, or with
        packed=True the packed sweep, staged (form 0) or direct (form 1) (None:
        whichever the tuner chose)."""
        form = sim.packed_form if packed is None and form is None else (form or 0)
        packed = sim.packed_sweep if packed is None else packed
        ev = []
        for _ in range(20):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            if packed:
                sx.sx_jacobi_sweep_packed_v(ptr(sim.x4), ptr(sim.y4), ptr(sim._y_other), ptr(sim.fixed),
                                            ptr(sim.adj_ptr), ptr(sim.adj_nbr16), ptr(sim.adj_rest32), V, ks, kb, 1,
                                            form, 1 if fast else 0, stream_handle())
            else:
                sx.sx_jacobi_sweep_mode(ptr(sim.x4), ptr(sim.y4), ptr(sim._y_other), ptr(sim.fixed),
                                        ptr(sim.adj_ptr), ptr(sim.adj), V, ks, kb, 1, sim.sweep_variant,
                                        1 if fast else 0, stream_handle())
            b.record(stream)
            ev.append((a, b))
        torch.cuda.synchronize()
        sweep_ms = sum(a.elapsed_time(b) for a, b in ev) / len(ev)
        kname = (("jacobi_sweep_packed_kernel" if form else "jacobi_sweep_staged_kernel") if packed
                 else "jacobi_sweep_kernel")
        return {"kernel": kname, "bound": "hbm",
                "achieved": round(alg / (sweep_ms / 1e3) / 1e9, 1), "peak": peak,
                "unit": "GB/s", "frac": round(alg / (sweep_ms / 1e3) / 1e9 / peak, 4),
                "algorithmic_bytes_per_launch": alg, "avg_launch_us": round(sweep_ms * 1e3, 2), "peak_source": kind}

    exact_sweep = sweep_roofline(False)
    sweeps = {"int2_exact": sweep_roofline(False, False), "int2_fast": sweep_roofline(True, False)}
    if sim.adj_nbr16 is not None:
        sweeps |= {"packed_exact": sweep_roofline(False, True, 0), "packed_fast": sweep_roofline(True, True, 0)}
        from starlab_physics_gb300.autotune import packed_forms

        for fast_, name in ((False, "packed_direct_exact"), (True, "packed_direct_fast")):
            best_ = None
            for f_ in range(1, packed_forms()):
                r_ = sweep_roofline(fast_, True, f_) | {"form": f_}
                if best_ is None or r_["avg_launch_us"] < best_["avg_launch_us"]:
                    best_ = r_
            sweeps[name] = best_
    status = int(sim.status.item())

    def timed_frames():
        sim.x4.copy_(x0)
        sim.v4.copy_(v0)
        sim.forward(S)  # capture
        tot_ = 0.0
        for _ in range(steps):
            sim.x4.copy_(x0)
            sim.v4.copy_(v0)
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            sim.forward(S)
            b.record(stream)
            torch.cuda.synchronize()
            tot_ += a.elapsed_time(b)
        return {"value": V * S * steps / (tot_ / 1e3), "unit": UNIT, "ms_per_step": tot_ / steps}

    # the same frames with the sweep's fast arithmetic (tolerance-validated,
    # not bit-identical)
    sim.fast_math = True
    exact_choice = (sim.sweep_variant, sim.packed_sweep, sim.packed_form)
    sim.x4.copy_(x0)
    sim.v4.copy_(v0)
    sim.forward(S)
    fast_variant, _ = sim.autotune()  # tuned for the fast arithmetic on the same batch
    fast = timed_frames() | {"sweep_roofline": sweep_roofline(True),
                             "sweep_variant": ((f"packed_direct_{sim.packed_form}" if sim.packed_form else "packed") if sim.packed_sweep
                                               else sim.sweep_variant)}
    sim.sweep_variant, sim.packed_sweep, sim.packed_form = exact_choice
    # one persistent launch per substep (an instance per CTA), exact and fast
    sim.fast_math = False
    sim.persistent = True
    sim.x4.copy_(x0)
    sim.v4.copy_(v0)
    pv, ptimes = sim.autotune_persistent()
    from starlab_physics_gb300._lib import load as _load

    def persistent_launch(variant):
        blk, bps = C.c_int(0), C.c_int(0)
        _load().sx_batched_substep_variant_info(variant, C.addressof(blk), C.addressof(bps))
        return {"launch": {"threads_per_cta": blk.value, "ctas_per_sm": bps.value,
                           "ctas_per_instance": int(_load().sx_batched_substep_variant_cluster(variant)),
                           "picked_by": "autotuner (fastest of %d identical variants, one "
                                        "substep each)" % len(ptimes)}}

    persistent = timed_frames() | persistent_launch(pv)
    sim.fast_math = True
    sim.x4.copy_(x0)
    sim.v4.copy_(v0)
    pv, ptimes = sim.autotune_persistent()
    persistent_fast = timed_frames() | persistent_launch(pv)
    sim.fast_math = False
    sim.persistent = False
    value, ms_job = replica_throughput(V * S * steps, tot, world)  # units summed over ranks / slowest rank
    if world > 1:
        import torch.distributed as dist

        t = torch.tensor([V], dtype=torch.float64, device="cuda")
        dist.all_reduce(t)
        value = float(t.item()) * S * steps / (ms_job / 1e3)
    return {"workload": f"512 cloths, {V} vertices on this rank, {sim.num_faces} faces, 10 substeps x 20 "
                        "iterations, obstacle contacts" + (f", instances split over {world} ranks" if world > 1
                                                            else ""),
            "value": value, "unit": UNIT,
            "ms_per_step": ms_job / steps, "steps": steps, "warmup": warmup,
            "sweep_variant": ((f"packed_direct_{sim.packed_form}" if sim.packed_form else "packed") if sim.packed_sweep
                              else sim.sweep_variant),
            "sweep_roofline": exact_sweep,
            "sweep_rooflines": sweeps,
            "fast_math": fast,
            "persistent": persistent,
            "persistent_fast_math": persistent_fast,
            "status_flags": status}


def coloring_timing(pkg, reps=5, with_cpu=True):
    """Constraint-graph colouring (sx_color_edges_greedy: first-fit in edge-id
    order, all parallel rounds in one cooperative launch, then the stable sort
    by colour) on the edges of the 64 x 64 and 256 x 256 cloths: ms per call
    (CUDA events, median of `reps`), colours, and the oracle's serial time."""
    import numpy as np
    import torch
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    out = {}
    for n in (64, 256):
        _, f = pkg.grid_cloth(n)
        e = pkg.mesh.edges_from_faces(f)
        E, V = e.shape[0], n * n
        et = torch.from_numpy(np.ascontiguousarray(e.astype(np.int32))).cuda()
        color = torch.empty(E, dtype=torch.int32, device="cuda")
        srt = torch.empty(E, dtype=torch.int32, device="cuda")
        prefix = torch.empty(100, dtype=torch.int32, device="cuda")
        wsb = int(sx.sx_color_workspace_bytes(V, E))
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")

        def call():
            sx.sx_color_edges_greedy(ptr(et), E, V, 100, ptr(color), ptr(srt), ptr(prefix), ptr(ws), wsb,
                                     stream_handle())

        call()
        ts = []
        for _ in range(reps):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        r = {"edges": E, "ms": round(sorted(ts)[reps // 2], 4), "colours": int(color.max().item()) + 1,
             "status": int(ws[:4].view(torch.int32).item())}
        if with_cpu:
            from oracle import pyoracle as po

            t0 = time.perf_counter()
            c_ref, s_ref, p_ref = po.color_edges(V, e)
            r["cpu_baseline_ms"] = round(1e3 * (time.perf_counter() - t0), 2)
            r["matches_oracle"] = bool(np.array_equal(color.cpu().numpy(), c_ref) and
                                       np.array_equal(srt.cpu().numpy(), s_ref))
        out[f"grid{n}"] = r
    return out


def gauss_seidel_drape(pkg, scene, x0, v0, jacobi_iters=30, max_gs=60, reps=5):
    """Colour-ordered Gauss-Seidel sweeps against the Jacobi sweep on the
    256 x 256 drape: from the timed frame's state, one substep's predicted
    positions are swept k times by each method (springs and bending pairs, no
    contacts) and the RMS constraint violation is read after every sweep.
    Reports the residual curves, the Gauss-Seidel sweeps needed to reach the
    residual of `jacobi_iters` Jacobi sweeps (the drape's count), each sweep's
    time (CUDA events over a captured graph of `jacobi_iters` sweeps, median of
    `reps`) and the time each method takes to that residual."""
    import torch

    sim = pkg.scenes.make_solver(scene, device="cuda")
    sim.bending_on = "y"
    m = sim.mesh_dy
    dt = scene.dt / scene.n_substeps
    sim.gauss_seidel = True
    n_colors = sim.gs_setup()[2]
    curves = {}
    for gs in (False, True):
        sim.gauss_seidel = gs
        m.x4.copy_(x0)
        m.v4.copy_(v0)
        sim.compute_y(dt)
        res = [float(sim.constraint_residual("y")[2].item())]
        for _ in range(max(jacobi_iters, max_gs)):
            sim.spring_sweep(dt)
            res.append(float(sim.constraint_residual("y")[2].item()))
        curves["gauss_seidel" if gs else "jacobi"] = res
    target = curves["jacobi"][jacobi_iters]
    gs_curve = curves["gauss_seidel"]
    gs_needed = next((k for k in range(len(gs_curve)) if gs_curve[k] <= target), None)
    ms = {}
    for gs in (False, True):
        sim.gauss_seidel = gs
        m.x4.copy_(x0)
        m.v4.copy_(v0)
        sim.compute_y(dt)
        g = torch.cuda.CUDAGraph()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(g, stream=side):
            for _ in range(jacobi_iters):
                sim.spring_sweep(dt)
        torch.cuda.current_stream().wait_stream(side)
        ts = []
        for _ in range(reps + 1):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b) / jacobi_iters)
        ms["gauss_seidel" if gs else "jacobi"] = sorted(ts[1:])[reps // 2]
    pick = (1, 2, 5, 10, 20, 30, 60)
    return {
        "workload": "256x256 drape, one substep's predicted positions from the timed frame, springs + bending pairs",
        "colours": n_colors,
        "residual_start": curves["jacobi"][0],
        "residual_jacobi": {str(k): curves["jacobi"][k] for k in pick if k < len(curves["jacobi"])},
        "residual_gauss_seidel": {str(k): gs_curve[k] for k in pick if k < len(gs_curve)},
        "target": f"residual of {jacobi_iters} Jacobi sweeps",
        "gauss_seidel_sweeps_to_target": gs_needed,
        "ms_per_sweep": {k: round(v, 5) for k, v in ms.items()},
        "ms_to_target": {"jacobi": round(jacobi_iters * ms["jacobi"], 4),
                         "gauss_seidel": round(gs_needed * ms["gauss_seidel"], 4) if gs_needed else None},
    }


def learned_batched(pkg, target_iters=100, train_frames=40, train_rows=65536, val_frames=40, val_rows=8192,
                    train_steps=6000, eval_start=10, eval_frames=6, rho=0.995, check_every=4, cap=400):
    """Learned warm start against the plain cold start on the 512-cloth batched
    workload, iterating every substep to the same relative residual.

    Training data: the plain solver (``target_iters`` Jacobi iterations per
    substep) runs the seed-0 scene from rest for ``train_frames`` frames (40
    frames x 10 substeps x 512 cloths = 204 800 cloth-substeps); every substep
    gives ``train_rows`` random free vertices (features, correction).  The MLP
    trains on them for ``train_steps`` Adam steps of 65 536 rows with the
    library's kernels.  Validation: the held-out seed-1 scene over the same
    frame range; the loss of predicting no correction is evaluated by the same
    masked loss.  Evaluation: the held-out seed-2 scene, from its state after
    ``eval_start`` frames, ``eval_frames`` consecutive frames for each solver,
    every substep iterated until the constraint residual is at most ``rho``
    times the residual of that substep's cold start (cap ``cap``, checks every
    ``check_every`` iterations, device-side loops); the learned solver starts
    from the network's prediction unless that raises the residual.  Reported:
    ms per frame, iterations, the end-state distance between the two runs.
    Why a relative tolerance: on these scenes Jacobi lowers the residual by
    0.5-2 % per 100 iterations once the cloths rest on their boxes (the
    compliant bending pairs hold it up), so an absolute 1e-5 is met before any
    iteration in free fall and never in contact."""
    import numpy as np
    import torch

    L = pkg.learned
    kw = dict(dHat=(4e-3) ** 2, stiffness_stretch=1e5, stiffness_bending=1e8, g=(0.0, 0.0, -9.81), dt=1.0 / 60.0,
              n_iter=20, padding=8e-3)
    A = pkg.BatchedSolver(pkg.batched_scene(512, seed=0), **kw)
    A.n_iter, A.persistent = target_iters, True
    t0 = time.time()
    feat, tgt = L.collect_samples(A, frames=train_frames, rows_per_substep=train_rows)
    torch.cuda.synchronize()
    collect_s = time.time() - t0
    n_train_substeps = train_frames * 10 * A.n_instances
    del A
    Bv = pkg.BatchedSolver(pkg.batched_scene(512, seed=1), **kw)
    Bv.n_iter, Bv.persistent = target_iters, True
    vf, vt = L.collect_samples(Bv, frames=val_frames, rows_per_substep=val_rows, seed=5)
    del Bv
    mlp = pkg.WarmStartMLP(seed=0)
    zero_net = pkg.WarmStartMLP(params=L.zero_output_params())  # predicts no correction
    loss0 = L.evaluate_loss(mlp, vf, vt)
    t0 = time.time()
    h1 = L.train(mlp, feat, tgt, train_steps // 2, batch=65536, lr=2e-3)
    h2 = L.train(mlp, feat, tgt, train_steps - train_steps // 2, batch=65536, lr=5e-4)
    torch.cuda.synchronize()
    train_s = time.time() - t0
    val = L.evaluate_loss(mlp, vf, vt)
    zero_val = L.evaluate_loss(zero_net, vf, vt)
    n_train_rows = int(feat.shape[0])
    del feat, tgt
    # inference alone, eager launches: the validation rows repeated to a batch
    # larger than L2, on the tcgen05 kernel and on the mma.sync kernel
    reps_ = max(1, (3 << 20) // vf.shape[0] + 1)
    big = torch.cat([vf] * reps_)
    n_big = big.shape[0]
    out_big = torch.empty((n_big, 4), dtype=torch.float32, device="cuda")
    flush_inf = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    inf = {"rows": n_big, "flop_per_row": 2 * (24 * 64 + 64 * 64 + 64 * 3), "bytes_per_row": 64 + 16}
    for name, tc in (("tcgen05", True), ("mma_sync", False)):
        mlp.tcgen05 = tc
        mlp.forward(big, out_big)
        ts = []
        for _ in range(5):
            flush_inf.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            mlp.forward(big, out_big)
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        ms_inf = sorted(ts)[2]
        inf[name] = {"us": round(ms_inf * 1e3, 1),
                     "tflops": round(inf["flop_per_row"] * n_big / (ms_inf / 1e3) / 1e12, 1),
                     "gbs": round(inf["bytes_per_row"] * n_big / (ms_inf / 1e3) / 1e9, 1)}
    mlp.tcgen05 = True
    inf["tcgen05_status"] = int(mlp.status.item())
    del big, out_big, flush_inf
    # evaluation scene: seed 2, state after eval_start plain frames
    B = pkg.BatchedSolver(pkg.batched_scene(512, seed=2), **kw)
    rec = L.WarmStart(B, mode="record")
    B.warm, B.persistent = rec, True
    for _ in range(eval_start):
        B.forward(10)
    B.warm, B.persistent = None, False
    snap = (B.x4.clone(), B.v4.clone(), rec.c4.clone())

    def restore(warm=None):
        B.x4.copy_(snap[0])
        B.v4.copy_(snap[1])
        if warm is not None:
            warm.c4.copy_(snap[2])

    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    out = {"workload": f"512 cloths ({B.num_verts} vertices), held-out seed 2, frames {eval_start + 1}-"
                       f"{eval_start + eval_frames} run in sequence, 10 substeps, each iterated to residual <= "
                       f"{rho} x its cold-start residual (cap {cap}, checks every {check_every} iterations)",
           "training": {"cloth_substeps": n_train_substeps, "frames": train_frames, "samples": n_train_rows,
                        "target_iterations": target_iters, "adam_steps": train_steps, "batch": 65536,
                        "collect_s": round(collect_s, 2), "train_s": round(train_s, 2),
                        "train_loss_first": float(h1[:10].mean()), "train_loss_last": float(h2[-100:].mean()),
                        "validation": f"held-out seed 1, frames 1-{val_frames}, {int(vf.shape[0])} rows",
                        "val_loss_untrained": loss0, "val_loss": val, "val_loss_zero_prediction": zero_val,
                        "val_loss_vs_zero": val / zero_val if zero_val > 0 else None},
           "inference": inf, "tolerance": {"relative_to_cold_start": rho}}
    finals = {}
    for mode in ("plain", "learned"):
        B.tol, B.tol_relative, B.check_every, B.n_iter, B.use_graph = rho, True, check_every, cap, True
        B.warm = L.WarmStart(B, mlp) if mode == "learned" else None
        restore(B.warm)
        B.forward(10)  # capture
        restore(B.warm)
        B.convergence_stats(reset=True)
        if B.warm is not None:
            B.warm.flags.zero_()
        times = []
        for _ in range(eval_frames):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            B.forward(10)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        st = B.convergence_stats()
        ms = sum(times) / len(times)
        finals[mode] = B.x4[:, :3].clone()
        out[mode] = {"ms_per_frame": round(ms, 3), "value": B.num_verts * 10 / (ms / 1e3), "unit": UNIT,
                     "converged_substeps": st["converged_substeps"], "substeps": 10 * eval_frames,
                     "mean_stop_iteration": st["mean_stop_iteration"],
                     "final_residual": float(B.constraint_residual("x")[2].item())}
        if B.warm is not None:
            out[mode].update(B.warm.fallback_counts())
    # the reference trajectory: the plain solver with target_iters iterations per substep
    B.warm, B.tol, B.use_graph, B.n_iter = None, None, True, target_iters
    restore()
    B.forward(10)  # capture
    restore()
    for _ in range(eval_frames):
        B.forward(10)
    torch.cuda.synchronize()
    finals["plain_fixed"] = B.x4[:, :3].clone()
    diag = float(np.sqrt(2.0))  # every instance is a unit square cloth

    def dist(a, b):
        d = (finals[a] - finals[b]).norm(dim=1)
        return {"max_abs_dx": float(d.max()), "rms_dx": float(d.pow(2).mean().sqrt()),
                "max_over_diagonal": float(d.max()) / diag}

    out["end_state"] = {"learned_vs_plain": dist("learned", "plain"),
                        f"plain_vs_plain_{target_iters}_iterations": dist("plain", "plain_fixed"),
                        f"learned_vs_plain_{target_iters}_iterations": dist("learned", "plain_fixed"),
                        "criterion_over_diagonal": 1e-4,
                        "note": "positions that differ when a substep's solve stops become velocities that "
                                "differ (v = (y - x) / dt), so two runs stopped at the same residual in different "
                                "states drift apart over frames; the per-substep comparison is in accuracy"}
    out["speedup"] = out["learned"]["value"] / out["plain"]["value"]
    out["accuracy"] = solve_accuracy(B, mlp, L, snap, target_iters=target_iters)
    return out


def solve_accuracy(B, mlp, L, snap, target_iters=100, ref_iters=400, ks=(4, 8, 16, 32, 64, 100), substeps=20):
    """What the warm start gains at equal iterations.  Along the reference
    trajectory (plain solver, target_iters iterations per substep) from the
    snapshot, for each of `substeps` substeps: from that substep's start, a
    tightly converged solve (ref_iters iterations) and plain and learned solves
    with k iterations each; error = RMS over vertices of the distance of the
    substep's end positions to the converged solve's.  Reported: mean errors
    per k and, for each learned k, the plain iteration count with the same
    error (log-linear interpolation; None past max(ks))."""
    import numpy as np
    import torch

    dt = B.dt / 10
    B.tol, B.use_graph = None, False
    rec = L.WarmStart(B, mode="record")
    warm = L.WarmStart(B, mlp)
    rec.c4.copy_(snap[2])
    x, v = snap[0].clone(), snap[1].clone()
    err_p = np.zeros(len(ks))
    err_l = np.zeros(len(ks))
    for _ in range(substeps):
        c4 = rec.c4.clone()

        def run(n_iter, w=None):
            B.x4.copy_(x)
            B.v4.copy_(v)
            B.n_iter = n_iter
            B.warm = w
            if w is not None:
                w.c4.copy_(c4)
            B.substep(dt)
            return B.x4[:, :3].clone()

        ref = run(ref_iters)
        for j, k in enumerate(ks):
            err_p[j] += float((run(k) - ref).norm(dim=1).pow(2).mean())
            err_l[j] += float((run(k, warm) - ref).norm(dim=1).pow(2).mean())
        run(target_iters, rec)  # advance the reference trajectory (and the recorded correction)
        x, v = B.x4.clone(), B.v4.clone()
    B.warm = None
    err_p = np.sqrt(err_p / substeps)
    err_l = np.sqrt(err_l / substeps)
    lk, lp = np.log(np.asarray(ks, float)), np.log(np.maximum(err_p, 1e-30))
    equal = {}
    for j, k in enumerate(ks):
        e = err_l[j]
        if e >= err_p[0]:
            equal[str(k)] = float(ks[0])
            continue
        hit = np.flatnonzero(err_p <= e)
        if not len(hit):
            equal[str(k)] = None
            continue
        i = hit[0]
        t = (np.log(e) - lp[i - 1]) / (lp[i] - lp[i - 1])
        equal[str(k)] = round(float(np.exp(lk[i - 1] + t * (lk[i] - lk[i - 1]))), 1)
    return {"substeps": substeps, "reference": f"{ref_iters} plain iterations from the same start",
            "iterations": list(ks), "rms_error_plain": [float(e) for e in err_p],
            "rms_error_learned": [float(e) for e in err_l],
            "plain_iterations_for_the_learned_error": equal}


def run_reference(args):
    """The reference arm: the CPU port of the reference's substep (the
    reference's Taichi path cannot run here) on all host cores, on the state
    the GPU arm times: the scene advanced by `warmup` frames, then `steps`
    substeps of the next frame(s) timed one by one (a bounded sample; at most
    about 150 s of timing)."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    pkg, scene = build_scene(args.workload)
    cores = os.cpu_count() or 1
    orc = _oracle_solver(pkg, scene, cores)
    t0 = time.perf_counter()
    for _ in range(args.warmup):
        orc.forward(scene.n_substeps)
    warm_s = time.perf_counter() - t0
    dt_sub = scene.dt / scene.n_substeps
    times = []
    budget = 150.0
    t_all = time.perf_counter()
    for _ in range(args.steps):
        t0 = time.perf_counter()
        orc.substep(dt_sub)
        times.append(time.perf_counter() - t0)
        if time.perf_counter() - t_all > budget:
            break
    V = scene.cloth_x.shape[0]
    tot = sum(times)
    val = V * len(times) / tot
    line = {
        "impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": args.gpus,
        "steps": len(times), "warmup": args.warmup, "ms_per_step": 1e3 * tot / len(times),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": workload_config(scene, args.workload) | {
            "step": f"one substep of frame {args.warmup + 1} onward (the state the GPU arm times, reached by "
                    f"{args.warmup} untimed frames, {warm_s:.1f} s)"},
        "cpu_baseline": {"value": val, "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"{len(times)} substeps from frame {args.warmup + 1} of the same scene on the "
                                   f"CPU oracle, {cores} threads (the reference's Taichi path cannot run here)"},
        "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


def main():
    args = parse_args()
    if args.profile_case:
        run_profile_case(args.profile_case)
        return
    if args.impl == "reference":
        run_reference(args)
        return
    import torch

    world, rank, local = dist_setup(args.gpus)
    pkg, scene = build_scene(args.workload)
    from starlab_physics_gb300 import _lib

    _lib.load()
    if args.only_batched:
        print(json.dumps({"batched512": batched512(pkg, steps=args.steps, warmup=args.warmup)}))
        return
    if args.only_lbvh:
        print(json.dumps({"lbvh_soup": lbvh_soup(pkg, with_cpu=False)}))
        return
    if args.only_learned:
        print(json.dumps({"learned_batched512": learned_batched(pkg)}))
        return
    if args.only_plain64:
        print(json.dumps({"plain64": plain64_timing(pkg, with_cpu=not args.no_cpu_baseline)}))
        return
    if args.only_color:
        print(json.dumps({"coloring": coloring_timing(pkg, with_cpu=not args.no_cpu_baseline)}))
        return
    if args.only_gs:
        sim = pkg.scenes.make_solver(scene, device="cuda")
        sim.bending_on = "y"
        sim.use_graph = True
        for _ in range(3):
            sim.forward(scene.n_substeps)
        print(json.dumps({"gauss_seidel": gauss_seidel_drape(pkg, scene, sim.mesh_dy.x4.clone(),
                                                             sim.mesh_dy.v4.clone())}))
        return
    sim = pkg.scenes.make_solver(scene, device="cuda")
    sim.bending_on = "y"
    V = sim.mesh_dy.num_verts
    S = scene.n_substeps
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream()

    # the frame runs as one captured CUDA graph (captured on the first call)
    sim.use_graph = not args.eager
    sim.forward(S)
    # the sweep's launch configuration is picked by the autotuner on this mesh
    # (the fastest alone, then the four best timed in whole frames)
    variant, vtimes = sim.autotune(S)
    from starlab_physics_gb300.autotune import variants as sweep_variants

    from starlab_physics_gb300.autotune import variant_forms

    sweep_cfg = (((f"packed_direct_{sim.packed_form}" if sim.packed_form else "packed"), 256, 1, 0) if sim.packed_sweep
                 else sweep_variants()[variant] + variant_forms()[variant])
    from starlab_physics_gb300.autotune import pairs_project_variants

    pp_variants = pairs_project_variants()
    # the projection's launch configuration: whole frames timed per variant
    pp_variant, pp_times = sim.autotune_contacts(S)
    for _ in range(args.warmup - 1):
        sim.forward(S)
    torch.cuda.synchronize()
    # every timed step simulates the same frame: the one after the warm-up frames
    x0 = sim.mesh_dy.x4.clone()
    v0 = sim.mesh_dy.v4.clone()

    # ---- device-resident timed region ----
    starts = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    barrier(world)
    torch.cuda.synchronize()
    lib = _lib.load()
    l0 = lib.sx_kernel_launches()
    with ClockSampler(local) as clk:
        for k in range(args.steps):
            sim.mesh_dy.x4.copy_(x0)
            sim.mesh_dy.v4.copy_(v0)
            flush.zero_()
            starts[k].record(stream)
            sim.forward(S)
            ends[k].record(stream)
        torch.cuda.synchronize()
    # graph replays bypass the host-side launch counter: each replay runs the
    # library kernels recorded at capture
    launches = lib.sx_kernel_launches() - l0 + (0 if args.eager else args.steps * sim.graph_kernel_launches)
    barrier(world)
    value, ms = replica_throughput(V * S * args.steps, sum(s.elapsed_time(e) for s, e in zip(starts, ends)), world)
    status = sim.status_flags()

    # ---- end-to-end through the public API with host buffers ----
    xh = x0.cpu().pin_memory()
    vh = v0.cpu().pin_memory()
    xo = torch.empty_like(xh).pin_memory()
    vo = torch.empty_like(vh).pin_memory()
    e_st = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    e_en = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    barrier(world)
    torch.cuda.synchronize()
    with ClockSampler(local) as clk2:
        for k in range(args.steps):
            flush.zero_()
            e_st[k].record(stream)
            sim.mesh_dy.x4.copy_(xh, non_blocking=True)
            sim.mesh_dy.v4.copy_(vh, non_blocking=True)
            sim.forward(S)
            xo.copy_(sim.mesh_dy.x4, non_blocking=True)
            vo.copy_(sim.mesh_dy.v4, non_blocking=True)
            e_en[k].record(stream)
        torch.cuda.synchronize()
    e2e_val, ms_e2e = replica_throughput(V * S * args.steps, sum(s.elapsed_time(e) for s, e in zip(e_st, e_en)),
                                         world)
    bytes_io = 2 * V * 16

    # ---- the same frame with the sweep's fast arithmetic (not bit-identical;
    # held to the substep tolerance by the GPU tests), sweep re-tuned for it ----
    exact_sweep = (sim.sweep_variant, sim.packed_sweep, sim.packed_form)
    sim.fast_math = True
    sim.mesh_dy.x4.copy_(x0)
    sim.mesh_dy.v4.copy_(v0)
    fast_variant, _ = sim.autotune(S)
    sim.forward(S)  # captures the fast frame
    f_st = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    f_en = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    torch.cuda.synchronize()
    for k in range(args.steps):
        sim.mesh_dy.x4.copy_(x0)
        sim.mesh_dy.v4.copy_(v0)
        flush.zero_()
        f_st[k].record(stream)
        sim.forward(S)
        f_en[k].record(stream)
    torch.cuda.synchronize()
    f_ms = sum(s_.elapsed_time(e_) for s_, e_ in zip(f_st, f_en))
    drape_fast = {"value": V * S * args.steps / (f_ms / 1e3), "unit": UNIT, "ms_per_step": f_ms / args.steps,
                  "sweep_config": {"variant": ((f"packed_direct_{sim.packed_form}" if sim.packed_form else "packed") if sim.packed_sweep
                                               else fast_variant),
                                   "lanes_per_vertex": 1 if sim.packed_sweep else variant_forms()[fast_variant][0]},
                  "note": "the sweep with fused multiply-adds, rsqrtf and a fast divide; contacts unchanged"}
    sim.fast_math = False
    sim.sweep_variant, sim.packed_sweep, sim.packed_form = exact_sweep
    sim.mesh_dy.x4.copy_(x0)
    sim.mesh_dy.v4.copy_(v0)

    # ---- dominant kernel: Jacobi sweep, instrumented pass ----
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    sweeps = []
    orig = sim.spring_sweep

    def timed_sweep(dt, iteration=0, loop=0):
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        a.record(stream)
        orig(dt, iteration, loop)
        b.record(stream)
        sweeps.append((a, b))

    sim.spring_sweep = timed_sweep
    sim.use_graph = False
    n_inst = max(1, min(args.steps, 5))
    for _ in range(n_inst):
        sim.forward(S)
    torch.cuda.synchronize()
    del sim.spring_sweep  # the solver's own again, which the chunk heads ask for
    eager_ms = sum(a.elapsed_time(b) for a, b in sweeps) / len(sweeps)
    # the same sweeps back to back as they run inside the frame's graph: a graph
    # of 30 sweeps (alternating buffers) on the frame's state, replayed and timed
    m = sim.mesh_dy
    dt_sub = scene.dt / S
    ks_, kb_ = sim.stiffness_bending * dt_sub * dt_sub, sim.stiffness_stretch * dt_sub * dt_sub
    ya, yb = m.y4.clone(), torch.empty_like(m.y4)

    def burst():
        for k in range(30):
            src, dst = (ya, yb) if k % 2 == 0 else (yb, ya)
            if sim.packed_sweep:
                sx.sx_jacobi_sweep_packed_v(ptr(m.x4), ptr(src), ptr(dst), ptr(m.fixed), ptr(m.adj_ptr),
                                            ptr(m.adj_nbr16), ptr(m.adj_rest32), V, ks_, kb_, 1, sim.packed_form, 0,
                                            stream_handle())
            else:
                sx.sx_jacobi_sweep_v(ptr(m.x4), ptr(src), ptr(dst), ptr(m.fixed), ptr(m.adj_ptr), ptr(m.adj), V,
                                     ks_, kb_, 1, sim.sweep_variant, stream_handle())

    side = torch.cuda.Stream()
    side.wait_stream(stream)
    with torch.cuda.stream(side):
        burst()
    stream.wait_stream(side)
    gb = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gb):
        burst()
    reps = []
    for _ in range(5):
        flush.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        gb.replay()
        b.record(stream)
        torch.cuda.synchronize()
        reps.append(a.elapsed_time(b) / 30)
    sweep_ms = sorted(reps)[len(reps) // 2]
    E, B = m.num_edges, m.bending_constraint_count
    alg_bytes = 12 * (E + B) + 28 * V
    achieved = alg_bytes / (sweep_ms / 1e3) / 1e9
    peak, peak_kind = measured_peak()
    frame_ms = ms / args.steps
    sweep_kname = (("jacobi_sweep_packed_kernel" if sim.packed_form else "jacobi_sweep_staged_kernel")
                   if sim.packed_sweep else "jacobi_sweep_kernel")
    roofline_sweep = {"kernel": sweep_kname,
                "bound": "hbm", "achieved": round(achieved, 1),
                "peak": peak, "unit": "GB/s", "frac": round(achieved / peak, 4),
                "traffic": ncu_traffic(sweep_kname + "_drape256.md"),
                "algorithmic_bytes_per_launch": alg_bytes, "avg_launch_us": round(sweep_ms * 1e3, 3),
                "timing": "CUDA events around a graph of 30 back-to-back sweeps on the frame's state (L2 flushed "
                          "before each replay), median of 5; one eager launch between events: "
                          f"{eager_ms * 1e3:.2f} us",
                "launches_per_step": len(sweeps) // n_inst,
                "share_of_step": round(sweep_ms * (len(sweeps) / n_inst) / frame_ms, 4),
                "peak_source": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs)" if peak_kind == "measured" else "fallback"}

    # ---- dominant kernel: the contact-pair projection (about half of a frame) ----
    # the pair list of one substep (its first iteration), then a graph of 30
    # projections back to back on that state; the projections only add to the
    # fixed-point accumulators, which are cleared afterwards
    sim.mesh_dy.x4.copy_(x0)
    sim.mesh_dy.v4.copy_(v0)
    sim.build_bvhs()
    sim.compute_y(dt_sub)
    sim._in_substep = True  # as within a substep: the chunk heads are written where a frame uses them
    for it in range(2):
        sim.solve_constraints_jacobi_x(dt_sub, first_iteration=it == 0, iteration=it)
    headed = sim._heads_on
    sim._in_substep = sim._heads_on = False
    torch.cuda.synchronize()
    n_pairs = sim.contact_pair_count()
    st_mesh = sim.mesh_st
    Vs = st_mesh.num_verts if st_mesh is not None else 0

    def project(heads):
        sx.sx_contact_pairs_project_headed(V, Vs, ptr(sim._pairs), ptr(sim._pairs_ws), ptr(m.y4),
                                           ptr(st_mesh.x4) if st_mesh is not None else None, ptr(m.fixed),
                                           ptr(m.m_inv), sim.dHat, float(sim.compliance_collision),
                                           sim.contact_cull_d2(), ptr(sim._dx_fix), ptr(sim._nc), ptr(sim.status),
                                           None, 0, pp_variant, ptr(sim._heads[0]) if heads else None,
                                           ptr(sim._heads[2]) if heads else None, stream_handle())

    def project_ms(heads):
        side = torch.cuda.Stream()
        side.wait_stream(stream)
        with torch.cuda.stream(side):
            project(heads)
        stream.wait_stream(side)
        gp = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gp):
            for _ in range(30):
                project(heads)
        preps = []
        for _ in range(5):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            gp.replay()
            b.record(stream)
            torch.cuda.synchronize()
            preps.append(a.elapsed_time(b) / 30)
        return sorted(preps)[len(preps) // 2]

    proj_ms = project_ms(False)
    headed_ms = project_ms(True) if headed else None
    sim._dx_fix.zero_()
    sim._nc.zero_()
    proj_bytes = 16 * n_pairs + 16 * V + 16 * Vs
    proj_gbs = proj_bytes / (proj_ms / 1e3) / 1e9
    pp_kernel = "pairs_project_kernel"
    roofline = {"kernel": pp_kernel, "bound": "hbm", "achieved": round(proj_gbs, 1), "peak": peak,
                "unit": "GB/s", "frac": round(proj_gbs / peak, 4),
                "traffic": ncu_traffic(pp_kernel + "_drape256.md"),
                "algorithmic_bytes_per_launch": proj_bytes, "pairs_per_launch": n_pairs,
                "avg_launch_us": round(proj_ms * 1e3, 3),
                "timing": "CUDA events around a graph of 30 back-to-back projections of one substep's pair list "
                          "(L2 flushed before each replay), median of 5",
                "launches_per_step": roofline_sweep["launches_per_step"],
                "headed_avg_launch_us": None if headed_ms is None else round(headed_ms * 1e3, 3),
                "share_of_step": round((headed_ms or proj_ms) * roofline_sweep["launches_per_step"] / frame_ms, 4),
                "peak_source": roofline_sweep["peak_source"]}

    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": frame_ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded scene generators)",
        "config": workload_config(scene, args.workload) | {
            "execution": "eager launches" if args.eager else "one CUDA graph per frame",
            "sweep_config": {"entries_per_load_batch": sweep_cfg[0], "threads_per_block": sweep_cfg[1],
                             "lanes_per_vertex": sweep_cfg[2], "streaming_adjacency": bool(sweep_cfg[3]),
                             "picked_by": "autotuner (%d bit-identical variants timed alone, the 4 fastest "
                                          "then in whole frames)" % len(vtimes)},
            "pairs_project_config": {"pair_batches_per_warp_step": pp_variants[pp_variant][0],
                                     "blocks_per_sm": pp_variants[pp_variant][1],
                                     "pipelined": bool(sx.sx_contact_pairs_project_variant_pipelined(pp_variant)),
                                     "picked_by": "autotuner (fastest of %d identical variants in whole-frame "
                                                  "timing)" % len(pp_times)},
            "step": f"frame {args.warmup + 1} of the scene, restored from a snapshot before each step"},
        "gpu_launches": int(launches),
        "e2e": {"value": e2e_val, "unit": UNIT, "h2d_bytes_per_step": bytes_io, "d2h_bytes_per_step": bytes_io},
        "roofline": roofline,
        "roofline_sweep": roofline_sweep,
        "fast_math": drape_fast,
        "clocks": clk.summary(),
        "status_flags": status,
    }
    line["clocks_e2e"] = clk2.summary()
    if rank == 0 and not args.no_lbvh:
        line["lbvh_soup"] = lbvh_soup(pkg, with_cpu=not args.no_cpu_baseline)
    if not args.no_batched:
        b512 = batched512(pkg, world=world, rank=rank)
        if rank == 0:
            line["batched512"] = b512
    if rank == 0:
        line["coloring"] = coloring_timing(pkg, with_cpu=not args.no_cpu_baseline)
        line["plain64"] = plain64_timing(pkg, with_cpu=not args.no_cpu_baseline)
        line["gauss_seidel"] = gauss_seidel_drape(pkg, scene, x0, v0)
    if rank == 0 and not args.no_learned:
        line["learned_batched512"] = learned_batched(pkg)
    if rank == 0 and world >= 1 and not args.no_cpu_baseline and world == 1:
        # the GPU's frame from the timed snapshot, for the comparison
        sim.use_graph = True
        sim.mesh_dy.x4.copy_(x0)
        sim.mesh_dy.v4.copy_(v0)
        sim.forward(S)
        torch.cuda.synchronize()
        line["cpu_baseline"] = cpu_baseline(pkg, scene, x0.cpu().numpy(), v0.cpu().numpy(),
                                            sim.mesh_dy.x4.cpu().numpy(), args.warmup + 1)
    if rank == 0:
        print(json.dumps(line))
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()


if __name__ == "__main__":
    main()
