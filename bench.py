#!/usr/bin/env python
"""Throughput benchmark: 64 independent scenes rendered in one batched wavefront.

Workload (one step): 64 seeded synthetic scenes (fumeng_b200.synth.batch_scene: 1-40
displaced icospheres / subdivided boxes per scene, 1k-200k triangles each, 2.4M in
total; Disney / Lambert / dielectric materials; one area light and a 512x256 HDR sky;
resolutions 128^2-512^2, 4-64 spp, depth 8) rendered once through fm_render_batch.
Metric: camera paths per second (a path = one pixel sample, counted when complete).

    python bench.py [--steps K] [--warmup W] [--impl ours|reference]
    torchrun --nproc-per-node N bench.py --gpus N ...   (replicas: each rank renders its own batch)

value  : device-resident scenes, device output images; time = device time of the K
         timed steps (CUDA events, max over ranks).
roofline: the trace kernel's algorithmic bytes (fixed per-ray formula, live ray counts)
         over its device time in the timed steps, taken from the GPU's global timer
         inside the kernel (earliest block start to latest block end of each launch;
         the render runs as one conditional CUDA graph, which admits no event nodes).
         The kernel is bound by instruction issue: most of these bytes come from caches,
         dram_frac is the share of the measured HBM rate that reaches DRAM.
e2e    : the same metric through the C-ABI from host memory: every step creates the 64
         scenes from host descriptors in one fm_scene_create_batch call (upload + device
         BVH builds + env tables), renders and reads the images back into host arrays
         (allocated once, written by every step) and destroys the scenes.
The plain per-pixel megakernel is timed on the same batch for comparison, and the
path-replay adjoint against its own forward pass on the inverse-rendering workload
(fumeng_b200.synth.inverse_scene: 120k triangles, 512^2 basecolor and roughness /
metallic textures, 16 views of 256^2, 32 spp forward and 32 spp adjoint, depth 6).
"""
from __future__ import annotations

import argparse
import json
import math
import os
import subprocess
import sys
import tempfile
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "Mpaths/s batched wavefront vs plain megakernel at relMSE≤1e-3; adjoint/fwd ratio"
WORKLOAD = "batched: 64 scenes x (1-40 displaced icosphere/box meshes, 1k-200k tris), 512x256 HDR env + 1 area light, 128^2-512^2, 4-64 spp, depth 8"
NSCENES = 64
# DRAM bytes the trace kernel moves per traced ray (read + write, cold L2 at each
# launch), from an ncu capture of two trace launches of the 8-scene case of this
# workload (66.7 and 61.7 B per ray); traffic grows with the rays a launch traces.
TRACE_DRAM_BYTES_PER_RAY = 64.2


def dram_frac(rays, trace_ms, peak):
    """The trace kernel's DRAM bytes as a share of the measured HBM rate."""
    return TRACE_DRAM_BYTES_PER_RAY * rays / (trace_ms / 1e3) / 1e9 / peak if trace_ms > 0 else None


def measured_peak_hbm():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return float(json.loads(p.read_text())["hbm_gbs"]), "measured"
        except Exception:
            pass
    return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the timed region."""

    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.path = Path(tempfile.mkstemp(prefix="fm_clocks_", suffix=".csv")[1])

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.QUERY}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        try:
            rows = [r.split(",") for r in self.path.read_text().strip().splitlines() if r.strip()]
        except Exception:
            rows = []
        finally:
            try:
                self.path.unlink()
            except Exception:
                pass
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"]}
        sm = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if len(r) > 5 + k and "Active" in r[5 + k]
                          and "Not" not in r[5 + k]})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


def bvh_depth_estimate(nprims: int) -> int:
    return max(1, math.ceil(math.log(max(nprims, 5) / 4.0, 8)))


def desc_bytes(holder) -> int:
    n = 0
    for name in ("obj_material", "obj_emission", "tri_pos", "tri_normal", "tri_has_normal", "tri_uv", "tri_object",
                 "tri_vattr", "rect_pts", "rect_object", "sphere_radius", "sphere_xform", "sphere_object"):
        a = getattr(holder, name, None)
        if a is not None:
            n += a.nbytes
    n += sum(a.nbytes for a in holder.tex_arrays)
    return n


# ---- reference arm (CPU) ---------------------------------------------------------------

# Camera paths per scene and step in the CPU sample: about this many pixels of each of
# the 64 scenes, spread over the image (every k-th pixel in row-major order, k odd so
# that the sample runs diagonally across rows), at 1 spp.
REF_PIXELS_PER_SCENE = 1024


def run_reference(args, steps=None, warmup=None, per_scene=REF_PIXELS_PER_SCENE):
    """The reference's own CPU integrator (oracle/_ref float build: its RenderPixel per
    camera sample, on all host threads) on a bounded sample of the workload per step:
    about `per_scene` pixels of every one of the 64 scenes at 1 spp.  The reference's
    speed differs by three orders of magnitude between scenes, so the sample measures
    each scene's rate r_s and reports the rate of the whole workload, whose scene s has
    P_s = width x height x spp paths: sum_s P_s / sum_s (P_s / r_s).  Scene loading (the
    reference's loader and BVH build) happens before the timed steps."""
    sys.path.insert(0, str(ROOT / "oracle"))
    import fmref  # noqa: E402  (test/baseline infrastructure)
    from fumeng_b200 import synth
    if not fmref.available("float"):
        return {"impl": "reference", "unavailable": "oracle/_ref/libfmref_f.so was not built (no reference sources)"}
    steps = args.steps if steps is None else steps
    warmup = args.warmup if warmup is None else warmup
    threads = os.cpu_count() or 1
    tmp = Path(tempfile.mkdtemp(prefix="fm_ref_"))
    loaded, workload_paths = [], np.zeros(NSCENES)
    for s in range(NSCENES):
        spec = synth.batch_scene(s)
        workload_paths[s] = float(spec.renderer["width"]) * float(spec.renderer["height"]) * float(spec.renderer["spp"])
        loaded.append(fmref.RefScene(spec.write(tmp / f"s{s}"), "float"))
    times = []
    per_scene_t = np.zeros(NSCENES)
    per_scene_p = np.zeros(NSCENES)
    sample_paths = 0
    for it in range(warmup + steps):
        t_step = 0.0
        for s, rs in enumerate(loaded):
            w, h, _ = rs.image_size()
            stride = max(1, (w * h) // per_scene) | 1
            n = (w * h + stride - 1) // stride
            t0 = time.perf_counter()
            rs.render(1, seed=it, threads=threads, stride=stride)
            dt = time.perf_counter() - t0
            t_step += dt
            if it >= warmup:
                per_scene_t[s] += dt
                per_scene_p[s] += n
        if it >= warmup:
            times.append(t_step)
        sample_paths = int(per_scene_p.sum() / max(1, it + 1 - warmup))
    for rs in loaded:
        rs.close()
    rates = per_scene_p / np.maximum(per_scene_t, 1e-12)
    value = float(workload_paths.sum() / np.sum(workload_paths / rates)) / 1e6
    return {"value": value, "unit": "Mpaths/s", "cores": threads, "kind": "reference",
            "sample": f"about {per_scene} pixels of each of the {NSCENES} scenes at 1 spp per step "
                      f"({sample_paths} paths), reference float build, all {threads} host threads, "
                      f"{warmup} warm-up step(s); value = workload paths / sum over scenes of "
                      f"(scene paths / scene rate)",
            "per_scene_mpaths": {"min": float(rates.min() / 1e6), "median": float(np.median(rates) / 1e6),
                                 "max": float(rates.max() / 1e6)},
            "ms_per_step": 1e3 * sum(times) / len(times)}


# ---- our arm (GPU) ---------------------------------------------------------------------

ADJ_WORKLOAD = ("inverse rendering: 120k-tri UV-mapped displaced plane + sphere, Disney with 512^2 basecolor and "
                "roughness(G)/metallic(B) textures, 16 views 256^2, 32 spp forward + 32 spp adjoint, depth 6")


def measure_adjoint(ctx, args, barrier, max_over_ranks):
    """Device time of the path-replay adjoint (gradients w.r.t. both 512^2 textures and
    the env texels) against the forward wavefront render of the same 16 views."""
    import fumeng_b200 as fb
    from fumeng_b200 import synth
    from fumeng_b200.scene import camera_struct
    spec = synth.inverse_scene(target=True)
    holder = spec.to_desc()
    ti = holder.texture_index
    sc = ctx.create_scene(holder)
    cams = [camera_struct(c) for c in synth.inverse_views(16)]
    fwd = [spec.render_params(spp=32, seed=100 + v) for v in range(16)]
    adj = [spec.render_params(spp=32, seed=5000 + v) for v in range(16)]
    tune = fb.Tuning(1 << 21, 128, 128, 8)
    d_rgb = [np.random.default_rng(v).standard_normal((p.height, p.width, 3)).astype(np.float32) * 1e-3
             for v, p in enumerate(adj)]
    shapes = {ti["basecolor"]: spec.textures["basecolor"].shape[:2], ti["rm"]: spec.textures["rm"].shape[:2],
              ti["sky"]: spec.textures["sky"].shape[:2]}
    prof = args.event_timing
    ctx.render_batch([sc] * 16, cams, fwd, tuning=tune, profile=prof)
    sc.render_adjoint(cams, adj, d_rgb, shapes, profile=prof)
    f_ms, a_ms, a_wall, nans = [], [], [], 0
    for _ in range(args.adjoint_steps):
        barrier()
        st = ctx.render_batch([sc] * 16, cams, fwd, tuning=tune, profile=prof)[3]
        f_ms.append(st.kernel_ms)
        t0 = time.perf_counter()
        _, _, _, sa = sc.render_adjoint(cams, adj, d_rgb, shapes, profile=prof)
        a_wall.append(1e3 * (time.perf_counter() - t0))
        a_ms.append(sa.kernel_ms)
        nans += sa.nan_samples
    sc.destroy()
    f, a = max_over_ranks(float(np.mean(f_ms))), max_over_ranks(float(np.mean(a_ms)))
    paths = sum(p.width * p.height * p.spp for p in fwd)
    return {"workload": ADJ_WORKLOAD, "forward_ms": f, "adjoint_ms": a, "adjoint_over_forward": a / f,
            "adjoint_wall_ms_host_buffers": float(np.mean(a_wall)), "forward_mpaths_s": paths / f / 1e3,
            "adjoint_mpaths_s": paths / a / 1e3, "grad_texels": int(sum(h * w for h, w in shapes.values())),
            "nan_samples": int(nans), "steps": args.adjoint_steps,
            "timing": "device time of the wavefront loop (CUDA events), same default tuning for both passes"}


LARGE_WORKLOAD = ("large: 8x8 grid of displaced meshes, 124,848 tris each (7.99 M), Disney (glass-like, diffuse, "
                  "general) + Lambert ground, 2048x1024 HDR env + 4 area lights, 8 views 1920x1080, 128 spp, depth 16")


def run_large(args, ctx, group, rank, world):
    """The large combined workload: forward Mpaths/s over the 8 views, a bounded
    megakernel sample, end to end from host memory, and the adjoint with respect to a
    512x256 env parameter grid (the 2048x1024 env map is that grid upsampled 4x by
    replication, so the grid's gradient is the sum of each 4x4 block of texel gradients)
    and the 64 per-mesh roughness values, against its forward at the same spp."""
    import torch
    import fumeng_b200 as fb
    from fumeng_b200 import synth
    from fumeng_b200.scene import camera_struct
    spec = synth.large_scene()
    holder = spec.to_desc()
    sc = ctx.create_scene(holder)
    build_ms = sc.bvh_stats()["build_ms"]
    cams = [camera_struct(c) for c in synth.large_views(8)]
    params = [spec.render_params(seed=1 + v) for v in range(8)]
    paths = sum(p.width * p.height * p.spp for p in params)
    outs = [torch.empty((p.height, p.width, 3), device="cuda") for p in params]
    ptrs = [o.data_ptr() for o in outs]
    tune = fb.Tuning(1 << 22, 128, 128, 8)

    def step():
        return ctx.render_batch([sc] * 8, cams, params, tuning=tune, device_outputs=ptrs)[3]
    for _ in range(args.warmup):
        step()
    group.barrier()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    tot = {"paths": 0, "closest": 0, "shadow": 0, "trace_ms": 0.0, "kernel_ms": 0.0, "launches": 0, "nans": 0}
    with ClockSampler(int(os.environ.get("LOCAL_RANK", "0"))) as clk:
        ev0.record()
        for _ in range(args.steps):
            st = step()
            tot["paths"] += st.paths
            tot["closest"] += st.closest_rays
            tot["shadow"] += st.shadow_rays
            tot["trace_ms"] += st.trace_ms
            tot["kernel_ms"] += st.kernel_ms
            tot["launches"] += st.launches
            tot["nans"] += st.nan_samples
        ev1.record()
        group.barrier()
    clocks = clk.summary()
    ms = group.max(ev0.elapsed_time(ev1))
    value = group.sum(float(tot["paths"])) / (ms / 1e3) / 1e6
    assert tot["paths"] == paths * args.steps
    # megakernel on one view at 8 spp (a bounded sample of the same work)
    mk_p = [spec.render_params(spp=8, seed=1, mode=fb.FM_MODE_MEGAKERNEL)]
    ctx.render_batch([sc], cams[:1], mk_p, device_outputs=ptrs[:1])
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    group.barrier()
    e0.record()
    ctx.render_batch([sc], cams[:1], mk_p, device_outputs=ptrs[:1])
    e1.record()
    group.barrier()
    mk_paths = mk_p[0].width * mk_p[0].height * mk_p[0].spp
    mk_value = group.sum(float(mk_paths)) / (group.max(e0.elapsed_time(e1)) / 1e3) / 1e6
    # roofline of the trace kernel
    D = bvh_depth_estimate(holder.desc.num_triangles + 2 * holder.desc.num_rects)
    closest_b, shadow_b = 32 + 16 + 80 * D + 160, 32 + 4 + 80 * D + 160
    peak, peak_kind = measured_peak_hbm()
    achieved = (tot["closest"] * closest_b + tot["shadow"] * shadow_b) / (tot["trace_ms"] / 1e3) / 1e9
    launches_trace = max(1, (tot["launches"] - args.steps * 9) * 8 // 49)
    roofline = {"bound": "issue", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "traffic": TRACE_DRAM_BYTES_PER_RAY * (tot["closest"] + tot["shadow"]) / launches_trace,
                "dram_frac": dram_frac(tot["closest"] + tot["shadow"], tot["trace_ms"], peak),
                "kernel": "k_wf_trace", "peak_source": f"{peak_kind} hbm_gbs (MEASURED_PEAKS.json)",
                "alg_bytes_per_closest_ray": closest_b, "alg_bytes_per_shadow_ray": shadow_b,
                "trace_share_of_step": tot["trace_ms"] / max(tot["kernel_ms"], 1e-9)}
    # end to end: scene from host descriptors, render into host images
    e2e = None
    if args.e2e_steps > 0:
        t0 = time.perf_counter()
        sc2 = ctx.create_scene(holder)
        ctx.render_batch([sc2] * 8, cams, params, tuning=tune)
        sc2.destroy()
        e2e_ms = group.max(1e3 * (time.perf_counter() - t0))
        e2e = {"value": group.sum(float(paths)) / (e2e_ms / 1e3) / 1e6, "unit": "Mpaths/s",
               "h2d_bytes_per_step": int(desc_bytes(holder)),
               "d2h_bytes_per_step": int(sum(p.width * p.height * 12 for p in params)), "ms_per_step": e2e_ms,
               "timing": "host wall clock around scene creation, render and image copies"}
    # adjoint w.r.t. the env parameter grid and the per-mesh roughness values, 32 spp
    adj = None
    if args.adjoint_steps > 0:
        ti, mi = holder.texture_index, holder.material_index
        fwd = [spec.render_params(spp=32, seed=100 + v) for v in range(8)]
        adjp = [spec.render_params(spp=32, seed=900 + v) for v in range(8)]
        d_rgb = [np.random.default_rng(v).standard_normal((p.height, p.width, 3)).astype(np.float32) * 1e-4
                 for v, p in enumerate(adjp)]
        sky = spec.textures["sky"]
        f_st = ctx.render_batch([sc] * 8, cams, fwd, tuning=tune, device_outputs=ptrs)[3]
        tg, mg, _, a_st = sc.render_adjoint(cams, adjp, d_rgb, {ti["sky"]: sky.shape[:2]}, material_grads=True)
        grid = tg[ti["sky"]].reshape(sky.shape[0] // 4, 4, sky.shape[1] // 4, 4, 3).sum(axis=(1, 3))
        rough = np.array([mg[mi[f"m{k}"], 4] for k in range(64)])
        adj = {"workload": "large scene, 8 views 1080p, 32 spp forward + 32 spp adjoint, depth 16; gradients of a "
                           "random linear loss w.r.t. the 512x256x3 env grid and the 64 per-mesh roughness values",
               "forward_ms": f_st.kernel_ms, "adjoint_ms": a_st.kernel_ms,
               "adjoint_over_forward": a_st.kernel_ms / f_st.kernel_ms, "env_grid_shape": list(grid.shape),
               "env_grid_grad_l2": float(np.linalg.norm(grid)), "roughness_grad_l2": float(np.linalg.norm(rough)),
               "nan_samples": int(a_st.nan_samples)}
    sc.destroy()
    if rank == 0:
        print(json.dumps({
            "metric": METRIC, "value": value, "unit": "Mpaths/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": LARGE_WORKLOAD, "triangles": int(holder.desc.num_triangles), "views": 8,
                       "paths_per_step": int(paths), "depth": 16, "parallelism": f"replicas x{world}",
                       "l2": "inputs larger than L2", "bvh_build_ms": build_ms, "tuning": tune.as_dict()},
            "roofline": roofline, "cpu_baseline": None, "e2e": e2e, "gpu_launches": int(tot["launches"]),
            "clocks": clocks, "megakernel": {"value": mk_value, "sample": "1 view at 8 spp"},
            "wavefront_vs_megakernel": value / mk_value, "adjoint": adj, "nan_samples": int(tot["nans"]),
            "render_device_ms_per_step": tot["kernel_ms"] / args.steps}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=2)
    ap.add_argument("--mk-steps", type=int, default=1)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--scenes", type=int, default=NSCENES, help="batch size (profiling runs use fewer)")
    ap.add_argument("--adjoint-steps", type=int, default=2, help="timed adjoint/forward pairs (0 skips)")
    ap.add_argument("--no-autotune", action="store_true", help="default tuning instead of the autotuner's")
    ap.add_argument("--tuning", default=None, metavar="POOL,TRACE_BLOCK,SHADE_BLOCK,ITERS",
                    help="fixed wavefront tuning instead of the autotuner's (profiling runs pass the "
                         "autotuned values, so that ncu sees the timed step without the trial renders)")
    ap.add_argument("--event-timing", action="store_true",
                    help="time renders with CUDA event nodes and a host loop over ordinary graphs "
                         "(FM_FLAG_PROFILE) instead of the one-launch conditional graph; ncu lists and "
                         "captures only these, since it does not see kernels launched by conditional nodes")
    ap.add_argument("--workload", default="batched", choices=["batched", "large"],
                    help="batched: 64 scenes (the headline); large: 8 M triangles, 8 views of 1080p, depth 16")
    args = ap.parse_args()

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        if rank != 0:
            return
        r = run_reference(args)
        if "unavailable" in r:
            print(json.dumps(r))
            return
        line = {"impl": "reference", "metric": METRIC, "value": r["value"], "unit": "Mpaths/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": r["ms_per_step"],
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
                "data": "synthetic", "config": {"workload": WORKLOAD, "scenes": NSCENES},
                "cpu_baseline": {k: r[k] for k in ("value", "unit", "cores", "kind", "sample", "per_scene_mpaths")},
                "e2e": {"value": r["value"], "unit": "Mpaths/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
        print(json.dumps(line))
        return

    import torch
    import fumeng_b200 as fb
    from fumeng_b200 import synth

    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=600))

    from fumeng_b200.replicas import RankGroup, batch_indices
    group = RankGroup(dist, "cuda")
    barrier, max_over_ranks, sum_over_ranks = group.barrier, group.max, group.sum

    ctx = fb.Context(local_rank)
    if args.workload == "large":
        run_large(args, ctx, group, rank, world)
        ctx.close()
        if dist is not None:
            dist.destroy_process_group()
        return
    specs = [synth.batch_scene(s) for s in batch_indices(rank, args.scenes, NSCENES)]
    holders = [s.to_desc() for s in specs]
    cams = [s.camera_struct() for s in specs]
    params_wf = [s.render_params(seed=1, mode=fb.FM_MODE_WAVEFRONT) for s in specs]
    params_mk = [s.render_params(seed=1, mode=fb.FM_MODE_MEGAKERNEL) for s in specs]
    paths_per_step = sum(p.width * p.height * p.spp for p in params_wf)
    tris = sum(h.desc.num_triangles for h in holders)
    scenes = [ctx.create_scene(h) for h in holders]
    build_ms = sum(s.bvh_stats()["build_ms"] for s in scenes)
    outs = [torch.empty((p.height, p.width, 3), device="cuda", dtype=torch.float32) for p in params_wf]
    out_ptrs = [o.data_ptr() for o in outs]

    if args.tuning:
        tuning = fb.Tuning(*(int(x) for x in args.tuning.split(",")))
    elif args.no_autotune:
        tuning = fb.Tuning(1 << 21, 128, 128, 8)
    else:
        tuning = ctx.autotune_batch(scenes, cams, params_wf)

    def step_wf(profile=False):
        return ctx.render_batch(scenes, cams, params_wf, tuning=tuning, device_outputs=out_ptrs, profile=profile)[3]

    for _ in range(args.warmup):
        step_wf()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    totals = {"paths": 0, "closest": 0, "shadow": 0, "bounces": 0, "nans": 0, "trace_ms": 0.0, "shade_ms": 0.0,
              "launches": 0, "kernel_ms": 0.0}
    barrier()
    with ClockSampler(local_rank) as clk:
        ev0.record()
        for _ in range(args.steps):
            st = step_wf(profile=args.event_timing)
            totals["paths"] += st.paths
            totals["closest"] += st.closest_rays
            totals["shadow"] += st.shadow_rays
            totals["bounces"] += st.bounces
            totals["nans"] += st.nan_samples
            totals["trace_ms"] += st.trace_ms
            totals["shade_ms"] += st.shade_ms
            totals["launches"] += st.launches
            totals["kernel_ms"] += st.kernel_ms
        ev1.record()
        barrier()
    clocks = clk.summary()
    elapsed_ms = max_over_ranks(ev0.elapsed_time(ev1))
    all_paths = sum_over_ranks(float(totals["paths"]))
    value = all_paths / (elapsed_ms / 1e3) / 1e6
    assert totals["paths"] == paths_per_step * args.steps, (totals["paths"], paths_per_step)

    # megakernel on the same batch
    mk = None
    if args.mk_steps > 0:
        ctx.render_batch(scenes, cams, params_mk, device_outputs=out_ptrs)   # warm-up
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.mk_steps):
            ctx.render_batch(scenes, cams, params_mk, device_outputs=out_ptrs)
        e1.record()
        barrier()
        mk_ms = max_over_ranks(e0.elapsed_time(e1))
        mk = {"value": sum_over_ranks(float(paths_per_step * args.mk_steps)) / (mk_ms / 1e3) / 1e6,
              "ms_per_step": mk_ms / args.mk_steps, "steps": args.mk_steps}

    # roofline of the trace kernel (algorithmic bytes per the fixed per-ray formula)
    depth_eff = sum(bvh_depth_estimate(h.desc.num_triangles + 2 * h.desc.num_rects) * p.width * p.height * p.spp
                    for h, p in zip(holders, params_wf)) / paths_per_step
    closest_b = 32 + 16 + 80 * depth_eff + 160
    shadow_b = 32 + 4 + 80 * depth_eff + 160
    alg_bytes = totals["closest"] * closest_b + totals["shadow"] * shadow_b
    peak, peak_kind = measured_peak_hbm()
    achieved = alg_bytes / (totals["trace_ms"] / 1e3) / 1e9 if totals["trace_ms"] > 0 else None
    # six launches per wavefront iteration (trace, two resolve kernels, two shade kernels,
    # logic), one loop-condition kernel per graph body of iters_per_graph iterations (made even),
    # and per step one init, one counter copy and one reduce per view
    it = tuning.iters_per_graph + (tuning.iters_per_graph & 1)
    launches_trace = max(1, (totals["launches"] - args.steps * (2 + len(specs))) * it // (6 * it + 1))
    traffic = None
    if TRACE_DRAM_BYTES_PER_RAY is not None:
        traffic = TRACE_DRAM_BYTES_PER_RAY * (totals["closest"] + totals["shadow"]) / launches_trace
    roofline = {"bound": "issue", "achieved": achieved, "peak": peak, "unit": "GB/s",
                "frac": (achieved / peak) if achieved else None, "traffic": traffic,
                "dram_frac": dram_frac(totals["closest"] + totals["shadow"], totals["trace_ms"], peak),
                "kernel": "k_wf_trace", "peak_source": f"{peak_kind} hbm_gbs (MEASURED_PEAKS.json)",
                "alg_bytes_per_closest_ray": closest_b, "alg_bytes_per_shadow_ray": shadow_b,
                "trace_share_of_step": totals["trace_ms"] / max(totals["kernel_ms"], 1e-9)}

    # end to end through the C-ABI from host memory
    e2e = None
    if args.e2e_steps > 0:
        h2d = sum(desc_bytes(h) for h in holders)
        d2h = sum(p.width * p.height * 3 * 4 for p in params_wf)

        # the host images are allocated once and written by every step's read-back
        host_rgb = [np.empty(p.out_shape() + (3,), np.float32) for p in params_wf]

        def step_e2e():
            sc = ctx.create_scenes(holders)
            ctx.render_batch(sc, cams, params_wf, tuning=tuning, out=host_rgb)
            for s in sc:
                s.destroy()
        step_e2e()
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.e2e_steps):
            step_e2e()
        e1.record()
        barrier()
        e2e_ms = max_over_ranks(e0.elapsed_time(e1))
        e2e = {"value": sum_over_ranks(float(paths_per_step * args.e2e_steps)) / (e2e_ms / 1e3) / 1e6,
               "unit": "Mpaths/s", "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h),
               "ms_per_step": e2e_ms / args.e2e_steps}

    adj = measure_adjoint(ctx, args, barrier, max_over_ranks) if args.adjoint_steps > 0 else None

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        r = run_reference(args, steps=2, warmup=1)
        cpu = ({k: r[k] for k in ("value", "unit", "cores", "kind", "sample", "per_scene_mpaths")}
               if "unavailable" not in r else r)

    for s in scenes:
        s.destroy()
    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": "Mpaths/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": elapsed_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": WORKLOAD, "scenes": len(specs), "triangles": int(tris),
                       "paths_per_step": int(paths_per_step), "depth": 8,
                       "parallelism": f"replicas x{world} (each rank renders its own 64-scene batch)",
                       "l2": "inputs larger than L2 (scene data + path state exceed 126 MB)",
                       "bvh_build_ms_total": build_ms, "tuning": tuning.as_dict()},
            "roofline": roofline, "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": int(totals["launches"]),
            "clocks": clocks, "megakernel": mk,
            "wavefront_vs_megakernel": (value / mk["value"]) if mk else None,
            "per_path": {"closest_rays": totals["closest"] / totals["paths"],
                         "shadow_rays": totals["shadow"] / totals["paths"],
                         "bounces": totals["bounces"] / totals["paths"]},
            "nan_samples": int(totals["nans"]),
            # device time inside the render calls (first kernel to last) against the
            # timed steps: the difference is host time between calls
            "render_device_ms_per_step": totals["kernel_ms"] / args.steps,
            "trace_ms_per_step": totals["trace_ms"] / args.steps,
            "adjoint": adj,
        }
        print(json.dumps(line))
    ctx.close()
    if dist is not None:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
