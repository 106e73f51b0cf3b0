"""Benchmark: fwd+bwd Mpix/s of rasterize -> interpolate -> texture on the batched multi-view
workload (200k-triangle displaced sphere with packed chart UVs, 64 views at 1024x1024, 3-channel
vertex attributes, 4096x4096x4 fp32 atlas, N(0,1) upstream gradients; seeded synthetic data).

One step = the forward and backward pass over all 64 views. `value` is timed with CUDA events on
device-resident inputs; `e2e` runs the same pass through the public autograd API
(photara_drender_gb300.torch) with the inputs copied from pinned host memory and the gradients read
back every step. `--impl reference` times the CPU restatement of the reference (oracle/, all host
threads) on a bounded sample of the same workload.

Run: python bench.py [--gpus N] [--steps K] [--warmup W] [--impl gb300|reference]
"""
from __future__ import annotations

import argparse
import ctypes as C
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = dict(name="c2_fwdbwd_200k_64x1024sq_atlas4096", triangles=200_000, views=64, height=1024, width=1024,
                attributes=3, atlas=4096, channels=4, seed=0)
METRIC = "fwd+bwd Mpix/s"
CPU_SAMPLE_SECONDS = 10.0  # bounded CPU-baseline sample: whole views until this much oracle time
SKIP_CPU = False  # set by --skip-cpu: no CPU-baseline legs beside the GPU legs


def scene(w=WORKLOAD):
    from photara_drender_gb300 import synthetic as S

    pos3, nrm, uv, idx, chart, remap = S.displaced_sphere(w["triangles"], seed=w["seed"], atlas_size=w["atlas"])
    mats, eyes = S.orbit_cameras(w["views"], radius=3.0, fov_y_deg=45.0, aspect=w["width"] / w["height"])
    rng = np.random.default_rng(w["seed"])
    attrs = rng.uniform(size=(pos3.shape[0], w["attributes"])).astype(np.float32)
    return pos3, uv, idx, mats, attrs


def load_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


class ClockSampler:
    """Samples SM clocks and throttle reasons with nvidia-smi while the timed region runs."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.device_index = device_index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device_index), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


def dist_setup(args):
    import torch

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist

        dist.barrier()


def max_over_ranks(x: float, world: int) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist

    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ---- CPU restatement (reference arm and cpu_baseline) -------------------------------------------------

def cpu_fwdbwd_sample(clip, uv, idx, attrs, tex, rng, res=None):
    """One view's forward + backward through the oracle (clip positions [V, 4] of the view, resolution
    `res`, default the workload's), returns seconds. Every stage runs on the oracle's host threads (forward
    per pixel, adjoints by owner partitions that keep the reference's summation order)."""
    w = WORKLOAD
    from oracle import api

    t0 = time.perf_counter()
    raster, deriv = api.rasterize_forward(clip, idx, res or (w["height"], w["width"]))
    a = api.interpolate_forward(attrs, idx, raster)
    u = api.interpolate_forward(uv, idx, raster)
    s = api.texture_forward(tex, u, raster)
    t1 = time.perf_counter()
    ga = rng.standard_normal(a.shape, dtype=np.float32)
    gs = rng.standard_normal(s.shape, dtype=np.float32)
    t2 = time.perf_counter()
    gt, gu = api.texture_backward(tex, u, raster, gs)
    guv, gr1 = api.interpolate_backward(uv, idx, raster, gu)
    gatt, gr2 = api.interpolate_backward(attrs, idx, raster, ga)
    gp = api.rasterize_backward(clip, idx, raster, gr1 + gr2)
    t3 = time.perf_counter()
    return (t1 - t0) + (t3 - t2)


def oracle_threads(n: int) -> None:
    """Host threads of the oracle's parallel loops (0: all); its results do not depend on it."""
    from oracle import api

    api.lib().ora_set_threads(int(n))


def cpu_sample_views(clips, uv, idx, attrs, tex, threads: int, budget_s: float, res=None):
    """Whole views (clips: [views, V, 4]) through the oracle's forward + backward with `threads` host threads
    until `budget_s` seconds of work (at least one view): (views done, seconds)."""
    oracle_threads(threads)
    rng = np.random.default_rng(1)
    secs, done = 0.0, 0
    try:
        while done < len(clips) and (done == 0 or secs < budget_s):
            secs += cpu_fwdbwd_sample(np.ascontiguousarray(clips[done]), uv, idx, attrs, tex, rng, res)
            done += 1
    finally:
        oracle_threads(0)
    return done, secs


def cpu_refine_sample(st, tv_weight, nsteps, threads):
    """Seconds per step of the refiner on the host: for each of the first `nsteps` steps, the oracle's
    photometric gradient over the step's batch views (the refine state's own view caches), the chart-aware
    TV gradient when tv_weight is set, and the dense Adam update, with `threads` host threads."""
    from oracle import api

    o = st.options
    n, B = len(st.weights), int(o.batch_size)
    need = sorted({(k * B + b) % n for k in range(nsteps) for b in range(B)})
    caches = {k: tuple(st.keep[3 * k + j].cpu().numpy() for j in range(3)) for k in need}
    th, tw = int(o.height), int(o.width)
    tex = np.full((th, tw, 3), 0.5, np.float32)
    g, m, v = np.zeros_like(tex), np.zeros_like(tex), np.zeros_like(tex)
    valid = st.tv_valid.cpu().numpy() if st.tv_valid is not None else None
    chart = st.tv_chart.cpu().numpy() if st.tv_chart is not None else None
    oracle_threads(threads)
    secs = 0.0
    try:
        for k in range(nsteps):
            t0 = time.perf_counter()
            bvw = sum(st.weights[(k * B + b) % n] for b in range(B))
            norm = float(np.float32(1.0 / (bvw * 3.0))) if bvw > 0 else 0.0
            for b in range(B):
                uv, tgt, msk = caches[(k * B + b) % n]
                api.photometric_gradient(tex, uv, tgt, msk, float(o.photometric_epsilon), norm, grad=g)
            if tv_weight and valid is not None:
                api.tv_gradient(tex, valid=valid, chart=chart, eps=float(o.tv_epsilon), weight=tv_weight, grad=g)
            lr = float(o.minimum_learning_rate) + 0.5 * (float(o.learning_rate) - float(o.minimum_learning_rate)) * (
                1.0 + np.cos(np.pi * k / max(int(o.steps), 1)))
            b1, b2 = float(o.adam_beta1), float(o.adam_beta2)
            api.adam_update(tex, g, m, v, lr, b1, b2, float(o.adam_epsilon), 1.0 - b1 ** (k + 1), 1.0 - b2 ** (k + 1),
                            float(o.clamp_min), float(o.clamp_max))
            secs += time.perf_counter() - t0
    finally:
        oracle_threads(0)
    return secs / nsteps


def run_reference(args, world, rank):
    if rank != 0:
        return
    from oracle import api  # builds the oracle when needed

    w = WORKLOAD
    pos3, uv, idx, mats, attrs = scene()
    rng = np.random.default_rng(1)
    tex = rng.uniform(size=(w["atlas"], w["atlas"], w["channels"])).astype(np.float32)
    cores = os.cpu_count() or 1
    clips = [api.transform_positions(pos3, mats[k]) for k in range(w["views"])]
    for k in range(args.warmup):
        cpu_fwdbwd_sample(clips[k % w["views"]], uv, idx, attrs, tex, rng)
    times = [cpu_fwdbwd_sample(clips[k % w["views"]], uv, idx, attrs, tex, rng) for k in range(args.steps)]
    per_view = float(np.mean(times))
    mpix = w["height"] * w["width"] / 1e6 / per_view
    sample = (f"one of the {w['views']} views per step (view k mod {w['views']}), full forward+backward at "
              f"{w['height']}x{w['width']}; every stage on all {cores} host threads (OpenMP: forward per pixel, "
              f"adjoints partitioned by texel rows / vertices / triangles so sums keep the reference's order)")
    line = {
        "metric": METRIC, "value": mpix, "unit": "Mpix/s", "n_gpus": args.gpus, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": per_view * 1e3, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic", "impl": "reference",
        "config": {"workload": w["name"], "views": w["views"], "resolution": [w["height"], w["width"]],
                   "triangles": int(idx.shape[0]), "atlas": [w["atlas"], w["atlas"], w["channels"]],
                   "attributes": w["attributes"], "l2": "inputs larger than L2"},
        "cpu_baseline": {"value": mpix, "unit": "Mpix/s", "cores": cores, "kind": "port", "sample": sample},
        "e2e": {"value": mpix, "unit": "Mpix/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "note": "the reference's Vulkan path cannot run here (no graphics stack); its shader arithmetic runs as "
                "the oracle's C restatement, pinned bit-exact to the reference shaders compiled for the CPU",
    }
    print(json.dumps(line), flush=True)


# ---- bake (200k triangles, 64 views 1024^2 -> 4096^2 atlas) and refine (500k triangles, 32 views 2048x1536,
# ---- 4096^2 atlas, 1000 steps as one CUDA graph) legs -----------------------------------------------------

BAKE = dict(name="c2_bake_200k_64x1024sq_atlas4096", triangles=200_000, views=64, height=1024, width=1024, atlas=4096,
            seed=0)
REFINE = dict(name="c3_refine_500k_32x2048x1536_atlas4096_1000steps", triangles=500_000, views=32, height=1536,
              width=2048, atlas=4096, steps=1000, batch=4, lr=1e-2, min_lr=2.5e-4, tv_weight=1e-4, seam_steps=30,
              seam_lr=1e-3, seed=1)


def smooth_noise_atlas(size, seed, dev):
    """Ground-truth atlas [size, size, 3]: 0.5 plus a few random low-frequency cosines per channel."""
    import torch

    g = torch.Generator(device="cpu").manual_seed(seed)
    y = torch.linspace(0.0, 1.0, size, device=dev)[:, None]
    x = torch.linspace(0.0, 1.0, size, device=dev)[None, :]
    out = torch.empty((size, size, 3), device=dev)
    for c in range(3):
        acc = torch.zeros((size, size), device=dev)
        for _ in range(6):
            fx, fy = (torch.rand(2, generator=g) * 12.0 + 1.0).tolist()
            ph = float(torch.rand(1, generator=g)) * 2.0 * np.pi
            acc += torch.cos(2.0 * np.pi * (fx * x + fy * y) + ph)
        out[..., c] = 0.5 + 0.06 * acc
    return out.clamp_(0.02, 0.98)


def render_views(r, t_pos, t_uv, t_idx, mats, H, W, atlas_rgb, dev):
    """Images of the ground-truth atlas through the library's own forward path: (rgb [n,H,W,3], raster)."""
    import torch

    from photara_drender_gb300 import _native
    from photara_drender_gb300.rasterizer import _ptr

    n, V = mats.shape[0], t_pos.shape[0]
    clip = torch.empty((n, V, 4), dtype=torch.float32, device=dev)
    t_mats = torch.tensor(mats, device=dev)
    _native.call("pdr_transform_positions", _ptr(t_pos), V, _ptr(t_mats), n, _ptr(clip),
                 C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    raster, _ = r.forward(clip, t_idx, (H, W), output_barycentric_derivatives=False)
    uv_img = r.interpolate_forward(t_uv, t_idx, raster)
    rgba = torch.cat([atlas_rgb, torch.ones_like(atlas_rgb[..., :1])], -1).contiguous()
    color = r.texture_forward(rgba, uv_img, raster)[..., :3]
    return color, raster


C1 = dict(name="c1_fwdbwd_ico4_8x512sq_tex1024", subdivisions=4, views=8, height=512, width=512, attributes=3,
          texture=1024, channels=4, seed=0, steps=200, e2e_steps=50)


def c1_leg(dev, hbm):
    """C1: icosphere subdivision 4 (2562 vertices, 5120 triangles), 8 Fibonacci orbit views at 512x512,
    3 attributes, 1024x1024x4 texture, N(0,1) upstream gradients. Small enough to be launch-bound, so
    it is timed both as plain launches and as one CUDA-graph replay per step."""
    import torch

    from photara_drender_gb300 import Rasterizer, _native
    from photara_drender_gb300 import synthetic as S
    from photara_drender_gb300.pipeline import RenderFwdBwd
    from photara_drender_gb300.rasterizer import _ptr

    c = C1
    pos3, idx = S.icosphere(c["subdivisions"])
    mats, _ = S.orbit_cameras(c["views"], radius=3.0, fov_y_deg=45.0, aspect=1.0)
    rng = np.random.default_rng(c["seed"])
    attrs = torch.tensor(rng.uniform(size=(pos3.shape[0], c["attributes"])).astype(np.float32), device=dev)
    tex = torch.tensor(rng.uniform(size=(c["texture"], c["texture"], c["channels"])).astype(np.float32), device=dev)
    uv = torch.tensor(S.spherical_uv(pos3), device=dev)
    clip = torch.tensor(S.clip_positions(pos3, mats), device=dev)
    t_idx = torch.tensor(idx.astype(np.int32), device=dev)
    views, H, W = c["views"], c["height"], c["width"]
    g_attr = torch.tensor(rng.standard_normal((views, H, W, c["attributes"])).astype(np.float32), device=dev)
    g_samp = torch.tensor(rng.standard_normal((views, H, W, c["channels"])).astype(np.float32), device=dev)
    r = Rasterizer(dev.index or 0)
    V, T = pos3.shape[0], idx.shape[0]
    pipe = RenderFwdBwd(r, t_idx, V, views, H, W, c["attributes"], tuple(tex.shape), direct=True)
    pipe.step(clip, attrs, uv, tex, g_attr, g_samp)

    def timed(fn, n):
        for _ in range(5):
            fn()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize(dev)
        e0.record()
        for _ in range(n):
            fn()
        e1.record()
        torch.cuda.synchronize(dev)
        return e0.elapsed_time(e1) / n

    ms_launch = timed(lambda: pipe.step(clip, attrs, uv, tex, g_attr, g_samp), c["steps"])
    graph = pipe.capture(clip, attrs, uv, tex, g_attr, g_samp)
    ms_graph = timed(graph.replay, c["steps"])
    P = views * H * W
    alg = P * 96 + 2 * c["texture"] ** 2 * c["channels"] * 4 + views * V * 16 * 2 + T * 12 + V * (c["attributes"] + 2) * 8
    best = min(ms_launch, ms_graph)
    res = {"workload": c["name"], "mpix_per_s": P / 1e6 / (best / 1e3), "ms_per_step_graph": ms_graph,
           "ms_per_step_launches": ms_launch, "algorithmic_bytes": alg,
           "achieved_gbs": alg / (best / 1e3) / 1e9, "frac": alg / (best / 1e3) / 1e9 / hbm,
           "timing": f"CUDA events over {c['steps']} fused fwd+bwd steps, device-resident inputs (which fit in L2)"}
    host = {k: v.cpu().pin_memory() for k, v in dict(clip=clip, attrs=attrs, uv=uv, tex=tex, g_attr=g_attr,
                                                     g_samp=g_samp).items()}
    host["idx"] = torch.tensor(idx.astype(np.int64)).pin_memory()
    e2e_ms, h2d, d2h = e2e_render(dev, r, host, H, W, c["e2e_steps"])
    res["e2e"] = {"value": P / 1e6 / (e2e_ms / 1e3), "unit": "Mpix/s", "ms_per_step": e2e_ms,
                  "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h),
                  "api": f"photara_drender_gb300.torch.render + backward with host buffers, {c['e2e_steps']} steps"}
    if not SKIP_CPU:
        args_h = (clip.cpu().numpy(), S.spherical_uv(pos3).astype(np.float32), idx, attrs.cpu().numpy(),
                  tex.cpu().numpy())
        done, secs = cpu_sample_views(*args_h, 0, 5.0, res=(H, W))
        done1, secs1 = cpu_sample_views(*args_h, 1, 5.0, res=(H, W))
        cores = os.cpu_count() or 1
        res["cpu_baseline"] = {
            "value": done * H * W / 1e6 / secs, "unit": "Mpix/s", "cores": cores, "kind": "port",
            "sample": f"{done} of the {views} views (until 5 s of work), full forward+backward through the oracle "
                      f"on all {cores} host threads, {secs:.2f} s",
            "one_core": {"value": done1 * H * W / 1e6 / secs1, "unit": "Mpix/s", "cores": 1,
                         "sample": f"{done1} views on one thread, {secs1:.2f} s"}}
    return res


def bake_leg(dev, hbm):
    """C2 bake: weighted-average projection of 64 noisy views, PCF 1, in the reference's default ray-query
    visibility (device BVH + any-hit rays per texel and view) and with shadow maps; then padding
    (margin 4, unobserved texels filled) and surface fill of the ray-query atlas."""
    import torch

    from photara_drender_gb300 import TextureBaker
    from photara_drender_gb300 import padding as PAD
    from photara_drender_gb300 import synthetic as S

    b = BAKE
    pos3, nrm, uv, idx, _, remap = S.displaced_sphere(b["triangles"], seed=b["seed"], atlas_size=b["atlas"])
    mats, eyes = S.orbit_cameras(b["views"], radius=3.0, fov_y_deg=45.0, aspect=b["width"] / b["height"])
    baker = TextureBaker(dev.index or 0)
    t_pos, t_nrm, t_uv = (torch.tensor(a, device=dev) for a in (pos3, nrm, uv))
    t_idx = torch.tensor(idx.astype(np.int32), device=dev)
    gt = smooth_noise_atlas(b["atlas"], b["seed"], dev)
    color, _ = render_views(baker.rasterizer, t_pos, t_uv, t_idx, mats, b["height"], b["width"], gt, dev)
    g = torch.Generator(device=dev).manual_seed(b["seed"])
    images = (color + 0.01 * torch.randn(color.shape, device=dev, generator=g)).contiguous()
    views = [images[k] for k in range(b["views"])]
    N = b["atlas"] ** 2
    P = b["views"] * b["height"] * b["width"]

    def timed(fn, reps=3):
        out = fn()
        torch.cuda.synchronize(dev)
        times = []
        for _ in range(reps):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize(dev)
            e0.record()
            out = fn()
            e1.record()
            torch.cuda.synchronize(dev)
            times.append(e0.elapsed_time(e1) / 1e3)
        return out, float(np.median(times))

    res = {"workload": b["name"], "timing": "median of 3 TextureBaker.bake_output calls on device-resident views "
                                            "(host validation, BVH build or per-view shadow rasters included)"}
    outs = {}
    for mode in ("ray_query", "shadow_map"):
        out, s = timed(lambda: baker.bake_output(t_pos, t_nrm, t_uv, t_idx, views, mats, eyes,
                                                 resolution=(b["atlas"], b["atlas"]), blend_mode="weighted_average",
                                                 visibility_mode=mode, pcf_radius=1))
        # atlas G-buffer read 28 B/texel, outputs 36 B/texel, per view pixel: photo 12 + mask 4 (+ shadow depth 4)
        alg = N * (28 + 36) + P * (16 if mode == "ray_query" else 20)
        valid = out.valid_mask > 0.5
        err = (out.color[..., :3] - gt).abs()[valid].mean().item() if bool(valid.any()) else None
        res[mode] = {"seconds": s, "gtexel_views_per_s": N * b["views"] / s / 1e9, "algorithmic_bytes": alg,
                     "achieved_gbs": alg / s / 1e9, "frac": alg / s / 1e9 / hbm,
                     "valid_texels": int(valid.sum().item()), "mean_abs_error_vs_ground_truth": err}
        outs[mode] = out
    out = outs["ray_query"]
    cov = out.coverage_mask.contiguous()
    valid = out.valid_mask.contiguous()
    work = out.color.clone()
    filled = torch.zeros_like(valid)

    def pad():
        work.copy_(out.color)
        filled.zero_()
        return PAD.pad_texture_atlas_device(work, valid, 4, cov, True, 0, filled_mask=filled)

    st, s_pad = timed(pad)
    copy_s = timed(lambda: work.copy_(out.color))[1]
    s_pad = max(s_pad - copy_s, 1e-9)
    # colour read once and written once, valid / coverage / filled read, filled written: 16+16+4+4+4+4 B
    pad_bytes = N * 48
    res["padding"] = {"seconds": s_pad, "texels_per_s": N / s_pad, "stats": list(st), "algorithmic_bytes": pad_bytes,
                      "achieved_gbs": pad_bytes / s_pad / 1e9,
                      "note": "pad_texture_atlas(margin=4, fill_unobserved) on the ray-query atlas; the copy that "
                              "restores the input each repetition is timed separately and subtracted"}
    welded = torch.tensor(remap[idx].astype(np.int32), device=dev)
    faces = out.face_ids.contiguous()
    sf, s_fill = timed(lambda: PAD.fill_texture_on_surface(out.color, valid, faces, welded))
    res["surface_fill"] = {"seconds": s_fill, "stats": list(sf[2]),
                           "note": "fill_texture_on_surface on the ray-query atlas with the welded mesh topology "
                                   "(copies of colour and filled_mask included)"}
    if not SKIP_CPU:
        from oracle import api as oracle_api

        try:
            cores = os.cpu_count() or 1
            imgs_h = [images[k].cpu().numpy() for k in range(4)]
            bake_args = (pos3, nrm, uv, idx)

            def cpu_bake(nv, threads):
                oracle_threads(threads)
                try:
                    t0 = time.perf_counter()
                    oracle_api.bake(*bake_args, imgs_h[:nv], mats[:nv], eyes[:nv], resolution=(b["atlas"], b["atlas"]),
                                    blend_mode="weighted_average", pcf_radius=1)
                    return time.perf_counter() - t0
                finally:
                    oracle_threads(0)

            s1, s4 = cpu_bake(1, 0), cpu_bake(4, 0)
            per_view = max((s4 - s1) / 3.0, 1e-9)
            one = cpu_bake(1, 1)
            res["cpu_baseline"] = {
                "value": N / 1e9 / per_view, "unit": "Gtexel-views/s", "cores": cores, "kind": "port",
                "sample": f"the oracle's shadow-map bake (weighted average, PCF 1) of views 0-3 into the "
                          f"{b['atlas']}^2 atlas on all {cores} host threads: 1 view {s1:.2f} s, 4 views {s4:.2f} s "
                          f"(per view {per_view:.2f} s after the atlas G-buffer); all {b['views']} views would take "
                          f"{s1 + per_view * (b['views'] - 1):.1f} s",
                "one_core": {"value": None, "unit": "Gtexel-views/s", "cores": 1,
                             "sample": f"1 view on one thread (G-buffer included): {one:.2f} s"}}
        except Exception as e:
            res["cpu_baseline"] = {"value": None, "kind": "port", "sample": f"failed: {e}"}

        host = (out.color.cpu().numpy(), valid.cpu().numpy(), cov.cpu().numpy())
        t0 = time.perf_counter()
        oracle_api.pad_texture_atlas(host[0], host[1], 4, coverage_mask=host[2], fill_unobserved=True)
        res["padding"]["cpu_oracle_seconds"] = time.perf_counter() - t0
        res["padding"]["cpu_oracle"] = "oracle restatement of texture_padding.cpp, one host thread (as the reference)"
    return res


def refine_scene(c, dev, baker):
    """A refinement scene of config `c` (triangles, views, height, width, atlas, seed): the displaced
    sphere with six packed charts, views rendered from a smooth-noise ground-truth atlas with a per-view
    exposure gain U[0.8, 1.2], binary foreground masks (silhouette eroded by 2 pixels and a random
    ellipse), the atlas valid mask and chart ids, and the seam pairs."""
    import torch
    import torch.nn.functional as F

    from photara_drender_gb300 import synthetic as S
    from photara_drender_gb300.precond import atlas_layout

    pos3, _, uv, idx, chart, remap = S.displaced_sphere(c["triangles"], seed=c["seed"], atlas_size=c["atlas"])
    mats, _ = S.orbit_cameras(c["views"], radius=3.0, fov_y_deg=45.0, aspect=c["width"] / c["height"])
    r = baker.rasterizer
    t_pos, t_uv = torch.tensor(pos3, device=dev), torch.tensor(uv, device=dev)
    t_idx = torch.tensor(idx.astype(np.int32), device=dev)
    gt = smooth_noise_atlas(c["atlas"], c["seed"], dev)
    color, raster = render_views(r, t_pos, t_uv, t_idx, mats, c["height"], c["width"], gt, dev)
    rng = np.random.default_rng(c["seed"])
    gain = torch.tensor(rng.uniform(0.8, 1.2, size=c["views"]).astype(np.float32), device=dev)
    images = (color * gain[:, None, None, None]).contiguous()
    sil = (raster[..., 3] > 0).float()
    eroded = 1.0 - F.max_pool2d((1.0 - sil)[:, None], 5, stride=1, padding=2)[:, 0]
    yy = torch.arange(c["height"], device=dev, dtype=torch.float32)[:, None] / c["height"]
    xx = torch.arange(c["width"], device=dev, dtype=torch.float32)[None, :] / c["width"]
    ell = torch.empty_like(sil)
    for k in range(c["views"]):
        cx, cy, rx, ry = rng.uniform(0.35, 0.65), rng.uniform(0.35, 0.65), rng.uniform(0.3, 0.6), rng.uniform(0.3, 0.6)
        ell[k] = (((xx - cx) / rx) ** 2 + ((yy - cy) / ry) ** 2 <= 1.0).float()
    masks = (eroded * ell).contiguous()
    del raster, color, sil, eroded, ell
    valid, charts = atlas_layout(r, t_uv, t_idx, chart, c["atlas"], c["atlas"])
    pairs = torch.tensor(S.seam_uv_pairs(uv, idx, remap, chart), device=dev)
    return dict(pos=t_pos, uv=t_uv, idx=t_idx, mats=mats, images=[images[k] for k in range(c["views"])],
                masks=[masks[k] for k in range(c["views"])], valid=valid, charts=charts, pairs=pairs, gt=gt)


def refine_args(c, sc, steps):
    """Positional arguments of TextureBaker._refine_prepare for scene `sc` with the config's schedule."""
    import torch

    init = torch.full((c["atlas"], c["atlas"], 3), 0.5, device=sc["pos"].device)
    return (init, sc["pos"], sc["uv"], sc["idx"], sc["images"], sc["mats"], sc["masks"], None, sc["pairs"], steps,
            c["batch"], c["lr"], c["min_lr"], 1e-3, c["seam_steps"], c["seam_lr"], 0.9, 0.999, 1e-8, 0.0, 1.0, 1e-4,
            c["tv_weight"], sc["valid"].float(), sc["charts"], 1e-4)


def refine_leg(dev, hbm):
    """C3 refine: 1000 masked photometric Adam steps with chart-aware TV, then the seam polish, recorded and
    launched as one CUDA graph."""
    import torch

    from photara_drender_gb300 import TextureBaker

    c = REFINE
    baker = TextureBaker(dev.index or 0)
    sc = refine_scene(c, dev, baker)
    with baker.context.lock:
        st = baker._refine_prepare(*refine_args(c, sc, c["steps"]))
        tex, hist, seam, pre_s, opt_s = baker._refine_finish(st, True)
    torch.cuda.synchronize(dev)
    pairs = sc["pairs"]
    steps = c["steps"] + (c["seam_steps"] if pairs.shape[0] else 0)
    P = c["views"] * c["height"] * c["width"]
    n = c["atlas"] ** 2 * 3
    # per photometric step: batch views x pixels x (uv 8 + target 12 + mask 4) + atlas gather + dense Adam 32 B/value
    step_bytes = c["batch"] * (P // c["views"]) * 24 + n * 4 + n * 32
    vmask = sc["valid"].bool()
    err = (tex - sc["gt"]).abs()[vmask].mean().item()
    return {"workload": c["name"], "optimization_seconds": opt_s, "precompute_seconds": pre_s,
            "ms_per_step": opt_s / steps * 1e3, "steps": steps, "final_loss": float(hist[-1]),
            "first_loss": float(hist[0]), "seam_pairs": int(pairs.shape[0]),
            "final_seam_loss": float(seam[-1]) if len(seam) else None,
            "algorithmic_bytes_per_step": step_bytes, "achieved_gbs": step_bytes * c["steps"] / opt_s / 1e9,
            "frac": step_bytes * c["steps"] / opt_s / 1e9 / hbm, "mean_abs_error_vs_ground_truth": err,
            "timing": "TextureBaker refinement optimisation wall time (graph record + instantiate + launch + "
                      "sync), texture starting at 0.5",
            "cpu_baseline": refine_cpu_baseline(st, c),
            "photometric_reductions": photometric_reduction_rate(dev, st)}


def photometric_reduction_rate(dev, st):
    """The photometric gradient kernel of step 0 (its batch of views) timed alone: its bilinear-tap
    reductions (four red.v4 per masked pixel) per second against the calibrated scattered-reduction rates."""
    import torch

    from photara_drender_gb300 import _native
    from photara_drender_gb300.rasterizer import _ptr

    o = st.options
    n, B = len(st.weights), int(o.batch_size)
    masked = sum(int((st.keep[3 * (b % n) + 2] > 0).sum().item()) for b in range(B))
    tex = torch.full((int(o.height), int(o.width), 3), 0.5, device=dev)
    grad = torch.zeros((int(o.height), int(o.width), 4), device=dev)
    loss = torch.zeros(1, device=dev)
    stream = C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)

    def run():
        _native.call("pdr_refine_photometric", _ptr(tex), int(o.width), int(o.height), _ptr(st.table_dev), n,
                     st.max_pixels, 0, B, float(o.photometric_epsilon), 1e-6, _ptr(grad), _ptr(loss), stream)

    run()
    times = []
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize(dev)
        e0.record()
        run()
        e1.record()
        torch.cuda.synchronize(dev)
        times.append(e0.elapsed_time(e1) / 1e3)
    t = float(np.median(times))
    peaks = reduction_peaks(dev)
    rate = 4 * masked / t
    return {"kernel": "photometric_kernel (one step: batch views of step 0)", "seconds": t,
            "reductions": 4 * masked, "reductions_per_s": rate, "calibrated_peaks_per_s": peaks,
            "frac_of_l2_resident_peak": rate / peaks["l2_resident_32MB"],
            "frac_of_hbm_peak": rate / peaks["hbm_268MB"],
            "note": "peaks: pdr_calibrate_reductions (red.global.add.v4.f32 to pseudo-random 16-byte slots) into "
                    "a 32 MB buffer that stays in L2 and a 268 MB one that does not"}


def reduction_peaks(dev):
    """Scattered red.global.add.v4.f32 rates (reductions / s) of pdr_calibrate_reductions: into a 32 MB
    buffer that stays in L2, and into a 268 MB one (the size of a 4096^2 RGBA gradient) that does not."""
    import torch

    from photara_drender_gb300 import _native
    from photara_drender_gb300.rasterizer import _ptr

    stream = C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    out = {}
    for name, mb in (("l2_resident_32MB", 32), ("hbm_268MB", 268)):
        slots = mb * 1024 * 1024 // 16
        buf = torch.zeros((slots, 4), dtype=torch.float32, device=dev)
        n = 64 * 1024 * 1024
        _native.call("pdr_calibrate_reductions", _ptr(buf), slots, n, 1, stream)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize(dev)
        e0.record()
        for k in range(3):
            _native.call("pdr_calibrate_reductions", _ptr(buf), slots, n, 2 + k, stream)
        e1.record()
        torch.cuda.synchronize(dev)
        out[name] = 3 * n / (e0.elapsed_time(e1) / 1e3)
        del buf
    return out


def refine_cpu_baseline(st, c):
    """The refiner's photometric + TV + Adam steps on the host (the oracle's restatement of the shaders), a
    reduced number of steps timed and stated, with all host threads and with one."""
    if SKIP_CPU:
        return None
    try:
        cores = os.cpu_count() or 1
        all_s = cpu_refine_sample(st, c["tv_weight"], 2, 0)
        one_s = cpu_refine_sample(st, c["tv_weight"], 1, 1)
        return {"value": all_s, "unit": "s/step", "cores": cores, "kind": "port",
                "sample": f"steps 0-1 of {c['steps']} (batch {c['batch']} views of {c['height']}x{c['width']}, "
                          f"{c['atlas']}^2 atlas): photometric gradient, chart-aware TV and dense Adam through the "
                          f"oracle on all {cores} host threads; {c['steps']} steps would take "
                          f"{all_s * c['steps']:.0f} s",
                "one_core": {"value": one_s, "unit": "s/step", "cores": 1, "sample": "step 0 on one thread"}}
    except Exception as e:  # the CPU leg never hides a GPU result
        return {"value": None, "unit": "s/step", "kind": "port", "sample": f"failed: {e}"}


C4 = dict(name="c4_uneven_batch_16_meshes", meshes=16, tri_min=10_000, tri_max=1_000_000, views=(4, 48),
          resolutions=((512, 512), (1024, 1024), (1536, 2048)), textures=(2048, 4096), attributes=8, seed=0, reps=3)


def c4_leg(dev, hbm):
    """C4: 16 meshes of log-uniform 10k-1M triangles, 4-48 views each at 512^2, 1024^2 or 2048x1536,
    8-channel attributes, 2048^2 or 4096^2 RGBA textures, forward + backward in one batch (one
    visibility pass, one shading launch, one adjoint launch); each mesh is also timed alone for the per-mesh p50 / p99."""
    import torch

    from photara_drender_gb300 import Rasterizer
    from photara_drender_gb300 import synthetic as S
    from photara_drender_gb300.batch import BatchMesh, MeshBatch

    c = C4
    rng = np.random.default_rng(c["seed"])
    g = torch.Generator(device=dev).manual_seed(c["seed"])
    r = Rasterizer(dev.index or 0)
    meshes, desc = [], []
    for k in range(c["meshes"]):
        T = int(np.exp(rng.uniform(np.log(c["tri_min"]), np.log(c["tri_max"]))))
        views = int(rng.integers(c["views"][0], c["views"][1] + 1))
        h, w = c["resolutions"][int(rng.integers(len(c["resolutions"])))]
        ts = int(c["textures"][int(rng.integers(len(c["textures"])))])
        pos3, _, uv, idx, _, _ = S.displaced_sphere(T, seed=k, atlas_size=ts)
        mats, _ = S.orbit_cameras(views, radius=3.0, fov_y_deg=45.0, aspect=w / h)
        V = pos3.shape[0]
        m = BatchMesh(clip=torch.tensor(S.clip_positions(pos3, mats), device=dev),
                      indices=torch.tensor(idx.astype(np.int32), device=dev), height=h, width=w,
                      attributes=torch.rand((V, c["attributes"]), device=dev, generator=g),
                      uv_attributes=torch.tensor(uv, device=dev),
                      texture=torch.rand((ts, ts, 4), device=dev, generator=g))
        m.grads["interp"] = torch.randn((views, h, w, c["attributes"]), device=dev, generator=g)
        m.grads["sampled"] = torch.randn((views, h, w, 4), device=dev, generator=g)
        if k == 0:
            first = (m.clip.cpu().numpy(), uv, idx, m.attributes.cpu().numpy(), m.texture.cpu().numpy(), (h, w))
        meshes.append(m)
        desc.append({"triangles": int(idx.shape[0]), "views": views, "resolution": [h, w], "texture": ts})
    batch = MeshBatch(r, meshes)

    def timed(b):
        b.forward()
        b.backward()
        out = []
        for _ in range(c["reps"]):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize(dev)
            e0.record()
            b.forward()
            b.backward()
            e1.record()
            torch.cuda.synchronize(dev)
            out.append(e0.elapsed_time(e1))
        return float(np.median(out))

    batch_ms = timed(batch)
    per_mesh = []
    for m in meshes:
        single = MeshBatch(r, [m])
        per_mesh.append(timed(single))
        del single
    P = sum(d["views"] * d["resolution"][0] * d["resolution"][1] for d in desc)
    A = c["attributes"]
    # forward outputs 16 + 16 + 4A + 8 + 16, backward inputs 4A + 16 per pixel; textures read and
    # their gradients written once
    alg = P * (16 + 16 + 4 * A + 8 + 16 + 4 * A + 16) + sum(2 * d["texture"] ** 2 * 16 for d in desc)
    cpu = None
    if not SKIP_CPU:
        clips, uv0, idx0, attrs0, tex0, res0 = first
        cores = os.cpu_count() or 1
        done, secs = cpu_sample_views(clips, uv0, idx0, attrs0, tex0, 0, 5.0, res=res0)
        done1, secs1 = cpu_sample_views(clips, uv0, idx0, attrs0, tex0, 1, 5.0, res=res0)
        px = res0[0] * res0[1]
        cpu = {"value": done * px / 1e6 / secs, "unit": "Mpix/s", "cores": cores, "kind": "port",
               "sample": f"mesh 0 of the batch ({desc[0]['triangles']} triangles, {desc[0]['texture']}^2 texture, "
                         f"8 attributes): {done} of its {desc[0]['views']} views at {res0[0]}x{res0[1]} (until 5 s "
                         f"of work), forward+backward through the oracle on all {cores} host threads, {secs:.2f} s; "
                         f"the whole batch at this rate: {P / (done * px / secs):.0f} s",
               "one_core": {"value": done1 * px / 1e6 / secs1, "unit": "Mpix/s", "cores": 1,
                            "sample": f"{done1} views on one thread, {secs1:.2f} s"}}
    return {"workload": c["name"], "batch_ms": batch_ms, "mpix_per_s": P / 1e6 / (batch_ms / 1e3), "cpu_baseline": cpu,
            "pixels": P, "meshes": desc,
            "per_mesh_ms_p50": float(np.percentile(per_mesh, 50)), "per_mesh_ms_p99": float(np.percentile(per_mesh, 99)),
            "per_mesh_ms": per_mesh, "per_mesh_sum_ms": float(np.sum(per_mesh)),
            "algorithmic_bytes": alg, "achieved_gbs": alg / (batch_ms / 1e3) / 1e9,
            "frac": alg / (batch_ms / 1e3) / 1e9 / hbm,
            "timing": "CUDA events, median of 3 forward+backward passes (host plan upload included); per mesh: the "
                      "same batch API with one mesh"}


# C5: the preconditioner is trained on plain trajectories of 64 seeded scenes of the C2 kind (smaller, so the
# training data is collected in seconds) and evaluated on a held-out 1M-triangle, 48-view 2048x1536 scene.
PRECOND_TRAIN = dict(triangles=50_000, views=16, height=512, width=512, atlas=1024, steps=1000, batch=4, lr=1e-2,
                     min_lr=2.5e-4, tv_weight=1e-4, seam_steps=30, seam_lr=1e-3, scenes=64, interval=25,
                     samples=4096, fit_steps=600, fit_batch=65536, fit_lr=2e-3)
PRECOND_EVAL = dict(name="c5_learned_precond_1M_48x2048x1536_atlas4096", triangles=1_000_000, views=48, height=1536,
                    width=2048, atlas=4096, steps=1000, batch=4, lr=1e-2, min_lr=2.5e-4, tv_weight=1e-4,
                    seam_steps=30, seam_lr=1e-3, seed=1000, budgets=(60, 125, 250, 500), refresh=25, tolerance=0.02)


def c5_leg(dev, hbm):
    """Learned vs plain refinement: time for the learned refiner to reach the plain 1000-step photometric loss
    (within 1%), with plain runs of the same shortened schedules as a control."""
    import torch

    from photara_drender_gb300 import TextureBaker
    from photara_drender_gb300.precond import (PrecondMLP, photometric_loss, plain_trajectory_samples,
                                               refine_learned, texel_stats)

    tr, ev = PRECOND_TRAIN, PRECOND_EVAL
    baker = TextureBaker(dev.index or 0)
    t0 = time.perf_counter()
    feats, targets, weights = [], [], []
    with baker.context.lock:
        for k in range(tr["scenes"]):
            sc = refine_scene(dict(tr, seed=k), dev, baker)
            st = baker._refine_prepare(*refine_args(tr, sc, tr["steps"]))
            stats = texel_stats(st, sc["valid"], sc["charts"])
            f, t, w, _ = plain_trajectory_samples(st, stats, sc["valid"], interval=tr["interval"],
                                                  samples=tr["samples"], seed=k)
            feats.append(f)
            targets.append(t)
            weights.append(w)
            del sc, st, stats
    torch.cuda.synchronize(dev)
    t1 = time.perf_counter()
    F_, T_, W_ = torch.cat(feats), torch.cat(targets), torch.cat(weights)
    mlp = PrecondMLP(dev.index or 0, seed=0)
    fit = mlp.fit(F_, T_, W_, steps=tr["fit_steps"], batch=tr["fit_batch"], lr=tr["fit_lr"])
    torch.cuda.synchronize(dev)
    t2 = time.perf_counter()

    sc = refine_scene(ev, dev, baker)
    runs = {}
    with baker.context.lock:
        def plain(steps):
            st = baker._refine_prepare(*refine_args(ev, sc, steps))
            out = baker._refine_finish(st, True)
            return {"steps": steps, "seconds": out[4], "loss": photometric_loss(st, out[0])}

        def learned(steps):
            st = baker._refine_prepare(*refine_args(ev, sc, steps))
            stats = texel_stats(st, sc["valid"], sc["charts"])
            out = refine_learned(baker, st, mlp, stats, refresh_interval=ev["refresh"],
                                 fallback_tolerance=ev["tolerance"], use_graph=True)
            return {"steps": steps, "seconds": out[4], "loss": photometric_loss(st, out[0]), "fell_back": out[5]}

        plain(ev["budgets"][0])  # warm-up (graph instantiation paths, caches)
        runs["plain"] = plain(ev["steps"])
        for b in ev["budgets"]:
            runs[f"learned_{b}"] = learned(b)
            runs[f"plain_{b}"] = plain(b)
    cpu = None
    if not SKIP_CPU:
        with baker.context.lock:
            st = baker._refine_prepare(*refine_args(ev, sc, ev["steps"]))
            try:
                cores = os.cpu_count() or 1
                per = cpu_refine_sample(st, ev["tv_weight"], 1, 0)
                cpu = {"value": per, "unit": "s/step", "cores": cores, "kind": "port",
                       "sample": f"one plain refine step at this size (batch {ev['batch']} views of "
                                 f"{ev['height']}x{ev['width']}, {ev['atlas']}^2 atlas, photometric + TV + Adam) "
                                 f"through the oracle on all {cores} host threads; the plain {ev['steps']}-step "
                                 f"schedule would take {per * ev['steps']:.0f} s"}
            except Exception as e:
                cpu = {"value": None, "kind": "port", "sample": f"failed: {e}"}
            del st
    target = runs["plain"]["loss"] * 1.01
    hit = [runs[f"learned_{b}"] for b in ev["budgets"] if runs[f"learned_{b}"]["loss"] <= target]
    best = min(hit, key=lambda r: r["seconds"]) if hit else None
    plain_hit = [runs[f"plain_{b}"] for b in ev["budgets"] if runs[f"plain_{b}"]["loss"] <= target]
    # the fair control: the fastest plain schedule (of the same budgets, or the full one) that reaches the target
    best_plain = min(plain_hit + [runs["plain"]], key=lambda r: r["seconds"])
    ratio_best = best["seconds"] / best_plain["seconds"] if best else None
    return {"workload": ev["name"], "cpu_baseline": cpu, "plain_loss": runs["plain"]["loss"],
            "plain_seconds": runs["plain"]["seconds"],
            "target_loss": target,
            "learned_seconds_to_target": best["seconds"] if best else None,
            "learned_steps_to_target": best["steps"] if best else None,
            "time_ratio_vs_plain": best["seconds"] / runs["plain"]["seconds"] if best else None,
            "best_plain_steps_to_target": best_plain["steps"], "best_plain_seconds_to_target": best_plain["seconds"],
            "time_ratio_vs_best_plain": ratio_best,
            "target_met": bool(ratio_best is not None and ratio_best <= 0.5),
            "fell_back": {f"learned_{b}": runs[f"learned_{b}"]["fell_back"] for b in ev["budgets"]},
            "plain_short_schedule_reaches_target": [r["steps"] for r in plain_hit],
            "runs": runs, "training": {"scenes": tr["scenes"], "samples": int(F_.shape[0]),
                                       "collect_seconds": t1 - t0, "fit_seconds": t2 - t1,
                                       "fit_loss_first": float(np.mean(fit[:10])),
                                       "fit_loss_last": float(np.mean(fit[-10:]))},
            "loss": "masked Charbonnier photometric loss over all views, each view normalised as one refiner batch"}


# ---- GPU arm ------------------------------------------------------------------------------------------

STAGES = ["visibility+shade", "render_backward"]
# Source files each timed stage is compiled from (its launches' files and what they include; render_backward's order of
# tiles is launched from visibility.cu), and its DRAM bytes (dram__bytes_read.sum +
# dram__bytes_write.sum over its kernels) on this 64-view workload from an ncu capture of the
# full-size run, recorded with the SHA-256 of those sources at capture time. A capture cannot run
# inside the timed region; when the sources no longer hash to the recorded value the figure belongs to
# other code and the line reports traffic as null.
KERNEL_SOURCES = {
    "visibility+shade": ["visibility.cu", "visibility.cuh", "raster_tile.cuh", "bin_rect.cuh", "ndc_axis.cuh",
                         "tile_order.cuh", "pdr_common.cuh", "pdr_internal.h"],
    "render_backward": ["fused.cu", "visibility.cu", "render_bwd_tile.cuh", "ndc_axis.cuh", "tile_order.cuh",
                        "pdr_common.cuh", "pdr_internal.h"],
}
# stage -> (sha256 of its sources, bytes)
KERNEL_TRAFFIC = {
    "visibility+shade": ("e8b231d59d198ff3", 7327000000),
    "render_backward": ("72fb25e21c5dec5b", 4748200000),
}


def kernel_source_hash(stage: str) -> str:
    import hashlib

    h = hashlib.sha256()
    for f in KERNEL_SOURCES[stage]:
        with open(os.path.join(ROOT, "photara_drender_gb300", "csrc", f), "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()


def recorded_traffic(stage: str):
    """The recorded DRAM bytes of `stage`, when its sources are those the capture ran; else None."""
    rec = KERNEL_TRAFFIC.get(stage)
    return rec[1] if rec and kernel_source_hash(stage).startswith(rec[0]) else None


def stage_bytes(w, T, V):
    """Algorithmic bytes of each timed stage: API-boundary tensors, each read or written once."""
    P = w["views"] * w["height"] * w["width"]
    A, Cc = w["attributes"], w["channels"]
    tex = w["atlas"] * w["atlas"] * Cc * 4
    mesh = w["views"] * V * 16 + T * 12
    return {
        # inputs: clip, indices, attributes, uv attributes, texture; outputs raster, derivatives,
        # attributes, uv, sampled
        "visibility+shade": mesh + V * (A + 2) * 4 + tex + P * (16 + 16 + A * 4 + 8 + Cc * 4),
        # inputs: raster, uv, grad_interpolated, grad_sampled, texture, clip, attributes;
        # outputs: grad_texture, grad_clip, grad_attributes, grad_uv_attributes
        "render_backward": P * (16 + 8 + A * 4 + Cc * 4) + 2 * tex + 2 * mesh + 2 * V * (A + 2) * 4,
    }


def e2e_render(dev, r, host, H, W, steps, world=1):
    """The fused pass through the public autograd API (photara_drender_gb300.torch.render + backward) with
    host buffers: every step copies its inputs (`host`: pinned clip, attrs, uv, tex, g_attr, g_samp, idx)
    to the device and reads the clip, attribute, uv and texture gradients back, all inside the timed
    region. The copies of step k+1 run on a copy stream while step k computes (two device buffer sets),
    so the step costs the larger of the two instead of their sum. Returns (median ms per step over five
    timed runs or None, host to device bytes per step, device to host bytes per step)."""
    import torch

    from photara_drender_gb300 import torch as pdr_torch

    h2d = sum(t.numel() * t.element_size() for t in host.values())
    grads_host = {k: torch.empty(host[k].shape, dtype=torch.float32).pin_memory() for k in ("clip", "attrs", "uv", "tex")}
    d2h = sum(t.numel() * t.element_size() for t in grads_host.values())
    if not steps:
        return None, h2d, d2h
    bufs = [{k: torch.empty_like(v, device=dev) for k, v in host.items()} for _ in range(2)]
    copy_stream = torch.cuda.Stream(dev)
    compute = torch.cuda.current_stream(dev)
    copied = [torch.cuda.Event() for _ in range(2)]
    released = [torch.cuda.Event() for _ in range(2)]
    computed = [torch.cuda.Event() for _ in range(2)]
    in_flight = [None, None]  # the gradients a slot's readback still reads

    def upload(slot):
        with torch.cuda.stream(copy_stream):
            copy_stream.wait_event(released[slot])
            for k, v in host.items():
                bufs[slot][k].copy_(v, non_blocking=True)
            copied[slot].record(copy_stream)

    def step(i, total):
        slot = i % 2
        compute.wait_event(copied[slot])
        if i + 1 < total:
            upload((i + 1) % 2)
        d = bufs[slot]
        leaves = {k: d[k].detach().requires_grad_(True) for k in ("clip", "attrs", "uv", "tex")}
        out = pdr_torch.render(leaves["clip"], d["idx"], (H, W), rasterizer=r, vertex_attributes=leaves["attrs"],
                               vertex_uv=leaves["uv"], texture=leaves["tex"], deferred_errors=True)
        torch.autograd.backward([out.interpolated, out.sampled], [d["g_attr"], d["g_samp"]])
        released[slot].record(compute)
        # gradients go back on the copy stream, after the next step's upload and overlapping its compute:
        # the host link runs one direction at a time (pinned copies measured at 211 GB/s up and 194 GB/s
        # down alone, 170 GB/s each way when both run), so the step costs upload + readback, not more
        computed[slot].record(compute)
        grads = {k: t.grad for k, t in leaves.items()}
        with torch.cuda.stream(copy_stream):
            copy_stream.wait_event(computed[slot])
            for k, t in grads.items():
                grads_host[k].copy_(t, non_blocking=True)
                t.record_stream(copy_stream)
        in_flight[slot] = grads

    def run(total):
        for e in released:
            e.record(compute)
        upload(0)
        for i in range(total):
            step(i, total)
        compute.wait_stream(copy_stream)

    # the host link on its own: pinned copies of the step's largest input up and of its gradient down
    big = max(host.values(), key=lambda t: t.numel() * t.element_size())
    dbuf = torch.empty_like(big, device=dev)
    link = {}
    for name, (dst, src) in (("h2d_gbs", (dbuf, big)), ("d2h_gbs", (big, dbuf))):
        dst.copy_(src, non_blocking=True)
        torch.cuda.synchronize(dev)
        t0 = time.perf_counter()
        for _ in range(3):
            dst.copy_(src, non_blocking=True)
        torch.cuda.synchronize(dev)
        link[name] = 3 * big.numel() * big.element_size() / (time.perf_counter() - t0) / 1e9
    e2e_render.last_link = link
    del dbuf
    run(2)  # warm-up: allocations and the tile-list capacity (reported back without a wait)
    torch.cuda.synchronize(dev)
    pdr_torch.check_deferred_errors(r)
    # five timed runs, the median reported: the host link is the bound, and its rate varies from run to run
    # on a machine whose host memory other jobs share (13.1 to 19.2 ms per step seen in one process)
    reps = []
    for _ in range(5):
        barrier(world)
        t0 = time.perf_counter()
        run(steps)  # no host wait inside: render(deferred_errors=True) queues its status checks
        torch.cuda.synchronize(dev)
        reps.append((time.perf_counter() - t0) * 1e3 / steps)
    pdr_torch.check_deferred_errors(r)
    e2e_render.last_reps = reps
    return max_over_ranks(float(np.median(reps)), world), h2d, d2h


def run_gpu(args, world, rank, local):
    import torch

    from photara_drender_gb300 import Rasterizer, _native
    from photara_drender_gb300.pipeline import RenderFwdBwd
    from photara_drender_gb300.rasterizer import _ptr

    w = WORKLOAD
    dev = torch.device("cuda", local)
    torch.cuda.set_device(dev)
    pos3, uv, idx, mats, attrs = scene()
    V, T = pos3.shape[0], idx.shape[0]
    views, H, W = w["views"], w["height"], w["width"]
    P = views * H * W
    r = Rasterizer(local)
    stream = C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    g = torch.Generator(device=dev)
    g.manual_seed(w["seed"] + rank)
    t_pos = torch.tensor(pos3, device=dev)
    t_mats = torch.tensor(mats, device=dev)
    clip = torch.empty((views, V, 4), dtype=torch.float32, device=dev)
    _native.call("pdr_transform_positions", _ptr(t_pos), V, _ptr(t_mats), views, _ptr(clip), stream)
    t_attrs = torch.tensor(attrs, device=dev)
    t_uv = torch.tensor(uv, device=dev)
    t_idx = torch.tensor(idx.astype(np.int32), device=dev)
    tex = torch.rand((w["atlas"], w["atlas"], w["channels"]), device=dev, generator=g)
    g_attr = torch.randn((views, H, W, w["attributes"]), device=dev, generator=g)
    g_samp = torch.randn((views, H, W, w["channels"]), device=dev, generator=g)

    if args.tile:  # the forward through tile lists of this shape and stage depth
        tw_th, k = args.tile.split("/")
        cfg = tuple(int(x) for x in tw_th.split("x")) + (int(k),)
        pipe = RenderFwdBwd(r, t_idx, V, views, H, W, w["attributes"], tuple(tex.shape), capacity=4 * T * views,
                            tile_config=cfg)
    else:  # through the visibility buffer, as the public render
        pipe = RenderFwdBwd(r, t_idx, V, views, H, W, w["attributes"], tuple(tex.shape), direct=True)
    pipe.step(clip, t_attrs, t_uv, tex, g_attr, g_samp, stream)
    if args.tile:
        pipe.set_tile_config(cfg, int(pipe.check_capacity() * 1.25) + 1024)
        pipe.step(clip, t_attrs, t_uv, tex, g_attr, g_samp, stream)
    pipe.check_capacity()
    for _ in range(args.warmup):
        pipe.step(clip, t_attrs, t_uv, tex, g_attr, g_samp, stream)
    torch.cuda.synchronize(dev)
    pipe.check_capacity()

    # ---- timed region: device-resident inputs ------------------------------------------------------
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier(world)
    torch.cuda.synchronize(dev)
    with ClockSampler(local) as clocks:
        start.record()
        for _ in range(args.steps):
            pipe.step(clip, t_attrs, t_uv, tex, g_attr, g_samp, stream)
        end.record()
        torch.cuda.synchronize(dev)
    barrier(world)
    ms = start.elapsed_time(end) / args.steps
    pipe.check_capacity()
    ms = max_over_ranks(ms, world)
    value = world * P / 1e6 / (ms / 1e3)

    # ---- per-stage attribution: replay each stage between events --------------------------------
    L = _native.lib()
    reps = 3
    stage_ms = np.zeros(len(STAGES))
    a = pipe._args(clip, t_attrs, t_uv, tex, g_attr, g_samp)
    timed = [
        lambda: _native.check((L.pdr_render_direct if pipe.direct else L.pdr_render_forward)(C.addressof(a), stream)),
        lambda: _native.check(L.pdr_render_backward(C.addressof(a), stream)),
    ]
    for _ in range(reps):
        for i, fn in enumerate(timed):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize(dev)
            e0.record()
            fn()
            e1.record()
            torch.cuda.synchronize(dev)
            stage_ms[i] += e0.elapsed_time(e1)
    stage_ms /= reps
    hbm, peak_kind = load_peaks()
    sbytes = stage_bytes(w, T, V)
    dom = int(np.argmax(stage_ms))
    dom_name = STAGES[dom]
    achieved = sbytes[dom_name] / (stage_ms[dom] / 1e3) / 1e9
    step_bytes = P * 96 + 2 * w["atlas"] ** 2 * w["channels"] * 4

    # ---- e2e: public autograd API with host buffers ---------------------------------------------------
    e2e_steps = 0 if args.skip_e2e else max(2, args.steps)
    host = {k: v.cpu().pin_memory() for k, v in dict(clip=clip, attrs=t_attrs, uv=t_uv, tex=tex, g_attr=g_attr,
                                                     g_samp=g_samp).items()}
    host["idx"] = torch.tensor(idx.astype(np.int64)).pin_memory()
    e2e_ms, h2d, d2h = e2e_render(dev, r, host, H, W, e2e_steps, world)
    e2e_value = world * P / 1e6 / (e2e_ms / 1e3) if e2e_ms else None

    # ---- CPU baseline (oracle restatement, bounded sample) --------------------------------------------
    cpu = None
    if rank == 0 and world == 1 and not args.skip_cpu:
        try:
            tex_h = tex.cpu().numpy()
            cores = os.cpu_count() or 1
            clips_h = clip.cpu().numpy()
            done, secs = cpu_sample_views(clips_h, uv, idx, attrs, tex_h, 0, CPU_SAMPLE_SECONDS)
            done1, secs1 = cpu_sample_views(clips_h, uv, idx, attrs, tex_h, 1, CPU_SAMPLE_SECONDS)
            cpu = {"value": done * H * W / 1e6 / secs, "unit": "Mpix/s", "cores": cores, "kind": "port",
                   "sample": f"views 0..{done - 1} of {views} (until {CPU_SAMPLE_SECONDS:.0f} s of work): full "
                             f"forward+backward at {H}x{W} through the oracle, every stage on all {cores} host "
                             f"threads, {secs:.1f} s",
                   "one_core": {"value": done1 * H * W / 1e6 / secs1, "unit": "Mpix/s", "cores": 1,
                                "sample": f"views 0..{done1 - 1}, the same path on one thread, {secs1:.1f} s"}}
        except Exception as e:  # the CPU leg never hides a GPU result
            cpu = {"value": None, "unit": "Mpix/s", "cores": os.cpu_count() or 1, "kind": "port",
                   "sample": f"failed: {e}"}
    # ---- parity at full size ---------------------------------------------------------------------------
    # (1) size-independent sums of the last backward: bilinear weights and barycentric weights each sum to
    # one, so the texture gradient summed over texels equals the sample gradient summed over covered
    # pixels, and the attribute gradient summed over vertices equals the attribute gradient summed over
    # covered pixels (errors relative to the sum of |terms|, float64 on the device);
    # (2) view 0's raster against the oracle at full size, with the tie counts.
    parity = None
    if rank == 0:
        cov = (pipe.raster[..., 3] != 0).unsqueeze(-1).double()
        ref_t, abs_t = (g_samp.double() * cov).sum((0, 1, 2)), (g_samp.double().abs() * cov).sum((0, 1, 2))
        ids = pipe.raster[..., 3]
        covv = ((ids >= 0.5) & (ids < T + 0.5)).unsqueeze(-1).double()
        ref_a, abs_a = (g_attr.double() * covv).sum((0, 1, 2)), (g_attr.double().abs() * covv).sum((0, 1, 2))
        parity = {"grad_texture_sum_err": float(((pipe.grad_tex.double().sum((0, 1)) - ref_t).abs() / abs_t).max()),
                  "grad_attribute_sum_err": float(((pipe.grad_attr.double().sum(0) - ref_a).abs() / abs_a).max())}
        del cov, covv
    if rank == 0 and world == 1 and not args.skip_cpu:
        try:
            from oracle import api

            clip0 = clip[0].cpu().numpy()
            o_r, _, counts = api.rasterize_tie_counts(clip0, idx, (H, W))
            g_r = pipe.raster[0].cpu().numpy()
            parity.update({"view": 0, "raster_bit_exact": bool(np.array_equal(o_r.view(np.uint32),
                                                                                 g_r.view(np.uint32))),
                           **counts, "note": "depth_ties: pixels the lowest-id rule decided; edge_ties: pixels whose "
                                             "winner passed an edge test inside the 1e-7 tolerance; *_sum_err: "
                                             "|sum of the GPU gradient - sum of the upstream gradient over covered "
                                             "pixels| / sum of |terms|, per channel, worst channel"})
        except Exception as e:
            parity.update({"view": 0, "failed": str(e)})

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": "Mpix/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded displaced sphere, orbit cameras)",
            "config": {"workload": w["name"], "views": views, "resolution": [H, W], "triangles": int(T),
                       "vertices": int(V), "atlas": [w["atlas"], w["atlas"], w["channels"]],
                       "attributes": w["attributes"],
                       "forward": "visibility buffer" if pipe.direct else f"tile lists {args.tile}",
                       "l2": "inputs larger than L2 (6.5 GB of per-view buffers per step)",
                       "parallelism": f"replicas x{world}"},
            "gpu_launches": pipe.kernels_per_step() * args.steps,
            "roofline": {"bound": "hbm", "kernel": dom_name, "achieved": achieved, "peak": hbm,
                         "peak_kind": peak_kind, "unit": "GB/s", "frac": achieved / hbm,
                         "traffic": recorded_traffic(dom_name)
                         if pipe.direct and views == 64 and w["atlas"] == 4096 else None,
                         "traffic_source_sha256": kernel_source_hash(dom_name),
                         "algorithmic_bytes": sbytes[dom_name], "ms": float(stage_ms[dom])},
            "stages_ms": {n: float(t) for n, t in zip(STAGES, stage_ms)},
            "pipeline": "fused" if pipe.fused else "separate kernels",
            "step_roofline": {"algorithmic_bytes": step_bytes, "achieved_gbs": step_bytes / (ms / 1e3) / 1e9,
                              "frac": step_bytes / (ms / 1e3) / 1e9 / hbm},
            "e2e": {"value": e2e_value, "unit": "Mpix/s", "h2d_bytes_per_step": int(h2d),
                    "d2h_bytes_per_step": int(d2h), "ms_per_step": e2e_ms,
                    "runs_ms_per_step": getattr(e2e_render, "last_reps", None),
                    "link": getattr(e2e_render, "last_link", None),
                    "link_floor_ms": (h2d / getattr(e2e_render, "last_link", {}).get("h2d_gbs", float("inf")) +
                                      d2h / getattr(e2e_render, "last_link", {}).get("d2h_gbs", float("inf"))) / 1e6
                    if getattr(e2e_render, "last_link", None) else None,
                    "api": "photara_drender_gb300.torch.render (fused autograd op, deferred_errors=True: no host "
                           "wait per call) + backward; inputs copied from pinned host memory every step "
                           "(double-buffered on a copy stream), gradients read back on the same copy stream after "
                           "the next step's upload (one link direction at a time)"},
            "cpu_baseline": cpu,
            "parity": parity,
            "clocks": clocks.summary(),
        }
        if world == 1:
            global SKIP_CPU
            SKIP_CPU = args.skip_cpu
            for key, skip, leg in (("c1", args.skip_c1, c1_leg), ("bake", args.skip_bake, bake_leg),
                                   ("refine", args.skip_refine, refine_leg), ("c4", args.skip_c4, c4_leg),
                                   ("precond", args.skip_precond, c5_leg)):
                if skip:
                    continue
                try:
                    line[key] = leg(dev, hbm)
                except Exception as e:  # a secondary leg never hides the headline number
                    line[key] = {"error": f"{type(e).__name__}: {e}"}
        print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["gb300", "reference"], default="gb300")
    ap.add_argument("--skip-cpu", action="store_true", help="omit the CPU-baseline leg")
    ap.add_argument("--skip-e2e", action="store_true", help="omit the end-to-end leg (profiling runs)")
    ap.add_argument("--views", type=int, default=None, help="override the view count (small profiling cases)")
    ap.add_argument("--atlas", type=int, default=None, help="override the atlas size (texture-gradient profiling)")
    ap.add_argument("--bake-views", type=int, default=None, help="override the bake leg's view count (profiling)")
    ap.add_argument("--skip-c1", action="store_true", help="omit the small-mesh (C1) leg")
    ap.add_argument("--skip-bake", action="store_true", help="omit the bake leg")
    ap.add_argument("--skip-refine", action="store_true", help="omit the refine leg")
    ap.add_argument("--skip-c4", action="store_true", help="omit the uneven multi-mesh batch leg")
    ap.add_argument("--skip-precond", action="store_true", help="omit the learned-preconditioner leg")
    ap.add_argument("--c4-meshes", type=int, default=None, help="override the C4 mesh count (small profiling cases)")
    ap.add_argument("--tile", default=None, help="forward through tile lists of this shape and stage depth, e.g. 16x8/128 (default: visibility "
                         "buffer)")
    ap.add_argument("--refine-steps", type=int, default=None, help="override the refine leg's step count (profiling)")
    args = ap.parse_args()
    if args.views:
        WORKLOAD["views"] = args.views
        WORKLOAD["name"] = WORKLOAD["name"].replace("64x", f"{args.views}x")
    if args.bake_views:
        BAKE["name"] = BAKE["name"].replace(f"{BAKE['views']}x", f"{args.bake_views}x")
        BAKE["views"] = args.bake_views
    if args.atlas:
        WORKLOAD["name"] = WORKLOAD["name"].replace(f"atlas{WORKLOAD['atlas']}", f"atlas{args.atlas}")
        WORKLOAD["atlas"] = args.atlas
    if args.c4_meshes:
        C4["meshes"] = args.c4_meshes
        C4["name"] = C4["name"].replace("16_meshes", f"{args.c4_meshes}_meshes")
    if args.refine_steps:
        REFINE["name"] = REFINE["name"].replace(f"{REFINE['steps']}steps", f"{args.refine_steps}steps")
        REFINE["steps"] = args.refine_steps
    if args.impl == "reference":
        world = int(os.environ.get("WORLD_SIZE", "1"))
        rank = int(os.environ.get("RANK", "0"))
        run_reference(args, world, rank)
        return
    import __graft_entry__ as g

    g.build()
    world, rank, local = dist_setup(args)
    run_gpu(args, world, rank, local)
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()


if __name__ == "__main__":
    main()
