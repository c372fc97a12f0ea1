"""Benchmark of the GB300 BIRP render path.

Headline workload (config 2 on config 1's cube): 512 renders of a 256^3
stretched-axis FP32 cube (x in [-40, 30], y, z in [-40, 40] Re, trilinear,
PREFIX march), poses on the SMILE-like orbit aimed at (9, 0, 0) with a roll
uniform in [-10, 10] deg, image sizes from {144x84, 288x168, 576x336,
1024x600} and steps from {0.025, 0.05, 0.1} Re, seeded. One step = one pass
over all 512 requests.

  value      images/s of the batched path (one persistent-kernel launch from a
             CUDA graph), device time, inputs resident, L2 flushed between steps
  e2e        the same through the C ABI birp_batch_render with HOST output
             buffers (descriptor H2D + image D2H + copies to the caller inside)
  plain      images/s of the one-render-per-call path (birp_render, host output)
  serving    p50/p99 latency of the continuous-batching server at 70% of the
             saturated rate (Poisson arrivals)
  parity     max and RMS relative error of EVERY timed image against the FP64
             oracle on a random pixel sample of each image, plus one whole
             image per size class
  roofline   the batched kernel against the slower of its FP32 work and its
             gathered bytes at the L2 read rate, both peaks measured in-run;
             roofline_issue: its warp instructions (per cell segment, from the
             committed ncu capture) against the SM issue rate at the sampled
             clock, the bound it actually runs into
  cpu_baseline  the reference's FP32 render arithmetic (oracle port) on all
             host cores over a bounded random pixel sample of the same
             workload, and on one core
  c3         config 3: 48 uneven stretched cubes x 16 cameras + 8 CMEM
             requests in one launch vs plain renders, with per-image parity
  c4         config 4: the serving sweep over 256 cubes of 512x384x384 (77 GB
             of host data) under a 60 GB device budget, Poisson arrivals at
             rising rates until the served rate falls behind the offered one,
             then p50/p99 at 70% of that saturated rate, with parity of
             served images

The result is one JSON line on stdout of at most 2400 characters, with the
single numbers of each block; `--details FILE` writes all of it (per-image
errors, every rate and size).

`--impl reference` times only the CPU implementation (bounded samples).
`--workload c3|c4` runs one of the extra blocks alone (`--c4-layout`,
`--c4-promote-layout`, `--c4-promote-gb`, `--c4-uploaders` vary the config-4
server); `--profile-case trilinear|nearest|compact|pairs|cmem|signed` runs a
small fixed batch to profile one kernel class. Multi-GPU (torchrun): replicas, one per rank, barrier + max
over ranks (the c3/c4 blocks run at N = 1 only).
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "images/s & p99 latency: batched/served vs plain GPU render at ≤1e-5 rel err"
UNIT = "images/s"
# Per trilinear ray-sample (the reference's formulation): 8 FP32 corners
# gathered, 6 position + 6 index + 3 fraction + 21 lerp + 4 Kahan flops.
FLOP_PER_SAMPLE = 40.0
BYTES_PER_SAMPLE = 32.0
# Per cell segment (what the kernel does: the samples inside one cell summed
# in closed form): one 32-byte coefficient record + one 8-byte walk-table
# entry for the face crossed into the cell; 45 FP32 operations for the run
# end, the closed-form sum about the run's middle and the Kahan update
# (FMA = 2) plus 3 for the new base offset and exit index of the crossed axis.
FLOP_PER_CELL = 48.0
BYTES_PER_CELL = 40.0


def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("gloo")
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


def allreduce_max(world, x: float) -> float:
    if world <= 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled every 200 ms."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except (OSError, ValueError):
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            p = [x.strip() for x in ln.split(",")]
            if len(p) < 9:
                continue
            try:
                sm.append(float(p[1]))
                smax = float(p[2])
            except ValueError:
                continue
            for n, v in zip(names, p[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"], "samples": 0}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": smax, "reasons": sorted(reasons), "samples": len(sm)}


# ---------------------------------------------------------------- oracle checks

def oracle():
    """The CPU oracle (test infrastructure): here only the checker of the
    timed images and the CPU baseline."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle as O
    O.build()
    return O


def o_camera(O, cam):
    """The FP64 oracle's camera for a C-ABI camera (roll included)."""
    return O.camera64(tuple(cam.pos), tuple(cam.aim), cam.fov_w_deg, cam.fov_h_deg, cam.nx, cam.ny, cam.n_samples,
                      cam.ray_length, cam.march, cam.roll_deg)


def image_error(O, space, cam, img, n_px: int, seed: int):
    """Max and RMS relative error of one image against the FP64 oracle on
    n_px random pixels (all pixels if the image has fewer), over the pixels
    above 1e-3 of the image maximum (the rendered image's, which is within
    the tolerance of the oracle's); also the worst pixel (i, j, rendered,
    oracle)."""
    rng = np.random.default_rng(seed)
    npx = cam.nx * cam.ny
    full = np.asarray(img).reshape(cam.ny, cam.nx)
    flat = np.arange(npx) if npx <= n_px else rng.choice(npx, n_px, replace=False)
    pi, pj = flat % cam.nx, flat // cam.nx
    ref = O.render64_pixels(space, o_camera(O, cam), pi, pj, threads=1)
    got = full[pj, pi].astype(np.float64)
    peak = float(np.abs(full).max()) if npx else 0.0
    m = np.abs(ref) > 1e-3 * peak if peak > 0 else np.zeros(len(ref), bool)
    if not m.any():
        # nothing bright enough: the sampled pixels must still agree closely
        bad = np.abs(got - ref).max() if len(ref) else 0.0
        return (0.0 if bad <= 1e-5 * max(peak, 1e-30) else float("inf")), 0.0, 0, None
    e = np.abs(got[m] - ref[m]) / np.abs(ref[m])
    w = int(np.argmax(e))
    worst = [int(pi[m][w]), int(pj[m][w]), float(got[m][w]), float(ref[m][w])]
    return float(e.max()), float(np.sqrt(np.mean(e * e))), int(m.sum()), worst


def parity_report(O, jobs, n_px: int, tol: float = 1e-5, label=None):
    """jobs: (oracle space, camera, image) per image; every image is checked
    on its own pixel sample, on all host cores (one oracle call per image)."""
    import concurrent.futures as cf
    t0 = time.perf_counter()
    with cf.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        res = list(ex.map(lambda a: image_error(O, a[1][0], a[1][1], a[1][2], n_px, 1000 + a[0]), enumerate(jobs)))
    mx = np.array([r[0] for r in res])
    rms = np.array([r[1] for r in res])
    cnt = np.array([r[2] for r in res])
    w = int(np.argmax(mx))
    wc = jobs[w][1]
    worst_px = res[w][3]
    out = {"images": len(jobs), "pixels_per_image": n_px, "pixels_checked": int(cnt.sum()),
           "max_rel_err": float(mx.max()), "rms_rel_err": float(np.sqrt(np.sum(rms * rms * cnt) / max(cnt.sum(), 1))),
           "per_image_max_quantiles": {q: float(np.quantile(mx, p)) for q, p in
                                       (("p50", .5), ("p90", .9), ("p99", .99), ("max", 1.0))},
           "worst_image": {"index": w, "size": f"{wc.nx}x{wc.ny}", "n_samples": int(wc.n_samples),
                           "max_rel_err": float(mx[w]), "rms_rel_err": float(rms[w]),
                           "worst_pixel_i_j_got_ref": worst_px},
           "images_within_tolerance": int(np.sum(mx <= tol)), "tolerance": tol,
           "per_image": [[float(f"{a:.3g}"), float(f"{b:.3g}")] for a, b in zip(mx, rms)],
           "check_s": time.perf_counter() - t0}
    if label:
        out["what"] = label
    return out


def full_image_checks(O, space, items, imgs):
    """One whole image per size class against the FP64 oracle."""
    seen, out = set(), []
    threads = os.cpu_count() or 4
    for (cam, img) in zip(items, imgs):
        key = (cam.nx, cam.ny)
        if key in seen:
            continue
        seen.add(key)
        t0 = time.perf_counter()
        ref = O.render64(space, o_camera(O, cam), threads=threads)
        got = np.asarray(img, np.float64).reshape(cam.ny, cam.nx)
        m = ref > 1e-3 * max(ref.max(), 1e-300)
        e = np.abs(got[m] - ref[m]) / ref[m] if m.any() else np.zeros(1)
        out.append({"size": f"{cam.nx}x{cam.ny}", "n_samples": int(cam.n_samples), "pixels": int(m.sum()),
                    "max_rel_err": float(e.max()), "rms_rel_err": float(np.sqrt(np.mean(e * e))),
                    "oracle_s": time.perf_counter() - t0})
    return out


# ---------------------------------------------------------------- workloads

def make_workload(B, n_req: int, seed_cube: int = 1, seed_req: int = 2):
    from birp_cpp_gb300 import synth
    xs, ys, zs, v64 = synth.cube_config1(seed=seed_cube)
    v32 = v64.astype(np.float32)
    cube = B.Cube(xs, ys, zs, v32)
    reqs = synth.config2_requests(n_req, seed=seed_req)
    rolls = synth.config2_rolls(n_req, seed=seed_req)
    cams = [B.camera(pos, aim, synth.FOV_W, synth.FOV_H, nx, ny, n_samples=synth.n_samples(step),
                     ray_length=synth.RAY_LENGTH, trilinear=True, roll=float(r))
            for (pos, aim, nx, ny, step), r in zip(reqs, rolls)]
    return dict(cube=cube, cams=cams, reqs=reqs, host=(xs, ys, zs, v32))


def _gen_cube(spec):
    from birp_cpp_gb300 import synth
    nx, ny, nz, r0, seed = spec
    xs, ys, zs, v = synth.cube_stretched(nx, ny, nz, r0, seed)
    return xs, ys, zs, v.astype(np.float32)


def gen_c3_host():
    """Config 3's 48 cubes, generated in a spawned process pool (safe before
    or after the first GPU call)."""
    import concurrent.futures as cf
    import multiprocessing as mp
    from birp_cpp_gb300 import synth
    cube_specs, specs = synth.config3_specs()
    with cf.ProcessPoolExecutor(max_workers=os.cpu_count() or 4, mp_context=mp.get_context("spawn")) as ex:
        host = list(ex.map(_gen_cube, cube_specs))
    return host, specs


def run_c3(args, B, O, host, specs):
    """Config 3: 48 uneven stretched cubes (16 cameras each) + 8 CMEM requests
    in one launch, against one plain call per request; every image checked
    against the FP64 oracle on a pixel sample."""
    from birp_cpp_gb300 import synth
    cubes = [B.Cube(*hc) for hc in host]
    cmem = B.Cmem()
    items = []
    for src, pos, aim, nx, ny, step in specs:
        cam = B.camera(pos, aim, synth.FOV_W, synth.FOV_H, nx, ny, n_samples=synth.n_samples(step),
                       ray_length=synth.RAY_LENGTH, trilinear=True)
        items.append((cubes[src] if src >= 0 else cmem, cam))
    total_px = sum(c.nx * c.ny for _, c in items)
    batch = B.Batch(len(items), total_px)
    for _ in range(max(args.warmup, 3)):
        batch.render(items)
    km = []
    for _ in range(args.steps):
        B.flush_l2()
        batch.submit(items)
        batch.wait()
        km.append(batch.last_ms()[0])
    ms = float(np.mean(km))
    imgs = batch.render(items)
    # plain: one birp_render per request, host outputs
    outs = [np.empty((c.ny, c.nx), np.float32) for _, c in items]
    for (sp, c), o in zip(items[:8], outs[:8]):
        B.render(sp, c, out=o)
    pt = []
    for _ in range(2):
        B.flush_l2()
        t0 = time.perf_counter()
        for (sp, c), o in zip(items, outs):
            B.render(sp, c, out=o)
        pt.append(time.perf_counter() - t0)
    plain_s = min(pt)
    dev_bytes = sum(c.info().device_bytes for c in cubes)
    batch.close()
    # parity: cube by cube (one FP64 oracle copy at a time), then CMEM
    jobs_err = [None] * len(items)
    reports = []
    t0 = time.perf_counter()
    for ci, (xs, ys, zs, v32) in enumerate(host):
        idx = [k for k, (src, *_r) in enumerate(specs) if src == ci]
        if not idx:
            continue
        oc = O.Cube64(xs, ys, zs, v32.astype(np.float64), 1)
        rep = parity_report(O, [(oc, items[k][1], imgs[k]) for k in idx], args.parity_px)
        rep["worst_image"]["source"] = f"cube {ci}"
        reports.append(rep)
        for k, (a, b) in zip(idx, rep["per_image"]):
            jobs_err[k] = (a, b)
        del oc
    idx = [k for k, (src, *_r) in enumerate(specs) if src < 0]
    rep_cmem = parity_report(O, [(O.Cmem64(), items[k][1], imgs[k]) for k in idx], args.parity_px)
    rep_cmem["worst_image"]["source"] = "cmem"
    reports.append(rep_cmem)
    for k, (a, b) in zip(idx, rep_cmem["per_image"]):
        jobs_err[k] = (a, b)
    mx = np.array([e[0] for e in jobs_err])
    w = int(np.argmax(mx))
    parity = {"images": len(items), "pixels_per_image": args.parity_px, "max_rel_err": float(mx.max()),
              "per_image_max_quantiles": {q: float(np.quantile(mx, p)) for q, p in
                                          (("p50", .5), ("p90", .9), ("p99", .99), ("max", 1.0))},
              "worst_image": dict(max(reports, key=lambda r: r["max_rel_err"])["worst_image"], request=w),
              "cmem_max_rel_err": rep_cmem["max_rel_err"],
              "images_within_tolerance": int(np.sum(mx <= 1e-5)), "tolerance": 1e-5,
              "per_image": [list(e) for e in jobs_err], "check_s": time.perf_counter() - t0}
    for c in cubes:
        c.close()
    cmem.close()
    n = len(items)
    return {"workload": "config 3: 48 uneven stretched cubes (dims multiples of 16 in [96, 320], r0 in U[7, 12]) "
                        "x 16 orbit cameras + 8 CMEM requests, one launch",
            "requests": n, "images_s": n / (ms / 1000), "ms_per_launch": ms, "plain_images_s": n / plain_s,
            "batched_vs_plain": (n / (ms / 1000)) / (n / plain_s), "cube_device_bytes": dev_bytes,
            "total_pixels": total_px, "parity": parity}


def run_c4(args, B, O):
    """Config 4, the serving sweep: Poisson arrivals at each offered rate for a
    fixed time; each request picks a cube by Zipf(1.1) popularity over a pool
    of cubes held in host (pinned) memory, rendered through the server under a
    GPU byte budget with LRU eviction; poses, sizes and steps from the orbit
    sampler. The sweep rises until the served rate falls behind the offered
    one (saturation); then one run at 70% of the saturated rate gives the
    p50/p99 the target is stated at. Served images of a few cubes (popular
    and rarely used, so some were evicted and re-uploaded) are checked
    against the FP64 oracle."""
    import concurrent.futures as cf
    from birp_cpp_gb300 import synth
    nx, ny, nz = (int(v) for v in args.c4_dims.split("x"))
    n_cubes = args.c4_cubes
    t_setup = time.perf_counter()
    xs, ys, zs, bases = synth.serving_bases(nx, ny, nz)
    codes = {"compact": B.CUBE_COMPACT, "pairs": B.CUBE_PAIRS, "records": B.CUBE_RECORDS}
    layout, promoted = codes[args.c4_layout], codes[args.c4_promote_layout]
    share = int(args.c4_promote_gb * (1 << 30)) if promoted != layout and layout != B.CUBE_RECORDS else 0
    srv = B.Server(B.server_config(cube_budget_bytes=int(args.c4_budget_gb * (1 << 30)), slots=3,
                                   max_batch_requests=64, max_batch_pixels=16 << 20, max_wait_ms=1.0,
                                   max_queue=1 << 17, cube_layout=layout, promoted_layout=promoted,
                                   promoted_budget_bytes=share, uploaders=args.c4_uploaders))

    def add(i):
        return srv.add_cube(xs, ys, zs, synth.serving_cube(i, bases))

    with cf.ThreadPoolExecutor(max_workers=8) as ex:
        ids = list(ex.map(add, range(n_cubes)))
    setup_s = time.perf_counter() - t_setup
    zipf_w = 1.0 / np.arange(1, n_cubes + 1) ** 1.1
    zipf_w /= zipf_w.sum()
    rng = np.random.default_rng(4)
    reqs = synth.config2_requests(8192, seed=44)
    rolls = synth.config2_rolls(8192, seed=44)
    cams = [B.camera(p, a, synth.FOV_W, synth.FOV_H, w, h, n_samples=synth.n_samples(st), roll=float(r))
            for (p, a, w, h, st), r in zip(reqs, rolls)]
    max_px = max(c.nx * c.ny for c in cams)
    # written once here: a client reuses its result buffers, and the first
    # touch of fresh pages is allocation cost, not serving latency
    bufs = [np.full(max_px, 0.0, np.float32) for _ in range(1024)]
    # warm start: the most popular cubes resident (requests in reverse
    # popularity order, so the LRU keeps the popular ones)
    t0 = time.perf_counter()
    small = [c for c in cams if c.nx == 144][:1]
    tk = [srv.submit(ids[r], small[0], bufs[r % len(bufs)]) for r in range(n_cubes - 1, -1, -1)]
    for t in tk:
        srv.wait(t, 600000)
    warm_s = time.perf_counter() - t0
    st_warm = srv.stats()
    # parity probes: the first requests to these popularity ranks in each
    # phase get their own buffers
    probe_ranks = sorted({0, 1, 4, min(30, n_cubes - 1), min(120, n_cubes - 1), n_cubes - 1})
    probes = []

    def phase(rate, seconds, max_probes_per_rank=1):
        picks = rng.choice(n_cubes, size=int(rate * seconds * 1.3) + 64, p=zipf_w)
        gaps = rng.exponential(1.0 / rate, size=len(picks))
        per_rank = {}
        st0 = srv.stats()
        t_start = time.perf_counter()
        nxt, k, tickets = t_start, 0, []
        rejected = 0
        while k < len(picks) and nxt - t_start < seconds:
            now = time.perf_counter()
            if now < nxt:
                if nxt - now > 0.0005:
                    time.sleep(min(nxt - now, 0.002))
                continue
            r = int(picks[k])
            cam = cams[k % len(cams)]
            out = bufs[k % len(bufs)]
            probe = r in probe_ranks and per_rank.get(r, 0) < max_probes_per_rank
            if probe:
                out = np.empty(cam.nx * cam.ny, np.float32)
            try:
                t = srv.submit(ids[r], cam, out)
                tickets.append(t)
                if probe:
                    per_rank[r] = per_rank.get(r, 0) + 1
                    probes.append({"rank": r, "cam": cam, "out": out, "ticket": t, "status": None})
            except B.BirpError:
                rejected += 1
            k += 1
            nxt += gaps[k - 1]
        t_offer = time.perf_counter() - t_start
        done, lat, qms = 0, [], []
        mine = {p["ticket"]: p for p in probes if p["status"] is None}
        for t in tickets:
            res = srv.wait(t, 600000)
            if res.status == 0:
                done += 1
                lat.append(res.latency_ms)
                qms.append(res.queue_ms)
            if t in mine:
                mine[t]["status"] = int(res.status)
        t_all = time.perf_counter() - t_start
        st1 = srv.stats()
        lat = np.array(lat) if lat else np.zeros(1)
        qms = np.array(qms) if qms else np.zeros(1)
        return {"offered_req_s": rate, "submitted": len(tickets), "completed": done,
                "served_images_s": done / t_all, "offer_s": t_offer, "drain_s": t_all - t_offer,
                "p50_ms": float(np.percentile(lat, 50)), "p99_ms": float(np.percentile(lat, 99)),
                "queue_p99_ms": float(np.percentile(qms, 99)),
                "uploads": st1.cube_uploads - st0.cube_uploads, "evictions": st1.cube_evictions - st0.cube_evictions,
                "rejected": rejected + (st1.rejected - st0.rejected)}

    sweep = []
    sat = 0.0
    for rate in (float(r) for r in args.c4_rates.split(",")):
        r = phase(rate, args.c4_seconds)
        sweep.append(r)
        print("c4 rate:", json.dumps(r), file=sys.stderr, flush=True)
        sat = max(sat, r["served_images_s"])
        if r["served_images_s"] < 0.9 * rate:
            break
    saturated = bool(sweep) and sweep[-1]["served_images_s"] < 0.9 * sweep[-1]["offered_req_s"]
    at70 = phase(0.7 * sat, 2 * args.c4_seconds, max_probes_per_rank=2) if sat > 0 else None
    st_end = srv.stats()
    srv.close()
    # parity of the probe images (each probe cube regenerated from its seed)
    t0 = time.perf_counter()
    parity = None
    if O is not None and probes:
        jobs, meta = [], []
        for rank in sorted({p["rank"] for p in probes}):
            v = synth.serving_cube(rank, bases)
            oc = O.Cube64(xs, ys, zs, v.astype(np.float64), 1)
            del v
            sel = [p for p in probes if p["rank"] == rank and p["status"] == 0]
            if sel:
                rep = parity_report(O, [(oc, p["cam"], p["out"]) for p in sel], args.parity_px)
                jobs += rep["per_image"]
                meta += [rank] * len(sel)
            del oc
        mx = np.array([j[0] for j in jobs]) if jobs else np.zeros(1)
        parity = {"images": len(jobs), "cube_ranks": sorted(set(meta)), "pixels_per_image": args.parity_px,
                  "max_rel_err": float(mx.max()), "images_within_tolerance": int(np.sum(mx <= 1e-5)),
                  "tolerance": 1e-5, "failed_requests": int(sum(1 for p in probes if p["status"] != 0)),
                  "per_image": jobs, "check_s": time.perf_counter() - t0}
    # plain per-call latency on one resident cube of the same layout
    cube = B.Cube(xs, ys, zs, synth.serving_cube(0, bases), layout=layout)
    for c in cams[:5]:
        B.render(cube, c, out=bufs[0][: c.nx * c.ny].reshape(c.ny, c.nx))
    pl = []
    for c in cams[:300]:
        t = time.perf_counter()
        B.render(cube, c, out=bufs[0][: c.nx * c.ny].reshape(c.ny, c.nx))
        pl.append(1000 * (time.perf_counter() - t))
    # the GPU's own rate on these requests: 256 of them batched on that one
    # resident cube (device time, L2 flushed), the ceiling a server can reach
    # (and the same in the promoted layout)
    def batched_rate(c3d):
        its = [(c3d, c) for c in cams[:256]]
        cb = B.Batch(len(its), sum(c.nx * c.ny for _, c in its))
        cb.render(its)
        bms = []
        for _ in range(3):
            B.flush_l2()
            cb.submit(its)
            cb.wait()
            bms.append(cb.last_ms()[0])
        cb.close()
        return len(its) / (min(bms) / 1000)

    ceiling = batched_rate(cube)
    cube_bytes = cube.info().device_bytes
    cube.close()
    ceiling_promoted = None
    if share:
        cube = B.Cube(xs, ys, zs, synth.serving_cube(0, bases), layout=promoted)
        ceiling_promoted = batched_rate(cube)
        cube.close()
    return {"workload": f"config 4 serving sweep: {n_cubes} cubes of {nx}x{ny}x{nz} FP32 "
                        f"({n_cubes * nx * ny * nz * 4 / 1e9:.1f} GB of pinned host copies), Zipf(1.1) popularity, "
                        f"{args.c4_budget_gb:g} GiB device budget, {args.c4_layout} layout"
                        + (f" (up to {args.c4_promote_gb:g} GiB of it for the most-requested cubes, promoted to "
                           f"the {args.c4_promote_layout} layout)" if share else "")
                        + f", Poisson arrivals, {args.c4_seconds:g} s per offered rate (70% run: "
                          f"{2 * args.c4_seconds:g} s)",
            "cube_device_bytes": cube_bytes,
            "resident_cubes_in_budget": int(args.c4_budget_gb * (1 << 30) // max(cube_bytes, 1)),
            "setup_s": setup_s, "warm_s": warm_s, "warm_uploads": int(st_warm.cube_uploads),
            "sweep": sweep, "saturated": saturated, "saturation_images_s": sat,
            "gpu_batched_one_cube_images_s": ceiling,
            "gpu_batched_one_cube_promoted_images_s": ceiling_promoted,
            "at_70pct_of_saturation": at70,
            "uploads_total": int(st_end.cube_uploads), "evictions_total": int(st_end.cube_evictions),
            "promoted_share_gb": args.c4_promote_gb if share else 0,
            "promoted_layout": args.c4_promote_layout if share else None, "uploaders": args.c4_uploaders,
            "promotions": int(st_end.cube_promotions), "promoted_bytes_end": int(st_end.promoted_bytes),
            "plain": {"p50_ms": float(np.percentile(pl, 50)), "p99_ms": float(np.percentile(pl, 99)),
                      "images_s": len(pl) / (sum(pl) / 1000)},
            "parity": parity}


def run_profile_case(args):
    """A small fixed batch for profiling one kernel class: the first
    --requests requests of the orbit sampler on the 256^3 stretched cube
    (trilinear or nearest, records, pairs or compact layout; signed: 1e-5 of
    its nodes negative) or on the default CMEM model, launched --launches
    times."""
    import birp_cpp_gb300 as B
    from birp_cpp_gb300 import build, synth
    build.build()
    B.init(0)
    mode = args.profile_case
    reqs = synth.config2_requests(args.requests, seed=2)
    if mode == "cmem":
        space = B.Cmem()
    else:
        xs, ys, zs, v = synth.cube_config1(seed=1)
        if mode == "signed":
            v = np.where(np.random.default_rng(5).random(v.shape) < 1e-5, -0.01 * v - 1e-4, v)
        layout = {"compact": B.CUBE_COMPACT, "pairs": B.CUBE_PAIRS}.get(mode, B.CUBE_RECORDS)
        space = B.Cube(xs, ys, zs, v.astype(np.float32), layout=layout)
    cams = [B.camera(p, a, synth.FOV_W, synth.FOV_H, nx, ny, n_samples=synth.n_samples(s),
                     ray_length=synth.RAY_LENGTH, trilinear=mode != "nearest") for p, a, nx, ny, s in reqs]
    items = [(space, c) for c in cams]
    batch = B.Batch(len(items), sum(c.nx * c.ny for c in cams))
    B.kernel_stats(reset=True)
    for _ in range(args.launches):
        batch.submit(items)
        batch.wait()
    ks = B.kernel_stats(reset=True)
    print(json.dumps({"profile_case": mode, "requests": len(items), "last_launch_ms": batch.last_ms()[0],
                      "cells_per_launch": ks["cells"] / args.launches,
                      "samples_per_launch": ks["samples"] / args.launches,
                      "exact_cmem_per_launch": ks["exact_cmem"] / args.launches,
                      "exact_range_rays_per_launch": ks["exact_range_rays"] / args.launches}))
    batch.close()


def cpu_sample(reqs, host, seconds: float, threads: int, seed: int = 7):
    """The reference's FP32 render arithmetic (oracle port, per-cell lookup on
    the stretched axes) over random pixels drawn uniformly from all pixels of
    all requests, until `seconds` of wall time; returns (images/s, pixels,
    wall s). images/s = n_requests / (time per pixel * total pixels). The
    requests of a round are spread over `threads` host threads, one oracle
    call (one thread inside) per request: the library call releases the GIL,
    and a round holds ~1000 pixels per thread, so every thread has work."""
    import concurrent.futures as cf
    from birp_cpp_gb300 import synth
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle as O
    O.build()
    xs, ys, zs, v32 = host
    cube = O.Cube32(xs.astype(np.float32), ys.astype(np.float32), zs.astype(np.float32), v32, 1, 1)
    cams = [O.camera32(pos, aim, synth.FOV_W, synth.FOV_H, nx, ny, n_samples=synth.n_samples(step), ray_max=44)
            for pos, aim, nx, ny, step in reqs]
    npx = np.array([nx * ny for _, _, nx, ny, _ in reqs], np.int64)
    total_px = int(npx.sum())
    cum = np.cumsum(npx)
    rng = np.random.default_rng(seed)
    done_px, t_used = 0, 0.0
    chunk = 1024 * max(1, threads)

    def job(args):
        r, loc = args
        nx = reqs[r][2]
        O.render32_pixels(cube, cams[r], loc % nx, loc // nx, threads=1)

    t_start = time.perf_counter()
    with cf.ThreadPoolExecutor(max_workers=max(1, threads)) as ex:
        while t_used < seconds or done_px == 0:
            flat = rng.integers(0, total_px, chunk)
            which = np.searchsorted(cum, flat, side="right")
            local = flat - np.concatenate([[0], cum[:-1]])[which]
            jobs = [(int(r), local[which == r]) for r in np.unique(which)]
            t0 = time.perf_counter()
            list(ex.map(job, jobs))
            t_used += time.perf_counter() - t0
            done_px += chunk
            if time.perf_counter() - t_start > 4 * seconds + 30:
                break
    per_px = t_used / done_px
    return len(reqs) / (per_px * total_px), done_px, t_used


def run_reference(args, world, rank):
    """--impl reference: the reference's CPU render arithmetic (oracle port).
    A step is a bounded sample: --ref-seconds of random pixels of the
    workload on all host threads; ms_per_step is that step's measured time,
    images_per_step the images its pixels amount to (pixels / the workload's
    mean pixels per image), and value their ratio, images/s."""
    if rank != 0:
        return
    from birp_cpp_gb300 import synth
    reqs = synth.config2_requests(args.requests, seed=2)
    xs, ys, zs, v64 = synth.cube_config1(seed=1)
    host = (xs, ys, zs, v64.astype(np.float32))
    threads = os.cpu_count() or 1
    for _ in range(args.warmup):
        cpu_sample(reqs, host, 0.5, threads, seed=100)
    vals, pxs, t_tot, walls = [], 0, 0.0, []
    for k in range(args.steps):
        t0 = time.perf_counter()
        v, px, t = cpu_sample(reqs, host, args.ref_seconds, threads, seed=200 + k)
        walls.append(time.perf_counter() - t0)
        vals.append(v)
        pxs += px
        t_tot += t
    value = float(np.mean(vals))
    mean_px = float(np.mean([nx * ny for _, _, nx, ny, _ in reqs]))
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000.0 * float(np.mean(walls)),
        "images_per_step": pxs / args.steps / mean_px,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": config_dict(args),
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": f"{pxs} random pixels of the workload ({t_tot:.1f} s); images/s extrapolated "
                                   f"by total pixels"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


def config_dict(args):
    return {"workload": f"{args.requests} orbit renders of a 256^3 stretched FP32 cube (config 2 on config 1's "
                        "cube): 144x84..1024x600 px, step 0.025-0.1 Re, roll U[-10, 10] deg, trilinear, PREFIX",
            "cube": "256x256x256 stretched axes, FP32 (FP64 oracle copy)", "requests": args.requests,
            "fov_deg": [27.0, 16.0], "ray_length_re": 44.0,
            "l2": "flushed between timed steps (512 MB write); images (~445 MB) exceed L2",
            "parallelism": f"replicas x{args.gpus}" if args.gpus > 1 else "1 GPU"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="birp", choices=["birp", "reference"])
    ap.add_argument("--requests", type=int, default=None, help="requests of the headline workload (512) or of "
                                                                 "--profile-case (64)")
    ap.add_argument("--ref-seconds", type=float, default=3.0)
    ap.add_argument("--cpu-seconds", type=float, default=10.0)
    ap.add_argument("--serve-seconds", type=float, default=3.0)
    ap.add_argument("--parity-px", type=int, default=256, help="pixels checked per image against the FP64 oracle")
    ap.add_argument("--details", help="file for everything measured (per-image errors, every rate and size), as JSON; "
                                      "the line on stdout has the single numbers")
    ap.add_argument("--no-plain", action="store_true")
    ap.add_argument("--no-c3", action="store_true", help="skip the config-3 block of the default run")
    ap.add_argument("--no-c4", action="store_true", help="skip the config-4 block of the default run")
    ap.add_argument("--workload", default="c2", choices=["c2", "c3", "c4"],
                    help="c2: the default run (headline on config 2, plus the c3 and c4 blocks); c3 / c4: that "
                         "block alone")
    ap.add_argument("--profile-case", choices=["trilinear", "nearest", "compact", "pairs", "cmem", "signed"],
                    help="run a small fixed batch of one kernel class (for a profiler) and exit")
    ap.add_argument("--launches", type=int, default=4, help="launches of --profile-case")
    ap.add_argument("--c4-cubes", type=int, default=256)
    ap.add_argument("--c4-dims", default="512x384x384")
    ap.add_argument("--c4-budget-gb", type=float, default=60.0)
    ap.add_argument("--c4-rates", default="50,200,500,1000,2000,3000,4000,6000,8000,12000,16000")
    ap.add_argument("--c4-seconds", type=float, default=4.0)
    ap.add_argument("--c4-layout", default="compact", choices=["compact", "pairs", "records"],
                    help="device layout of the served cubes")
    ap.add_argument("--c4-uploaders", type=int, default=1, help="the server's parallel cube uploads")
    ap.add_argument("--c4-promote-layout", default="pairs", choices=["pairs", "records"],
                    help="faster layout the server promotes its most-requested cubes to")
    ap.add_argument("--c4-promote-gb", type=float, default=0.0,
                    help="share of the budget for promoted cubes (0: no promotion)")
    args = ap.parse_args()
    world, rank, local = dist_setup()
    if args.requests is None:
        args.requests = 64 if args.profile_case else 512
    if args.impl == "reference":
        run_reference(args, world, rank)
        return
    if args.profile_case:
        run_profile_case(args)
        return
    import birp_cpp_gb300 as B
    from birp_cpp_gb300 import build
    if args.workload in ("c3", "c4"):
        O = oracle()
        host_c3 = gen_c3_host() if args.workload == "c3" else None
        build.build()
        B.init(0)
        out = run_c3(args, B, O, *host_c3) if args.workload == "c3" else run_c4(args, B, O)
        print(json.dumps(out))
        return

    extra_blocks = world == 1 and rank == 0
    # the oracle is built, and config 3's cubes generated in spawned
    # processes, before the first GPU call
    O = oracle() if rank == 0 else None
    host_c3 = gen_c3_host() if extra_blocks and not args.no_c3 else None
    build.build()
    B.init(local)
    W = make_workload(B, args.requests)
    cube, cams = W["cube"], W["cams"]
    npx = [c.nx * c.ny for c in cams]
    total_px = int(sum(npx))
    batch = B.Batch(len(cams), total_px)
    items = [(cube, c) for c in cams]

    for _ in range(max(args.warmup, 3)):
        batch.render(items)

    # ---- device-timed batched steps (inputs resident, L2 flushed before each)
    B.kernel_stats(reset=True)
    barrier(world)
    kern_ms, dev_ms = [], []
    with ClockSampler(local) as clocks:
        for _ in range(args.steps):
            B.flush_l2()
            batch.submit(items)
            batch.wait()
            k, t = batch.last_ms()
            kern_ms.append(k)
            dev_ms.append(t)
    barrier(world)
    ks = B.kernel_stats(reset=True)
    step_ms = allreduce_max(world, float(np.mean(kern_ms)))
    value = world * args.requests / (step_ms / 1000.0)
    samples_per_step = ks["samples"] / args.steps

    # ---- end to end through the C ABI with host buffers
    outs = [np.empty((c.ny, c.nx), np.float32) for c in cams]
    e2e_t = []
    import ctypes as C
    arr = B.Batch._reqs(items)
    ptrs = (C.c_void_p * len(items))(*[o.ctypes.data for o in outs])
    # untimed calls with the same output buffers (their pages are then mapped,
    # as in a serving loop that reuses its buffers)
    for _ in range(max(args.warmup, 1)):
        B.check(B.lib().birp_batch_render(batch.h, arr, len(items), ptrs))
    e2e_dev = []
    for _ in range(args.steps):
        B.flush_l2()
        barrier(world)
        t0 = time.perf_counter()
        B.check(B.lib().birp_batch_render(batch.h, arr, len(items), ptrs))
        e2e_t.append(time.perf_counter() - t0)
        e2e_dev.append(batch.last_ms())
    e2e_s = allreduce_max(world, float(np.mean(e2e_t)))
    e2e = world * args.requests / e2e_s
    # where the end-to-end time goes: kernel, device->host copy, host side
    k_mean = float(np.mean([k for k, _ in e2e_dev]))
    t_mean = float(np.mean([t for _, t in e2e_dev]))
    e2e_breakdown = {"kernel_ms": k_mean, "d2h_ms": t_mean - k_mean,
                     "host_ms": float(np.mean(e2e_t)) * 1e3 - t_mean}

    # ---- parity of every timed image against the FP64 oracle
    parity = None
    if rank == 0:
        xs, ys, zs, v32 = W["host"]
        oc = O.Cube64(xs, ys, zs, v32.astype(np.float64), 1)
        parity = parity_report(O, [(oc, c, o) for c, o in zip(cams, outs)], args.parity_px,
                               label="every image of the last e2e step, a random pixel sample each")
        parity["full_images"] = full_image_checks(O, oc, cams, outs)
        del oc

    # ---- plain per-call path on the same requests
    plain = None
    if not args.no_plain:
        pt = []
        for rep in range(2):
            B.flush_l2()
            t0 = time.perf_counter()
            for c, o in zip(cams, outs):
                B.render(cube, c, out=o)
            pt.append(time.perf_counter() - t0)
        plain_s = allreduce_max(world, min(pt))
        plain = world * args.requests / plain_s

    # ---- batched vs plain per image size (each class alone)
    by_size = None
    if not args.no_plain and rank == 0:
        by_size = {}
        img_buf = np.empty(max(c.nx * c.ny for c in cams), np.float32)
        for sz in sorted({(c.nx, c.ny) for c in cams}):
            sel = [c for c in cams if (c.nx, c.ny) == sz]
            its = [(cube, c) for c in sel]
            tb, tp = [], []
            for rep in range(2):
                B.flush_l2()
                batch.submit(its)
                batch.wait()
                tb.append(batch.last_ms()[0])
                B.flush_l2()
                t0 = time.perf_counter()
                for c in sel:
                    B.render(cube, c, out=img_buf[: c.nx * c.ny].reshape(c.ny, c.nx))
                tp.append(1000 * (time.perf_counter() - t0))
            bi, pi = len(sel) / (min(tb) / 1000), len(sel) / (min(tp) / 1000)
            by_size[f"{sz[0]}x{sz[1]}"] = {"requests": len(sel), "batched_images_s": bi, "plain_images_s": pi,
                                          "batched_vs_plain": bi / pi}

    # ---- roofline of the batched kernel (measured peaks)
    fp32_tflops, l2_gbs, l2_buf = B.measure_peaks()
    t_k = step_ms / 1000.0
    cells_per_step = ks["cells"] / args.steps

    def roof(units, flop_per, bytes_per, label):
        af = units * flop_per / t_k / 1e12
        ab = units * bytes_per / t_k / 1e9
        if units * flop_per / (fp32_tflops * 1e12) >= units * bytes_per / (l2_gbs * 1e9):
            r = {"bound": "fp32", "achieved": af, "peak": fp32_tflops, "unit": "TFLOP/s", "frac": af / fp32_tflops}
        else:
            r = {"bound": "l2", "achieved": ab, "peak": l2_gbs, "unit": "GB/s", "frac": ab / l2_gbs}
        r["units"] = label
        return r

    roofline = roof(cells_per_step, FLOP_PER_CELL, BYTES_PER_CELL,
                    f"{cells_per_step:.4g} cell segments/launch x {FLOP_PER_CELL:.0f} flop, {BYTES_PER_CELL:.0f} B")
    roofline.update({"traffic": traffic_from_profile(), "kernel": "render_batch_kernel",
                     "peak_source": f"measured in-run: FP32 FMA loop and L2-resident read (birp_measure_peaks: "
                                    f"loads that bypass L1, best of 16, 32 and 64 MB buffers, set by the "
                                    f"{l2_buf >> 20} MB one)",
                     "fp32_frac": cells_per_step * FLOP_PER_CELL / t_k / 1e12 / fp32_tflops,
                     "l2_frac": cells_per_step * BYTES_PER_CELL / t_k / 1e9 / l2_gbs})
    # the kernel is bound by instruction issue: warp instructions per cell
    # segment (ncu, profiles/) against one warp instruction per scheduler and
    # cycle (4 per SM) at the SM clock sampled during the timed steps
    wipc = profile_value("warp_instructions_per_cell")

    def issue_roofline(sm_mhz):
        if not wipc or not sm_mhz:
            return None
        try:
            import torch
            sms = torch.cuda.get_device_properties(local).multi_processor_count
        except Exception as e:  # a reporting extra: never fails the run
            return {"bound": "issue", "achieved": None, "error": str(e)[:120]}
        ai, peak = wipc * cells_per_step / t_k, 4.0 * sms * sm_mhz * 1e6
        return {"bound": "issue", "achieved": ai, "peak": peak, "unit": "warp-inst/s", "frac": ai / peak,
                "note": f"{wipc:.3f} warp instructions per cell segment (ncu, 64-request launch); peak = 4 x "
                        f"{sms} SMs x {sm_mhz:.0f} MHz (median SM clock of the timed steps)"}
    roofline_per_sample = roof(samples_per_step, FLOP_PER_SAMPLE, BYTES_PER_SAMPLE,
                               f"{samples_per_step:.4g} ray-samples/launch x {FLOP_PER_SAMPLE:.0f} flop, "
                               f"{BYTES_PER_SAMPLE:.0f} B (per-sample formulation; the kernel sums "
                               f"{samples_per_step / max(cells_per_step, 1):.2f} samples per cell in closed form)")
    peaks_file = os.path.join(ROOT, "MEASURED_PEAKS.json")
    hbm = None
    if os.path.exists(peaks_file):
        hbm = json.load(open(peaks_file)).get("hbm_gbs")
    unique_bytes = cube.info().device_bytes + 4 * total_px
    roofline_hbm = {"bound": "hbm", "achieved": unique_bytes / t_k / 1e9, "peak": hbm, "unit": "GB/s",
                    "frac": (unique_bytes / t_k / 1e9 / hbm) if hbm else None,
                    "note": "unique bytes: cube read once + images written; peak of measured (MEASURED_PEAKS.json)"}

    # ---- serving at 70% of the saturated batched rate: three runs (a run's
    # p99 is the 1% tail of ~17 k requests, which one host-side stall of a
    # few tens of ms can set); the run with the median p99 is reported,
    # with every run's p50/p99
    serving = None
    if args.serve_seconds > 0:
        runs = [serve_latency(B, W, rate=0.7 * value / world, seconds=args.serve_seconds, seed=13 + k)
                for k in range(3)]
        serving = dict(sorted(runs, key=lambda r: r["p99_ms"] or 0.0)[1])
        serving["runs_p50_p99_ms"] = [[r["p50_ms"], r["p99_ms"]] for r in runs]

    # ---- CPU baseline (rank 0, N = 1)
    cpu = None
    if rank == 0 and world == 1 and args.cpu_seconds > 0:
        threads = os.cpu_count() or 1
        v, px, t = cpu_sample(W["reqs"], W["host"], args.cpu_seconds, threads)
        cpu = {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
               "sample": f"{px} random pixels of the {args.requests}-request workload, {t:.1f} s on {threads} "
                         f"threads; images/s extrapolated by total pixels (the reference has no roll input; the "
                         f"cost of a pixel does not depend on it)"}
        v1, px1, t1 = cpu_sample(W["reqs"], W["host"], max(2.0, args.cpu_seconds / 3), 1, seed=11)
        cpu["single_core"] = {"value": v1, "unit": UNIT, "cores": 1,
                              "sample": f"{px1} random pixels, {t1:.1f} s on 1 thread"}
    clock_summary = clocks.summary()
    h2d = batch.upload_bytes()  # request descriptors and work tables, copied each step
    batch.close()
    cube.close()

    # ---- the config-3 and config-4 blocks (one GPU only)
    c3 = c4 = None
    if extra_blocks and host_c3 is not None:
        c3 = run_c3(args, B, O, *host_c3)
        del host_c3
    if extra_blocks and not args.no_c4:
        c4 = run_c4(args, B, O)

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": step_ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic", "config": config_dict(args),
            "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": 4 * total_px},
            "plain": {"value": plain, "unit": UNIT} if plain else None,
            "batched_vs_plain": (value / plain) if plain else None,
            "by_size": by_size,
            "e2e_vs_plain": (e2e / plain) if plain else None,
            "e2e_breakdown": e2e_breakdown,
            "serving": serving,
            "ray_samples_per_s": samples_per_step * world / (step_ms / 1000.0),
            "roofline": roofline, "roofline_issue": issue_roofline(clock_summary.get("sm_mhz")),
            "roofline_per_sample": roofline_per_sample,
            "roofline_hbm": roofline_hbm,
            "cpu_baseline": cpu,
            # each step replays one graph with six kernels: the CMEM, signed,
            # nearest, compact- and pairs-layout ones (no work here) and the
            # records-layout trilinear one
            "gpu_launches": 6 * args.steps, "clocks": clock_summary,
            "exact_fp64_rays_per_step": ks["exact_range_rays"] / args.steps,
            "samples_per_cell": (ks["samples"] / ks["cells"]) if ks.get("cells") else None,
            "c3": c3, "c4": c4,
            "parity": parity,
        }
        print_result(line, args.details)


# What the result line keeps of its larger blocks, and the longest it may get:
# programs that read the end of a run's output keep 2 to 3 KB of it.
BRIEF = {
    "e2e_breakdown": ("kernel_ms", "host_ms"), "serving": ("achieved_images_s", "p50_ms", "p99_ms"),
    "roofline": ("bound", "achieved", "peak", "unit", "frac"), "roofline_issue": ("achieved", "peak", "unit", "frac"),
    "cpu_baseline": ("value", "unit", "cores", "kind"), "c3": ("requests", "images_s", "batched_vs_plain", "parity"),
    "c4": ("saturation_images_s", "at_70pct_of_saturation", "parity"),
    "parity": ("images", "pixels_checked", "max_rel_err", "rms_rel_err", "images_within_tolerance", "tolerance"),
}
BRIEF_NESTED = ("max_rel_err", "images_within_tolerance", "served_images_s", "p50_ms", "p99_ms")
WHOLE = ("config", "e2e", "clocks", "plain")
MAX_LINE = 2400


def result_line(full: dict) -> str:
    """The result as one JSON line of at most MAX_LINE characters: every plain
    value and the config, clocks, end-to-end and launch counts in full, of the
    other blocks the numbers BRIEF names."""
    def short(v):
        return float(f"{v:.6g}") if isinstance(v, float) else v

    line = {}
    for k, v in full.items():
        if not isinstance(v, (dict, list)):
            line[k] = v if k in ("value", "ms_per_step") else short(v)
        elif k in WHOLE:
            line[k] = v
        elif k in BRIEF:
            line[k] = {a: {n: short(x[n]) for n in BRIEF_NESTED if n in x} if isinstance(x, dict) else short(x)
                       for a, x in ((a, v[a]) for a in BRIEF[k] if a in v)}
    for k in ("e2e_breakdown", "c4", "c3", "serving", "roofline_issue"):  # (not reached by the blocks as they are)
        if len(json.dumps(line)) > MAX_LINE:
            line.pop(k, None)
    return json.dumps(line)


def print_result(full: dict, details: str | None) -> None:
    """The result line on stdout; everything measured in the file `details`."""
    if details:
        with open(details, "w") as f:
            json.dump(full, f)
    print(result_line(full), flush=True)


def serve_latency(B, W, rate: float, seconds: float, seed: int = 13):
    """Poisson arrivals at `rate` req/s for `seconds` into the server; returns
    p50/p99 latency and achieved throughput."""
    from birp_cpp_gb300 import synth
    srv = B.Server(B.server_config(slots=3, max_batch_requests=64, max_batch_pixels=16 << 20, max_wait_ms=1.0))
    sid = srv.add_cube(*W["host"])
    reqs = synth.config2_requests(4096, seed=seed)
    rng = np.random.default_rng(seed)
    cams = [B.camera(p, a, synth.FOV_W, synth.FOV_H, nx, ny, n_samples=synth.n_samples(s)) for p, a, nx, ny, s in reqs]
    # one buffer per in-flight request slot, each large enough for any image
    max_px = max(c.nx * c.ny for c in cams)
    bufs = [np.full(max_px, 0.0, np.float32) for _ in range(256)]  # pages resident before the timed arrivals
    # warm the cube into GPU memory
    t = srv.submit(sid, cams[0], bufs[0])
    srv.wait(t)
    tickets = []
    t0 = time.perf_counter()
    next_t = t0
    k = 0
    while next_t - t0 < seconds:
        now = time.perf_counter()
        if now < next_t:
            time.sleep(min(next_t - now, 0.002))
            continue
        c = cams[k % len(cams)]
        try:
            tickets.append(srv.submit(sid, c, bufs[k % len(bufs)]))
        except B.BirpError:
            pass
        k += 1
        next_t += rng.exponential(1.0 / rate)
    lat = []
    for t in tickets:
        r = srv.wait(t, 60000)
        if r.status == 0:
            lat.append(r.latency_ms)
    t_end = time.perf_counter()
    st = srv.stats()
    srv.close()
    lat = np.array(lat)
    return {"offered_rate": rate, "requests": len(tickets), "completed": int(len(lat)),
            "achieved_images_s": len(lat) / (t_end - t0), "p50_ms": float(np.percentile(lat, 50)) if len(lat) else None,
            "p99_ms": float(np.percentile(lat, 99)) if len(lat) else None, "batches": int(st.batches),
            "load": "70% of the saturated batched rate, Poisson"}


def profile_value(key):
    """One figure of the batched kernel from the committed ncu summary
    (profiles/render_batch_kernel_traffic.json), or None."""
    p = os.path.join(ROOT, "profiles", "render_batch_kernel_traffic.json")
    if os.path.exists(p):
        try:
            return json.load(open(p)).get(key)
        except (OSError, ValueError):
            return None
    return None


def traffic_from_profile():
    """DRAM bytes per launch of the batched kernel (ncu), if recorded."""
    return profile_value("dram_bytes_per_launch")


if __name__ == "__main__":
    main()
