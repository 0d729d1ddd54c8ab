#!/usr/bin/env python3
"""Benchmark: Gpixels/s of bit-exact reconstruction by dilation on GB300.

Headline workload (one "step"): the plain 16384 x 16384 uint8 8-connected
reconstruction of the spiral-corridor image -- smoothed noise (seed 2,
sigma 16) with a one-pixel square spiral corridor at 255 (arm pitch 256,
1 048 194 pixels) and a marker that is 0 except 64 seeds, one at the
spiral's start -- the largest configuration that fits one GPU, through the
C ABI (async queue by default; --variant picks mutex / double / unique).
The library's autotuner is run once on the image class before the timed
region (as a user would, once per class); every step then restores the
marker from a pristine device copy and reconstructs with the default
configuration fields, which the tuning table fills.

  value : device-resident throughput (inputs already in HBM), CUDA events
          around K steps on the launching stream, max over ranks.
  e2e   : the same reconstruction from pinned HOST buffers through the
          per-image C-ABI call: H2D of marker + mask and D2H of the result
          inside the timed region, copies on their own streams and
          double-buffered so that one step's copies overlap its neighbours'
          reconstructions.
  roofline : one reconstruction (front stage: seed check, top-level
          labelling, whole-image passes where the configuration has them;
          then the tile engine -- all of this library's kernels of the
          call) as the unit: algorithmic bytes
          = 3 * W * H * bytes/pixel (read mask, read marker, write result)
          over its CUDA-event duration, against the measured HBM copy
          bandwidth.
  cpu_baseline : the CPU oracle (Vincent 1993 hybrid, single thread) on the
          same image, which also checks the GPU output bit for bit.

Sub-results in the same line (skipped with --no-extras):
  config1 : the six 4096^2 uint8 reconstructions (connectivity {4, 8} x
          h-dome h {10, 40, 100}), device-resident and end to end, after
          the autotuner has seen each connectivity's image class once
          (--config1-only: the untuned default, or --config1-solver's
          solver, the profiled launches).
  batched : 64 uneven images in one CUDA-graph plan vs 64 sequential plain
          calls, Gpixels/s of each, bit-exact against each other and the
          oracle.
  served : a 2000 req/s Poisson stream through the serving loop (open loop:
          p50 / p99 latency; closed loop: saturated Gpixels/s) vs plain
          per-request calls, with host buffers, every result bit-exact.
  spiral_types : the 16384^2 spiral in uint16 and int32, each checked
          against the oracle.

--impl reference times the reference's CPU path for the same workload.  The
reference has no CPU implementation, so that is the oracle port: one copy
of the headline reconstruction per host core at once, on the same metric
and config.

Multi-GPU (torchrun, N > 1): replicas only -- every rank reconstructs its own
copy of the workload, no collective on the data path; value = all ranks'
pixels / max time.
"""
from __future__ import annotations

import argparse
import gc
import json
import os
import statistics
import subprocess
import sys
import threading
import time

REPO = os.path.dirname(os.path.abspath(__file__))
for p in (os.path.join(REPO, "iwpp-mp_gb300"), REPO):
    if p not in sys.path:
        sys.path.insert(0, p)

METRIC = "Gpixels/s bit-exact reconstruction (plain vs batched); served p50/p99 latency"
UNIT = "Gpixels/s"
WORKLOAD = ("16384x16384 uint8 8-connected spiral-corridor reconstruction: smoothed noise (seed 2, sigma 16), "
            "1-px square spiral corridor at 255 (arm pitch 256), marker 0 but 64 seeds (one per step)")
CONFIG1 = ("4096x4096 uint8 plain reconstruction, seed 1, sigma 8, 2000 discs, h-dome h in {10,40,100} x "
           "connectivity {4,8} (6 images per step)")


def _dist_env():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


def max_over_ranks(x: float, device=None) -> float:
    """The largest x over all ranks of the default process group (x itself
    without one): the job's time is its slowest replica's."""
    import torch
    import torch.distributed as dist

    if not (dist.is_available() and dist.is_initialized()) or dist.get_world_size() == 1:
        return x
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_gpx(world: int, px_per_rank_step: int, steps: int, elapsed_ms: float) -> float:
    """Replicas: every rank processes its own copy of the workload, so the
    job processed world x the pixels of one rank in the slowest rank's time."""
    return world * px_per_rank_step * steps / (elapsed_ms / 1e3) / 1e9


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled under load.

    Every sample carries nvidia-smi's own timestamp, so the samples taken
    inside a region (region_begin() .. region_end(), host wall clock) are
    told apart from the one taken at start-up, before the GPU is loaded."""

    FIELDS = ("timestamp,index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    PERIOD_MS = 100

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.lines = []
        self.thread = None
        self.t_begin = None
        self.t_end = None

    def start(self):
        """Starts sampling and returns once the first sample has arrived:
        nvidia-smi's start-up takes driver locks that stall CUDA calls for
        tens of milliseconds, which must not fall inside a timed region."""
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), "--query-gpu=" + self.FIELDS,
                                          "--format=csv,noheader,nounits", "-lms", str(self.PERIOD_MS)],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except (OSError, FileNotFoundError):
            self.proc = None
            return
        self.thread = threading.Thread(target=self._read, daemon=True)
        self.thread.start()
        t0 = time.perf_counter()
        while not self.lines and self.proc.poll() is None and time.perf_counter() - t0 < 10.0:
            time.sleep(0.01)
        time.sleep(0.05)

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def region_begin(self):
        self.t_begin = time.time()

    def region_end(self):
        self.t_end = time.time()

    @staticmethod
    def _stamp(text):
        import datetime

        for fmt in ("%Y/%m/%d %H:%M:%S.%f", "%Y/%m/%d %H:%M:%S"):
            try:
                return datetime.datetime.strptime(text, fmt).timestamp()
            except ValueError:
                pass
        return None

    def _samples(self):
        out = []
        for line in list(self.lines):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 10:
                continue
            try:
                out.append((self._stamp(parts[0]), float(parts[2]), float(parts[3]), parts[6:10]))
            except ValueError:
                continue
        return out

    def since_begin(self):
        """Samples taken since region_begin()."""
        if self.t_begin is None:
            return 0
        return sum(1 for ts, *_ in self._samples() if ts is not None and ts >= self.t_begin)

    def stop(self):
        """Median SM clock and the throttle reasons seen, over the samples
        taken since region_begin() (all samples when no region was marked);
        `in_region` counts those taken before region_end()."""
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        if self.thread:
            self.thread.join(timeout=2)
        samples = self._samples()
        if self.t_begin is not None:
            samples = [x for x in samples if x[0] is not None and x[0] >= self.t_begin]
        if not samples:
            return None
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for *_, flags in samples:
            for name, val in zip(names, flags):
                if val.lower().startswith("active"):
                    reasons.add(name)
        info = {"sm_mhz": statistics.median(x[1] for x in samples), "sm_max_mhz": max(x[2] for x in samples),
                "samples": len(samples), "reasons": sorted(reasons)}
        if self.t_begin is not None and self.t_end is not None:
            info["in_region"] = sum(1 for x in samples if x[0] <= self.t_end)
        return info


def load_headline():
    """(marker, mask, corridor pixels) of the headline image."""
    from iwpp import synth

    return synth.config2(synth.U8)


def load_config1():
    from iwpp import synth

    mask = synth.config1_mask()
    cases = []
    for conn, h in synth.CONFIG1_CASES:
        cases.append((conn, h, synth.hdome_marker(mask, h)))
    return mask, cases


def timed_oracle(marker, mask, conn):
    """(result, seconds) of one oracle reconstruction (one host thread)."""
    import oracle

    t0 = time.perf_counter()
    res = oracle.reconstruct(marker, mask, conn)
    return res, time.perf_counter() - t0


def inputs_sha256(*arrays):
    """sha256 over the bytes of the generated input arrays, in order (the
    record of which synthetic inputs a result was measured on)."""
    import hashlib

    h = hashlib.sha256()
    for a in arrays:
        h.update(a.tobytes())
    return h.hexdigest()


def traffic_from_profile(key):
    """DRAM bytes per launch recorded from an ncu capture (profiles/)."""
    path = os.path.join(REPO, "profiles", "dram_traffic.json")
    try:
        with open(path) as f:
            return json.load(f)[key]["bytes_per_launch"]
    except (OSError, ValueError, KeyError, TypeError):
        return None


def peak_hbm():
    try:
        with open(os.path.join(REPO, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except (OSError, ValueError, KeyError):
        return 6800.0, "fallback"


def run_reference(args):
    """The reference has no CPU path (its only implementation is CUDA), so the
    reference arm times the oracle port: one copy of the headline
    reconstruction per host thread at once (the oracle is sequential), on
    every host core, once -- about 20-40 s of CPU work."""
    world, rank, _ = _dist_env()
    if rank != 0:
        return 0
    from concurrent.futures import ThreadPoolExecutor

    marker, mask, _ = load_headline()
    px = marker.size
    threads = min(os.cpu_count() or 1, 16)
    with ThreadPoolExecutor(max_workers=threads) as ex:  # ctypes releases the GIL
        t0 = time.perf_counter()
        list(ex.map(lambda _: timed_oracle(marker, mask, 8), range(threads)))
        t_total = time.perf_counter() - t0
    value = threads * px / t_total / 1e9
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": px / (value * 1e9) * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u8", "data": "synthetic",
        "config": {"workload": WORKLOAD, "l2": "n/a (host)"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": f"{threads} concurrent reconstructions of the 16384x16384 uint8 spiral image, one "
                                   "per host thread (the reference has no CPU path; this is the oracle "
                                   "restatement, Vincent 1993 hybrid)"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


def _to_dev(a, dev):
    import numpy as np
    import torch

    return torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).to(dev)


def _from_dev(t, dtype):
    import numpy as np

    a = t.cpu().numpy()
    return a.view(np.uint16) if dtype == np.uint16 else a


def _pinned(a):
    """A page-locked copy of a numpy array (through torch), same dtype."""
    import numpy as np
    import torch

    t = torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).pin_memory()
    n = t.numpy()
    return n.view(np.uint16) if a.dtype == np.uint16 else n


def bench_batched(args, dev, variant):
    """64 images of uneven sizes (uint8 / uint16, 4/8-connectivity, h-dome
    h in [5, 120], seed 3): one CUDA-graph plan (one persistent launch over
    all tiles) against 64 sequential plain synchronous calls on the same
    device-resident inputs."""
    import numpy as np
    import torch

    import iwpp
    from iwpp import synth

    specs = synth.config3_specs(64)
    imgs = [synth.spec_images(s, nthreads=os.cpu_count() or 1) for s in specs]
    px = sum(s.pixels for s in specs)
    nbytes = sum(3 * s.pixels * s.bpp for s in specs)
    h = iwpp.Handle(dev.index or 0)
    pm = [_to_dev(m, dev) for m, _ in imgs]
    pk = [_to_dev(k, dev) for _, k in imgs]
    work = [p.clone() for p in pm]
    reps = max(args.warmup, 3) + 5

    def restore():
        for w, p in zip(work, pm):
            w.copy_(p)
        torch.cuda.synchronize()

    seq = []
    for _ in range(reps):
        restore()
        t = time.perf_counter()
        for w, k, s in zip(work, pk, specs):
            iwpp.reconstruct(w, k, connectivity=s.conn, variant=variant, handle=h)
        seq.append(time.perf_counter() - t)
    seq_out = [_from_dev(w, m.dtype) for w, (m, _) in zip(work, imgs)]
    # the autotuner picks tile rows / solver / initial passes for this batch
    # class; the plan below is built with default fields, so it uses them
    restore()
    tuned = iwpp.autotune([(w, k, s.conn) for w, k, s in zip(work, pk, specs)], variant=variant, handle=h)
    tune_ok = all(np.array_equal(_from_dev(w, m.dtype), ref) for w, (m, _), ref in zip(work, imgs, seq_out))
    plan = iwpp.Plan(h, [(w, k, s.conn) for w, k, s in zip(work, pk, specs)], variant=variant)
    graph = []
    for _ in range(reps):
        restore()
        t = time.perf_counter()
        plan.launch()
        st = plan.sync()
        graph.append(time.perf_counter() - t)
    plan_ok = all(np.array_equal(_from_dev(w, m.dtype), ref) for w, (m, _), ref in zip(work, imgs, seq_out))
    oracle_ok = None
    if not args.no_cpu:
        import oracle
        from concurrent.futures import ThreadPoolExecutor

        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
            refs = list(ex.map(lambda i: oracle.reconstruct(imgs[i][0], imgs[i][1], specs[i].conn),
                               range(len(specs))))
        oracle_ok = all(np.array_equal(a, b) for a, b in zip(seq_out, refs))
    plan.close()
    h.close()
    t_seq = statistics.median(seq[max(args.warmup, 3):])
    t_plan = statistics.median(graph[max(args.warmup, 3):])
    return {"workload": f"64 images, sizes log-uniform 512..4096 x 512..3072 (seed 3, {px / 1e6:.1f} Mpx), "
                        "uint8/uint16, 4/8-conn, h-dome h in [5,120]; device-resident",
            "inputs_sha256": inputs_sha256(*[a for pair in imgs for a in pair]),
            "plan_gpx_s": px / t_plan / 1e9, "sequential_gpx_s": px / t_seq / 1e9, "speedup": t_seq / t_plan,
            "plan_ms": t_plan * 1e3, "sequential_ms": t_seq * 1e3,
            "plan_hbm_frac": nbytes / t_plan / 1e9 / peak_hbm()[0], "tiles": st.tiles, "visits": st.visits,
            "bitexact_plan_vs_sequential": plan_ok and tune_ok, "bitexact_vs_oracle": oracle_ok,
            "autotuned": tuned,
            "timing": f"median of {reps - max(args.warmup, 3)} after {max(args.warmup, 3)} warm-up, host clock "
                      "around launch + sync, markers restored before each"}


def bench_served(args, dev, variant):
    """Poisson request stream (2000 req/s, seed 4) of 8-connected uint8 (80 %)
    / uint16 images, sides log-uniform 256..8192, h-dome or sparse-seed
    markers, through the serving loop (iwpp_server_*) with pinned host
    buffers; against plain per-request synchronous calls (H2D, reconstruct,
    D2H) on the same requests."""
    import numpy as np
    import torch

    import iwpp
    from iwpp import synth

    n_req = args.served_requests
    times, which, specs = synth.config4_stream(n_req, args.served_pool)
    imgs = [synth.spec_images(s, nthreads=os.cpu_count() or 1) for s in specs]
    pin = [(_pinned(m), _pinned(k)) for m, k in imgs]
    outs = [_pinned(np.zeros_like(m)) for m, _ in imgs]
    px = sum(specs[w].pixels for w in which)
    h = iwpp.Handle(dev.index or 0)
    refs = []
    for (m, k), s in zip(pin, specs):  # one plain call per distinct image
        dm, dk = _to_dev(m, dev), _to_dev(k, dev)
        iwpp.reconstruct(dm, dk, connectivity=8, variant=variant, handle=h)
        refs.append(_from_dev(dm, m.dtype))
    oracle_ok = None
    if not args.no_cpu:
        import oracle
        from concurrent.futures import ThreadPoolExecutor

        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
            orefs = list(ex.map(lambda i: oracle.reconstruct(imgs[i][0], imgs[i][1], 8), range(len(specs))))
        oracle_ok = all(np.array_equal(a, b) for a, b in zip(refs, orefs))

    # plain per-request calls, closed loop, same pinned host buffers
    torch.cuda.synchronize()
    gc.collect()
    gc.disable()
    try:
        t = time.perf_counter()
        for w in which:
            m, k = pin[w]
            dm, dk = _to_dev(m, dev), _to_dev(k, dev)
            iwpp.reconstruct(dm, dk, connectivity=8, variant=variant, handle=h)
            o = outs[w]
            torch.from_numpy(o.view(np.int16) if o.dtype == np.uint16 else o).copy_(dm)
        t_plain = time.perf_counter() - t
    finally:
        gc.enable()
    plain_ok = all(np.array_equal(outs[w], refs[w]) for w in set(which))
    h.close()

    def run(open_loop):
        clocks = ClockSampler(dev.index or 0)
        for o in outs:
            o.fill(0)
        with iwpp.Server(device=dev.index or 0, lanes=args.lanes, variant=variant) as srv:
            for w in range(len(specs)):  # warm the pool and the lanes
                srv.wait(srv.submit(pin[w][0], pin[w][1], 8, out=outs[w]))
            # no collector pauses in the submitting loop: a pause would turn
            # the Poisson stream into bursts
            gc.collect()
            gc.disable()
            clocks.start()
            clocks.region_begin()
            try:
                tickets = []
                t0 = time.perf_counter()
                for i, w in enumerate(which):
                    if open_loop:
                        while time.perf_counter() - t0 < times[i]:
                            pass
                    tickets.append(srv.submit(pin[w][0], pin[w][1], 8, out=outs[w]))
                lat, queue, service, status_ok = [], [], [], True
                for tk in tickets:
                    _, info = srv.wait(tk)
                    lat.append(info["latency_us"] / 1e3)
                    queue.append(info["queue_us"] / 1e3)
                    service.append(info["service_us"] / 1e3)
                    status_ok &= info["status"] == 0
                dt = time.perf_counter() - t0
            finally:
                gc.enable()
                clocks.region_end()
                clock_info = clocks.stop()
            st = srv.stats()
        ok = status_ok and all(np.array_equal(outs[w], refs[w]) for w in set(which))
        lat = np.array(lat)
        return {"gpx_s": px / dt / 1e9, "seconds": dt, "p50_ms": float(np.percentile(lat, 50)),
                "p99_ms": float(np.percentile(lat, 99)),
                "queue_p50_ms": float(np.percentile(queue, 50)), "queue_p99_ms": float(np.percentile(queue, 99)),
                "service_p50_ms": float(np.percentile(service, 50)),
                "service_p99_ms": float(np.percentile(service, 99)), "batches": st["batches"],
                "largest_batch": st["largest_batch"], "device_bytes_peak": st["bytes_peak"], "bitexact": ok,
                "clocks": clock_info}

    # the open loop three times, the run with the median p99 reported: the
    # host-to-device path of a shared box has slow moments of its own
    opens = sorted((run(True) for _ in range(3)), key=lambda r: r["p99_ms"])
    served = dict(opens[1])
    served["p99_ms_of_runs"] = [r["p99_ms"] for r in opens]
    served["bitexact"] = all(r["bitexact"] for r in opens)
    saturated = run(False)
    return {"workload": f"{n_req} requests over {len(set(which))} distinct images, Poisson 2000/s (seed 4), "
                        "sides log-uniform 256..8192 "
                        f"({px / n_req / 1e6:.2f} Mpx mean), uint8 80% / uint16 20%, 8-conn, "
                        "h-dome or 0.01% sparse seeds; pinned host buffers, H2D + D2H included",
            "offered_gpx_s": px / times[-1] / 1e9, "lanes": args.lanes, "distinct_images": len(set(which)),
            "inputs_sha256": inputs_sha256(*[a for pair in imgs for a in pair]),
            "open_loop": served, "closed_loop": saturated,
            "plain_per_request_gpx_s": px / t_plain / 1e9, "plain_bitexact": plain_ok,
            "speedup_vs_plain": saturated["gpx_s"] / (px / t_plain / 1e9),
            "bitexact_vs_oracle": oracle_ok}


def bench_config1(args, dev, variant, handle, tune=True):
    """The six 4096^2 uint8 reconstructions of configuration 1 per step:
    device-resident (events on the launching stream) and end to end from
    pinned host buffers, each image through the per-image C-ABI call with
    the default configuration, after the autotuner has seen each
    connectivity's image class once."""
    import numpy as np
    import torch

    import iwpp

    lib = iwpp.load()
    mask_np, cases = load_config1()
    H, W = mask_np.shape
    px_step = W * H * len(cases)
    vcode = iwpp._variant(variant)
    mask = torch.from_numpy(mask_np).to(dev)
    pristine = [torch.from_numpy(m).to(dev) for _, _, m in cases]
    work = [p.clone() for p in pristine]
    conns = [c for c, _, _ in cases]
    stream = torch.cuda.Stream(dev)
    steps = max(args.steps, 20)
    solver = getattr(args, "config1_solver", None)
    tile_rows = getattr(args, "config1_tile_rows", 0)
    cfg = None if solver is None else __import__("ctypes").byref(iwpp.Config.make(solver=solver, tile_rows=tile_rows))

    # the autotuner once per image class (4096^2 uint8 at each connectivity,
    # tuned on its h = 40 image); the default calls below read its table
    tuned = {}
    for conn in sorted(set(conns)) if tune else ():
        i = next(j for j, (c, h, _) in enumerate(cases) if c == conn and h == 40)
        probe = pristine[i].clone()
        with torch.cuda.stream(stream):
            t = iwpp.autotune([(probe, mask, conn)], variant=variant, handle=handle, stream=stream)
        tuned[f"conn{conn}"] = {k_: t[k_] for k_ in ("tile_rows", "solver", "init_passes", "front_passes")}
        del probe
    torch.cuda.synchronize()

    def step(ev_pairs=None):
        for i in range(len(cases)):
            work[i].copy_(pristine[i], non_blocking=True)
            if ev_pairs is not None:
                ev_pairs[i][0].record(stream)
            st = lib.iwpp_reconstruct_async(handle.ptr, work[i].data_ptr(), mask.data_ptr(), W, W, W, H, 0, conns[i],
                                            vcode, cfg, stream.cuda_stream)
            if st != 0:
                raise iwpp.IwppError(st, "iwpp_reconstruct_async")
            if ev_pairs is not None:
                ev_pairs[i][1].record(stream)

    with torch.cuda.stream(stream):
        for _ in range(max(args.warmup, 3)):
            step()
        stream.synchronize()
        results = [w.cpu().numpy() for w in work]
    bitexact = None
    if not args.no_cpu:
        import oracle
        from concurrent.futures import ThreadPoolExecutor

        with ThreadPoolExecutor(max_workers=len(cases)) as ex:
            refs = list(ex.map(lambda c: oracle.reconstruct(c[2], mask_np, c[0]), cases))
        bitexact = all(np.array_equal(a, b) for a, b in zip(results, refs))
    ev = [[(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in cases]
          for _ in range(steps)]
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        t0.record(stream)
        for k in range(steps):
            step(ev[k])
        t1.record(stream)
    torch.cuda.synchronize()
    elapsed = t0.elapsed_time(t1)
    recon_ms = [a.elapsed_time(b) for row in ev for (a, b) in row]
    mean_ms = sum(recon_ms) / len(recon_ms)
    peak = peak_hbm()[0]

    # end to end: H2D / reconstruction / D2H on three streams, double-buffered
    host_m = [torch.from_numpy(m).pin_memory() for _, _, m in cases]
    host_k = torch.from_numpy(mask_np).pin_memory()
    host_out = [torch.empty(h.shape, dtype=h.dtype, pin_memory=True) for h in host_m]
    s_in, s_run, s_out = (torch.cuda.Stream(dev) for _ in range(3))
    dmb = [torch.empty((H, W), dtype=torch.uint8, device=dev) for _ in range(2)]
    dkb = [torch.empty((H, W), dtype=torch.uint8, device=dev) for _ in range(2)]
    ev_in = [torch.cuda.Event() for _ in range(2)]
    ev_run = [torch.cuda.Event() for _ in range(2)]
    ev_out = [torch.cuda.Event() for _ in range(2)]
    for e in ev_out:
        e.record(s_out)

    def pipelined_step(finish=True):
        for i in range(len(cases)):
            b = i & 1
            with torch.cuda.stream(s_in):
                s_in.wait_event(ev_out[b])
                dmb[b].copy_(host_m[i], non_blocking=True)
                dkb[b].copy_(host_k, non_blocking=True)
                ev_in[b].record(s_in)
            s_run.wait_event(ev_in[b])
            st = lib.iwpp_reconstruct_async(handle.ptr, dmb[b].data_ptr(), dkb[b].data_ptr(), W, W, W, H, 0,
                                            conns[i], vcode, cfg, s_run.cuda_stream)
            if st != 0:
                raise iwpp.IwppError(st, "iwpp_reconstruct_async")
            ev_run[b].record(s_run)
            with torch.cuda.stream(s_out):
                s_out.wait_event(ev_run[b])
                host_out[i].copy_(dmb[b], non_blocking=True)
                ev_out[b].record(s_out)
        if finish:
            s_out.synchronize()
            st = lib.iwpp_handle_sync(handle.ptr, None)
            if st != 0:
                raise iwpp.IwppError(st, "iwpp_handle_sync")

    for _ in range(max(args.warmup, 3)):
        pipelined_step()
    e2e_steps = min(steps, 40)
    torch.cuda.synchronize()
    ts = time.perf_counter()
    for k in range(e2e_steps):
        pipelined_step(finish=k == e2e_steps - 1)
    secs = time.perf_counter() - ts
    e2e_ok = all(np.array_equal(host_out[i].numpy(), results[i]) for i in range(len(cases)))
    return {"workload": CONFIG1, "variant": variant, "autotuned": tuned or None, "solver": solver,
            "tile_rows": tile_rows if solver is not None else None, "steps": steps,
            "gpx_s": px_step * steps / (elapsed / 1e3) / 1e9,
            "inputs_sha256": inputs_sha256(mask_np, *[m for _, _, m in cases]),
            "ms_per_step": elapsed / steps, "mean_reconstruction_ms": mean_ms,
            "hbm_frac": 3 * W * H / (mean_ms / 1e3) / 1e9 / peak, "bitexact_vs_oracle": bitexact,
            "dram_bytes_per_reconstruction": traffic_from_profile("config1"),
            "e2e": {"gpx_s": px_step * e2e_steps / secs / 1e9, "steps": e2e_steps, "bitexact": e2e_ok,
                    "h2d_bytes_per_step": len(cases) * 2 * W * H, "d2h_bytes_per_step": len(cases) * W * H}}


def bench_spiral_types(args, dev, variant, handle):
    """The 16384^2 spiral in uint16 and int32 (8-connectivity): untuned
    default, then autotuned; each result checked against the oracle, which
    runs on host threads while the GPU works."""
    import numpy as np
    import torch
    from concurrent.futures import ThreadPoolExecutor

    import iwpp
    from iwpp import synth

    res = {}
    peak = peak_hbm()[0]
    ex = ThreadPoolExecutor(max_workers=2)
    pending = []
    for name, dt in (("u16", synth.U16), ("i32", synth.I32)):
        marker, mask, _ = synth.config2(dt)
        H, W = mask.shape
        bpp = mask.dtype.itemsize
        fut = None if args.no_cpu else ex.submit(timed_oracle, marker, mask, 8)
        m0, k = _to_dev(marker, dev), _to_dev(mask, dev)
        m = m0.clone()
        st0 = iwpp.reconstruct(m, k, connectivity=8, variant=variant, handle=handle)
        m.copy_(m0)
        tuned = iwpp.autotune([(m, k, 8)], variant=variant, repeats=1, handle=handle)
        times = []
        for rep in range(1 + args.spiral_reps):
            m.copy_(m0)
            torch.cuda.synchronize()
            st = iwpp.reconstruct(m, k, connectivity=8, variant=variant, handle=handle)
            if rep:
                times.append(st.device_ms)
        t = statistics.median(times) / 1e3
        res[name] = {"ms": t * 1e3, "gpx_s": W * H / t / 1e9, "hbm_frac": 3 * W * H * bpp / t / 1e9 / peak,
                     "visits": st.visits, "tiles": st.tiles, "top_pixels": st.top_pixels,
                     "untuned_ms": st0.device_ms, "inputs_sha256": inputs_sha256(marker, mask),
                     "autotuned": {k_: tuned[k_] for k_ in ("tile_rows", "solver", "init_passes", "front_passes")}}
        pending.append((name, fut, _from_dev(m, marker.dtype)))
        del m, m0, k
        torch.cuda.empty_cache()
    for name, fut, out in pending:
        if fut is not None:
            ref, secs = fut.result()
            res[name]["bitexact_vs_oracle"] = bool(np.array_equal(out, ref))
            res[name]["cpu_oracle_s"] = secs
    ex.shutdown()
    res["workload"] = ("16384x16384, 8-conn, smoothed noise (seed 2, sigma 16) with a 1-px spiral corridor "
                       "(arm pitch 256) at the dtype maximum, marker the dtype minimum but 64 seeds; device time "
                       f"per reconstruction with the autotuned configuration, median of {args.spiral_reps}")
    return res


def run_ours(args):
    import numpy as np
    import torch
    from concurrent.futures import ThreadPoolExecutor

    import iwpp

    world, rank, local = _dist_env()
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl", init_method="env://")
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    variant = args.variant
    marker_np, mask_np, n_corridor = load_headline()
    H, W = mask_np.shape
    px = W * H
    bytes_per_recon = 3 * W * H * 1
    # the oracle (one host thread) runs while the GPU works: the CPU baseline
    # and the bit-exact check of the headline result
    oracle_ex = ThreadPoolExecutor(max_workers=1)
    oracle_fut = None
    if rank == 0 and not args.no_cpu:
        oracle_fut = oracle_ex.submit(timed_oracle, marker_np, mask_np, 8)

    mask = torch.from_numpy(mask_np).to(dev)
    pristine = torch.from_numpy(marker_np).to(dev)
    work = pristine.clone()
    handle = iwpp.Handle(local)
    lib = iwpp.load()
    stream = torch.cuda.Stream(dev)
    sptr = stream.cuda_stream
    vcode = iwpp._variant(variant)

    # the untuned default once, then the autotuner once for this image class
    # (its winner goes to the tuning table that the default calls below read)
    with torch.cuda.stream(stream):
        st_untuned = iwpp.reconstruct(work, mask, connectivity=8, variant=variant, handle=handle, stream=stream)
        work.copy_(pristine)
        # three repeats (median): the 2- and 3-pass candidates lie within 2 %
        tuned = iwpp.autotune([(work, mask, 8)], variant=variant, repeats=3, handle=handle, stream=stream)
    torch.cuda.synchronize()

    def step(ev_pair=None):
        work.copy_(pristine, non_blocking=True)
        if ev_pair is not None:
            ev_pair[0].record(stream)
        st = lib.iwpp_reconstruct_async(handle.ptr, work.data_ptr(), mask.data_ptr(), W, W, W, H, 0, 8, vcode, None,
                                        sptr)
        if st != 0:
            raise iwpp.IwppError(st, "iwpp_reconstruct_async")
        if ev_pair is not None:
            ev_pair[1].record(stream)

    with torch.cuda.stream(stream):
        for _ in range(max(args.warmup, 3)):
            step()
        stream.synchronize()
        result = work.cpu().numpy()
    fixed_point_ok = iwpp.fixed_point_violations(work, mask, 8) == 0

    # ---- device-resident timed region
    clocks = ClockSampler(local)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    t_start, t_end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    clocks.start()
    clocks.region_begin()
    with torch.cuda.stream(stream):
        t_start.record(stream)
        for k in range(args.steps):
            step(ev[k])
        t_end.record(stream)
    torch.cuda.synchronize()
    clocks.region_end()
    # a timed region shorter than a few sampling periods holds few samples:
    # the same reconstruction keeps running back to back, untimed, until
    # five samples were taken since the region began (at most 2 s)
    t_more = time.perf_counter()
    with torch.cuda.stream(stream):
        while clocks.since_begin() < 5 and time.perf_counter() - t_more < 2.0:
            for _ in range(8):
                step()
            stream.synchronize()
    clock_info = clocks.stop()
    if clock_info is not None:
        clock_info["window"] = ("the timed region, then the same reconstruction back to back (untimed) until "
                                "5 samples")
    elapsed_ms = t_start.elapsed_time(t_end)
    recon_ms = [a.elapsed_time(b) for a, b in ev]
    if world > 1:
        elapsed_ms = max_over_ranks(elapsed_ms, dev)
        torch.distributed.barrier()
    value = whole_job_gpx(world, px, args.steps, elapsed_ms)
    last = iwpp.Stats()
    if lib.iwpp_handle_sync(handle.ptr, __import__("ctypes").byref(last)) != 0:
        raise iwpp.IwppError(last.status, "iwpp_handle_sync")
    timed_ok = bool(np.array_equal(work.cpu().numpy(), result))

    # ---- serving sub-result before the copy-heavy end-to-end legs: the
    # host-to-device path of a shared box slows down for a while after them
    served = None
    if rank == 0 and not args.no_extras:
        try:
            served = bench_served(args, dev, variant)
        except Exception as exc:  # reported in the line, the headline stands
            served = {"error": f"{type(exc).__name__}: {exc}"}

    # ---- end to end: pinned host buffers in, host buffers out, every copy
    # inside the timed region, through the per-image C-ABI call; copies on
    # their own streams, two device buffer sets, so the next step's H2D and
    # the previous step's D2H overlap this step's reconstruction
    host_m = torch.from_numpy(marker_np).pin_memory()
    host_k = torch.from_numpy(mask_np).pin_memory()
    host_out = [torch.empty((H, W), dtype=torch.uint8, pin_memory=True) for _ in range(2)]
    s_in, s_run, s_out = (torch.cuda.Stream(dev) for _ in range(3))
    dmb = [torch.empty((H, W), dtype=torch.uint8, device=dev) for _ in range(2)]
    dkb = [torch.empty((H, W), dtype=torch.uint8, device=dev) for _ in range(2)]
    ev_in = [torch.cuda.Event() for _ in range(2)]
    ev_run = [torch.cuda.Event() for _ in range(2)]
    ev_out = [torch.cuda.Event() for _ in range(2)]
    for e in ev_out:
        e.record(s_out)

    def e2e_step(k, finish):
        b = k & 1
        with torch.cuda.stream(s_in):
            s_in.wait_event(ev_out[b])  # buffer b's previous result is home
            dmb[b].copy_(host_m, non_blocking=True)
            dkb[b].copy_(host_k, non_blocking=True)
            ev_in[b].record(s_in)
        s_run.wait_event(ev_in[b])
        st = lib.iwpp_reconstruct_async(handle.ptr, dmb[b].data_ptr(), dkb[b].data_ptr(), W, W, W, H, 0, 8, vcode,
                                        None, s_run.cuda_stream)
        if st != 0:
            raise iwpp.IwppError(st, "iwpp_reconstruct_async")
        ev_run[b].record(s_run)
        with torch.cuda.stream(s_out):
            s_out.wait_event(ev_run[b])
            host_out[b].copy_(dmb[b], non_blocking=True)
            ev_out[b].record(s_out)
        if finish:
            s_out.synchronize()
            st = lib.iwpp_handle_sync(handle.ptr, None)
            if st != 0:
                raise iwpp.IwppError(st, "iwpp_handle_sync")

    for k in range(max(args.warmup, 3)):
        e2e_step(k, k == max(args.warmup, 3) - 1)
    e2e_steps = min(args.steps, 30)  # bounded copy volume; the rate is per step
    for o in host_out:
        o.zero_()
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for k in range(e2e_steps):
        e2e_step(k, k == e2e_steps - 1)
    e2e_secs = time.perf_counter() - t0
    if world > 1:
        e2e_secs = max_over_ranks(e2e_secs, dev)
    e2e_ok = all(np.array_equal(o.numpy(), result) for o in host_out)
    e2e = {"value": whole_job_gpx(world, px, e2e_steps, e2e_secs * 1e3), "unit": UNIT,
           "h2d_bytes_per_step": 2 * W * H, "d2h_bytes_per_step": W * H,
           "path": "iwpp_reconstruct_async per step from pinned host buffers: H2D / reconstruction / D2H on three "
                   "streams, two device buffer sets, steps back to back (one host wait at the end)",
           "steps": e2e_steps, "bitexact_vs_device_path": e2e_ok}
    del dmb, dkb
    torch.cuda.empty_cache()

    if rank != 0:
        handle.close()
        if world > 1:
            torch.distributed.destroy_process_group()
        return 0
    extras = {}
    if not args.no_extras:
        for key, fn in (("config1", bench_config1), ("batched", None), ("spiral_types", bench_spiral_types)):
            try:
                extras[key] = fn(args, dev, variant, handle) if fn else bench_batched(args, dev, variant)
            except Exception as exc:  # reported in the line, the headline stands
                extras[key] = {"error": f"{type(exc).__name__}: {exc}"}
    cpu = None
    bitexact = None
    if oracle_fut is not None:
        ref, cpu_secs = oracle_fut.result()
        bitexact = bool(np.array_equal(result, ref))
        cpu = {"value": px / cpu_secs / 1e9, "unit": UNIT, "cores": 1, "kind": "port",
               "sample": "the same 16384x16384 uint8 spiral reconstruction once, oracle (Vincent 1993 hybrid), one "
                         f"host thread ({cpu_secs:.1f} s)"}
    oracle_ex.shutdown()
    peak, peak_kind = peak_hbm()
    mean_recon_ms = sum(recon_ms) / len(recon_ms)
    achieved = bytes_per_recon / (mean_recon_ms / 1e3) / 1e9
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": max(args.warmup, 3), "ms_per_step": elapsed_ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u8", "data": "synthetic",
        "config": {"workload": WORKLOAD, "variant": variant,
                   "autotuned": {k_: tuned[k_] for k_ in ("tile_rows", "solver", "init_passes", "front_passes")},
                   "l2": "inputs larger than L2: working + pristine marker + mask = 805 MB per step",
                   "inputs_sha256": {"marker": inputs_sha256(marker_np), "mask": inputs_sha256(mask_np)},
                   "parallelism": f"replicas x{world}" if world > 1 else "single GPU"},
        "bitexact": bitexact, "bitexact_timed_steps": timed_ok, "fixed_point": fixed_point_ok,
        "untuned_ms": st_untuned.device_ms,
        "reconstruction": {"tiles": last.tiles, "visits": last.visits, "top_pixels": last.top_pixels,
                           "front_stage": last.front_stage,
                           "launches": last.launches, "corridor_pixels": n_corridor},
        "e2e": e2e,
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "traffic": traffic_from_profile("headline"), "peak_source": peak_kind,
                     "kernel": "one reconstruction: all of libiwpp's kernels of the call (front stage, check, "
                               "engine init, tile engine), events around the call on its stream",
                     "algorithmic_bytes_per_launch": bytes_per_recon, "mean_launch_ms": mean_recon_ms},
        "cpu_baseline": cpu,
        "clocks": clock_info,
        "gpu_launches": args.steps * int(last.launches),
    }
    handle.close()
    if served is not None:
        line["served"] = served
    line.update(extras)
    print(json.dumps(line), flush=True)
    if world > 1:
        torch.distributed.destroy_process_group()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--variant", default="async", choices=["mutex", "double", "unique", "async"])
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline / bit-exact checks")
    ap.add_argument("--no-extras", action="store_true",
                    help="only the headline line (no config1 / batched / served / spiral-type sub-results)")
    ap.add_argument("--served-requests", type=int, default=4000)
    ap.add_argument("--served-pool", type=int, default=128,
                    help="distinct generated image pairs the served requests draw from")
    ap.add_argument("--lanes", type=int, default=3)
    ap.add_argument("--spiral-reps", type=int, default=3)
    ap.add_argument("--config1-only", action="store_true",
                    help="only the six 4096^2 configuration-1 reconstructions with --variant (one JSON line)")
    ap.add_argument("--config1-solver", type=int, default=None, choices=[0, 1, 2, 3],
                    help="with --config1-only: every call with this in-tile solver (the configuration the "
                         "autotuner picks, without its launches before the profiled ones)")
    ap.add_argument("--config1-tile-rows", type=int, default=0, choices=[0, 32, 64],
                    help="with --config1-solver: the tile height as well (0: the default)")
    ap.add_argument("--profile-headline", type=int, default=0, metavar="N",
                    help="only N reconstructions of the headline image with the front stage (for profilers)")
    ap.add_argument("--profile-passes", type=int, default=None,
                    help="whole-image passes of the front stage in --profile-headline (default: the untuned call)")
    args = ap.parse_args()
    if args.impl == "reference":
        return run_reference(args)
    import __graft_entry__ as ge

    ge.build()
    if args.config1_only:
        return run_config1_only(args)
    if args.profile_headline > 0:
        return run_profile_headline(args)
    return run_ours(args)


def run_profile_headline(args):
    """N reconstructions of the headline image in the untuned configuration
    (which the autotuner picks for this image class in a plain run; under a
    profiler, which serialises and replays every launch, its timings could
    pick another), or with the front stage and --profile-passes whole-image
    passes, and --variant, each from the pristine marker, nothing else."""
    import torch

    import iwpp

    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    marker_np, mask_np, _ = load_headline()
    mask = torch.from_numpy(mask_np).to(dev)
    pristine = torch.from_numpy(marker_np).to(dev)
    work = pristine.clone()
    cfg = iwpp.Config.make()
    if args.profile_passes is not None:
        cfg = iwpp.Config.make(front_passes=1, init_passes=args.profile_passes)
    for i in range(args.profile_headline):
        work.copy_(pristine)
        torch.cuda.synchronize()
        st = iwpp.reconstruct(work, mask, connectivity=8, variant=args.variant, config=cfg)
        print(json.dumps({"call": i, "device_ms": st.device_ms, "launches": st.launches, "visits": st.visits,
                          "front_stage": st.front_stage, "status": st.status}), flush=True)
    return 0


def run_config1_only(args):
    """The configuration-1 sub-result alone, for one queue variant (the form
    the per-variant profiles are captured with)."""
    import torch

    import iwpp

    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    handle = iwpp.Handle(0)
    res = bench_config1(args, dev, args.variant, handle, tune=False)
    handle.close()
    print(json.dumps({"config1": res}), flush=True)
    return 0


if __name__ == "__main__":
    sys.exit(main())
