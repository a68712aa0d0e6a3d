"""Benchmark: Mpix/s to the bit-exact min cut on one (or N) B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--config single|batch|strokes|serving] [--size 2048]

A step is one solve of one synthetic grid: capacities already resident in HBM (row-major
int32 planes) -> tile upload -> push-relabel with global relabels -> canonical cut flood
-> labels in a device buffer + the flow value on the host.  `value` is the whole-job
throughput (pixels solved by all ranks / max-over-ranks device time), timed with CUDA
events on the solver's stream; L2 is flushed (256 MiB write) between steps, outside the
timed region.  `e2e` is the same metric through the public API with host buffers: every
step copies the pinned RGBA image and t-link plane to the device, builds the graph there
(GraphCut.upload_image, n-links on the device), solves, and reads the flow and the
bit-packed cut back (pipeline.SolvePipeline, which overlaps step k+1's copies with step
k's solve); `e2e_serial` runs the same calls one step after another.
`e2e_image_and_models` starts one step earlier, from the image and the two colour models
(t-links from gmm_tlinks.tlinks).

Workload (`--config single`, the default): one 2048x2048 grid per rank built as in the
synthetic generator (12 blurred ellipses + noise, 2-component GMM t-links, exp n-links),
seed 1 + rank.  Multi-GPU runs are replicas (one independent grid per rank, weak scaling);
a single grid is not split across GPUs.

`--impl reference` times the reference schedule restated on the CPU (the oracle's
ref_tiled: GraphCut.cut + graphcut.cl in int32, OpenMP over tiles) on rank 0 with all host
threads, on the same workload and metric.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "cl-util_b200")
for _p in (PKG, ROOT):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import numpy as np  # noqa: E402

METRIC = "Mpix/s at bit-exact min cut"
UNIT = "Mpix/s"

# Algorithmic bytes per tile (32x32 pixels, int32 planes) of each kernel kind: the bytes a
# kernel must move for one tile, counting each plane it reads or writes once.
ALGO_BYTES_PER_TILE = {
    "upload": 1024 * 4 * (5 + 7),          # read 5 row-major planes, write 7 tile planes
    "discharge": 1024 * 4 * (6 + 6) + 4 * 32 * 4,  # read+write excess/height/4 caps, halo
    "edge_relabel_build": 124 * 4 * 2 + 16,  # edge excess+height, flags
    "masks": 1024 * 4 * 5 + 6 * 128 + 8,              # 5 planes in, 6 row masks + tile sum out
    "bfs_first": 6 * 128 + 1024 * 4,                  # masks in, distances out
    "bfs": 5 * 128 + 4 * 128 + 2 * 1024 * 4,          # masks, halo, distances in/out
    "flood_first": 1024 * 4 + 5 * 128 + 128,
    "flood": 5 * 128 + 4 * 256 + 128,
    "compact": 8,
    "labels": 1024 * 1 + 128,
}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--config", default="single",
                    choices=["single", "batch", "strokes", "serving"])
    ap.add_argument("--batch", type=int, default=64, help="grids in --config batch")
    ap.add_argument("--strokes", type=int, default=200, help="strokes in --config strokes")
    ap.add_argument("--size", type=int, default=2048)
    ap.add_argument("--duration", type=float, default=60.0, help="seconds of --config serving trace")
    ap.add_argument("--rate", type=float, default=200.0, help="requests/s of --config serving")
    ap.add_argument("--slots", type=int, default=1,
                    help="requests in flight, --config serving; only 1 is accepted (more "
                         "raised an intermittent device fault whose cause is not found)")
    ap.add_argument("--verify-s", type=float, default=90.0,
                    help="wall-time cap of the --config serving result verification")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--profile-solve", action="store_true",
                    help="warm up, then run one host-driven solve of the --size grid inside the "
                         "NVTX range 'profiled_solve' and print its per-kernel launches and "
                         "tiles (the command the ncu summaries are made from)")
    ap.add_argument("--profile-models", action="store_true",
                    help="one gc_tlinks_gmm launch on the --size image (two 2-component "
                         "full-covariance models) and one gc_gmm_fit launch (10000 samples, 4 "
                         "components, 65 iterations), after a warm-up of each: the command the "
                         "ncu summaries of those two kernels are made from")
    ap.add_argument("--host-driven", action="store_true",
                    help="solve loops decided by the host (use_graph=0); ncu does not profile "
                         "the steps of the one-launch solve apart, so profiling runs use this")
    return ap.parse_args()


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled every 200 ms during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
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
            time.sleep(0.25)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        if not self.lines:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax = float(parts[2])
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples": len(sm)}


def measured_peak():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def ncu_traffic():
    """DRAM bytes per tile of each kernel kind from the committed ncu summary (or {})."""
    path = os.path.join(ROOT, "profiles", "dram_traffic_per_tile.txt")
    try:
        with open(path) as f:
            return json.loads("".join(l for l in f if not l.startswith("#")))
    except Exception:
        return {}


def time_gmm_fit(g, stream, with_cpu):
    """The colour-model fit of the reference's own fit test (test_GMM.py:58-67: 20x500 = 10000
    samples, 4 components, 65 iterations, likelihood test 0.01), here on the pixels of the
    largest ellipse of the bench image: gc_gmm_fit's device time (CUDA events on its stream,
    one launch) and, as its CPU baseline, the float64 numpy restatement of the same EM."""
    import ctypes

    import torch

    import _gcut
    from GraphCut import _as_rgba32
    img = g.image
    h, w = img.shape[:2]
    rgba = _as_rgba32(img)
    # samples: a 20x500 window around the image centre (the reference test's rectangle shape)
    y0, x0 = h // 2 - 10, max(0, w // 2 - 250)
    s = np.ascontiguousarray(rgba[y0:y0 + 20, x0:x0 + 500]).reshape(-1)
    d = torch.from_numpy(s.view(np.int32)).cuda()
    res = torch.empty(ctypes.sizeof(_gcut.GcGmmFitResult), dtype=torch.uint8, device="cuda")
    L = _gcut.lib()
    ms = []
    for rep in range(6):
        ev0 = torch.cuda.Event(enable_timing=True)
        ev1 = torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        _gcut.check(L.gc_gmm_fit(_gcut.ptr(d), s.size, 4, 65, 0.01, 1e-3, 30.0, 0,
                                 _gcut.ptr(res), _gcut.stream_handle(stream)))
        ev1.record(stream)
        ev1.synchronize()
        if rep >= 2:
            ms.append(ev0.elapsed_time(ev1))
    r = _gcut.GcGmmFitResult.from_buffer_copy(res.cpu().numpy().tobytes())
    out = {"samples": int(s.size), "components": 4, "max_iterations": 65,
           "iterations": int(r.iterations), "converged": bool(r.converged),
           "ms": sum(ms) / len(ms), "launches": 1}
    if with_cpu:
        from oracle import oracle as O
        t0 = time.perf_counter()
        ref = O.gmm_fit(s, 4, 65, tolerance=0.01)
        out["cpu_baseline_ms"] = 1000 * (time.perf_counter() - t0)
        out["cpu_baseline"] = "float64 numpy EM restatement (oracle gmm_fit), 1 process"
        out["parity"] = bool(ref["iterations"] == r.iterations and np.allclose(
            ref["means"], np.array([list(r.means[k]) for k in range(4)]), rtol=1e-7, atol=1e-7))
    return out


def _cpu_build():
    from oracle import oracle as O
    return "-O3 -march=native (built on this host)" if O.native_lib() else \
        "-O3 -march=x86-64-v2 (portable build)"


# What pins the port to the reference's own code (tests/test_refcl_golden.py).
PORT_PINNED = ("ends in the same cut after the same push iterations and relabel passes as "
               "the reference's graphcut.cl run under its host loop")


def cpu_baseline(graph, threads, budget_s=12.0):
    """The reference schedule restated (oracle ref_tiled) on the host cores, built for this
    host's CPU."""
    from oracle import oracle as O
    build = _cpu_build()
    reps, t_total = 0, 0.0
    while t_total < budget_s and reps < 50:
        t0 = time.perf_counter()
        O.ref_tiled(*graph.planes(), bfs=5, threads=threads, native=True)
        t_total += time.perf_counter() - t0
        reps += 1
    mpix = graph.width * graph.height / 1e6
    return {"value": reps * mpix / t_total, "unit": UNIT, "cores": threads, "kind": "port",
            "build": build, "pinned": PORT_PINNED,
            "sample": f"{reps} full solves of the {graph.width}x{graph.height} grid "
                      f"({t_total:.1f} s), oracle ref_tiled (GraphCut.cut + graphcut.cl "
                      f"restated, int32, OpenMP)"}


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import synth
    threads = os.cpu_count() or 1
    g = synth.make_graph(args.size, args.size, 1)
    from oracle import oracle as O
    build = _cpu_build()
    for _ in range(max(1, args.warmup)):
        O.ref_tiled(*g.planes(), bfs=5, threads=threads, native=True)
    times = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        O.ref_tiled(*g.planes(), bfs=5, threads=threads, native=True)
        times.append(time.perf_counter() - t0)
    mpix = g.width * g.height / 1e6
    ms = 1000 * statistics.mean(times)
    value = mpix / (ms / 1000)
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT,
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
        "data": "synthetic",
        "config": {"workload": f"single {args.size}x{args.size} synthetic segmentation grid, seed 1",
                   "impl": "oracle ref_tiled: the reference schedule (GraphCut.pyx:348-418 + "
                           "graphcut.cl) restated in int32 C++, OpenMP over tiles"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "build": build, "pinned": PORT_PINNED,
                         "sample": f"{args.steps} full solves of the {args.size}^2 grid"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def spawn_ranks(args):
    """`--gpus N` without a launcher: re-run this command under torch.distributed.run with N
    processes on this node (one per GPU, rendezvous on 127.0.0.1) and return its exit code.
    The ranks print the JSON line (rank 0) exactly as under an external torchrun."""
    import socket

    import torch
    if torch.cuda.device_count() < args.gpus:
        sys.exit(f"bench.py: --gpus {args.gpus} needs {args.gpus} GPUs, "
                 f"{torch.cuda.device_count()} visible")
    with socket.socket() as so:
        so.bind(("127.0.0.1", 0))
        port = so.getsockname()[1]
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1",
           f"--nproc-per-node={args.gpus}", "--master-addr=127.0.0.1", f"--master-port={port}",
           os.path.abspath(__file__), *sys.argv[1:]]
    return subprocess.call(cmd)


def main():
    args = parse()
    if args.gpus > 1 and "WORLD_SIZE" not in os.environ:
        sys.exit(spawn_ranks(args))
    if args.slots != 1:
        sys.exit("bench.py: --slots must be 1 (concurrent serving slots raised an "
                 "intermittent device fault whose cause is not found)")
    if args.impl == "reference":
        return run_reference(args)
    if args.config == "batch":
        return run_batch(args)
    if args.config == "strokes":
        return run_strokes(args)
    if args.config == "serving":
        return run_serving(args)
    if args.profile_solve:
        return run_profile_solve(args)
    if args.profile_models:
        return run_profile_models(args)
    import torch
    import torch.distributed as dist

    import synth
    from GraphCut import GraphCut
    from sharding import reduce_max

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))

    def barrier():
        if world > 1:
            dist.barrier()

    W = H = args.size
    g = synth.make_graph(W, H, 1 + rank, keep_image=True)
    dev_planes = [torch.from_numpy(p).cuda() for p in g.planes()]
    stream = torch.cuda.Stream()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    labels = torch.empty((H, W), dtype=torch.uint8, device="cuda")
    gc = GraphCut(W, H, device=local, use_graph=not args.host_driven)

    def step():
        gc.upload_capacities(*dev_planes, stream=stream)
        gc.cut_labels(out=labels, stream=stream)   # solve + labels, one host wait
        return gc.flow

    with torch.cuda.stream(stream):
        for _ in range(max(3, args.warmup)):
            flow = step()
        stream.synchronize()
        # parity of this workload against the oracle (outside the timed region)
        lab = labels.cpu().numpy()
        from oracle import oracle as O
        f_ref, l_ref = O.maxflow_bk(*g.planes())
        parity = bool(flow == f_ref and np.array_equal(lab, l_ref))

        # timed region: one launch per solve (profiling off)
        step_ms = []
        launches = 0
        clocks = ClockSampler(local)
        barrier()
        torch.cuda.synchronize()
        with clocks:
            for _ in range(args.steps):
                flush.fill_(1)
                ev0 = torch.cuda.Event(enable_timing=True)
                ev1 = torch.cuda.Event(enable_timing=True)
                ev0.record(stream)
                step()
                ev1.record(stream)
                ev1.synchronize()
                step_ms.append(ev0.elapsed_time(ev1))
                # the upload and the solve, which writes the labels itself; the host-driven
                # loop launches every step, and the labels
                launches += 2 if not args.host_driven else gc.stats()["launches"] + 2
        torch.cuda.synchronize()
        barrier()
        total_ms = reduce_max(sum(step_ms), torch.device("cuda", local))
        mpix_all = world * args.steps * W * H / 1e6
        value = mpix_all / (total_ms / 1000)

        # the timeline from the device-side trace (start stamps of the steps inside the one
        # launch, which host profilers do not list): one solve, outside the timed region
        import _gcut
        gc.set_trace(True, stream=stream)
        step()   # a first traced step, not part of the timeline
        flush.fill_(1)
        stream.synchronize()
        gc.set_trace(True, stream=stream)   # a fresh trace
        step()
        trace = gc.trace(stream=stream)
        gc.set_trace(False, stream=stream)
        timeline = {k: [v[0], round(v[1] / 1000, 2)] for k, v in _gcut.trace_summary(trace).items()}
        timeline_total = round((trace[-1][1] - trace[0][1]) / 1000, 2) if len(trace) > 1 else None

        # per-kernel CUDA-event timing (host-driven loop, same kernels) for the roofline
        gc.set_profile(True)
        prof_tot = {}
        prof_ms = []
        for _ in range(args.steps):
            flush.fill_(1)
            ev0 = torch.cuda.Event(enable_timing=True)
            ev1 = torch.cuda.Event(enable_timing=True)
            ev0.record(stream)
            step()
            ev1.record(stream)
            ev1.synchronize()
            prof_ms.append(ev0.elapsed_time(ev1))
            for k, v in gc.profile().items():
                acc = prof_tot.setdefault(k, {"launches": 0, "ms": 0.0, "tiles": 0})
                for f in acc:
                    acc[f] += v[f]
        gc.set_profile(False)

        # e2e through the public API with host buffers
        e2e = e2e_serial = e2e_models = None
        if not args.no_e2e:
            # the reference's own inputs: the RGBA image (n-links are built on the device)
            # and the t-link plane, from pinned host memory; the cut comes back bit-packed
            from GraphCut import _as_rgba32, unpack_labels
            from pipeline import SolvePipeline
            rgba_pin = torch.from_numpy(np.ascontiguousarray(_as_rgba32(g.image))).pin_memory()
            exc_pin = torch.from_numpy(g.excess).pin_memory()
            rgba_host, exc_host = rgba_pin.numpy(), exc_pin.numpy()
            bits_host = torch.empty((H, (W + 7) // 8), dtype=torch.uint8).pin_memory().numpy()
            h2d, d2h = 2 * 4 * W * H, H * ((W + 7) // 8) + 8
            # pipelined: frame k+1's copies overlap frame k's solve (SolvePipeline)
            pipe = SolvePipeline(W, H, device=local)
            frames = [(rgba_host, exc_host)] * args.steps
            for fl, bits in pipe.run(frames[:3]):
                pass
            e2e_parity = bool(fl == f_ref and np.array_equal(unpack_labels(bits, W), l_ref))
            barrier()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            n_out = 0
            for fl, bits in pipe.run(frames):
                n_out += 1
            e_tot = reduce_max(1000 * (time.perf_counter() - t0), torch.device("cuda", local))
            e2e_parity &= bool(n_out == args.steps and fl == f_ref and
                               np.array_equal(unpack_labels(bits, W), l_ref))
            pipe.close()
            e2e = {"value": mpix_all / (e_tot / 1000), "unit": UNIT,
                   "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                   "ms_per_step": e_tot / args.steps, "parity": e2e_parity,
                   "api": "pipeline.SolvePipeline.run over pinned (RGBA, int32 t-links) frames: "
                          "per frame H2D copy, GraphCut.upload_image, cut, flow and packed "
                          "labels D2H; frame k+1's copies overlap frame k's solve"}
            # serial: one frame after another, every call blocking
            for _ in range(2):
                gc.upload_image(rgba_host, exc_host, stream=stream)
                gc.cut(stream=stream)
                gc.labels_packed_host(out=bits_host, stream=stream)
            s_parity = bool(gc.flow == f_ref and np.array_equal(unpack_labels(bits_host, W), l_ref))
            e_ms = []
            barrier()
            for _ in range(args.steps):
                flush.fill_(1)
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                gc.upload_image(rgba_host, exc_host, stream=stream)
                gc.cut(stream=stream)
                gc.labels_packed_host(out=bits_host, stream=stream)
                _ = gc.flow
                e_ms.append(1000 * (time.perf_counter() - t0))
            es_tot = reduce_max(sum(e_ms), torch.device("cuda", local))
            e2e_serial = {"value": mpix_all / (es_tot / 1000), "unit": UNIT,
                          "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                          "ms_per_step": es_tot / args.steps, "parity": s_parity,
                          "api": "GraphCut.upload_image (RGBA + int32 t-links, host) -> cut -> "
                                 "labels_packed_host + flow, one frame at a time, L2 flushed "
                                 "before each"}
            out_host = bits_host

            # one step further back in the reference's pipeline: the image and the two colour
            # models only (t-links from gc_tlinks_gmm, n-links from gc_upload_rgba; 4 B/px up)
            from gmm_tlinks import Mixture, tlinks
            models = tuple(Mixture.from_components(c) for c in g.models)
            rgba_pin32 = torch.from_numpy(
                np.ascontiguousarray(_as_rgba32(g.image)).view(np.int32)).pin_memory()
            rgba_dev = torch.empty((H, W), dtype=torch.int32, device="cuda")
            ex_dev = torch.empty((H, W), dtype=torch.int32, device="cuda")

            def model_step():
                rgba_dev.copy_(rgba_pin32, non_blocking=True)
                tlinks(rgba_dev, *models, out=ex_dev, stream=stream)
                gc.upload_image(rgba_dev, ex_dev, stream=stream)
                gc.cut(stream=stream)
                gc.labels_packed_host(out=out_host, stream=stream)
                return gc.flow

            for _ in range(2):
                fm = model_step()
            m_parity = bool(fm == f_ref and np.array_equal(unpack_labels(out_host, W), l_ref))
            m_ms = []
            barrier()
            for _ in range(args.steps):
                flush.fill_(1)
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                model_step()
                m_ms.append(1000 * (time.perf_counter() - t0))
            m_tot_serial = reduce_max(sum(m_ms), torch.device("cuda", local))
            # pipelined (SolvePipeline): frame k+1's image copy overlaps frame k's work
            pipe = SolvePipeline(W, H, device=local)
            mframes = [(rgba_host, models)] * args.steps
            for fm2, bits2 in pipe.run(mframes[:3]):
                pass
            m_parity &= bool(fm2 == f_ref and np.array_equal(unpack_labels(bits2, W), l_ref))
            barrier()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for fm2, bits2 in pipe.run(mframes):
                pass
            m_tot = reduce_max(1000 * (time.perf_counter() - t0), torch.device("cuda", local))
            m_parity &= bool(fm2 == f_ref and np.array_equal(unpack_labels(bits2, W), l_ref))
            pipe.close()
            # the t-link kernel alone (CUDA events on its stream, L2 flushed before each)
            tl_ms = []
            for _ in range(max(3, args.steps // 5)):
                flush.fill_(1)
                ev0 = torch.cuda.Event(enable_timing=True)
                ev1 = torch.cuda.Event(enable_timing=True)
                ev0.record(stream)
                tlinks(rgba_dev, *models, out=ex_dev, stream=stream)
                ev1.record(stream)
                ev1.synchronize()
                tl_ms.append(ev0.elapsed_time(ev1))
            tl_avg = sum(tl_ms) / len(tl_ms)
            e2e_models = {"value": mpix_all / (m_tot / 1000), "unit": UNIT,
                          "h2d_bytes_per_step": 4 * W * H, "d2h_bytes_per_step": d2h,
                          "ms_per_step": m_tot / args.steps, "parity": m_parity,
                          "serial_ms_per_step": m_tot_serial / args.steps,
                          "tlinks_gmm_ms": tl_avg,
                          "tlinks_gmm_gbs": 8 * W * H / (tl_avg / 1000) / 1e9,
                          "api": "pipeline.SolvePipeline.run over pinned (RGBA, (fg, bg) "
                                 "2-component full-covariance models) frames: per frame the "
                                 "image H2D, gmm_tlinks.tlinks, GraphCut.upload_image, cut, "
                                 "flow and packed labels D2H; serial_ms_per_step: the same "
                                 "calls one frame at a time"}
            e2e_models["gmm_fit"] = time_gmm_fit(g, stream, rank == 0 and world == 1
                                                 and not args.no_cpu_baseline)

    # roofline of the step's largest part: the upload by its span in the trace, a kind of solve
    # step by its event time as a kernel of its own (the host-driven loop's rounds that find
    # nothing to do would count there, so the choice is the trace's)
    peak, peak_kind = measured_peak()
    spans = {k: v for k, v in timeline.items() if k in ALGO_BYTES_PER_TILE}
    dname = max(spans, key=lambda k: spans[k][1]) if spans else "discharge"
    d = prof_tot.get(dname)
    if not d or not d["launches"]:
        n_dom, us_dom = spans.get(dname, [1, 0.0])
        d = {"launches": n_dom, "ms": us_dom / 1000, "tiles": n_dom * ((W + 31) // 32) * ((H + 31) // 32)}
    algo_bytes = d["tiles"] * ALGO_BYTES_PER_TILE.get(dname, 0)
    if dname == "compact":
        algo_bytes = d["launches"] * ((W // 32) * (H // 32)) * 8
    achieved = algo_bytes / (d["ms"] / 1000) / 1e9 if d["ms"] > 0 else 0.0
    traffic = None
    tr_all = ncu_traffic()
    if dname == "compact":
        traffic = tr_all.get("compact_per_launch")
    elif tr_all.get(dname) is not None and d["launches"]:
        traffic = tr_all[dname] * d["tiles"] / d["launches"]

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline(g, os.cpu_count() or 1)

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": max(3, args.warmup), "ms_per_step": total_ms / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
            "data": "synthetic",
            "config": {"workload": f"single {W}x{H} synthetic segmentation grid per GPU "
                                   "(12 blurred ellipses + N(0,8) noise, 2-component GMM "
                                   "t-links x100, 50*exp(-beta*dI^2) n-links), seed 1+rank",
                       "l2": "flushed between steps (256 MiB write, outside the timed region)",
                       "parallelism": f"replicas x{world}",
                       "loop": "host-driven" if args.host_driven else "one cooperative launch per solve",
                       "step": "GraphCut.upload_capacities from device planes, then "
                               "GraphCut.cut_labels (gc_solve_labels: the solve and the labels "
                               "into device memory, one host wait)",
                       "solver": {"discharge_iters": gc.opts.discharge_iters,
                                  "pulses_per_relabel": gc.opts.pulses_per_relabel,
                                  "initial_relabel": gc.opts.initial_relabel}},
            "parity": parity,
            "flow": flow,
            "e2e": e2e,
            "e2e_serial": e2e_serial,
            "e2e_image_and_models": e2e_models,
            "gpu_launches": launches,
            "ms_per_step_host_driven": sum(prof_ms) / len(prof_ms),
            "graph_timeline_us": {"kernels": timeline, "upload_start_to_labels_start": timeline_total,
                                  "how": "device-side trace of one solve: per step kind "
                                         "[steps, us from its start to the next step's start]"},
            "roofline": {"bound": "hbm", "kernel": dname, "achieved": achieved, "peak": peak,
                         "peak_kind": peak_kind, "unit": "GB/s",
                         "frac": achieved / peak if peak else None, "traffic": traffic,
                         # against the nominal HBM3e figure (8 TB/s), for context
                         "nominal_peak": 8000.0, "frac_of_nominal": achieved / 8000.0,
                         "algo_bytes_per_launch": algo_bytes / max(1, d["launches"]),
                         "avg_launch_us": 1000 * d["ms"] / max(1, d["launches"])},
            "kernels": {k: {"launches": v["launches"], "ms": round(v["ms"], 4), "tiles": v["tiles"]}
                        for k, v in prof_tot.items() if v["launches"]},
            "clocks": clocks.summary(),
            "cpu_baseline": cpu,
            "solve_stats": gc.stats(),
        }
        print(json.dumps(line), flush=True)
    gc.close()
    if world > 1:
        dist.destroy_process_group()


def run_profile_solve(args):
    """One host-driven solve of the --size synthetic grid (seed 1) in the NVTX range
    'profiled_solve', after `--warmup` solves; prints the per-kernel launches, tiles and
    event times of that solve.  ncu captures only that range (--nvtx --nvtx-include
    profiled_solve/), so launch lists and DRAM counters cover exactly one solve."""
    import torch

    import synth
    from GraphCut import GraphCut
    W = H = args.size
    g = synth.make_graph(W, H, 1)
    torch.cuda.set_device(0)
    planes = [torch.from_numpy(p).cuda() for p in g.planes()]
    labels = torch.empty((H, W), dtype=torch.uint8, device="cuda")
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    gc = GraphCut(W, H, use_graph=False)
    with torch.cuda.stream(stream):
        for _ in range(max(1, args.warmup)):
            gc.upload_capacities(*planes, stream=stream)
            gc.cut_labels(out=labels, stream=stream)
        flush.fill_(1)
        stream.synchronize()
        gc.set_profile(True)
        torch.cuda.nvtx.range_push("profiled_solve")
        gc.upload_capacities(*planes, stream=stream)
        gc.cut_labels(out=labels, stream=stream)
        stream.synchronize()
        torch.cuda.nvtx.range_pop()
        prof = gc.profile()
        gc.set_profile(False)
    print(json.dumps({"workload": f"{W}x{H} synthetic grid, seed 1, one host-driven solve",
                      "flow": gc.flow, "stats": gc.stats(),
                      "kernels": {k: v for k, v in prof.items() if v["launches"]}}), flush=True)
    gc.close()


def run_profile_models(args):
    """See --profile-models.  Prints the two kernels' CUDA-event times."""
    import torch

    import synth
    from gmm_tlinks import Mixture, tlinks
    from GraphCut import _as_rgba32
    W = H = args.size
    g = synth.make_graph(W, H, 1, keep_image=True)
    torch.cuda.set_device(0)
    stream = torch.cuda.Stream()
    rgba = torch.from_numpy(np.ascontiguousarray(_as_rgba32(g.image)).view(np.int32)).cuda()
    ex = torch.empty((H, W), dtype=torch.int32, device="cuda")
    models = tuple(Mixture.from_components(c) for c in g.models)
    with torch.cuda.stream(stream):
        tlinks(rgba, *models, out=ex, stream=stream)       # warm-up
        stream.synchronize()
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ev[0].record(stream)
        tlinks(rgba, *models, out=ex, stream=stream)
        ev[1].record(stream)
        ev[1].synchronize()
    fit = time_gmm_fit(g, stream, False)
    print(json.dumps({"tlinks_gmm_ms": ev[0].elapsed_time(ev[1]), "gmm_fit_ms": fit["ms"],
                      "size": [W, H], "fit": fit}), flush=True)


def _percentile(xs, p):
    return float(np.percentile(np.asarray(xs, dtype=np.float64), p))


def run_batch(args):
    """Config 2: `--batch` (64) independent grids, sides drawn from {256, 384, ..., 1536},
    solved together in one tile pool (one launch per solve over a shared tile
    worklist), against the same grids solved one at a time by the single-grid solver.
    Under torchrun each rank takes its LPT share of the grids (by pixel count); the job's
    time is the slowest rank's."""
    import torch
    import torch.distributed as dist

    import synth
    from GraphCut import GraphCut
    from GraphCutBatch import GraphCutBatch
    from oracle import oracle as O
    from sharding import lpt_assign, reduce_max, reduce_min
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))
    all_shapes = synth.batch_shapes(args.batch, seed=2)
    mine = lpt_assign([w * h for w, h in all_shapes], world)[rank]
    shapes = [all_shapes[i] for i in mine]
    graphs = synth.make_graphs([(all_shapes[i][0], all_shapes[i][1], 10_000 + i) for i in mine])
    planes = [[torch.from_numpy(p).cuda() for p in g.planes()] for g in graphs]
    mpix = sum(w * h for w, h in all_shapes) / 1e6
    stream = torch.cuda.Stream()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    labels = [torch.empty((h, w), dtype=torch.uint8, device="cuda") for w, h in shapes]
    b = GraphCutBatch(shapes, device=local)

    def step_batch():
        for i, pl in enumerate(planes):
            b.upload(i, *pl, stream=stream)
        b.cut(stream=stream)
        for i in range(len(shapes)):
            b.labels(i, out=labels[i], stream=stream)

    singles = [GraphCut(w, h, device=local) for w, h in shapes]

    def step_single():
        for i, (gc, pl) in enumerate(zip(singles, planes)):
            gc.upload_capacities(*pl, stream=stream)
            gc.cut(stream=stream)
            gc.labels(out=labels[i], stream=stream)

    def timed(fn):
        ms = []
        for _ in range(args.steps):
            flush.fill_(1)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            fn()
            e1.record(stream)
            e1.synchronize()
            ms.append(e0.elapsed_time(e1))
        return sum(ms) / len(ms)

    with torch.cuda.stream(stream):
        for _ in range(max(3, args.warmup)):
            step_batch()
            step_single()
        stream.synchronize()
        # parity: batch == per-image solves == oracle, bit-exact, every grid
        step_batch()
        stream.synchronize()
        bl = [(b.flow(i), labels[i].cpu().numpy()) for i in range(len(shapes))]
        parity = True
        for i, g in enumerate(graphs):
            f_ref, l_ref = O.maxflow_bk(*g.planes())
            parity &= bl[i][0] == f_ref and np.array_equal(bl[i][1], l_ref)
        if world > 1:
            dist.barrier()
        clocks = ClockSampler(local)
        with clocks:
            ms_batch = timed(step_batch)
        ms_single = timed(step_single)
        st = b.stats()
    dev = torch.device("cuda", local)
    ms_batch = reduce_max(ms_batch, dev)     # the job takes as long as its slowest rank
    ms_single = reduce_max(ms_single, dev)
    parity = reduce_min(1.0 if parity else 0.0, dev) > 0
    line = {
        "metric": METRIC + " (batched)", "value": mpix / (ms_batch / 1000), "unit": UNIT,
        "n_gpus": world, "steps": args.steps, "warmup": max(3, args.warmup), "ms_per_step": ms_batch,
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "int32",
        "data": "synthetic",
        "config": {"workload": f"{len(all_shapes)} independent grids, sides uniform in "
                               "{256,384,...,1536}, built as the synthetic generator, seeds "
                               "10000+i; one tile pool per rank, one launch a solve",
                   "total_mpix": mpix, "l2": "flushed between steps",
                   "parallelism": f"LPT split of the grids over {world} rank(s)"},
        "single_solver_one_at_a_time": {"value": mpix / (ms_single / 1000), "unit": UNIT,
                                         "ms_per_step": ms_single},
        "batch_over_single": ms_single / ms_batch,
        "parity": bool(parity), "solve_stats": st, "clocks": clocks.summary(),
    }
    b.close()
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def run_strokes(args):
    """Config 3: one 4096x4096 grid, then `--strokes` (200) sequential brush strokes (random
    polylines, radius 8-32, t-links set to +-10**6), each re-solved warm from the previous
    residual graph; latency per stroke (edit + solve + labels, CUDA events) and a cold solve
    of the same edited graph for every stroke (bit-exact check)."""
    import torch

    import strokes
    import synth
    from GraphCut import GraphCut
    from oracle import oracle as O
    W = H = args.size if args.size != 2048 else 4096
    g = synth.make_graph(W, H, 3)
    torch.cuda.set_device(0)
    planes = [torch.from_numpy(p).cuda() for p in g.planes()]
    stream = torch.cuda.Stream()
    rng = np.random.default_rng(77)
    strokes_list = [strokes.random_stroke(rng, W, H) for _ in range(args.strokes)]
    warm = GraphCut(W, H)
    cold = GraphCut(W, H)
    lab_w = torch.empty((H, W), dtype=torch.uint8, device="cuda")
    lab_c = torch.empty((H, W), dtype=torch.uint8, device="cuda")
    t_host = g.excess.copy()
    lat, cold_ms, mism = [], [], 0
    with torch.cuda.stream(stream):
        warm.upload_capacities(*planes, stream=stream)
        warm.cut(stream=stream)
        f0, l0 = O.maxflow_bk(*g.planes())
        parity0 = f0 == warm.flow and np.array_equal(warm.labels().cpu().numpy(), l0)
        checks = {0, len(strokes_list) // 2, len(strokes_list) - 1}
        oracle_ok = True
        clocks = ClockSampler(0)
        with clocks:
            for k, s in enumerate(strokes_list):
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                warm.edit_stroke(s.xs, s.ys, s.radius, s.value, stream=stream)
                warm.cut(stream=stream)
                warm.labels(out=lab_w, stream=stream)
                e1.record(stream)
                e1.synchronize()
                lat.append(e0.elapsed_time(e1))
                fw = warm.flow
                # cold solve of the same edited graph (not timed in the latency)
                t_host = strokes.apply(t_host, s)
                planes[4].copy_(torch.from_numpy(t_host))
                c0 = torch.cuda.Event(enable_timing=True)
                c1 = torch.cuda.Event(enable_timing=True)
                c0.record(stream)
                cold.upload_capacities(*planes, stream=stream)
                cold.cut(stream=stream)
                cold.labels(out=lab_c, stream=stream)
                c1.record(stream)
                c1.synchronize()
                cold_ms.append(c0.elapsed_time(c1))
                if fw != cold.flow or not torch.equal(lab_w, lab_c):
                    mism += 1
                if k in checks:
                    fr, lr = O.maxflow_bk(g.up, g.down, g.left, g.right, t_host)
                    oracle_ok &= fr == fw and np.array_equal(lab_w.cpu().numpy(), lr)
    mpix = W * H / 1e6
    line = {
        "metric": "p50/p99 stroke re-solve latency", "value": _percentile(lat, 99), "unit": "ms",
        "p50_ms": _percentile(lat, 50), "p99_ms": _percentile(lat, 99), "mean_ms": float(np.mean(lat)),
        "n_gpus": 1, "steps": len(lat), "warmup": 1, "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "int32", "data": "synthetic",
        "config": {"workload": f"{W}x{H} synthetic segmentation grid (seed 3) + {len(lat)} "
                               "random polyline strokes, radius 8-32, t-links +-10^6, warm "
                               "re-solve from the previous residual graph"},
        "warm_mpix_per_s": mpix / (np.mean(lat) / 1000),
        "cold_solve_ms_mean": float(np.mean(cold_ms)),
        "warm_vs_cold_mismatches": mism, "oracle_checks_ok": bool(oracle_ok and parity0),
        "clocks": clocks.summary(),
    }
    print(json.dumps(line), flush=True)


def serving_images(n=12, seed=4):
    """The image pool of --config serving: n grids with sides drawn uniformly from
    [256, 4096] (width and height independent), built as the synthetic generator, seeds
    20000+i, with their images.  New-image requests draw from this pool; each starts its own
    session."""
    import synth
    rng = np.random.default_rng(seed)
    shapes = [(int(rng.integers(256, 4097)), int(rng.integers(256, 4097))) for _ in range(n)]
    return synth.make_graphs([(w, h, 20_000 + i) for i, (w, h) in enumerate(shapes)],
                             keep_image=True)


def run_trace(graphs, host_planes, trace, server, budget, seed=5, solver_kw=None):
    """Replays a (time, kind, image) trace in real time against a server: "batching"
    (BatchingServer: continuous batching over one session pool) or "single"
    (GraphCutServer: one request at a time, one handle per session).  A stroke targets one
    of the 8 most recently opened sessions (random polyline, radius 8-32, t-links +-10**6).
    Returns (results, history, server counters, wall seconds)."""
    import strokes
    from serving import BatchingServer, GraphCutServer, NewImage, Stroke
    rng = np.random.default_rng(seed)
    if server == "batching":
        srv = BatchingServer(hbm_budget=budget, solver_kw=solver_kw)
    else:
        srv = GraphCutServer(slots=1, hbm_budget=budget, solver_kw=solver_kw)
    history = {}     # session -> (image index, [strokes in submission order])
    sid = 0
    t0 = time.perf_counter()
    for t, kind, img in trace:
        now = time.perf_counter() - t0
        if t > now:
            time.sleep(t - now)
        if kind == "image" or not history:
            history[sid] = (img, [])
            srv.submit(NewImage(sid, host_planes[img]), arrival=t0 + t)
            sid += 1
        else:
            recent = list(history)[-8:]
            target = recent[int(rng.integers(len(recent)))]
            g = graphs[history[target][0]]
            s = strokes.random_stroke(rng, g.width, g.height)
            history[target][1].append(s)
            srv.submit(Stroke(target, s.xs, s.ys, s.radius, s.value), arrival=t0 + t)
    srv.drain()
    wall = time.perf_counter() - t0
    results = sorted(srv.results, key=lambda r: r.arrival)
    counters = {"misses": srv.misses, "evictions": srv.evictions}
    if server == "batching":
        counters["launches"] = srv.ticks
        counters["requests_per_launch"] = len(results) / max(1, srv.ticks)
    srv.close()
    return results, history, counters, wall


def _latency_summary(results, wall):
    lat = {k: [r.latency_ms for r in results if r.kind == k] for k in ("image", "stroke")}
    big = [r.latency_ms for r in results if r.kind == "stroke" and r.pixels >= 3072 * 3072]
    svc = [1000.0 * (r.done - r.start) for r in results]
    pct = lambda xs, p: _percentile(xs, p) if xs else None  # noqa: E731
    first = min(r.arrival for r in results)
    last = max(r.done for r in results)
    return {
        "stroke_p50_ms": pct(lat["stroke"], 50), "stroke_p99_ms": pct(lat["stroke"], 99),
        "stroke_p99_ms_images_ge_3072sq": pct(big, 99), "strokes_on_images_ge_3072sq": len(big),
        "image_p50_ms": pct(lat["image"], 50), "image_p99_ms": pct(lat["image"], 99),
        "all_p50_ms": pct(lat["image"] + lat["stroke"], 50),
        "all_p99_ms": pct(lat["image"] + lat["stroke"], 99),
        "service_p50_ms": pct(svc, 50), "service_p99_ms": pct(svc, 99),
        "served_mpix_per_s": sum(r.pixels for r in results) / 1e6 / (last - first),
        "phases_p50_ms": {k: [round(_percentile([r.phases_ms[j] for r in results
                                                if r.kind == k], 50), 3) for j in range(3)]
                          for k in ("image", "stroke") if lat[k]},
        "phases": "(input upload or stroke edit, solve, labels to host) per request",
        "results": len(results), "images": len(lat["image"]), "strokes": len(lat["stroke"]),
        "wall_s": wall,
    }


def verify_results(graphs, dev_planes, results, history, cap_s):
    """Checks results against cold solves of the same edited graph (host stroke raster,
    fresh upload, one solve), session by session in random order, until cap_s seconds.
    Returns (checked, mismatches, examples)."""
    import torch

    import strokes
    from GraphCut import GraphCut
    by_session = {}
    for r in results:
        by_session.setdefault(r.session, []).append(r)
    order = list(by_session)
    np.random.default_rng(9).shuffle(order)
    cold = {}
    checked, bad, examples = 0, 0, []
    t0 = time.perf_counter()
    for sid in order:
        if time.perf_counter() - t0 > cap_s:
            break
        img, strks = history[sid]
        g = graphs[img]
        key = (g.width, g.height)
        if key not in cold:
            cold[key] = GraphCut(g.width, g.height)
        gc = cold[key]
        t = g.excess.copy()
        for k, r in enumerate(by_session[sid]):   # the k-th result follows the first k strokes
            if k:
                t = strokes.apply(t, strks[k - 1])
            pl = list(dev_planes[img][:4]) + [torch.from_numpy(t).cuda()]
            gc.upload_capacities(*pl)
            gc.cut()
            f, lab = gc.flow, gc.labels_host()
            checked += 1
            if f != r.flow or not np.array_equal(lab, r.labels):
                bad += 1
                if len(examples) < 5:
                    examples.append({"session": sid, "kind": r.kind, "k": k, "flow": r.flow,
                                     "cold": f, "size": list(key)})
    for gc in cold.values():
        gc.close()
    return checked, bad, examples


def run_serving(args):
    """Config 4: a Poisson request stream (`--rate` 200 req/s for `--duration` 60 s), 30 %
    new images (sides uniform in [256, 4096]) and 70 % brush strokes on resident sessions,
    served with continuous batching (BatchingServer: every session in one session pool under
    a 64 GiB HBM budget, each tick solves all ready requests in one launch), then the same
    trace served by the plain one-at-a-time solver (GraphCutServer, one handle per session).
    Latency = result on the host - arrival; every request's inputs come from pinned host
    memory and its labels go back to host memory.  A time-capped sample of the results
    (whole sessions) is checked bit-exactly against cold solves."""
    import torch

    from serving import poisson_trace
    from GraphCut import _as_rgba32
    graphs = serving_images()
    torch.cuda.set_device(0)
    # requests carry the reference's inputs: the image and the t-links (8 B/px); the device
    # builds the n-links, which equal the generator's planes the results are checked against
    pinned = [[torch.from_numpy(np.ascontiguousarray(_as_rgba32(g.image)).view(np.int32)).pin_memory(),
               torch.from_numpy(g.excess).pin_memory()] for g in graphs]
    host_planes = [(pl[0].numpy().view(np.uint32), pl[1].numpy()) for pl in pinned]
    dev_planes = [[torch.from_numpy(p).cuda() for p in g.planes()] for g in graphs]
    trace = poisson_trace(np.random.default_rng(6), args.rate, args.duration, len(graphs))
    budget = 64 << 30
    # warm-up: an untimed trace of another seed (up to 15 s): the first launches and pinned
    # allocations of a process are start-up, not serving
    warm = poisson_trace(np.random.default_rng(7), args.rate, min(args.duration, 15.0),
                         len(graphs))
    run_trace(graphs, host_planes, warm, "batching", budget, seed=8)
    clocks = ClockSampler(0)
    with clocks:
        res, hist, cnt, wall = run_trace(graphs, host_planes, trace, "batching", budget)
    main_sum = _latency_summary(res, wall)
    run_trace(graphs, host_planes, warm, "single", budget, seed=8)
    res1, hist1, cnt1, wall1 = run_trace(graphs, host_planes, trace, "single", budget)
    one_sum = _latency_summary(res1, wall1)
    checked, bad, examples = verify_results(graphs, dev_planes, res, hist, args.verify_s)
    line = {
        "metric": "p99 stroke re-solve latency, mixed-size load", "value": main_sum["stroke_p99_ms"],
        "unit": "ms", "n_gpus": 1, "steps": len(trace), "warmup": len(warm),
        "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
        "data": "synthetic",
        "config": {"workload": f"Poisson {args.rate:g} req/s for {args.duration:g} s: 30% new "
                               "image (pool of 12 synthetic grids, sides uniform in [256, 4096], "
                               "seeds 20000+i; each request opens its own session), 70% stroke "
                               "(radius 8-32, t-links +-10^6) on one of the 8 newest sessions",
                   "server": "continuous batching (BatchingServer, one session pool, one "
                             "launch per tick)", "hbm_budget_gib": budget >> 30,
                   "latency": "arrival to labels in host memory (queueing included)"},
        **main_sum, **cnt,
        "one_at_a_time": {**one_sum, **cnt1},
        "verified_results": checked, "mismatches": bad, "mismatch_examples": examples,
        "clocks": clocks.summary(),
    }
    print(json.dumps(line), flush=True)


if __name__ == "__main__":
    main()
