#!/usr/bin/env python3
"""STRIDE decode benchmark: one JSON line per run.

Workloads (``--workload``):
  heightfield   (default) one 2049 x 2049 heightfield mesh, 8,388,608
                triangles, 12-bit bbox quantisation (``--bits``), seeded
                value-noise heights, encoded by the project encoder.  One step
                = one decode of the whole stream (the scan kernel, then one
                fused connectivity + vertex kernel: one stride_decode call)
                into resident device buffers.
  icosphere     the level-8 displaced icosphere (1,310,720 triangles).
  batch         many meshes with log-uniform sizes decoded in one persistent
                launch (CUDA graph), next to per-mesh launches.
  serve         Poisson arrivals into the continuous-batching server.

Metric: decoded triangles per second (M tris/s).  ``value`` is device time
of the decode with the stream already in HBM and L2 flushed before every step
(a 256 MiB write, not timed); ``e2e`` goes through the public
ParaDeltaV5GpuDecoder API with pinned host buffers (upload, decode, download,
synchronise each step).  ``roofline`` relates the dominant kernel's duration
(CUDA events around each kernel, from separate untimed decodes) to the
measured HBM copy bandwidth; ``cpu_baseline`` times the CPU oracle (a C
restatement of the reference decoder) on all host cores.

``--impl reference`` times the CPU decoder (oracle) alone on the same
workload and prints the reference line.  Multi-GPU (torchrun): every rank
decodes its own replica; the step time is the max over ranks.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, REPO)

from meshpress_gb300 import encoder, synth  # noqa: E402

WORKLOADS = ("heightfield", "icosphere", "batch", "serve")


def parse_args(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=("ours", "reference"))
    ap.add_argument("--workload", default="heightfield", choices=WORKLOADS)
    ap.add_argument("--bits", type=int, default=12)
    ap.add_argument("--grid", type=int, default=2049)
    ap.add_argument("--tune", type=int, default=1, help="autotune the launch shape before timing")
    ap.add_argument("--shape", default=None,
                    help="launch shape warps_per_cta,persistent[,stage_bytes,code_bytes] instead of autotuning "
                         "(single-mesh workloads)")
    ap.add_argument("--batch-meshes", type=int, default=4096)
    ap.add_argument("--rates", default="50,100,200,500,1000,2000", help="serve: Poisson arrival rates (requests/s)")
    ap.add_argument("--serve-host-rate", type=float, default=500.0,
                    help="serve: one more pass at this rate with every response copied to host memory (0 = none)")
    ap.add_argument("--serve-seconds", type=float, default=3.0, help="serve: arrivals per rate span this long")
    ap.add_argument("--serve-pool", type=int, default=48, help="serve: distinct encoded blobs drawn from")
    ap.add_argument("--serve-budget-gb", type=int, default=40)
    ap.add_argument("--serve-burst", default="64,512",
                    help="serve: saturating passes that queue this many requests at once, then let the server "
                         "run them ('' = none)")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--write-stream", default=None, help=argparse.SUPPRESS)  # encode a workload's stream to a file
    ap.add_argument("--no-cpu-baseline", action="store_true")
    return ap.parse_args(argv)


# ---------------------------------------------------------------------------
# distributed helpers (replicas only: no data-path collective)
# ---------------------------------------------------------------------------
def dist_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("LOCAL_RANK", 0)), int(os.environ.get("WORLD_SIZE", 1))


def dist_init(backend: str):
    import torch.distributed as dist
    rank, local, world = dist_env()
    if world > 1 and not dist.is_initialized():
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        dist.init_process_group(backend=backend, rank=rank, world_size=world)
    return rank, local, world


def reduce_max(x: float, device=None) -> float:
    import torch
    import torch.distributed as dist
    if not (dist.is_available() and dist.is_initialized()):
        return float(x)
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(device=None):
    import torch.distributed as dist
    if dist.is_available() and dist.is_initialized():
        if device is not None:
            dist.barrier(device_ids=[device.index])
        else:
            dist.barrier()


def replica_value(units_per_rank: int, world: int, max_seconds: float) -> float:
    """Whole-job throughput of ``world`` replicas: all units / slowest rank."""
    return units_per_rank * world / max_seconds


def shard_range(n: int, rank: int, world: int) -> range:
    """Contiguous share of ``n`` independent meshes for ``rank`` (no exchange)."""
    lo = n * rank // world
    hi = n * (rank + 1) // world
    return range(lo, hi)


def shard_batch(blobs, rank: int, world: int):
    """The meshes of a batch that ``rank`` decodes: its contiguous share
    (every mesh decoded by exactly one rank; no data-path exchange)."""
    r = shard_range(len(blobs), rank, world)
    return blobs[r.start:r.stop]


def sharded_value(total_units: int, max_seconds: float) -> float:
    """Whole-job throughput of a sharded batch: every unit once, over the
    slowest rank's time (strong scaling: the total work is fixed)."""
    return total_units / max_seconds


# ---------------------------------------------------------------------------
# workloads
# ---------------------------------------------------------------------------
def heightfield_stream(n: int, bits: int):
    V, T = synth.noise_heightfield(n, seed=3)
    e = encoder.encode(V, T, precision_error=synth.bbox_bits_error(bits), precision_mode="bbox_frac")
    return e.data, {"workload": f"heightfield_{n}x{n}_{bits}bit", "grid": n, "bits": bits,
                    "triangles": int(len(T)), "source_vertices": int(len(V)),
                    "vertices_dup": int(e.n_v_dup), "meshlets": int(e.n_meshlets),
                    "stream_bytes": len(e.data),
                    "heights": "seeded 6-octave value noise (seed 3)",
                    "encoder": "project encoder, fitted IRLP, max_verts=max_tris=256"}


def icosphere_stream(bits: int):
    V, T = synth.icosphere(8, seed=2)
    e = encoder.encode(V, T, precision_error=synth.bbox_bits_error(bits), precision_mode="bbox_frac")
    return e.data, {"workload": f"icosphere_L8_{bits}bit", "bits": bits, "triangles": int(len(T)),
                    "source_vertices": int(len(V)), "vertices_dup": int(e.n_v_dup),
                    "meshlets": int(e.n_meshlets), "stream_bytes": len(e.data),
                    "displacement": "5-octave value noise, 5% of radius, seeded vertex shuffle",
                    "encoder": "project encoder, fitted IRLP, max_verts=max_tris=256"}


# ---------------------------------------------------------------------------
# clocks during the timed region
# ---------------------------------------------------------------------------
class ClockSampler:
    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def start(self):
        import tempfile
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
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
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"], "samples": 0}
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for _, _, r in rows for i, v in enumerate(r) if v.lower() == "active"})
        sm = [r[0] for r in rows]
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(r[1] for r in rows),
                "reasons": reasons, "samples": len(rows)}


def measured_peak():
    path = os.path.join(REPO, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs, burst copy)"
    return 6800.0, "fallback 6.8 TB/s"


def link_floor(h_in, h_idx, h_pos, d_idx, d_pos, stream, reps: int = 5) -> dict:
    """The host link alone: the step's upload (the stream, pinned) and its
    download (indices and positions into pinned memory) as plain copies,
    timed with CUDA events; their sum is the floor of an end-to-end step
    that waits for its inputs before decoding."""
    import torch
    d_in = torch.empty(h_in.numel(), dtype=torch.uint8, device=d_idx.device)

    def best(fn):
        ts = []
        for _ in range(reps):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with torch.cuda.stream(stream):  # the copies go to the timed stream
                e0.record(stream)
                fn()
                e1.record(stream)
            e1.synchronize()
            ts.append(e0.elapsed_time(e1))
        return min(ts)

    up = best(lambda: d_in.copy_(h_in, non_blocking=True))
    down = best(lambda: (h_idx.copy_(d_idx, non_blocking=True), h_pos.copy_(d_pos, non_blocking=True)))
    nb_up, nb_down = h_in.numel(), 4 * (h_idx.numel() + h_pos.numel())
    return {"h2d_ms": round(up, 4), "d2h_ms": round(down, 4), "h2d_gbs": round(nb_up / up / 1e6, 1),
            "d2h_gbs": round(nb_down / down / 1e6, 1), "floor_ms": round(up + down, 4),
            "what": "plain pinned copies of the step's bytes, CUDA events, best of %d" % reps}


def kernel_split(kern, fused: bool, stream_bytes: int, n_v: int, n_t: int, persistent: int = 2):
    """Names of the decode's kernels, the dominant one and its algorithmic
    bytes, from the per-kernel times (scan, connectivity, vertex; a one-kernel
    decode's time in the second slot: the group kernel, persistent 3, or the
    fused kernel, persistent 2)."""
    if fused:  # one kernel reads the stream and writes both outputs
        name = {3: "group_kernel", 4: "team_kernel"}.get(persistent, "flow_kernel")
        return ("scan_kernel", name), 1, stream_bytes + 12 * (n_v + n_t)
    # connectivity reads the stream and writes the indices (12 B per
    # triangle); the vertex kernel writes the positions (12 B per vertex)
    # from residual bits already counted in the stream
    dom = 1 + int(np.argmax(kern[1:3]))
    return ("scan_kernel", "conn_kernel", "vert_kernel"), dom, (stream_bytes + 12 * n_t) if dom == 1 else 12 * n_v


def ncu_traffic(kernel: str, workload: str):
    """DRAM bytes per launch from the committed ncu summary, if any."""
    path = os.path.join(REPO, "profiles", "traffic.json")
    if not os.path.exists(path):
        return None
    with open(path) as f:
        t = json.load(f)
    v = t.get(kernel, {}).get(workload)
    return None if v is None else float(v)


# ---------------------------------------------------------------------------
# CPU oracle (baseline leg only)
# ---------------------------------------------------------------------------
def cpu_oracle_rate(data: bytes, n_t: int, min_wall: float = 10.0, max_reps: int = 2000):
    import oracle
    oracle.build()
    cores = os.cpu_count() or 1
    h = oracle.parse_header(data)
    out = (np.empty((h.n_v_total, 3), np.float32), np.empty((h.n_t, 3), np.int64))
    oracle.decode_mt(data, cores, out=out)  # warm caches
    reps = 0
    t0 = time.perf_counter()
    while reps < 3 or (time.perf_counter() - t0 < min_wall and reps < max_reps):
        oracle.decode_mt(data, cores, out=out)
        reps += 1
    wall = time.perf_counter() - t0
    return n_t * reps / wall / 1e6, cores, reps, wall


# ---------------------------------------------------------------------------
# reference arm: the CPU decoder on all host cores
# ---------------------------------------------------------------------------
def run_reference(args):
    rank, _, world = dist_env()
    if rank != 0:
        return 0
    data, cfg = load_stream(args)
    import oracle
    oracle.build()
    cores = os.cpu_count() or 1
    h = oracle.parse_header(data)
    out = (np.empty((h.n_v_total, 3), np.float32), np.empty((h.n_t, 3), np.int64))
    for _ in range(max(1, args.warmup)):
        oracle.decode_mt(data, cores, out=out)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        oracle.decode_mt(data, cores, out=out)
    wall = time.perf_counter() - t0
    value = h.n_t * args.steps / wall / 1e6
    line = {
        "impl": "reference", "metric": "decoded triangles per second", "value": round(value, 3),
        "unit": "M tris/s", "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(wall / args.steps * 1e3, 4), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "int32+f64->f32", "data": "synthetic",
        "config": cfg,
        "cpu_baseline": {"value": round(value, 3), "unit": "M tris/s", "cores": cores, "kind": "port",
                         "sample": f"{args.steps} full decodes of the stream (C restatement of decode_dup, "
                                   f"meshlet-parallel over {cores} threads)"},
        "e2e": {"value": round(value, 3), "unit": "M tris/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


def encode_specs(specs, bits: int):
    """Build and encode mesh specs on all host cores (the encoder and most of
    the mesh generation run outside the GIL)."""
    from concurrent.futures import ThreadPoolExecutor

    def one(sp):
        V, T = synth.build_spec(*sp)
        e = encoder.encode(V, T, precision_error=synth.bbox_bits_error(bits), precision_mode="bbox_frac")
        return e.data, int(len(T)), int(e.n_v_dup)

    with ThreadPoolExecutor(os.cpu_count() or 1) as ex:
        return list(ex.map(one, specs))


def batch_streams(n_meshes: int, bits: int):
    specs = synth.mixed_batch_specs(n_meshes, seed=4)
    enc = encode_specs(specs, bits)
    kinds = {}
    for kind, _ in specs:
        kinds[kind] = kinds.get(kind, 0) + 1
    blobs = [e[0] for e in enc]
    cfg = {"workload": f"mixed_{n_meshes}_meshes_{bits}bit", "meshes": n_meshes, "bits": bits,
           "triangles": int(sum(e[1] for e in enc)), "vertices_dup": int(sum(e[2] for e in enc)),
           "stream_bytes": int(sum(len(b) for b in blobs)), "kinds": kinds,
           "sizes": "triangle counts log-uniform in [1K, 200K] (seed 4); 50% grids of random aspect, "
                    "30% displaced icospheres L3-L7, 20% tori R/r in [2, 5]",
           "encoder": "project encoder, fitted IRLP, max_verts=max_tris=256"}
    return blobs, cfg


def oracle_rate_meshes(blobs, tris, max_wall: float = 15.0):
    """CPU oracle (sequential decoder per mesh, meshes spread over all host
    cores) on a bounded prefix of the meshes -> (M tris/s, cores, sample)."""
    from concurrent.futures import ThreadPoolExecutor
    import oracle
    oracle.build()
    cores = os.cpu_count() or 1
    # sample: every 8th mesh (the same size mix), seconds of work
    pick = list(range(0, len(blobs), 8))
    acc = sum(tris[i] for i in pick)
    sample = [blobs[i] for i in pick]
    reps = 0
    t0 = time.perf_counter()
    with ThreadPoolExecutor(cores) as ex:
        while reps < 1 or time.perf_counter() - t0 < 10.0:  # about ten seconds of CPU work
            list(ex.map(oracle.decode, sample))
            reps += 1
    wall = time.perf_counter() - t0
    return acc * reps / wall / 1e6, cores, f"every 8th mesh: {len(pick)} of {len(blobs)} meshes ({acc} triangles), " \
                                           f"{reps} passes in {wall:.2f} s (C restatement of decode_dup, one mesh " \
                                           f"per thread)"


def make_stream(args):
    if args.workload == "heightfield":
        return heightfield_stream(args.grid, args.bits)
    if args.workload == "icosphere":
        return icosphere_stream(args.bits)
    raise ValueError(args.workload)


def stream_file(args) -> str:
    """Where the encoded stream of a single-mesh workload is kept (git-ignored
    build output): both arms read the same bytes from it."""
    name = f"{args.workload}_{args.grid if args.workload == 'heightfield' else 'l8'}_{args.bits}bit"
    return os.path.join(REPO, "_build", "bench_streams", name + ".dpr4")


def write_stream(args, path: str):
    data, cfg = make_stream(args)
    os.makedirs(os.path.dirname(path), exist_ok=True)
    with open(path + ".tmp", "wb") as f:
        f.write(data)
    with open(path + ".json.tmp", "w") as f:
        json.dump(cfg, f)
    os.replace(path + ".json.tmp", path + ".json")
    os.replace(path + ".tmp", path)


def load_stream(args):
    """The workload's stream and its description.  A missing file is made by
    a child process, so the caller never loads the encoder library (the
    reference arm depends on no product code of this repository)."""
    path = stream_file(args)
    if not (os.path.exists(path) and os.path.exists(path + ".json")):
        cmd = [sys.executable, os.path.abspath(__file__), "--write-stream", path, "--workload", args.workload,
               "--grid", str(args.grid), "--bits", str(args.bits)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"could not encode the workload: {r.stderr[-2000:]}")
    with open(path, "rb") as f:
        data = f.read()
    with open(path + ".json") as f:
        cfg = json.load(f)
    return data, cfg


# ---------------------------------------------------------------------------
# our arm
# ---------------------------------------------------------------------------
def run_single(args):
    import torch
    from meshpress_gb300 import ParaDeltaV5GpuDecoder, _lib
    rank, local, world = dist_init("nccl")
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    data, cfg = load_stream(args)
    lib = _lib.load()
    dec = ParaDeltaV5GpuDecoder(data)
    n_t, n_v = dec.n_t_total, dec.n_v_total
    idx = torch.empty((n_t, 3), dtype=torch.int32, device=dev)
    pos = torch.empty((n_v, 3), dtype=torch.float32, device=dev)
    stream = torch.cuda.current_stream()
    sh = ctypes.c_void_p(int(stream.cuda_stream))

    # launch shape: as given, or autotuned over a one-mesh batch; applied to the handle
    launch = None
    if args.shape:
        v = [int(x) for x in args.shape.split(",")]
        c = _lib.LaunchCfg()
        c.warps_per_cta, c.persistent = v[0], v[1]
        c.ctas_per_sm = 0
        c.stage_bytes = v[2] if len(v) > 2 else 16 * 1024
        c.code_bytes = v[3] if len(v) > 3 else 12 * 1024
        dec.set_launch_config(c)
        launch = c.as_dict()
    elif args.tune:
        from meshpress_gb300.batch import BatchDecoder
        b = BatchDecoder([data])
        best, best_ms = b.autotune(iters=3)
        b.close()
        dec.set_launch_config(best)
        launch = dict(best.as_dict(), tuned_ms=round(best_ms, 4))

    # parity before timing: bit-exact against the CPU oracle
    dec.decode_into(idx, pos)
    exact = None
    if rank == 0:
        import oracle
        opos, oidx = oracle.decode_mt(data, 0)
        exact = bool(np.array_equal(pos.cpu().numpy().view(np.uint32), opos.view(np.uint32)) and
                     np.array_equal(idx.cpu().numpy().view(np.uint32).astype(np.int64), oidx))

    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    kms = (ctypes.c_float * 3)()
    for _ in range(max(args.warmup, 3)):
        flush.fill_(1)
        _lib.check(lib.stride_decode_timed(dec._h, sh, ctypes.c_void_p(idx.data_ptr()),
                                           ctypes.c_void_p(pos.data_ptr()), kms), "decode")
    dec.check()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    kern_ms = []
    clocks = ClockSampler(local)
    barrier(dev)
    torch.cuda.synchronize()
    clocks.start()
    time.sleep(0.3)
    t_wall = time.perf_counter()
    # the timed step is the plain decode call (stride_decode, as
    # decode_into makes it); per-kernel events inside the step would add
    # about 20 us, so the kernel split comes from separate timed decodes
    for k in range(args.steps):
        flush.fill_(k & 0xFF)
        ev[k][0].record(stream)
        _lib.check(lib.stride_decode(dec._h, sh, ctypes.c_void_p(idx.data_ptr()),
                                     ctypes.c_void_p(pos.data_ptr()), None), "decode")
        ev[k][1].record(stream)
    torch.cuda.synchronize()
    wall = time.perf_counter() - t_wall
    barrier(dev)
    clk = clocks.stop()
    dec.check()
    for k in range(args.steps):  # untimed: the kernel split, same L2 flush
        flush.fill_(k & 0xFF)
        _lib.check(lib.stride_decode_timed(dec._h, sh, ctypes.c_void_p(idx.data_ptr()),
                                           ctypes.c_void_p(pos.data_ptr()), kms), "decode")
        kern_ms.append(tuple(kms))
    dec.check()
    step_ms = [a.elapsed_time(b) for a, b in ev]
    mean_step = reduce_max(sum(step_ms) / len(step_ms), dev)
    value = replica_value(n_t, world, mean_step / 1e3) / 1e6

    # Dominant kernel and its algorithmic bytes; the step's algorithmic
    # bytes are stream + both outputs.
    alg_bytes = len(data) + 12 * (n_v + n_t)
    peak, peak_src = measured_peak()
    k = np.array(kern_ms).mean(axis=0)
    names, dom, dom_bytes = kernel_split(k, int(dec.info.kernels) == 2, len(data), n_v, n_t,
                                         int(dec.launch_config().persistent))
    achieved = dom_bytes / (k[dom] / 1e3) / 1e9
    roofline = {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                "frac": round(achieved / peak, 4), "traffic": ncu_traffic(names[dom], cfg["workload"]),
                "kernel": names[dom], "kernel_ms": {n: round(float(v), 4) for n, v in zip(names, k)},
                "kernel_alg_bytes": int(dom_bytes), "step_alg_bytes": int(alg_bytes),
                "peak_source": peak_src,
                "step_achieved": round(alg_bytes / (mean_step / 1e3) / 1e9, 1),
                "step_frac": round(alg_bytes / (mean_step / 1e3) / 1e9 / peak, 4)}

    # end to end through the public API with pinned host buffers
    e2e = None
    if not args.no_e2e:
        h_blob = torch.empty(len(data), dtype=torch.uint8, pin_memory=True)
        h_blob.numpy()[:] = np.frombuffer(data, np.uint8)
        h_pos = torch.empty((n_v, 3), dtype=torch.float32, pin_memory=True)
        h_idx = torch.empty((n_t, 3), dtype=torch.int32, pin_memory=True)
        blob_ptr = ctypes.c_void_p(h_blob.data_ptr())
        for _ in range(2):
            _lib.check(lib.stride_reload(dec._h, blob_ptr, len(data), sh), "reload")
            _lib.check(lib.stride_decode_host(dec._h, sh, ctypes.c_void_p(h_idx.data_ptr()),
                                              ctypes.c_void_p(h_pos.data_ptr())), "decode_host")
        ts = []
        for _ in range(args.steps):
            t0 = time.perf_counter()
            _lib.check(lib.stride_reload(dec._h, blob_ptr, len(data), sh), "reload")
            _lib.check(lib.stride_decode_host(dec._h, sh, ctypes.c_void_p(h_idx.data_ptr()),
                                              ctypes.c_void_p(h_pos.data_ptr())), "decode_host")
            ts.append(time.perf_counter() - t0)
        e2e_s = reduce_max(sum(ts) / len(ts), dev)
        e2e = {"value": round(replica_value(n_t, world, e2e_s) / 1e6, 3), "unit": "M tris/s",
               "h2d_bytes_per_step": len(data), "d2h_bytes_per_step": 12 * (n_v + n_t),
               "ms_per_step": round(e2e_s * 1e3, 4), "path": "ParaDeltaV5GpuDecoder C ABI: stride_reload + "
                                                              "stride_decode_host, pinned host buffers",
               "link": link_floor(h_blob, h_idx, h_pos, idx, pos, stream)}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        v, cores, reps, w = cpu_oracle_rate(data, n_t)
        cpu = {"value": round(v, 3), "unit": "M tris/s", "cores": cores, "kind": "port",
               "sample": f"{reps} full decodes of the same stream in {w:.2f} s wall "
                         f"(C restatement of decode_dup, meshlet-parallel)"}

    if rank == 0:
        cfg = dict(cfg)
        cfg["l2"] = "flushed before every step (256 MiB write, untimed)"
        cfg["launch"] = launch
        cfg["parallelism"] = f"replicas x{world}"
        cfg["parity"] = "bit-exact vs CPU oracle (positions, indices)" if exact else f"MISMATCH ({exact})"
        line = {
            "metric": "decoded triangles per second", "value": round(value, 3), "unit": "M tris/s",
            "n_gpus": world, "steps": args.steps, "warmup": max(args.warmup, 3),
            "ms_per_step": round(mean_step, 4), "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int32+f32 (exact f64 expression)",
            "data": "synthetic (seeded heightfield; reference meshes not available)",
            "config": cfg, "roofline": roofline, "cpu_baseline": cpu, "e2e": e2e,
            "gpu_launches": int(dec.info.kernels) * args.steps, "clocks": clk, "wall_s": round(wall, 3),
        }
        print(json.dumps(line), flush=True)
    return 0


def run_batch(args):
    """Many meshes: one persistent launch over all of them (CUDA graph)
    against one plain decode launch per mesh, same outputs."""
    import torch
    from meshpress_gb300 import ParaDeltaV5GpuDecoder, _lib
    from meshpress_gb300.batch import BatchDecoder
    rank, local, world = dist_init("nccl")
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    blobs, cfg = batch_streams(args.batch_meshes, args.bits)
    n_t_all = cfg["triangles"]  # the whole batch: every rank decodes its share once
    blobs = shard_batch(blobs, rank, world)
    lib = _lib.load()
    b = BatchDecoder(blobs)
    launch = None
    if args.tune:
        best, best_ms = b.autotune(iters=2)
        launch = dict(best.as_dict(), tuned_ms=round(best_ms, 4))
    # scan (with the dequantisation tables), then the fused kernel or the
    # connectivity and vertex kernels
    fused = int(b.config().persistent) >= 2
    per_step_kernels = 2 if fused else 3
    stream = torch.cuda.Stream(device=dev)
    with torch.cuda.stream(stream):
        b.capture_graph(stream)
    stream.synchronize()
    b.check()

    # parity: every mesh bit-exact against the oracle
    exact = None
    if rank == 0:
        from concurrent.futures import ThreadPoolExecutor
        import oracle
        oracle.build()
        t_all = b.d_tris.view(torch.int32).cpu().numpy().view(np.uint32)
        v_all = b.d_verts.cpu().numpy()

        def same(i):
            opos, oidx = oracle.decode(blobs[i])
            return (np.array_equal(t_all[b.t_offset[i]:b.t_offset[i + 1]].astype(np.int64), oidx) and
                    np.array_equal(v_all[b.v_offset[i]:b.v_offset[i + 1]].view(np.uint32), opos.view(np.uint32)))

        with ThreadPoolExecutor(os.cpu_count() or 1) as ex:
            exact = all(ex.map(same, range(len(blobs))))
        del t_all, v_all

    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    clocks = ClockSampler(local)
    with torch.cuda.stream(stream):
        for _ in range(max(args.warmup, 3)):
            flush.fill_(1)
            b.launch_graph(stream)
        barrier(dev)
        torch.cuda.synchronize()
        clocks.start()
        time.sleep(0.3)
        for k in range(args.steps):
            flush.fill_(k & 0xFF)
            ev[k][0].record(stream)
            b.launch_graph(stream)
            ev[k][1].record(stream)
        torch.cuda.synchronize()
    clk = clocks.stop()
    b.check()
    batched_ms = reduce_max(sum(a.elapsed_time(c) for a, c in ev) / args.steps, dev)
    value = sharded_value(n_t_all, batched_ms / 1e3) / 1e6
    kern = np.array([b.decode_timed(stream=stream) for _ in range(3)]).mean(axis=0)

    # per-mesh plain launches (one ParaDeltaV5GpuDecoder per mesh, own outputs)
    decs = [ParaDeltaV5GpuDecoder(x) for x in blobs]
    per_mesh_launches = sum(int(d.info.kernels) for d in decs)
    outs = [(torch.empty((d.n_t_total, 3), dtype=torch.int32, device=dev),
             torch.empty((d.n_v_total, 3), dtype=torch.float32, device=dev)) for d in decs]
    sh = ctypes.c_void_p(int(stream.cuda_stream))
    ptrs = [(ctypes.c_void_p(t.data_ptr()), ctypes.c_void_p(v.data_ptr())) for t, v in outs]

    def per_mesh_pass():
        for d, (pt, pv) in zip(decs, ptrs):
            _lib.check(lib.stride_decode(d._h, sh, pt, pv, None), "stride_decode")

    with torch.cuda.stream(stream):
        per_mesh_pass()
        torch.cuda.synchronize()
        pm_ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
                 for _ in range(args.steps)]
        for k in range(args.steps):
            flush.fill_(k & 0xFF)
            pm_ev[k][0].record(stream)
            per_mesh_pass()
            pm_ev[k][1].record(stream)
        torch.cuda.synchronize()
    for d in decs:
        d.check()
    per_mesh_ms = reduce_max(sum(a.elapsed_time(c) for a, c in pm_ev) / args.steps, dev)
    same_as_batch = (torch.equal(torch.cat([t for t, _ in outs]), b.d_tris.view(torch.int32)) and
                     torch.equal(torch.cat([v for _, v in outs]).view(torch.int32), b.d_verts.view(torch.int32)))
    for d in decs:
        d.close()
    del outs, decs

    # end to end: pinned host image -> device, decode with the outputs copied to pinned host memory
    e2e = None
    if not args.no_e2e:
        img = b.make_image()
        h_img = torch.empty(img.size, dtype=torch.uint8, pin_memory=True)
        h_img.numpy()[:] = img
        h_t = torch.empty(b.d_tris.shape, dtype=torch.int32, pin_memory=True)
        h_v = torch.empty(b.d_verts.shape, dtype=torch.float32, pin_memory=True)
        out = (h_v.numpy(), h_t.numpy().view(np.uint32))
        ts = []
        with torch.cuda.stream(stream):
            for k in range(args.steps + 2):
                t0 = time.perf_counter()
                b.upload(h_img.data_ptr(), img.size, stream=stream)
                b.decode_to_host(out=out, stream=stream)
                if k >= 2:
                    ts.append(time.perf_counter() - t0)
        b.check()
        e2e_s = reduce_max(sum(ts) / len(ts), dev)
        e2e = {"value": round(sharded_value(n_t_all, e2e_s) / 1e6, 3), "unit": "M tris/s",
               "h2d_bytes_per_step": int(img.size), "d2h_bytes_per_step": 12 * (b.n_t_total + b.n_v_total),
               "ms_per_step": round(e2e_s * 1e3, 4),
               "path": "BatchDecoder: stride_batch_upload (pinned arena image) + stride_batch_decode_to_host "
                       "(pinned outputs, copies beside the decode)",
               "link": link_floor(h_img, h_t, h_v, b.d_tris.view(torch.int32), b.d_verts, stream)}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        tris = [int(b.t_offset[i + 1] - b.t_offset[i]) for i in range(len(blobs))]
        v, cores, sample = oracle_rate_meshes(blobs, tris)
        cpu = {"value": round(v, 3), "unit": "M tris/s", "cores": cores, "kind": "port", "sample": sample}

    if rank == 0:
        peak, peak_src = measured_peak()
        names, dom, dom_bytes = kernel_split(kern, fused, cfg["stream_bytes"], b.n_v_total, b.n_t_total,
                                             int(b.config().persistent))
        achieved = dom_bytes / (kern[dom] / 1e3) / 1e9
        alg = cfg["stream_bytes"] + 12 * (b.n_t_total + b.n_v_total)
        cfg = dict(cfg)
        cfg.update(l2="inputs larger than L2 (and a 256 MiB flush before every step)", launch=launch,
                   parallelism=f"meshes sharded over {world} ranks (contiguous shares, no exchange)",
                   parity=("bit-exact vs CPU oracle, every mesh of rank 0's share" if exact
                           else f"MISMATCH ({exact})"))
        line = {
            "metric": "decoded triangles per second", "value": round(value, 3), "unit": "M tris/s",
            "n_gpus": world, "steps": args.steps, "warmup": max(args.warmup, 3),
            "ms_per_step": round(batched_ms, 4), "higher_is_better": True, "scaling": "strong",
            "vs_baseline": None, "dtype": "int32+f32 (exact f64 expression)",
            "data": "synthetic (seeded mixed meshes; reference meshes not available)", "config": cfg,
            "per_mesh": {"value": round(sharded_value(n_t_all, per_mesh_ms / 1e3) / 1e6, 3),
                         "unit": "M tris/s", "ms_per_step": round(per_mesh_ms, 4),
                         "launches_per_step": per_mesh_launches, "same_output_as_batched": bool(same_as_batch)},
            "batched_over_per_mesh": round(per_mesh_ms / batched_ms, 3),
            "roofline": {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                         "frac": round(achieved / peak, 4), "traffic": ncu_traffic(names[dom], cfg["workload"]),
                         "kernel": names[dom], "kernel_ms": {n: round(float(x), 4) for n, x in zip(names, kern)},
                         "kernel_alg_bytes": int(dom_bytes), "step_alg_bytes": int(alg), "peak_source": peak_src,
                         "step_achieved": round(alg / (batched_ms / 1e3) / 1e9, 1),
                         "step_frac": round(alg / (batched_ms / 1e3) / 1e9 / peak, 4)},
            "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": per_step_kernels * args.steps, "clocks": clk,
        }
        print(json.dumps(line), flush=True)
    b.close()
    return 0


def run_serve(args):
    """Poisson arrivals into the continuous-batching server, then closed-loop
    passes that keep a fixed number of requests outstanding (the saturating
    rate); one line per pass with p50/p99 latency, aggregate throughput,
    requests per launch and the arena's high-water mark.  Every response is
    compared with the same mesh decoded alone."""
    import threading
    import torch
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    from meshpress_gb300.serve import DecodeServer
    rank, local, world = dist_init("nccl")
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    specs = synth.mixed_batch_specs(args.serve_pool, seed=5, t_min=5e3, t_max=2e6)
    enc = encode_specs(specs, args.bits)
    blobs = [e[0] for e in enc]
    tris = [e[1] for e in enc]
    # every pool entry decoded alone once, and that checked against the oracle
    import oracle
    oracle.build()
    alone = []
    pool_exact = True
    for x in blobs:
        d = ParaDeltaV5GpuDecoder(x)
        t, v = d.decode_to_device()
        alone.append((t.view(torch.int32).clone(), v.view(torch.int32).clone()))
        if rank == 0:
            opos, oidx = oracle.decode_mt(x, 0)
            ti = t.view(torch.int32).cpu().numpy().view(np.uint32).astype(np.int64)
            pool_exact = pool_exact and np.array_equal(ti, oidx) and \
                np.array_equal(v.cpu().numpy().view(np.uint32), opos.view(np.uint32))
        d.close()
    rates = [float(r) for r in args.rates.split(",")]
    rng = np.random.default_rng(11)
    with DecodeServer(4 << 30) as warm:  # first launches set kernel attributes
        for rid in [warm.submit(x) for x in blobs[:4]]:
            assert warm.wait(rid).ok
            warm.release(rid)
    runs = [("rate", r, False) for r in rates]
    runs += [("rate", args.serve_host_rate, True)] if args.serve_host_rate > 0 else []
    runs += [("burst", int(q), False) for q in args.serve_burst.split(",") if q.strip()]
    alone_host = None
    for mode, knob, to_host in runs:
        if mode == "rate":
            n_req = max(20, int(knob * args.serve_seconds))
            gaps = rng.exponential(1.0 / knob, n_req)
        else:  # bursts of `knob` requests, as many in all as the 2000 rps pass
            n_req = max(1, int(2000 * args.serve_seconds) // knob) * knob
            gaps = None
        picks = rng.integers(0, len(blobs), n_req)
        if to_host and alone_host is None:
            alone_host = [(t.cpu().numpy(), v.cpu().numpy()) for t, v in alone]
        srv = DecodeServer(args.serve_budget_gb << 30, n_streams=3, max_batch=256, copy_to_host=to_host)
        ids = [None] * n_req
        ok, failed = [0, 0], {}
        times = np.zeros((n_req, 3))  # server clock (us): submit, admit, done
        # device results are compared on the device and read back in chunks
        # (one synchronisation per chunk), then released
        pending = []

        def settle():
            if not pending:
                return
            flags = torch.stack([f for _, f in pending]).cpu().tolist()
            for (i, _), bad in zip(pending, flags):
                ok[1 if bad else 0] += 1
                srv.release(ids[i])
            pending.clear()

        def collect(i):
            r = srv.wait(ids[i])
            if not r.ok:
                failed[r.status] = failed.get(r.status, 0) + 1
                srv.release(ids[i])
            elif to_host:
                at, av = alone_host[picks[i]]
                good = np.array_equal(r.host_tris.view(np.int32), at) and \
                    np.array_equal(r.host_verts.view(np.int32), av)
                ok[0 if good else 1] += 1
                srv.release(ids[i])
            else:
                at, av = alone[picks[i]]
                bad = torch.ne(r.tris.view(torch.int32), at).any() | torch.ne(r.verts.view(torch.int32), av).any()
                pending.append((i, bad))
                if len(pending) >= 32:
                    settle()
            times[i] = (r.t_submit_us, r.t_admit_us, r.t_done_us)

        torch.cuda.synchronize()
        t0 = time.perf_counter()
        if mode == "rate":
            def feed():
                t_next = time.perf_counter()
                for i in range(n_req):
                    t_next += gaps[i]
                    dt = t_next - time.perf_counter()
                    if dt > 0:
                        time.sleep(dt)
                    ids[i] = srv.submit(blobs[picks[i]])

            th = threading.Thread(target=feed)
            th.start()
            for i in range(n_req):
                while ids[i] is None:
                    time.sleep(0.0002)
                collect(i)
            th.join()
        else:
            # the server holds each burst's requests until all are queued, so
            # it forms its launches from a full queue (the client's own
            # per-request cost -- payload copies, checks -- stays outside the
            # server's busy time measured below)
            busy_us = 0.0
            for b0 in range(0, n_req, knob):
                srv.hold(True)
                for i in range(b0, b0 + knob):
                    ids[i] = srv.submit(blobs[picks[i]])
                srv.hold(False)
                for i in range(b0, b0 + knob):
                    collect(i)
                seg = times[b0:b0 + knob]
                busy_us += seg[:, 2].max() - seg[:, 1].min()
        settle()
        wall = time.perf_counter() - t0
        st = srv.stats()
        srv.close()
        if mode == "rate":
            span_s = (times[:, 2].max() - times[:, 0].min()) / 1e6
            lat = (times[:, 2] - times[:, 0]) / 1e3
        else:
            span_s = busy_us / 1e6
            lat = (times[:, 2] - times[:, 1]) / 1e3
        total_t = int(sum(tris[j] for j in picks))
        if rank == 0:
            if mode == "rate":
                name = f"serve_poisson_{int(knob)}rps" + ("_to_host" if to_host else "")
                load = {"rate_rps": knob}
            else:
                name = f"serve_burst{knob}"
                load = {"burst": knob, "arrivals": "bursts: the server holds each burst of requests until all "
                                                   "are queued; throughput over the server's busy time (first "
                                                   "admission to last completion of each burst)"}
            line = {
                "metric": "served decode latency p50/p99 and throughput", "value": round(total_t / span_s / 1e6, 3),
                "unit": "M tris/s", "n_gpus": world, "higher_is_better": True, "scaling": "weak",
                "vs_baseline": None, "dtype": "int32+f32 (exact f64 expression)",
                "data": "synthetic (seeded mixed meshes)",
                "config": {"workload": name, **load, "requests": n_req,
                           "pool": len(blobs), "pool_triangles": int(sum(tris)),
                           "sizes": "log-uniform [5K, 2M] triangles from the many-mesh generator (seed 5)",
                           "hbm_budget_gb": args.serve_budget_gb, "streams": 3, "max_batch": 256},
                "latency_ms": {"p50": round(float(np.percentile(lat, 50)), 3),
                               "p99": round(float(np.percentile(lat, 99)), 3),
                               "max": round(float(np.max(lat)), 3),
                               "from": "submit" if mode == "rate" else "admission",
                               "to": "outputs in pinned host memory" if to_host
                               else "outputs resident on the device"},
                "achieved_rps": round(n_req / span_s, 1), "launches": st["launches"],
                "mean_requests_per_launch": round(n_req / max(1, st["launches"]), 2),
                "arena_peak_gb": round(st["arena_peak_bytes"] / 2 ** 30, 3),
                "exact_responses": ok[0], "mismatched_responses": ok[1],
                "failed_responses": {str(k): v for k, v in failed.items()},
                "pool_bit_exact_vs_oracle": bool(pool_exact), "wall_s": round(wall, 3),
            }
            print(json.dumps(line), flush=True)
    return 0


def run_reference_batch(args):
    rank, _, world = dist_env()
    if rank != 0:
        return 0
    blobs, cfg = batch_streams(args.batch_meshes, args.bits)
    from concurrent.futures import ThreadPoolExecutor
    import oracle
    oracle.build()
    cores = os.cpu_count() or 1
    # bounded sample per step: every 16th mesh (the same size mix)
    sample_blobs = blobs[::16]
    acc = sum(oracle.parse_header(x).n_t for x in sample_blobs)
    with ThreadPoolExecutor(cores) as ex:
        for _ in range(max(1, args.warmup)):
            list(ex.map(oracle.decode, sample_blobs))
        t0 = time.perf_counter()
        for _ in range(args.steps):
            list(ex.map(oracle.decode, sample_blobs))
        wall = time.perf_counter() - t0
    value = acc * args.steps / wall / 1e6
    sample = f"per step every 16th mesh: {len(sample_blobs)} of {len(blobs)} meshes ({acc} triangles), " \
             f"one mesh per thread"
    line = {
        "impl": "reference", "metric": "decoded triangles per second", "value": round(value, 3),
        "unit": "M tris/s", "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(wall / args.steps * 1e3, 4), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "int64+f64->f32", "data": "synthetic", "config": cfg,
        "cpu_baseline": {"value": round(value, 3), "unit": "M tris/s", "cores": cores, "kind": "port",
                         "sample": sample},
        "e2e": {"value": round(value, 3), "unit": "M tris/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


def main(argv=None):
    args = parse_args(argv)
    if args.write_stream:
        write_stream(args, args.write_stream)
        return 0
    if args.impl == "reference":
        if args.workload == "batch":
            return run_reference_batch(args)
        if args.workload == "serve":
            print(json.dumps({"impl": "reference", "unavailable": "the reference has no serving path "
                                                                  "(one decoder object per stream)"}))
            return 0
        return run_reference(args)
    if args.workload == "batch":
        return run_batch(args)
    if args.workload == "serve":
        return run_serve(args)
    return run_single(args)


if __name__ == "__main__":
    sys.exit(main())
