"""Benchmark of the P-frame inter-analysis stage at 1080p (1920x1080, QP 27, 1 reference, 8 slice bands).

One step = one P picture through the stage: the half-sample planes of its reference (K1) and the
analysis of all 8160 macroblocks (P_Skip vector + SAD, best_inter with its motion searches; K2), in
replay mode: each macroblock is analysed against its neighbours' final decisions (made beforehand by
the stage's own auto mode, outside the timed region), so all macroblocks are independent.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

- ``value``: macroblocks per second over all ranks, inputs resident in device memory (device-pointer
  entry points), K steps timed with CUDA events between a barrier + synchronize on both sides, the max
  over ranks;
- ``e2e``: the same through the host-buffer C ABI calls (ironav_set_source, ironav_push_reference,
  ironav_analyse_picture_replay) from pinned host memory, copies included;
- ``roofline``: the analysis kernel against the measured 32-bit integer issue rate; ``roofline_planes``:
  the plane kernel against the measured HBM bandwidth (the 6.65 TB/s fallback when no measurement is
  at hand, named in ``peak_source``); ``traffic``: each kernel's DRAM bytes per launch from one ncu
  capture of the 8-bit workload;
- ``cpu_baseline``: the C restatement of the reference's stage (oracle/) over all host cores on a
  bounded sample of the same workload, rank 0 only.
- ``--impl reference``: the reference's algorithm on the host cores (the oracle port: the Rust
  reference cannot be built here), same workload and metric.

Multi-GPU: the stage does not shard within a stream (each picture depends on the previous one and all
slice bands read the whole reference), so N GPUs run N independent replicas (weak scaling).
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "1080p inter-analysis MB/s: plain bit-exact vs learned at ≤1% bitrate delta"
WIDTH, HEIGHT, QP, NSLICES = 1920, 1080, 27, 8
RING = 40  # frames in the ring: luma + decisions + results of the ring exceed the 126 MB L2
E2E_MIN_S = 0.5  # the shortest wall-clock window of the host-buffer (e2e) pass


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=20)
    p.add_argument("--warmup", type=int, default=5)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--cpu-seconds", type=float, default=12.0, help="bound on the CPU baseline sample")
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--ring", type=int, default=RING,
                   help="pictures in the ring (fewer than 36 fits in L2: for profiling runs only)")
    p.add_argument("--no-e2e", action="store_true", help="skip the host-buffer pass (profiling runs)")
    p.add_argument("--workload", default="1080p", choices=["1080p", "batched", "scenecut", "deblock", "bpicture", "residual", "decide",
                                                         "decide_batched", "inloop", "encode", "learned"],
                   help="1080p: one stream, replay mode (the headline); batched: 64 mixed-resolution streams in auto "
                        "mode, one launch per stage and frame step, against the per-stream launch loop")
    p.add_argument("--streams", type=int, default=64, help="streams of the batched workload")
    p.add_argument("--replay-form", type=int, default=None, choices=[0, 1, 2, 3],
                   help="replay mode's kernel (ironav_set_replay_form): 0 8-lane groups, 1 one macroblock a warp, 2 16-lane "
                        "groups, 3 4-lane groups; default the library's choice for the picture (at 1080p 0 at 8 bits, 1 at 10)")
    p.add_argument("--learned-samples", type=int, default=2_000_000, help="training samples of the learned workload's proposer")
    p.add_argument("--e2e-threads", type=int, default=8, help="host threads (each with a context) of the e2e pass")
    p.add_argument("--cabac", action="store_true",
                   help="decide, decide_batched and encode workloads: CABAC with rate-distortion decisions and the 8x8 "
                        "transform (the reference encoder's default entropy coding) instead of CAVLC")
    p.add_argument("--bd", type=int, default=8, choices=[8, 10],
                   help="sample depth of the 1080p workload: 8 (Yuv420p) or 10 (Yuv420p10, QP' = QP + 12)")
    return p.parse_args()


def dist_setup(args):
    import torch
    import torch.distributed as dist

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        from datetime import timedelta

        backend = "nccl" if (args.impl == "ours" and torch.cuda.is_available()) else "gloo"
        if backend == "nccl":
            torch.cuda.set_device(local)
        dist.init_process_group(backend, timeout=timedelta(seconds=120))
    elif torch.cuda.is_available() and args.impl == "ours":
        torch.cuda.set_device(0)
    return rank, world, local


class Clocks:
    """nvidia-smi samples during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = os.path.join("/tmp", f"ironav_clocks_{os.getpid()}.csv")

    def start(self):
        try:
            self.out = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=self.out, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.out.close()
        sm, smax, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax = max(smax, float(parts[2]))
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": smax, "reasons": sorted(reasons), "samples": len(sm),
                "window": "0.6 s of untimed steps, then the timed steps"}


def max_over_ranks(value: float, world: int, device) -> float:
    """The largest of every rank's value: a job's time is its slowest rank's. A tensor on `device` (the
    GPU for NCCL, the CPU for gloo); one all-reduce when there are several ranks."""
    import torch

    t = torch.tensor([value], dtype=torch.float64, device=device)
    if world > 1:
        import torch.distributed as dist

        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def sum_over_ranks(value: float, world: int, device) -> float:
    """The sum of every rank's value (the macroblocks all ranks processed); one all-reduce when there are
    several ranks."""
    import torch

    t = torch.tensor([value], dtype=torch.float64, device=device)
    if world > 1:
        import torch.distributed as dist

        dist.all_reduce(t, op=dist.ReduceOp.SUM)
    return float(t.item())


def split_streams(streams, rank: int, world: int):
    """This rank's share of the batched configuration's streams: every stream goes to exactly one rank,
    the largest first to the rank with the fewest macroblocks so far (ties to the lower rank), so the
    ranks' shares of macroblocks stay close and the slowest rank's time, which the job's time is, is not
    one rank's accident of resolutions. Deterministic: every rank computes the same split."""
    load = [0] * world
    owner = [0] * len(streams)
    order = sorted(range(len(streams)), key=lambda i: (-((streams[i][0] + 15) // 16) * ((streams[i][1] + 15) // 16), i))
    for i in order:
        r = min(range(world), key=lambda k: (load[k], k))
        owner[i] = r
        load[r] += ((streams[i][0] + 15) // 16) * ((streams[i][1] + 15) // 16)
    return [s for i, s in enumerate(streams) if owner[i] == rank]


def make_frames(rank: int, n: int, bd: int = 8):
    """The 1080p sequence of one rank: each replica analyses its own seeded sequence (weak scaling)."""
    from ironav_b200.synth import CONFIGS, Sequence

    w, h, seed, pan_q, nobj, vmax, sigma = CONFIGS["1080p"]
    seq = Sequence(w, h, n, seed + 0x1000 * rank, pan_q, nobj, vmax, sigma)
    return np.stack([seq.frame10(t) if bd > 8 else seq.frame(t) for t in range(n)])


def qp_prime(bd: int) -> int:
    """QP'Y of the workload's P pictures: QP + 6 * (bd - 8) (FrameCoder::new, enc/frame.rs:381-412)."""
    return QP + 6 * (bd - 8)


def cpu_baseline(frames, states, seconds: float, bd: int = 8):
    """The oracle (C restatement of the reference's stage) in replay mode over all host cores, on as
    many of the ring's pictures as fit in `seconds`."""
    from tests.oracle_lib import oracle_library
    from ironav_b200.inter import InterStage

    lib = oracle_library()
    cores = host_cores()
    st = InterStage(WIDTH, HEIGHT, nslices=NSLICES, lib=lib, bd=bd)
    lib.oracle_set_threads(st.ctx, cores)
    done_mb, elapsed, pics = 0, 0.0, 0
    while elapsed < seconds:
        t = 1 + pics % (len(frames) - 1)
        st.clear_references()
        st.push_reference(frames[t - 1], col=states[t - 1] if t >= 2 else None)
        st.set_source(frames[t])
        st.begin_p_picture(qp_prime(bd))
        t0 = time.perf_counter()
        st.analyse_replay(states[t])
        elapsed += time.perf_counter() - t0
        done_mb += st.nmb
        pics += 1
    st.close()
    return {"value": done_mb / elapsed, "unit": "MB/s", "cores": cores, "kind": "port",
            "sample": f"{pics} pictures of the 1080p {bd}-bit ring ({done_mb} macroblocks), replay mode, "
                      f"{cores} threads, {elapsed:.2f} s; half-sample planes built outside the timing"}


def cpu_slice_threads(frames, seconds: float, bd: int = 8):
    """The reference-faithful CPU form: the oracle's slice loop (auto mode: each band's macroblocks in
    raster order, deciding as it goes) with one thread per slice band, as the reference's slice threads
    run (enc/mod.rs:620-628), on as many of the ring's pictures as fit in `seconds`."""
    from tests.oracle_lib import oracle_library
    from ironav_b200.inter import InterStage

    lib = oracle_library()
    threads = min(host_cores(), NSLICES)
    st = InterStage(WIDTH, HEIGHT, nslices=NSLICES, lib=lib, bd=bd)
    lib.oracle_set_threads(st.ctx, threads)
    done_mb, elapsed, pics, prev = 0, 0.0, 0, None
    while elapsed < seconds:
        t = 1 + pics % (len(frames) - 1)
        st.clear_references()
        st.push_reference(frames[t - 1], col=prev if t >= 2 else None)
        st.set_source(frames[t])
        st.begin_p_picture(qp_prime(bd))
        t0 = time.perf_counter()
        prev, _ = st.analyse_auto()
        elapsed += time.perf_counter() - t0
        done_mb += st.nmb
        pics += 1
    st.close()
    return {"value": done_mb / elapsed, "unit": "MB/s", "cores": threads, "kind": "port",
            "sample": f"{pics} pictures of the 1080p {bd}-bit ring, auto mode, {NSLICES} slice bands on {threads} threads, "
                      f"{elapsed:.2f} s; less work a macroblock than the replay workload: macroblocks under the P_Skip "
                      f"threshold are not searched"}


def host_cores() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def run_reference(args, rank, world):
    """The reference's algorithm on the host cores (the C port: the Rust reference cannot be built here)."""
    if rank != 0:
        return
    from tests.oracle_lib import oracle_library
    from ironav_b200.inter import InterStage

    lib = oracle_library()
    cores = host_cores()
    nfr = args.steps + args.warmup + 2
    frames = make_frames(0, min(nfr, RING), args.bd)
    qpp = qp_prime(args.bd)
    # decisions of every picture by the oracle's own auto mode (the reference's slice loop)
    st = InterStage(WIDTH, HEIGHT, nslices=NSLICES, lib=lib, bd=args.bd)
    lib.oracle_set_threads(st.ctx, cores)
    states = [None]
    for t in range(1, len(frames)):
        st.clear_references()
        st.push_reference(frames[t - 1], col=states[t - 1])
        st.set_source(frames[t])
        st.begin_p_picture(qpp)
        s, _ = st.analyse_auto()
        states.append(s)
    times = []
    for i in range(args.warmup + args.steps):
        t = 1 + i % (len(frames) - 1)
        st.clear_references()
        t0 = time.perf_counter()
        st.push_reference(frames[t - 1], col=states[t - 1])
        st.set_source(frames[t])
        st.begin_p_picture(qpp)
        st.analyse_replay(states[t])
        dt = time.perf_counter() - t0
        if i >= args.warmup:
            times.append(dt)
    total = sum(times)
    value = st.nmb * len(times) / total
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "MB/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * total / len(times),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u8" if args.bd == 8 else "u16",
        "data": data_desc(args.bd),
        "config": config_dict(args.bd),
        "cpu_baseline": {"value": value, "unit": "MB/s", "cores": cores, "kind": "port",
                         "sample": f"each step one 1080p picture (8160 macroblocks): planes + replay analysis, "
                                   f"{cores} threads"},
        "e2e": {"value": value, "unit": "MB/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def data_desc(bd: int = 8) -> str:
    d = "synthetic: seeded 4-octave value noise panned per frame + 8 moving rectangles, sigma 3"
    return d if bd == 8 else d + "; 10-bit: the 8-bit frame x 4 + 2 seeded low bits per sample"


def config_dict(bd: int = 8):
    return {"workload": f"1080p {bd}-bit P-picture inter analysis, replay mode: half-sample planes (K1) + all 8160 "
                        "macroblocks' P_Skip test and best_inter (K2) per step",
            "width": WIDTH, "height": HEIGHT, "bit_depth": bd, "qp": QP, "qp_prime": qp_prime(bd), "refs": 1,
            "slices": NSLICES, "mode": "replay",
            "l2": f"inputs larger than L2: ring of {RING} pictures (luma, decisions, results ~140 MB)",
            "parallelism": "replicas"}


def main():
    global RING
    args = parse()
    RING = max(3, args.ring)
    rank, world, local = dist_setup(args)
    if args.impl == "reference":
        run_reference(args, rank, world)
        return finish(world)
    if args.workload == "batched":
        run_batched(args, rank, world)
        return finish(world)
    if args.workload == "scenecut":
        run_scenecut(args, rank, world)
        return finish(world)
    if args.workload == "deblock":
        run_deblock(args, rank, world)
        return finish(world)
    if args.workload == "bpicture":
        run_bpicture(args, rank, world)
        return finish(world)
    if args.workload == "residual":
        run_residual(args, rank, world)
        return finish(world)
    if args.workload == "decide":
        run_decide(args, rank, world)
        return finish(world)
    if args.workload == "decide_batched":
        run_decide_batched(args, rank, world)
        return finish(world)
    if args.workload == "inloop":
        run_inloop(args, rank, world)
        return finish(world)
    if args.workload == "encode":
        run_encode(args, rank, world)
        return finish(world)
    if args.workload == "learned":
        run_learned(args, rank, world)
        return finish(world)

    import torch
    import torch.distributed as dist
    from ironav_b200.inter import MBRESULT_DTYPE, MBSTATE_DTYPE, InterStage, cuda_library

    lib = cuda_library()
    dev = torch.device("cuda", torch.cuda.current_device())
    bd, qpp = args.bd, qp_prime(args.bd)
    frames = make_frames(rank, RING, bd)
    stream = torch.cuda.Stream()
    st = InterStage(WIDTH, HEIGHT, nslices=NSLICES, lib=lib, bd=bd)
    st.set_stream(stream.cuda_stream)
    if args.replay_form is not None:
        st._check(lib.ironav_set_replay_form(st.ctx, args.replay_form), "ironav_set_replay_form")
    nmb = st.nmb
    d_frames = torch.from_numpy(frames.view(np.int16) if bd > 8 else frames).to(dev)
    d_states = torch.zeros((RING, nmb * 72), dtype=torch.uint8, device=dev)
    d_res = torch.zeros((RING, nmb * 104), dtype=torch.uint8, device=dev)
    fp = lambda t: d_frames[t].data_ptr()
    # decisions of every picture of the ring by the stage's auto mode (untimed set-up)
    with torch.cuda.stream(stream):
        for t in range(1, RING):
            st.clear_references()
            st.push_reference_device(fp(t - 1), WIDTH, WIDTH, HEIGHT, d_states[t - 1].data_ptr() if t >= 2 else None)
            st.set_source_device(fp(t), WIDTH)
            st.begin_p_picture(qpp)
            st.analyse_auto_device(d_states[t].data_ptr(), d_res[t].data_ptr())
        st.sync()

    def step(i, ev=None):
        t = 1 + i % (RING - 1)
        st.clear_references()
        st.push_reference_device(fp(t - 1), WIDTH, WIDTH, HEIGHT, d_states[t - 1].data_ptr() if t >= 2 else None)
        st.set_source_device(fp(t), WIDTH)
        st.begin_p_picture(qpp)
        if ev is not None:
            ev[0].record(stream)
        st.analyse_replay_device(d_states[t].data_ptr(), d_res[t].data_ptr())
        if ev is not None:
            ev[1].record(stream)

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    with torch.cuda.stream(stream):
        for i in range(args.warmup):
            step(i)
        # nvidia-smi samples every 100 ms, longer than a few timed steps: keep the GPU busy with untimed
        # steps for half a second before the timed ones so the samples cover the load around them
        clocks = Clocks(local)
        clocks.start()
        t_load = time.perf_counter()
        i = 0
        while time.perf_counter() - t_load < 0.6:
            for _ in range(8):
                step(args.warmup + i)
                i += 1
            torch.cuda.synchronize()
        barrier()
        k2_ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for i in range(args.steps):
            step(args.warmup + i, k2_ev[i])
        e1.record(stream)
        barrier()
        clk = clocks.stop()
    st.sync()
    ms = e0.elapsed_time(e1)
    k2_ms = [a.elapsed_time(b) for a, b in k2_ev]
    ms_max = max_over_ranks(ms, world, dev)
    value = world * nmb * args.steps / (ms_max * 1e-3)

    # algorithmic work of the timed launches (from the kernel's own per-macroblock counts)
    ops = []
    for i in range(args.steps):
        t = 1 + (args.warmup + i) % (RING - 1)
        r = d_res[t].cpu().numpy().view(MBRESULT_DTYPE)
        ops.append(3.0 * r["sad_px"].astype(np.float64).sum() + 9.0 * r["satd_px"].astype(np.float64).sum())
    k2_mean = float(np.mean(k2_ms))
    achieved = float(np.mean(ops)) / (k2_mean * 1e-3) / 1e12
    peak = ctypes_peak(lib)

    # the plane kernel alone, for its HBM roofline (one launch per picture, timed in isolation)
    planes_ms = time_planes(st, fp, stream, torch)
    planes_bytes = (WIDTH * HEIGHT + 4 * st.sw * st.sh) * (2 if bd > 8 else 1)  # luma read once + 4 planes written
    hbm = measured_hbm()

    # end to end through the host-buffer C ABI, pinned host memory
    e2e = None if args.no_e2e else run_e2e(args, st, frames, d_states, nmb, world, torch, dist, dev, stream)

    line = {
        "metric": METRIC, "value": value, "unit": "MB/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_max / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "u8" if bd == 8 else "u16",
        "data": data_desc(bd),
        "config": config_dict(bd),
        "e2e": e2e,
        "gpu_launches": 3 * args.steps,  # per step: half-sample planes (+ co-located vectors), the source copied with its padding, analysis
        "roofline": {"bound": "int32", "kernel": replay_kernel_name(args.replay_form if args.replay_form is not None else (1 if bd > 8 else 0), bd), "achieved": achieved, "peak": peak,
                     "unit": "Tops/s", "frac": achieved / peak if peak else None,
                     # DRAM bytes per launch (dram__bytes_read.sum + write.sum) of one ncu capture of this
                     # workload at 8 bits (ncu --set full, one launch of a 6-picture ring): the source and the
                     # reference's planes read once
                     "traffic": 11637248 + 2304 if bd == 8 else None,
                     "traffic_source": "one ncu capture of this kernel on this workload (8-bit)" if bd == 8 else None,
                     "ms_per_launch": k2_mean,
                     "note": "achieved = algorithmic ops (3 per SAD sample, 9 per SATD sample, counted by the "
                             "kernel in the reference's evaluation order) / event time; peak = measured 32-bit "
                             "integer issue rate (add+xor chains on every SM)"},
        "roofline_planes": {"bound": "hbm", "kernel": f"halfpel_planes_kernel<{'uint8_t' if bd == 8 else 'uint16_t'}>",
                            "achieved": planes_bytes / (planes_ms * 1e-3) / 1e9, "peak": hbm[0], "unit": "GB/s",
                            "frac": planes_bytes / (planes_ms * 1e-3) / 1e9 / hbm[0], "peak_source": hbm[1],
                            "ms_per_launch": planes_ms,
                            # one ncu capture at 8 bits: the luma read once; the 9.5 MB of planes written stay
                            # in L2 (the analysis reads them from there)
                            "traffic": 2670336 if bd == 8 else None,
                            "traffic_source": "one ncu capture of this kernel on this workload (8-bit)" if bd == 8 else None},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        host_states = [None] + [d_states[t].cpu().numpy().view(MBSTATE_DTYPE) for t in range(1, RING)]
        line["cpu_baseline"] = cpu_baseline(frames, host_states, args.cpu_seconds, bd)
        line["cpu_slice_threads"] = cpu_slice_threads(frames, min(args.cpu_seconds, 6.0), bd)
    if rank == 0:
        print(json.dumps(line), flush=True)
    st.close()
    return finish(world)


def run_inloop(args, rank, world):
    """In-loop mode, the drop-in as the reference's encoder would drive it (FrameCoder::encode's slice loop,
    enc/frame.rs:467-478, on one thread per slice band, enc/mod.rs:620-628): 1080p, QP 27, one reference,
    eight bands; one native host thread per band reads each macroblock's analysis, decides it (the auto
    policy standing in for the host's rate-distortion choice) and commits it through mapped host memory,
    and the device analyses a macroblock once its left and top-right neighbours are committed. One step is
    one P picture; wall clock (the picture is host-synchronous by nature), max over ranks. Against the
    reference-faithful CPU form, the oracle's own slice loop on the same number of threads."""
    import torch
    import torch.distributed as dist
    from ironav_b200.inter import MBRESULT_DTYPE, MBSTATE_DTYPE, InterStage, cuda_library, default_bands, inloop_caller

    lib, drv = cuda_library(), inloop_caller()
    dev = torch.device("cuda", torch.cuda.current_device())
    ring = min(RING, 12)
    frames = make_frames(rank, ring)
    st = InterStage(WIDTH, HEIGHT, nslices=NSLICES, lib=lib)
    nmb, thr = st.nmb, lib.ironav_skip_threshold(QP)
    bands = np.asarray(default_bands(st.mb_h, NSLICES), dtype=np.int32)
    d_frames = torch.from_numpy(frames).to(dev)
    fp = lambda t: d_frames[t].data_ptr()
    # the co-located decisions of each reference: the stage's auto mode (the in-loop decisions under the auto
    # policy are the same ones; checked below)
    d_states = torch.zeros((ring, nmb * 72), dtype=torch.uint8, device=dev)
    d_res = torch.zeros(nmb * 104, dtype=torch.uint8, device=dev)
    for t in range(1, ring):
        st.clear_references()
        st.push_reference_device(fp(t - 1), WIDTH, WIDTH, HEIGHT, d_states[t - 1].data_ptr() if t >= 2 else None)
        st.set_source_device(fp(t), WIDTH)
        st.begin_p_picture(QP)
        st.analyse_auto_device(d_states[t].data_ptr(), d_res.data_ptr())
    st.sync()
    states = np.zeros(nmb, dtype=MBSTATE_DTYPE)
    results = np.zeros(nmb, dtype=MBRESULT_DTYPE)

    def picture(i, host=False):
        t = 1 + i % (ring - 1)
        st.clear_references()
        col = d_states[t - 1].data_ptr() if t >= 2 else None
        if host:  # the host-buffer calls: the source and the reference luma from host memory
            st.push_reference(frames[t - 1], col=d_states[t - 1].cpu().numpy().view(MBSTATE_DTYPE) if t >= 2 else None)
            st.set_source(frames[t])
        else:
            st.push_reference_device(fp(t - 1), WIDTH, WIDTH, HEIGHT, col)
            st.set_source_device(fp(t), WIDTH)
        st.begin_p_picture(QP)
        s_ = drv.ironav_inloop_drive_bands(st.ctx, st.mb_w, NSLICES, bands.ctypes.data, thr, states.ctypes.data, results.ctypes.data)
        if s_ != 0:
            raise RuntimeError(f"ironav_inloop_drive_bands: status {s_}")
        return t

    t = picture(0)
    assert np.array_equal(states, d_states[t].cpu().numpy().view(MBSTATE_DTYPE)), "in-loop decisions differ from auto mode's"

    def timed(k, host):
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        t0 = time.perf_counter()
        for i in range(k):
            picture(args.warmup + i, host)
        torch.cuda.synchronize()
        return max_over_ranks(time.perf_counter() - t0, world, dev)

    for i in range(args.warmup):
        picture(i)
    clocks = Clocks(int(os.environ.get("LOCAL_RANK", "0")))
    clocks.start()
    t_load = time.perf_counter()
    i = 0
    while time.perf_counter() - t_load < 0.6:
        picture(i)
        i += 1
    el = timed(args.steps, False)
    clk = clocks.stop()
    el_host = timed(args.steps, True)
    total = sum_over_ranks(nmb, world, dev)
    line = {
        "metric": "1080p in-loop inter analysis MB/s (the host decides and commits every macroblock)", "value": total * args.steps / el,
        "unit": "MB/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * el / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u8", "data": data_desc(8),
        "config": {"workload": f"1080p 8-bit P pictures in in-loop mode, QP {QP}, one reference, {NSLICES} slice bands, one native host "
                               "thread per band (ironav_inloop_result / decide / ironav_inloop_commit per macroblock)",
                   "width": WIDTH, "height": HEIGHT, "qp": QP, "slices": NSLICES, "mode": "in-loop",
                   "l2": f"ring of {ring} pictures; the analysis reads each picture once", "parallelism": "replicas"},
        "e2e": {"value": total * args.steps / el_host, "unit": "MB/s", "h2d_bytes_per_step": 2 * WIDTH * HEIGHT + nmb * 72,
                "d2h_bytes_per_step": nmb * 104, "ms_per_step": 1e3 * el_host / args.steps,
                "note": "the source and reference luma and the reference's decisions through the host-buffer calls each step; "
                        "results reach the host and commits the device through mapped host memory (counted: one result and one "
                        "decision per macroblock)"},
        "gpu_launches": 3 * args.steps,  # per picture: planes (+ co-located vectors), source copy and padding, the in-loop analysis
        "roofline": {"bound": "latency", "kernel": "analyse_kernel<MODE_INLOOP, uint8_t>", "achieved": None, "peak": None, "unit": None,
                     "frac": None, "traffic": None,
                     "note": "each band is a chain of host round trips through mapped memory (commit -> device sees it -> analysis -> "
                             "result -> host sees it), one per macroblock"},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_slice_threads(frames, min(args.cpu_seconds, 6.0))
        line["cpu_slice_threads"] = cpu
        line["cpu_baseline"] = cpu
        line["ratio_to_cpu_slice_threads"] = line["value"] / cpu["value"]
    st.close()
    if rank == 0:
        print(json.dumps(line), flush=True)


def run_encode(args, rank, world):
    """The CAVLC encoder's whole P picture on the device (ironav_b200.encoder.DeviceEncoder.encode_device):
    scene-cut measure, decide mode (code_mb of every macroblock), the slices written on the device from the
    codes and their bytes brought back as Annex B NAL units, the filter's records, the deblocking filter, and
    the filtered picture pushed as the next reference. 1080p, QP 27, one reference, eight bands; the IDR
    picture is coded first, untimed; one step is one P picture. `value` has the sources in device memory;
    `e2e` uploads each picture's planes from host memory (DeviceEncoder.encode). Against the oracle's encoder
    loop (the same steps on the host, the decision on one thread per band). With --cabac, the default
    encoder's stream instead (High: CABAC decisions by rate-distortion cost, the CABAC writer)."""
    import torch
    import torch.distributed as dist
    from ironav_b200.encoder import DeviceEncoder, Encoder
    from ironav_b200.synth import Sequence

    dev = torch.device("cuda", torch.cuda.current_device())
    n = args.warmup + 2 * args.steps + 2
    from ironav_b200.synth import CONFIGS

    w, h, seed, pan_q, nobj, vmax, sigma = CONFIGS["1080p"]
    seq = Sequence(w, h, n, seed + 0x1000 * rank, pan_q, nobj, vmax, sigma)
    ys = [seq.frame(t) for t in range(n)]
    cs = [seq.chroma(t) for t in range(n)]
    d_y = torch.from_numpy(np.stack(ys)).to(dev)
    d_c = torch.from_numpy(np.stack([np.stack(c) for c in cs])).to(dev)
    enc = DeviceEncoder(w, h, qp=QP, keyint=10 ** 6, refs=1, nslices=NSLICES, cabac=args.cabac)
    how = "CABAC (High)" if args.cabac else "CAVLC"
    nbytes = [0]

    def picture(t):
        prev = d_y[t - 1].data_ptr() if t > 0 else None
        nbytes[0] += len(enc.encode_device(d_y[t].data_ptr(), d_c[t][0].data_ptr(), d_c[t][1].data_ptr(), w, prev))

    picture(0)  # the IDR picture
    t = 1
    for _ in range(args.warmup):
        picture(t)
        t += 1
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    clocks = Clocks(int(os.environ.get("LOCAL_RANK", "0")))
    clocks.start()
    nbytes[0] = 0
    t0 = time.perf_counter()
    for _ in range(args.steps):
        picture(t)
        t += 1
    torch.cuda.synchronize()
    el = max_over_ranks(time.perf_counter() - t0, world, dev)
    clk = clocks.stop()
    bits_per_picture = 8.0 * nbytes[0] / args.steps
    # end to end: each picture's planes uploaded from host memory by the encoder itself
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        enc.encode(ys[t], *cs[t])
        t += 1
    el_host = max_over_ranks(time.perf_counter() - t0, world, dev)
    enc.close()
    nmb = ((w + 15) // 16) * ((h + 15) // 16)
    total = sum_over_ranks(nmb, world, dev)
    line = {
        "metric": f"1080p {how} encoding MB/s on the device (decide, slices written, deblocking, next reference)",
        "value": total * args.steps / el, "unit": "MB/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * el / args.steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
        "data": data_desc(8) + "; chroma from the 2x2 luma means",
        "config": {"workload": f"1080p 8-bit P pictures through DeviceEncoder.encode_device, QP {QP}, one reference, {NSLICES} slice "
                               f"bands: scene cut, decide mode, {how} slices (device writer, NAL framing on the host), records, "
                               "deblocking, reference planes", "width": w, "height": h, "qp": QP, "slices": NSLICES,
                   "bits_per_picture": bits_per_picture, "l2": "each picture read once from a ring in device memory",
                   "parallelism": "replicas"},
        "e2e": {"value": total * args.steps / el_host, "unit": "MB/s", "h2d_bytes_per_step": w * h * 3 // 2,
                "d2h_bytes_per_step": int(bits_per_picture / 8), "ms_per_step": 1e3 * el_host / args.steps,
                "note": "DeviceEncoder.encode: the picture's three planes from host memory, the stream's bytes back"},
        # per picture: scene cut 2, source copy 1, chroma 2, decide 1, writer 3 (CABAC: 1), records 1, deblocking 2, planes 1, chroma
        # copies 2 (and their padding)
        "gpu_launches": (14 if args.cabac else 16) * args.steps,
        "roofline": {"bound": "latency", "kernel": "decide_rdw_kernel<uint8_t>" if args.cabac else "decide_kernel<uint8_t>", "achieved": None,
                     "peak": None, "unit": None, "frac": None, "traffic": None,
                     "note": ("one stream's slice bands under CABAC: 8 chains of ~1020 dependent macroblocks bound the picture"
                              if args.cabac else "one stream's decide wavefront (a chain of ~136 dependent macroblocks) bounds the picture")},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from tests.oracle_lib import oracle_library

        lib = oracle_library()
        threads = min(host_cores(), NSLICES)
        o = Encoder(w, h, qp=QP, keyint=10 ** 6, refs=1, nslices=NSLICES, lib=lib, cabac=args.cabac)
        lib.oracle_set_threads(o.st.ctx, threads)
        o.encode(ys[0], *cs[0])
        k, t0, el_o = 1, time.perf_counter(), 0.0
        while el_o < min(args.cpu_seconds, 6.0) and k < n:
            o.encode(ys[k], *cs[k])
            k += 1
            el_o = time.perf_counter() - t0
        o.close()
        line["cpu_baseline"] = {"value": (k - 1) * nmb / el_o, "unit": "MB/s", "cores": threads, "kind": "port",
                                "sample": f"{k - 1} P pictures of the same sequence through the oracle's encoder loop (host buffers), "
                                          f"decide mode on {threads} threads, {el_o:.2f} s"}
    if rank == 0:
        print(json.dumps(line), flush=True)


def run_learned(args, rank, world):
    """The learned form (ironav_b200.learned, the north star's form 4) on the 1080p sequence. Untimed first: the
    training data from the plain search on three unseen-seed 1080p sequences (11 pictures each at QP 22, 27
    and 32, eight bands), Adam on `--learned-samples` samples, and the quality of both forms through the
    device encoder at QP 22, 27 and 32 (bytes and luma PSNR of the benchmark's sequence, 11 pictures). Timed:
    one step is one 1080p P picture in auto mode (QP 27, eight bands): the reference's half-sample planes, then
    the proposer's input, four tcgen05 conv layers, head and proposals, then the analysis with the exact-cost
    judge; the plain auto-mode step (planes + analysis) is timed the same way beside it. `e2e` uploads each
    picture from pinned host memory and brings its results back."""
    import torch
    import torch.distributed as dist
    from ironav_b200 import learned
    from ironav_b200.inter import MBRESULT_DTYPE, MBSTATE_DTYPE, InterStage
    from ironav_b200.proposer import Proposer
    from ironav_b200.synth import CONFIGS, Sequence

    dev = torch.device("cuda", torch.cuda.current_device())
    t0 = time.perf_counter()
    data = learned.TrainingSet().collect(sequences=3, frames=11, qps=(22, 27, 32), nslices=NSLICES)
    collect_s = time.perf_counter() - t0
    n_train = len(data)
    prop = Proposer(max_batch=512)
    hist = learned.train(prop, data, samples=args.learned_samples, batch=512, lr=1e-3, log_every=1000)
    train_s = time.perf_counter() - t0 - collect_s
    del data
    torch.cuda.empty_cache()
    seq_eval = Sequence.config("1080p", 11)
    quality = []
    for qp in (22, 27, 32):
        plain = learned.encode_sequence(seq_eval, qp, 11, nslices=NSLICES)
        lrn = learned.encode_sequence(seq_eval, qp, 11, prop=prop, nslices=NSLICES)
        searched = lrn["judged"] + lrn["class_fallback"] + lrn["cost_fallback"]
        quality.append({"qp": qp, "bytes_plain": plain["bytes"], "bytes_learned": lrn["bytes"],
                        "bytes_delta_pct": 100.0 * (lrn["bytes"] - plain["bytes"]) / plain["bytes"],
                        "psnr_y_plain": plain["psnr_y"], "psnr_y_learned": lrn["psnr_y"],
                        "psnr_delta_db": lrn["psnr_y"] - plain["psnr_y"],
                        "fallback_rate": (lrn["class_fallback"] + lrn["cost_fallback"]) / max(1, searched),
                        "judged": lrn["judged"], "class_fallback": lrn["class_fallback"], "cost_fallback": lrn["cost_fallback"]})

    # the timed pictures: a ring of the benchmark sequence in device memory (with its activations, far above L2)
    w, h, seed, pan_q, nobj, vmax, sigma = CONFIGS["1080p"]
    npic = args.warmup + args.steps + 1
    seq = Sequence(w, h, npic, seed + 0x1000 * rank, pan_q, nobj, vmax, sigma)
    host = [seq.frame(t) for t in range(npic)]
    d_pics = torch.from_numpy(np.stack(host)).to(dev)
    st = InterStage(w, h, nslices=NSLICES)
    stream = torch.cuda.Stream()
    st.set_stream(stream.cuda_stream)
    prop.stream = stream
    n = st.nmb
    d_states = torch.zeros(n * MBSTATE_DTYPE.itemsize, dtype=torch.uint8, device=dev)
    d_out = torch.zeros(n * MBRESULT_DTYPE.itemsize, dtype=torch.uint8, device=dev)
    cands = torch.zeros((n, 8), dtype=torch.int16, device=dev)
    cls = torch.zeros(n, dtype=torch.uint8, device=dev)
    stats = torch.zeros(3, dtype=torch.int32, device=dev)
    smp = [None] + [torch.from_numpy(learned.picture_samples(d_pics[t].data_ptr(), d_pics[t - 1].data_ptr(), w, h, w, w).view(np.uint8))
                    .to(dev) for t in range(1, npic)]
    conv_ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(npic)]

    def set_learned(on: bool):
        if on:
            st._check(st.lib.ironav_set_learned(st.ctx, cands.data_ptr(), cls.data_ptr(), 0, stats.data_ptr()), "ironav_set_learned")
        else:
            st._check(st.lib.ironav_set_learned(st.ctx, None, None, 0, None), "ironav_set_learned")

    def step(t: int, on: bool, d_cur=None, d_prev=None, d_smp=None):
        cur = d_pics[t].data_ptr() if d_cur is None else d_cur
        prev = d_pics[t - 1].data_ptr() if d_prev is None else d_prev
        st.clear_references()
        st.push_reference_device(prev, w, w, h, None)
        st.set_source_device(cur, w)
        st.begin_p_picture(QP, 1)
        if on:
            prop.set_samples_device((smp[t] if d_smp is None else d_smp).data_ptr(), n)
            prop.forward(n, conv_events=conv_ev[t] if d_cur is None else None)
            prop.propose(n, cands.data_ptr(), cls.data_ptr())
        st.analyse_auto_device(d_states.data_ptr(), d_out.data_ptr())

    def timed(on: bool):
        set_learned(on)
        for t in range(1, args.warmup + 1):
            step(t, on)
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for t in range(args.warmup + 1, npic):
            step(t, on)
        e1.record(stream)
        torch.cuda.synchronize()
        return max_over_ranks(e0.elapsed_time(e1) * 1e-3, world, dev)

    # the software pipeline: picture t + 1's proposals on a stream of their own while picture t is analysed
    # (auto mode's wavefront leaves most SMs idle); two sets of proposal buffers, handed over by events
    pstream = torch.cuda.Stream()
    pc = [cands, torch.zeros_like(cands)]
    pk = [cls, torch.zeros_like(cls)]
    pev = [torch.cuda.Event() for _ in range(2)]  # proposals of buffer k written
    aev = [torch.cuda.Event() for _ in range(2)]  # analysis that read buffer k done

    def propose_into(t: int, first: bool):
        k = t & 1
        if not first:
            pstream.wait_event(aev[k])
        prop.set_samples_device(smp[t].data_ptr(), n)
        prop.forward(n, conv_events=conv_ev[t])
        prop.propose(n, pc[k].data_ptr(), pk[k].data_ptr())
        pev[k].record(pstream)

    def analyse_with(t: int):
        k = t & 1
        stream.wait_event(pev[k])
        st._check(st.lib.ironav_set_learned(st.ctx, pc[k].data_ptr(), pk[k].data_ptr(), 0, stats.data_ptr()), "ironav_set_learned")
        st.clear_references()
        st.push_reference_device(d_pics[t - 1].data_ptr(), w, w, h, None)
        st.set_source_device(d_pics[t].data_ptr(), w)
        st.begin_p_picture(QP, 1)
        st.analyse_auto_device(d_states.data_ptr(), d_out.data_ptr())
        aev[k].record(stream)

    def timed_pipelined():
        prop.stream = pstream
        try:
            out = None
            for ts in (list(range(1, args.warmup + 1)), list(range(args.warmup + 1, npic))):
                torch.cuda.synchronize()
                timing = ts[0] == args.warmup + 1
                if timing and world > 1:
                    dist.barrier()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                pstream.wait_stream(stream)
                propose_into(ts[0], True)
                for i, t in enumerate(ts):
                    if i + 1 < len(ts):
                        propose_into(ts[i + 1], i + 1 < 2)
                    analyse_with(t)
                stream.wait_stream(pstream)
                e1.record(stream)
                torch.cuda.synchronize()
                if timing:
                    out = max_over_ranks(e0.elapsed_time(e1) * 1e-3, world, dev)
            return out
        finally:
            prop.stream = stream

    el_plain = timed(False)
    el_seq = timed(True)
    clocks = Clocks(int(os.environ.get("LOCAL_RANK", "0")))
    clocks.start()
    stats.zero_()
    el = timed_pipelined()
    clk = clocks.stop()
    conv_ms = float(np.mean([a.elapsed_time(b) for a, b in conv_ev[args.warmup + 1:]]))
    judge = stats.cpu().numpy()
    set_learned(True)

    # end to end: each picture uploaded from pinned host memory into a two-picture staging ring, the results
    # brought back to pinned host memory, in stream order
    pinned = [torch.from_numpy(host[t]).pin_memory() for t in range(npic)]
    stage = [torch.zeros((h, w), dtype=torch.uint8, device=dev) for _ in range(2)]
    stage_smp = [torch.from_numpy(learned.picture_samples(stage[k].data_ptr(), stage[k ^ 1].data_ptr(), w, h, w, w).view(np.uint8)).to(dev)
                 for k in range(2)]
    res_host = torch.zeros(n * MBRESULT_DTYPE.itemsize, dtype=torch.uint8).pin_memory()
    set_learned(True)
    with torch.cuda.stream(stream):
        stage[0].copy_(pinned[0], non_blocking=True)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for t in range(1, npic):
        k = t & 1
        with torch.cuda.stream(stream):
            stage[k].copy_(pinned[t], non_blocking=True)
        step(t, True, d_cur=stage[k].data_ptr(), d_prev=stage[k ^ 1].data_ptr(), d_smp=stage_smp[k])
        with torch.cuda.stream(stream):
            res_host.copy_(d_out, non_blocking=True)
    e1.record(stream)
    torch.cuda.synchronize()
    el_e2e = max_over_ranks(e0.elapsed_time(e1) * 1e-3, world, dev)
    prop.check_errors()

    steps = npic - 1 - args.warmup
    total = sum_over_ranks(n, world, dev)
    # the four layers' roofline. Their arithmetic intensity (layers 2-4: 2 * 9 * 32 * 32 FLOP per pixel against
    # 64 bytes read and 64 written) is below the B200's ridge point, so HBM bounds them: bytes per picture =
    # every layer's input planes read once and its 4 output planes written once, 16 bytes a plane a pixel of
    # the padded rasters; the tensor-pipe fraction is reported beside it
    flops = n * 48 * 48 * 9 * 32 * 2 * (2 + 3 * 32)
    conv_bytes = n * 2500 * 16 * ((2 + 4) + 3 * (4 + 4))
    peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json"))) if os.path.exists(os.path.join(ROOT, "MEASURED_PEAKS.json")) else {}
    peak = float(peaks.get("bf16_tflops_sustained", 1400.0))
    peak_source = ("MEASURED_PEAKS.json bf16_tflops_sustained (measured)" if "bf16_tflops_sustained" in peaks
                   else "fallback 1.4 PFLOP/s, the pool's sustained bf16 rate (MEASURED_PEAKS.json absent)")
    achieved = flops / (conv_ms * 1e-3) / 1e12
    hbm = measured_hbm()
    achieved_gbs = conv_bytes / (conv_ms * 1e-3) / 1e9
    line = {
        "metric": METRIC + " (learned form)",
        "value": total * (npic - 1 - args.warmup) / el, "unit": "MB/s", "n_gpus": world, "steps": steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * el / steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "bf16+u8",
        "data": data_desc(8) + "; proposer trained on three other seeds of the same generator",
        "config": {"workload": f"1080p 8-bit P pictures in auto mode, QP {QP}, {NSLICES} slice bands: half-sample planes, proposer "
                               "(input, 4 tcgen05 conv3x3 layers of 32 channels, head, proposals), analysis with the exact-cost judge",
                   "width": w, "height": h, "qp": QP, "slices": NSLICES,
                   "plain_mb_per_s": total * steps / el_plain, "plain_ms_per_step": 1e3 * el_plain / steps,
                   "learned_over_plain": el_plain / el,
                   "learned_sequential_ms_per_step": 1e3 * el_seq / steps,
                   "pipeline": "value: picture t + 1's proposer on a second stream while picture t is analysed (two proposal "
                               "buffers handed over by events); learned_sequential_ms_per_step: proposer then analysis, one "
                               "picture after the other",
                   "quality_vs_plain": quality,
                   "judge_timed": {"judged": int(judge[0]), "class_fallback": int(judge[1]), "cost_fallback": int(judge[2])},
                   "training": {"samples_available": n_train, "samples_seen": hist[-1]["samples"], "collect_s": collect_s, "train_s": train_s,
                                "first": hist[0], "last": hist[-1]},
                   "l2": "each step reads its own picture and activations (1.3 GB a layer), far above L2",
                   "parallelism": "replicas"},
        "e2e": {"value": total * steps / el_e2e, "unit": "MB/s", "h2d_bytes_per_step": w * h,
                "d2h_bytes_per_step": n * MBRESULT_DTYPE.itemsize, "ms_per_step": 1e3 * el_e2e / steps,
                "note": "each picture copied in from pinned host memory, its result records copied out, in stream order"},
        "gpu_launches": 10 * steps,  # per step: source copy 1, planes 1, prep 1, conv 4, head 1, propose 1, analysis 1
        "roofline": {"bound": "hbm", "kernel": "conv3x3p_kernel (4 layers)", "achieved": achieved_gbs, "peak": hbm[0], "unit": "GB/s",
                     "frac": achieved_gbs / hbm[0], "traffic": None, "peak_source": hbm[1],
                     "tensor": {"achieved": achieved, "peak": peak, "unit": "TFLOP/s", "frac": achieved / peak, "peak_source": peak_source},
                     "note": f"{conv_bytes / 1e9:.2f} GB a picture (each layer's input read and output written once) and "
                             f"{flops / 1e12:.3f} TFLOP of algorithmic work on the 48 x 48 interior over the four layers' "
                             f"CUDA-event time ({conv_ms:.3f} ms a step)"},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from tests.oracle_lib import oracle_library

        lib = oracle_library()
        threads = min(host_cores(), NSLICES)
        o = InterStage(w, h, nslices=NSLICES, lib=lib)
        lib.oracle_set_threads(o.ctx, threads)
        hc = np.zeros((n, 8), dtype=np.int16)
        hk = np.zeros(n, dtype=np.uint8)
        hs = np.zeros(3, dtype=np.uint32)
        assert lib.ironav_set_learned(o.ctx, hc.ctypes.data, hk.ctypes.data, 0, hs.ctypes.data) == 0
        k, el_o = 1, 0.0
        while el_o < min(args.cpu_seconds, 8.0) and k < npic:
            step(k, True)  # the proposals of picture k, on the GPU
            torch.cuda.synchronize()
            hc[:] = cands.cpu().numpy()
            hk[:] = cls.cpu().numpy()
            t1 = time.perf_counter()
            o.clear_references()
            o.push_reference(host[k - 1])
            o.set_source(host[k])
            o.begin_p_picture(QP, 1)
            o.analyse_auto()
            el_o += time.perf_counter() - t1
            k += 1
        o.close()
        line["cpu_baseline"] = {"value": (k - 1) * n / el_o, "unit": "MB/s", "cores": threads, "kind": "port",
                                "sample": f"{k - 1} P pictures of the same sequence, the oracle's auto-mode analysis with the GPU's "
                                          f"proposals on {threads} threads (the proposer itself untimed), {el_o:.2f} s"}
    st.close()
    if rank == 0:
        print(json.dumps(line), flush=True)


def run_batched(args, rank, world):
    """The batched configuration: streams with resolutions drawn from {640x360, 854x480, 1280x720,
    1920x1080}, QP 27, one reference, auto mode (the streams' wavefronts decide every macroblock). One
    step = every stream's next picture: sources, reference planes and the analysis, each one launch over
    all streams. Compared with the plain per-stream launch loop (each stream's own launches, one after
    another) and with the batched step replayed from a CUDA graph. Streams are split across ranks."""
    import torch
    import torch.distributed as dist
    from ironav_b200.inter import InterBatch, InterStage, cuda_library
    from ironav_b200.synth import Sequence, batch_streams

    lib = cuda_library()
    dev = torch.device("cuda", torch.cuda.current_device())
    mine = split_streams(batch_streams(args.streams), rank, world)
    stream = torch.cuda.Stream()
    stages, frames = [], []
    for (w, h, ns, seed) in mine:
        seq = Sequence.config("1080p", 3, seed=seed, size=(w, h))
        frames.append([torch.from_numpy(seq.frame(t)).to(dev) for t in range(3)])
        st = InterStage(w, h, nslices=ns, lib=lib)
        st.set_stream(stream.cuda_stream)
        st.push_reference_device(frames[-1][0].data_ptr(), w, w, h, None)
        st.begin_p_picture(QP)
        stages.append(st)
    n = len(stages)
    nmb = sum(st.nmb for st in stages)
    d_states = [[torch.zeros(st.nmb * 72, dtype=torch.uint8, device=dev) for _ in range(2)] for st in stages]
    d_res = [torch.zeros(st.nmb * 104, dtype=torch.uint8, device=dev) for st in stages]
    torch.cuda.synchronize()
    batch = InterBatch(stages)

    def args_of(i):
        t = 1 + i % 2
        col = [d_states[k][(i + 1) % 2].data_ptr() if i > 0 else None for k in range(n)]
        return ([f[t].data_ptr() for f in frames], [f[t - 1].data_ptr() for f in frames], col,
                [d_states[k][i % 2].data_ptr() for k in range(n)], [d.data_ptr() for d in d_res])

    def batched(i):
        batch.step(*args_of(i))

    def plain(i):
        src, ref, col, sts, res = args_of(i)
        for k, st in enumerate(stages):
            st.clear_references()
            st.push_reference_device(ref[k], st.width, st.width, st.height, col[k])
            st.set_source_device(src[k], st.width)
            st.begin_p_picture(QP)
            st.analyse_auto_device(sts[k], res[k])

    def timed(fn, k):
        with torch.cuda.stream(stream):
            for i in range(args.warmup):
                fn(i)
            torch.cuda.synchronize()
            if world > 1:
                dist.barrier()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for i in range(k):
                fn(args.warmup + i)
            e1.record(stream)
            torch.cuda.synchronize()
        return max_over_ranks(e0.elapsed_time(e1), world, dev)

    clocks = Clocks(int(os.environ.get("LOCAL_RANK", "0")))
    clocks.start()
    ms_fixed = timed(batched, args.steps)  # the default setting (4 CTAs an SM, 16-row plane tiles, order 0)
    batch.sync()
    # the project's tuner: every setting timed on this mix (untimed here), the fastest kept
    with torch.cuda.stream(stream):
        tune = batch.autotune(*args_of(args.warmup + args.steps), reps=5)
    ms_b = timed(batched, args.steps)
    batch.sync()
    ms_p = timed(plain, args.steps)
    for st in stages:
        st.sync()
    clk = clocks.stop()
    # the batched step replayed from a CUDA graph (fixed inputs)
    for k, st in enumerate(stages):
        st.clear_references()
        st.push_reference_device(frames[k][0].data_ptr(), st.width, st.width, st.height, None)
        st.begin_p_picture(QP)
    batched(0)
    batch.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        batch.step(*args_of(1))
    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            g.replay()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            g.replay()
        e1.record(stream)
    torch.cuda.synchronize()
    batch.sync()
    ms_g = e0.elapsed_time(e1)
    # the job's macroblocks: every rank's own share summed (the ranks' shares differ in size)
    total = sum_over_ranks(nmb, world, dev)
    mbs = lambda ms: total * args.steps / (ms * 1e-3)
    line = {
        "metric": f"batched inter-analysis MB/s: {args.streams} mixed-resolution streams, auto mode, one launch per stage and step",
        "value": mbs(ms_b), "unit": "MB/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": ms_b / args.steps, "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
        "dtype": "u8", "data": "synthetic: per-stream seeded value noise, pan, 8 moving rectangles, sigma 3",
        "config": {"workload": f"{args.streams} streams ({n} on rank 0), {nmb} macroblocks per step on rank 0, QP {QP}, "
                               "one reference, auto mode", "parallelism": "streams split across ranks"},
        "plain_loop": {"value": mbs(ms_p), "ms_per_step": ms_p / args.steps,
                       "note": "each stream's own launches (planes, source, auto-mode analysis), one after another"},
        "graph": {"value": nmb * args.steps / (ms_g * 1e-3), "ms_per_step": ms_g / args.steps,
                  "note": "the batched step captured once in a CUDA graph and replayed (rank 0's streams alone)"},
        "speedup_vs_plain_loop": ms_p / ms_b,
        "autotune": {"best": tune["best"], "fixed_value": mbs(ms_fixed), "fixed_ms_per_step": ms_fixed / args.steps,
                     "tuned_vs_fixed": ms_fixed / ms_b, "settings": tune["all"],
                     "note": "value is the tuned setting's; fixed is the default (4 CTAs an SM, 16-row plane tiles, order 0)"},
        "clocks": clk,
    }
    del g
    batch.close()
    if rank == 0:
        print(json.dumps(line), flush=True)


def run_scenecut(args, rank, world):
    """The scene-cut measure at 1080p (change_threads, codec/change.rs:56-90): low-resolution luma of two
    pictures and the +-4 search of every 8x8 low-resolution block, device-resident, against the oracle on
    the host. One step = one picture pair."""
    import torch
    from ironav_b200.inter import InterStage, cuda_library
    from tests.oracle_lib import oracle_library

    dev = torch.device("cuda", torch.cuda.current_device())
    frames = make_frames(rank, 8)
    d = torch.from_numpy(frames).to(dev)
    st = InterStage(WIDTH, HEIGHT, lib=cuda_library())
    out = np.zeros(2, dtype=np.int64)
    lib = st.lib
    for i in range(args.warmup):
        lib.ironav_scene_change_device(st.ctx, d[i % 7].data_ptr(), d[i % 7 + 1].data_ptr(), WIDTH, out.ctypes.data)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for i in range(args.steps):
        lib.ironav_scene_change_device(st.ctx, d[i % 7].data_ptr(), d[i % 7 + 1].data_ptr(), WIDTH, out.ctypes.data)
    el = time.perf_counter() - t0
    o = InterStage(WIDTH, HEIGHT, lib=oracle_library())
    t0 = time.perf_counter()
    n_cpu = 0
    while time.perf_counter() - t0 < 3.0:
        o.scene_change(frames[n_cpu % 7], frames[n_cpu % 7 + 1])
        n_cpu += 1
    el_cpu = time.perf_counter() - t0
    if rank == 0:
        print(json.dumps({
            "metric": "1080p scene-cut measure, picture pairs per second", "value": args.steps / el, "unit": "pairs/s",
            "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * el / args.steps,
            "higher_is_better": True, "scaling": "replicas", "vs_baseline": None, "dtype": "u8", "data": "synthetic",
            "config": {"workload": "low-resolution luma of both pictures + +-4 search of 2040 8x8 blocks, one call per pair "
                                   "(synchronous: returns the totals)"},
            "cpu_baseline": {"value": n_cpu / el_cpu, "unit": "pairs/s", "cores": 1, "kind": "port",
                             "sample": f"{n_cpu} pairs, one thread (the reference's non-live setting)"}}), flush=True)


def run_bpicture(args, rank, world):
    """The B-picture searches at 1080p (decide_b's 16x16 list 0 / list 1 / bi, best_b_parts, spatial direct;
    enc/frame.rs:1518-1747), replay mode, device-resident: one step = all 8160 macroblocks of one B picture
    (frames t, t+1, t+2 of a synthetic sequence: list 0, the B picture, list 1). A ring of contexts (each
    with its two reference pictures) larger than L2; the decisions replayed are those the B results favour,
    made before the timed region. The oracle runs the same pictures on all host cores."""
    import torch
    from ironav_b200.inter import BRESULT_DTYPE, MBSTATE_B_DTYPE, InterStage, b_decision_states, cuda_library
    from ironav_b200.synth import CONFIGS, Sequence

    lib = cuda_library()
    ring = max(2, min(args.ring, 6))
    w, h, seed, pan_q, nobj, vmax, sigma = CONFIGS["1080p"]
    seq = Sequence(w, h, 2 * ring + 1, seed + 0x1000 * rank, pan_q, nobj, vmax, sigma)
    qpp = QP + 2  # the encoder's B pictures: QP + 2
    stream = torch.cuda.Stream()
    stages, d_states, d_res, frames, states_h = [], [], [], [], []
    for k in range(ring):
        f = [seq.frame(2 * k + t) for t in range(3)]
        st = InterStage(w, h, max_refs=2, nslices=NSLICES, lib=lib)
        st.push_reference(f[0])
        st.set_source(f[2])
        st.begin_p_picture(QP)
        col, _ = st.analyse_auto()
        st.push_reference(f[2], col=col)
        st.set_source(f[1])
        st.begin_b_picture(qpp, ref_l0=1, ref_l1=0, col=col, tb=1, td=2)
        states = b_decision_states(st.analyse_b_replay(np.zeros(st.nmb, dtype=MBSTATE_B_DTYPE)))
        st.set_stream(stream.cuda_stream)
        stages.append(st)
        frames.append((f, col))
        states_h.append(states)
        d_states.append(torch.from_numpy(states.view(np.uint8)).cuda())
        d_res.append(torch.zeros(st.nmb * 200, dtype=torch.uint8, device="cuda"))
    nmb = stages[0].nmb

    def step(i, ev=None):
        k = i % ring
        if ev is not None:
            ev[0].record(stream)
        lib.ironav_analyse_b_replay_device(stages[k].ctx, d_states[k].data_ptr(), d_res[k].data_ptr())
        if ev is not None:
            ev[1].record(stream)

    with torch.cuda.stream(stream):
        for i in range(args.warmup):
            step(i)
        clocks = Clocks(int(os.environ.get("LOCAL_RANK", 0)))
        clocks.start()
        t_load = time.perf_counter()
        i = 0
        while time.perf_counter() - t_load < 0.6:
            step(args.warmup + i)
            i += 1
            if i % 8 == 0:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for i in range(args.steps):
            step(args.warmup + i, evs[i])
        e1.record(stream)
        torch.cuda.synchronize()
        clk = clocks.stop()
    ms = e0.elapsed_time(e1)
    k_ms = float(np.mean([a.elapsed_time(b) for a, b in evs]))
    value = world * nmb * args.steps / (ms * 1e-3)
    ops = []
    for i in range(args.steps):
        r = d_res[(args.warmup + i) % ring].cpu().numpy().view(BRESULT_DTYPE)
        ops.append(3.0 * r["sad_px"].astype(np.float64).sum() + 9.0 * r["satd_px"].astype(np.float64).sum())
    achieved = float(np.mean(ops)) / (k_ms * 1e-3) / 1e12
    peak = ctypes_peak(lib)
    # end to end: decisions in and results out through the host-buffer call, pinned memory
    pin_s = [torch.from_numpy(s_.view(np.uint8)).pin_memory() for s_ in states_h]
    pin_r = [torch.zeros(nmb * 200, dtype=torch.uint8).pin_memory() for _ in range(ring)]
    for st in stages:
        st.set_stream(None)
    for i in range(args.warmup):
        lib.ironav_analyse_b_replay(stages[i % ring].ctx, pin_s[i % ring].data_ptr(), pin_r[i % ring].data_ptr())
    t0 = time.perf_counter()
    for i in range(args.steps):
        k = i % ring
        s_ = lib.ironav_analyse_b_replay(stages[k].ctx, pin_s[k].data_ptr(), pin_r[k].data_ptr())
        if s_:
            raise RuntimeError(f"ironav_analyse_b_replay: {s_}")
    el = time.perf_counter() - t0
    line = {
        "metric": "1080p B-picture inter-analysis MB/s", "value": value, "unit": "MB/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u8",
        "data": "synthetic: seeded 4-octave value noise panned per frame + 8 moving rectangles, sigma 3",
        "config": {"workload": f"1080p B picture (list 0 = frame t, list 1 = frame t+2, QP' {qpp}, tb 1, td 2), replay mode: "
                               "spatial direct, 16x16 list 0 / list 1 / bi, best_b_parts for all 8160 macroblocks per step",
                   "slices": NSLICES, "mode": "replay", "l2": f"ring of {ring} contexts (two reference pictures each, > L2)"},
        "gpu_launches": args.steps,
        "e2e": {"value": world * nmb * args.steps / el, "unit": "MB/s", "h2d_bytes_per_step": nmb * 140,
                "d2h_bytes_per_step": nmb * 200, "ms_per_step": 1e3 * el / args.steps,
                "note": "ironav_analyse_b_replay on pinned host buffers, one thread"},
        "roofline": {"bound": "int32", "kernel": "analyse_b_kernel<uint8_t>", "achieved": achieved, "peak": peak,
                     "unit": "Tops/s", "frac": achieved / peak if peak else None, "traffic": None, "ms_per_launch": k_ms,
                     "note": "algorithmic ops: 3 per SAD sample, 9 per SATD sample (searches, bi and direct SATDs)"},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from tests.oracle_lib import oracle_library

        olib = oracle_library()
        cores = host_cores()
        f, col = frames[0]
        o = InterStage(w, h, max_refs=2, nslices=NSLICES, lib=olib)
        olib.oracle_set_threads(o.ctx, cores)
        o.push_reference(f[0])
        o.push_reference(f[2], col=col)
        o.set_source(f[1])
        o.begin_b_picture(qpp, ref_l0=1, ref_l1=0, col=col, tb=1, td=2)
        n_cpu, t_cpu = 0, 0.0
        while t_cpu < min(args.cpu_seconds, 10.0):
            t0 = time.perf_counter()
            o.analyse_b_replay(states_h[0])
            t_cpu += time.perf_counter() - t0
            n_cpu += 1
        line["cpu_baseline"] = {"value": n_cpu * nmb / t_cpu, "unit": "MB/s", "cores": cores, "kind": "port",
                                "sample": f"{n_cpu} B pictures (the ring's first), replay mode, {cores} threads, {t_cpu:.1f} s"}
    if rank == 0:
        print(json.dumps(line), flush=True)
    for st in stages:
        st.close()


def run_decide_batched(args, rank, world):
    """Decide mode for many streams in one launch (ironav_batch_decide): streams with resolutions drawn
    from {640x360, 854x480, 1280x720, 1920x1080} (the batched configuration's), QP 27, one reference each;
    one step = every stream's P picture decided and coded. Compared with the per-stream loop (each
    stream's own decide launch, one after another). Streams are split across ranks. With --cabac, the
    default encoder's decision (decide_rd under CABAC): every stream's slice bands as chains of one launch."""
    import torch
    from ironav_b200.inter import MBCODE_DTYPE, InterBatch, InterStage, cuda_library
    from ironav_b200.synth import Sequence, batch_streams

    lib = cuda_library()
    dev = torch.device("cuda", torch.cuda.current_device())
    mine = split_streams(batch_streams(args.streams), rank, world)
    stream = torch.cuda.Stream()
    stages, bufs, pin_src, d_src, seqs = [], [], [], [], []
    for (w, h, ns, seed) in mine:
        seq = Sequence.config("1080p", 2, seed=seed, size=(w, h))
        st = InterStage(w, h, nslices=ns, lib=lib)
        st.push_reference(seq.frame(0))
        st.push_reference_chroma(*seq.chroma(0))
        st.set_source(seq.frame(1))
        st.set_source_chroma(*seq.chroma(1))
        st.set_entropy(args.cabac, True)
        st.begin_p_picture(QP)
        st.set_stream(stream.cuda_stream)
        stages.append(st)
        seqs.append((seq.frame(0), seq.chroma(0), seq.frame(1), seq.chroma(1)))
        pin_src.append(torch.from_numpy(seq.frame(1)).pin_memory())
        d_src.append(torch.empty((h, w), dtype=torch.uint8, device=dev))
        bufs.append((torch.zeros(st.nmb * 72, dtype=torch.uint8, device=dev), torch.zeros(st.nmb * MBCODE_DTYPE.itemsize, dtype=torch.uint8, device=dev),
                     torch.zeros((st.mb_h * 16, st.mb_w * 16), dtype=torch.uint8, device=dev),
                     torch.zeros((2, st.mb_h * 8, st.mb_w * 8), dtype=torch.uint8, device=dev)))
    n = len(stages)
    nmb = sum(st.nmb for st in stages)
    torch.cuda.synchronize()
    batch = InterBatch(stages)
    dargs = ([b[0].data_ptr() for b in bufs], [b[1].data_ptr() for b in bufs], [b[2].data_ptr() for b in bufs],
             [b[2].shape[1] for b in bufs], [b[3][0].data_ptr() for b in bufs], [b[3][1].data_ptr() for b in bufs],
             [b[3].shape[2] for b in bufs])

    def batched():
        batch.decide(*dargs)

    def plain():
        for k, st in enumerate(stages):
            s_, c_, y, c = bufs[k]
            r = lib.ironav_decide_p_picture_device(st.ctx, s_.data_ptr(), c_.data_ptr(), y.data_ptr(), y.shape[1], c[0].data_ptr(),
                                                   c[1].data_ptr(), c.shape[2])
            if r:
                raise RuntimeError(f"ironav_decide_p_picture_device: {r}")

    def timed(fn, k):
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(k)]
        for i in range(k):
            evs[i][0].record(stream)
            fn()
            evs[i][1].record(stream)
        torch.cuda.synchronize()
        return [a.elapsed_time(b) for a, b in evs]

    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            batched()
        batch.sync()
        clocks = Clocks(int(os.environ.get("LOCAL_RANK", 0)))
        clocks.start()
        t_load = time.perf_counter()
        while time.perf_counter() - t_load < 0.6:
            batched()
            batch.sync()
        torch.cuda.synchronize()
        if world > 1:
            import torch.distributed as dist

            dist.barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        per = timed(batched, args.steps)
        e1.record(stream)
        batch.sync()
        clk = clocks.stop()
        ms = max_over_ranks(e0.elapsed_time(e1), world, dev)
        plain_ms = float(np.median(timed(plain, max(2, min(args.steps, 5)))))
        # end to end: every stream's source luma from pinned host memory, the launch, and the states, codes
        # and reconstructions back to pinned host memory, each step
        host = [(torch.empty(b[0].shape, dtype=torch.uint8).pin_memory(), torch.empty(b[1].shape, dtype=torch.uint8).pin_memory(),
                 torch.empty(b[2].shape, dtype=torch.uint8).pin_memory(), torch.empty(b[3].shape, dtype=torch.uint8).pin_memory())
                for b in bufs]

        def e2e_step():
            for k, st in enumerate(stages):
                d_src[k].copy_(pin_src[k], non_blocking=True)
                st.set_source_device(d_src[k].data_ptr(), d_src[k].shape[1])
            batched()
            for k in range(n):
                for a, b in zip(host[k], bufs[k]):
                    a.copy_(b, non_blocking=True)
        for _ in range(2):
            e2e_step()
        batch.sync()
        if world > 1:
            dist.barrier()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            e2e_step()
        batch.sync()
        el = max_over_ranks(time.perf_counter() - t0, world, dev)
    # the whole P picture of every stream: batched decide, each stream's filter records, batched deblocking
    from ironav_b200.inter import DBK_MB_DTYPE
    from ironav_b200.synth import dbk_encoder_slices

    d_mbs = [torch.zeros(st.nmb * DBK_MB_DTYPE.itemsize, dtype=torch.uint8, device=dev) for st in stages]
    slice_tabs = [dbk_encoder_slices(ns) for (_, _, ns, _) in mine]

    def pipeline():
        batched()
        for k, st in enumerate(stages):
            r = lib.ironav_decide_dbk_records_device(st.ctx, bufs[k][1].data_ptr(), bufs[k][0].data_ptr(), d_mbs[k].data_ptr())
            if r:
                raise RuntimeError(f"ironav_decide_dbk_records_device: {r}")
        batch.deblock(dargs[2], dargs[3], dargs[4], dargs[5], dargs[6], [t.data_ptr() for t in d_mbs], slice_tabs)

    with torch.cuda.stream(stream):
        for _ in range(2):
            pipeline()
        batch.sync()
        pipe_ms = float(np.median(timed(pipeline, max(2, min(args.steps, 5)))))
        batch.sync()
    # the job's macroblocks: every rank's own share summed (the ranks' shares differ in size)
    total = sum_over_ranks(nmb, world, dev)
    value = total * args.steps / (ms * 1e-3)
    line = {
        "metric": "P-picture macroblock decision + coding MB/s, many streams in one launch "
                  f"({'CABAC decide_rd, High' if args.cabac else 'CAVLC code_mb'})", "value": value,
        "unit": "MB/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps,
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "u8",
        "data": "synthetic: per-stream seeded value noise, pan, 8 moving rectangles, sigma 3; chroma from the 2x2 luma means",
        "config": {"workload": f"{args.streams} streams ({n} on rank 0) of 640x360..1920x1080, {nmb} macroblocks per step on rank 0, QP "
                               f"{QP}, one reference each, decide mode, ironav_batch_decide",
                   "per_stream_loop_ms": plain_ms, "batched_ms": float(np.median(per)),
                   "picture_pipeline_ms": pipe_ms,
                   "picture_pipeline_note": "ironav_batch_decide + each stream's ironav_decide_dbk_records_device + "
                                            "ironav_batch_deblock: every stream's P picture decided, coded and deblocked",
                   "l2": "inputs of all streams (planes, chroma, codes, reconstructions) exceed L2"},
        "gpu_launches": args.steps,
        "e2e": {"value": total * args.steps / el, "unit": "MB/s",
                "h2d_bytes_per_step": sum(int(p.numel()) for p in pin_src),
                "d2h_bytes_per_step": sum(sum(int(t.numel()) for t in b) for b in bufs), "ms_per_step": 1e3 * el / args.steps,
                "note": "each stream's source luma from pinned host memory (its chroma stays resident) + the launch + states, "
                        "codes and reconstructions back to pinned host memory"},
        "roofline": {"bound": "latency", "kernel": "decide_rdw_batch_kernel" if args.cabac else "decide_batch_kernel", "achieved": None,
                     "peak": None, "unit": None, "frac": None,
                     "traffic": None, "ms_per_launch": float(np.median(per)),
                     "note": "many wavefronts interleaved; the per-stream loop above is the same work one stream at a time"},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from tests.oracle_lib import oracle_library

        olib = oracle_library()
        cores = host_cores()
        (w, h, ns, seed) = mine[0]
        o = InterStage(w, h, nslices=ns, lib=olib)
        olib.oracle_set_threads(o.ctx, cores)
        o.set_entropy(args.cabac, True)
        f0, c0, f1, c1 = seqs[0]
        o.push_reference(f0)
        o.push_reference_chroma(*c0)
        o.set_source(f1)
        o.set_source_chroma(*c1)
        o.begin_p_picture(QP)
        n_cpu, t_cpu = 0, 0.0
        while t_cpu < min(args.cpu_seconds, 10.0):
            t0 = time.perf_counter()
            o.decide_p_picture()
            t_cpu += time.perf_counter() - t0
            n_cpu += 1
        line["cpu_baseline"] = {"value": n_cpu * o.nmb / t_cpu, "unit": "MB/s", "cores": min(cores, ns), "kind": "port",
                                "sample": f"{n_cpu} pictures of the first stream ({w}x{h}, {ns} slice bands on {min(cores, ns)} threads), {t_cpu:.1f} s"}
        o.close()
    if rank == 0:
        print(json.dumps(line), flush=True)
    batch.close()
    for st in stages:
        st.close()


def run_decide(args, rank, world):
    """The whole P macroblock decision of the CAVLC encoder at 1080p (code_mb, enc/frame.rs:715-790: P_Skip
    tests, best_i16, best_inter, the Intra4x4 trial, the coding of the chosen macroblock into the unfiltered
    reconstruction) in the device wavefront, device-resident: one step = every macroblock of one P picture.
    With --cabac, the default encoder's decision instead (decide_rd, enc/frame.rs:1462-1513: every candidate
    coded and the least SSD + lambda2 * CABAC bits kept), one chain per slice band. A ring of contexts
    (reference planes and chroma, states, codes, reconstructions) larger than L2. The oracle decides the same
    picture on all host cores (slice bands in parallel, as the reference's slice threads)."""
    import torch
    from ironav_b200.inter import MBCODE_DTYPE, InterStage, cuda_library
    from ironav_b200.synth import CONFIGS, Sequence

    bd = args.bd
    lib = cuda_library()
    ring = max(2, min(args.ring, 6))
    w, h, seed, pan_q, nobj, vmax, sigma = CONFIGS["1080p"]
    seq = Sequence(w, h, ring + 1, seed + 0x3000 * rank, pan_q, nobj, vmax, sigma)
    frame = (lambda t: seq.frame10(t)) if bd == 10 else seq.frame
    qpp = QP + 6 * (bd - 8)
    stream = torch.cuda.Stream()
    dev = torch.device("cuda", torch.cuda.current_device())
    stages, bufs, srcs = [], [], []
    dt = torch.uint8 if bd == 8 else torch.int16
    for k in range(ring):
        st = InterStage(w, h, max_refs=1, nslices=NSLICES, lib=lib, bd=bd)
        st.push_reference(frame(k))
        st.push_reference_chroma(*seq.chroma(k, bd))
        st.set_source(frame(k + 1))
        st.set_source_chroma(*seq.chroma(k + 1, bd))
        st.set_entropy(args.cabac, True)
        st.begin_p_picture(qpp)
        st.set_stream(stream.cuda_stream)
        stages.append(st)
        srcs.append((frame(k), seq.chroma(k, bd), frame(k + 1), seq.chroma(k + 1, bd)))
        bufs.append((torch.zeros(st.nmb * 72, dtype=torch.uint8, device=dev), torch.zeros(st.nmb * MBCODE_DTYPE.itemsize, dtype=torch.uint8, device=dev),
                     torch.zeros((st.mb_h * 16, st.mb_w * 16), dtype=dt, device=dev), torch.zeros((2, st.mb_h * 8, st.mb_w * 8), dtype=dt, device=dev)))
    nmb, mb_w, mb_h = stages[0].nmb, stages[0].mb_w, stages[0].mb_h

    def step(i, ev=None):
        k = i % ring
        s_, c_, y, c = bufs[k]
        if ev is not None:
            ev[0].record(stream)
        r = lib.ironav_decide_p_picture_device(stages[k].ctx, s_.data_ptr(), c_.data_ptr(), y.data_ptr(), y.shape[1], c[0].data_ptr(),
                                               c[1].data_ptr(), c.shape[2])
        if r:
            raise RuntimeError(f"ironav_decide_p_picture_device: {r}")
        if ev is not None:
            ev[1].record(stream)

    with torch.cuda.stream(stream):
        for i in range(args.warmup):
            step(i)
        clocks = Clocks(int(os.environ.get("LOCAL_RANK", 0)))
        clocks.start()
        t_load = time.perf_counter()
        i = 0
        while time.perf_counter() - t_load < 0.6:
            step(args.warmup + i)
            i += 1
            if i % 8 == 0:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for i in range(args.steps):
            step(args.warmup + i, evs[i])
        e1.record(stream)
        torch.cuda.synchronize()
        clk = clocks.stop()
    for st in stages:
        st.sync()
    ms = e0.elapsed_time(e1)
    k_ms = float(np.mean([a.elapsed_time(b) for a, b in evs]))
    value = world * nmb * args.steps / (ms * 1e-3)
    # the whole P picture on the device: decide, the filter's records, deblocking (the reference's order,
    # enc/mod.rs:633-655), one stream
    from ironav_b200.inter import DBK_MB_DTYPE
    from ironav_b200.synth import dbk_encoder_slices

    d_mbs = [torch.zeros(nmb * DBK_MB_DTYPE.itemsize, dtype=torch.uint8, device=dev) for _ in range(ring)]
    slices = dbk_encoder_slices(NSLICES)

    def picture(i):
        k = i % ring
        s_, c_, y, c = bufs[k]
        step(i)
        r = lib.ironav_decide_dbk_records_device(stages[k].ctx, c_.data_ptr(), s_.data_ptr(), d_mbs[k].data_ptr())
        if r:
            raise RuntimeError(f"ironav_decide_dbk_records_device: {r}")
        stages[k].deblock_device(y.data_ptr(), y.shape[1], c[0].data_ptr(), c[1].data_ptr(), c.shape[2], d_mbs[k].data_ptr(), slices)

    with torch.cuda.stream(stream):
        for i in range(args.warmup):
            picture(i)
        torch.cuda.synchronize()
        p0, p1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        p0.record(stream)
        for i in range(args.steps):
            picture(args.warmup + i)
        p1.record(stream)
        torch.cuda.synchronize()
    pic_ms = p0.elapsed_time(p1) / args.steps
    codes = bufs[0][1].cpu().numpy().view(MBCODE_DTYPE)
    kinds = {"skip": int(codes["skip"].sum()), "inter": int(((codes["kind"] == 5) & (codes["skip"] == 0)).sum()),
             "i16": int((codes["kind"] == 3).sum()), "i4": int((codes["kind"] == 1).sum())}
    if args.cabac:
        kinds["i8"] = int((codes["kind"] == 2).sum())
        kinds["inter_t8"] = int(((codes["kind"] == 5) & (codes["res"]["t8x8"] != 0)).sum())
    how = "CABAC decide_rd, High" if args.cabac else "CAVLC code_mb"
    # end to end through the host-buffer call (states, codes and the reconstruction back every step)
    for st in stages:
        st.set_stream(None)
    for i in range(args.warmup):
        stages[i % ring].decide_p_picture()
    t0 = time.perf_counter()
    for i in range(args.steps):
        stages[i % ring].decide_p_picture()
    el = time.perf_counter() - t0
    B = 1 if bd == 8 else 2
    line = {
        "metric": f"1080p P-picture macroblock decision + coding MB/s ({bd}-bit, {how})", "value": value, "unit": "MB/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "int32",
        "data": "synthetic: seeded 4-octave value noise panned per frame + 8 moving rectangles, sigma 3; chroma from the 2x2 "
                "luma means",
        "config": {"workload": f"decide and code every macroblock of one 1920x1088 {bd}-bit P picture per step (QP {QP}, one "
                               f"reference, 8 slice bands, {'one chain a band' if args.cabac else 'wavefront'}); decisions: {kinds}",
                   "slices": NSLICES, "mode": "decide (device pointers)",
                   "l2": f"ring of {ring} contexts (reference planes, chroma, states, codes, reconstructions > L2)"},
        "picture_pipeline": {"ms_per_picture": pic_ms, "MB/s": world * nmb / (pic_ms * 1e-3),
                             "note": "decide + ironav_decide_dbk_records_device + the deblocking filter (two launches), "
                                     "device pointers, the same ring, timed after the main region"},
        "gpu_launches": args.steps,
        "e2e": {"value": world * nmb * args.steps / el, "unit": "MB/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": nmb * (72 + MBCODE_DTYPE.itemsize + 384 * B), "ms_per_step": 1e3 * el / args.steps,
                "note": "ironav_decide_p_picture with host buffers (sources and references already held by the contexts)"},
        "roofline": {"bound": "latency", "kernel": f"{'decide_rdw_kernel' if args.cabac else 'decide_kernel'}<{'uint8_t' if bd == 8 else 'uint16_t'}>",
                     "achieved": None, "peak": None, "unit": None, "frac": None, "traffic": None, "ms_per_launch": k_ms,
                     "note": (f"one chain a slice band: {nmb // NSLICES} dependent macroblocks (each macroblock's CABAC cost reads "
                              "the contexts every earlier one in its slice left), five warps each"
                              if args.cabac else
                              f"one stream's wavefront: a critical path of mb_w + 2 (band rows - 1) = {mb_w + 2 * (-(-mb_h // NSLICES) - 1)} "
                              "dependent macroblocks; see the per-macroblock latency in the profile")},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from tests.oracle_lib import oracle_library

        olib = oracle_library()
        cores = host_cores()
        o = InterStage(w, h, max_refs=1, nslices=NSLICES, lib=olib, bd=bd)
        olib.oracle_set_threads(o.ctx, cores)
        o.set_entropy(args.cabac, True)
        f0, c0, f1, c1 = srcs[0]
        o.push_reference(f0)
        o.push_reference_chroma(*c0)
        o.set_source(f1)
        o.set_source_chroma(*c1)
        o.begin_p_picture(qpp)
        n_cpu, t_cpu = 0, 0.0
        while t_cpu < min(args.cpu_seconds, 10.0):
            t0 = time.perf_counter()
            o.decide_p_picture()
            t_cpu += time.perf_counter() - t0
            n_cpu += 1
        line["cpu_baseline"] = {"value": n_cpu * nmb / t_cpu, "unit": "MB/s", "cores": min(cores, NSLICES), "kind": "port",
                                "sample": f"{n_cpu} P pictures (the ring's first), slice bands on {min(cores, NSLICES)} threads, {t_cpu:.1f} s"}
        o.close()
    if rank == 0:
        print(json.dumps(line), flush=True)
    for st in stages:
        st.close()


def run_residual(args, rank, world):
    """Inter residual coding and reconstruction at 1080p (code_inter / code_inter_residual / code_luma8 /
    code_chroma, enc/frame.rs:1202-1305, 1856-1915), device-resident: one step = every macroblock of one P
    picture coded from its decision (P_Skip prediction, or luma and chroma motion compensation, 4x4 or 8x8
    transform, quantisation, decimation, chroma DC/AC, dequantisation, inverse transform into the
    reconstruction). The decisions are those of the stage's own auto-mode analysis (8x8 transform allowed),
    made before the timed region. A ring of contexts (reference planes, chroma, codes, reconstructions) larger
    than L2. The oracle codes the same picture on all host cores."""
    import torch
    from ironav_b200.inter import INTERCODE_DTYPE, InterStage, cuda_library, inter_decisions
    from ironav_b200.synth import CONFIGS, Sequence

    bd = args.bd
    lib = cuda_library()
    ring = max(2, min(args.ring, 6))
    w, h, seed, pan_q, nobj, vmax, sigma = CONFIGS["1080p"]
    seq = Sequence(w, h, ring + 1, seed + 0x2000 * rank, pan_q, nobj, vmax, sigma)
    qp = QP
    frame = (lambda t: seq.frame10(t)) if bd == 10 else seq.frame
    stream = torch.cuda.Stream()
    dev = torch.device("cuda", torch.cuda.current_device())
    stages, d_decs, d_codes, d_rec, decs_h, srcs = [], [], [], [], [], []
    for k in range(ring):
        st = InterStage(w, h, max_refs=1, nslices=NSLICES, lib=lib, bd=bd)
        st.push_reference(frame(k))
        st.push_reference_chroma(*seq.chroma(k, bd))
        st.set_source(frame(k + 1))
        st.set_source_chroma(*seq.chroma(k + 1, bd))
        st.begin_p_picture(qp + 6 * (bd - 8))
        _, res = st.analyse_auto()
        decs = inter_decisions(res, t8=True)
        st.set_stream(stream.cuda_stream)
        stages.append(st)
        decs_h.append(decs)
        srcs.append((frame(k), seq.chroma(k, bd), frame(k + 1), seq.chroma(k + 1, bd)))
        d_decs.append(torch.from_numpy(decs.view(np.uint8)).to(dev))
        d_codes.append(torch.zeros(st.nmb * INTERCODE_DTYPE.itemsize, dtype=torch.uint8, device=dev))
        dt = torch.uint8 if bd == 8 else torch.int16
        d_rec.append((torch.zeros((st.mb_h * 16, st.mb_w * 16), dtype=dt, device=dev),
                      torch.zeros((2, st.mb_h * 8, st.mb_w * 8), dtype=dt, device=dev)))
    nmb, mb_w, mb_h = stages[0].nmb, stages[0].mb_w, stages[0].mb_h
    modes = np.bincount(decs_h[0]["mode"], minlength=3)

    def step(i, ev=None):
        k = i % ring
        y, c = d_rec[k]
        if ev is not None:
            ev[0].record(stream)
        s_ = lib.ironav_code_inter_picture_device(stages[k].ctx, qp + 6 * (bd - 8), d_decs[k].data_ptr(), d_codes[k].data_ptr(),
                                                  y.data_ptr(), y.shape[1], c[0].data_ptr(), c[1].data_ptr(), c.shape[2])
        if s_:
            raise RuntimeError(f"ironav_code_inter_picture_device: {s_}")
        if ev is not None:
            ev[1].record(stream)

    with torch.cuda.stream(stream):
        for i in range(args.warmup):
            step(i)
        clocks = Clocks(int(os.environ.get("LOCAL_RANK", 0)))
        clocks.start()
        t_load = time.perf_counter()
        i = 0
        while time.perf_counter() - t_load < 0.6:
            step(args.warmup + i)
            i += 1
            if i % 8 == 0:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for i in range(args.steps):
            step(args.warmup + i, evs[i])
        e1.record(stream)
        torch.cuda.synchronize()
        clk = clocks.stop()
    for st in stages:
        st.sync()
    ms = e0.elapsed_time(e1)
    k_ms = float(np.mean([a.elapsed_time(b) for a, b in evs]))
    value = world * nmb * args.steps / (ms * 1e-3)
    B = 1 if bd == 8 else 2
    # algorithmic bytes of one picture: every decision read and code record written; per P_Skip or inter
    # macroblock its reference samples read once (luma 16x16, chroma 2 x 8x8) and its reconstruction written;
    # per inter macroblock its source luma and chroma read
    def algo_bytes(m):
        return nmb * (78 + 1324) + int(m[1] + m[2]) * 2 * 384 * B + int(m[2]) * 384 * B
    bytes_per = algo_bytes(modes)
    hbm = measured_hbm()

    # the residual path everywhere: the same vectors, every macroblock coded with its residual (no P_Skip)
    coded = []
    for k in range(ring):
        d = decs_h[k].copy()
        d["mode"] = 2
        coded.append(torch.from_numpy(d.view(np.uint8)).to(dev))
    ev_c = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    with torch.cuda.stream(stream):
        for i in range(args.warmup + args.steps):
            k = i % ring
            y, c = d_rec[k]
            if i >= args.warmup:
                ev_c[i - args.warmup][0].record(stream)
            s_ = lib.ironav_code_inter_picture_device(stages[k].ctx, qp + 6 * (bd - 8), coded[k].data_ptr(), d_codes[k].data_ptr(),
                                                      y.data_ptr(), y.shape[1], c[0].data_ptr(), c[1].data_ptr(), c.shape[2])
            if s_:
                raise RuntimeError(f"ironav_code_inter_picture_device: {s_}")
            if i >= args.warmup:
                ev_c[i - args.warmup][1].record(stream)
        torch.cuda.synchronize()
    kc_ms = float(np.mean([a.elapsed_time(b) for a, b in ev_c]))
    bytes_c = algo_bytes([0, 0, nmb])

    # end to end through the host-buffer call: decisions and the reconstruction planes in, codes and planes out
    ho = [InterStage(w, h, max_refs=1, nslices=NSLICES, lib=lib, bd=bd) for _ in range(2)]
    for k, o_ in enumerate(ho):
        f0, c0, f1, c1 = srcs[k]
        o_.push_reference(f0)
        o_.push_reference_chroma(*c0)
        o_.set_source(f1)
        o_.set_source_chroma(*c1)
        o_.begin_p_picture(qp + 6 * (bd - 8))
    tnp = (lambda a: torch.from_numpy(a).pin_memory())
    pin_d = [tnp(decs_h[k].view(np.uint8)) for k in range(2)]
    pin_c = [torch.zeros(nmb * INTERCODE_DTYPE.itemsize, dtype=torch.uint8).pin_memory() for _ in range(2)]
    dt_np = np.uint8 if bd == 8 else np.int16
    pin_y = [tnp(np.zeros((mb_h * 16, mb_w * 16), dt_np)) for _ in range(2)]
    pin_ch = [tnp(np.zeros((2, mb_h * 8, mb_w * 8), dt_np)) for _ in range(2)]

    def host_call(k):
        return lib.ironav_code_inter_picture(ho[k].ctx, qp + 6 * (bd - 8), pin_d[k].data_ptr(), pin_c[k].data_ptr(),
                                             pin_y[k].data_ptr(), mb_w * 16, pin_ch[k][0].data_ptr(), pin_ch[k][1].data_ptr(),
                                             mb_w * 8)
    for i in range(args.warmup):
        host_call(i % 2)
    t0 = time.perf_counter()
    for i in range(args.steps):
        s_ = host_call(i % 2)
        if s_:
            raise RuntimeError(f"ironav_code_inter_picture: {s_}")
    el = time.perf_counter() - t0
    plane_bytes = nmb * 384 * B
    line = {
        "metric": f"1080p P-picture inter residual coding + reconstruction MB/s ({bd}-bit)", "value": value, "unit": "MB/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
        "data": "synthetic: seeded 4-octave value noise panned per frame + 8 moving rectangles, sigma 3; chroma "
                "from the 2x2 luma means",
        "config": {"workload": f"code every macroblock of one 1920x1088 {bd}-bit P picture per step (QP {qp}, 8x8 "
                               f"transform allowed) from the stage's own decisions: {int(modes[1])} P_Skip, "
                               f"{int(modes[2])} inter, {int(modes[0])} left to intra",
                   "slices": NSLICES, "mode": "device pointers",
                   "l2": f"ring of {ring} contexts (reference planes, chroma, codes, reconstructions > L2)"},
        "gpu_launches": args.steps,
        "e2e": {"value": world * nmb * args.steps / el, "unit": "MB/s",
                "h2d_bytes_per_step": nmb * 78 + plane_bytes, "d2h_bytes_per_step": nmb * 1324 + plane_bytes,
                "ms_per_step": 1e3 * el / args.steps,
                "note": "ironav_code_inter_picture on pinned host buffers, one thread"},
        "roofline": {"bound": "hbm", "kernel": f"code_inter_kernel<{'uint8_t' if bd == 8 else 'uint16_t'}>",
                     "achieved": bytes_per / (k_ms * 1e-3) / 1e9, "peak": hbm[0], "unit": "GB/s",
                     "frac": bytes_per / (k_ms * 1e-3) / 1e9 / hbm[0], "peak_source": hbm[1], "ms_per_launch": k_ms,
                     "traffic": None,
                     "note": "algorithmic bytes: decisions, source, reference samples once, codes and reconstruction"},
        "all_coded": {"ms_per_launch": kc_ms, "MB/s": nmb / (kc_ms * 1e-3), "achieved_gbs": bytes_c / (kc_ms * 1e-3) / 1e9,
                      "frac": bytes_c / (kc_ms * 1e-3) / 1e9 / hbm[0],
                      "note": "the same vectors with every macroblock coded with its residual (mode 2), timed after the "
                              "timed region with the same events and ring"},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from tests.oracle_lib import oracle_library

        olib = oracle_library()
        cores = host_cores()
        o = InterStage(w, h, max_refs=1, nslices=NSLICES, lib=olib, bd=bd)
        olib.oracle_set_threads(o.ctx, cores)
        f0, c0, f1, c1 = srcs[0]
        o.push_reference(f0)
        o.push_reference_chroma(*c0)
        o.set_source(f1)
        o.set_source_chroma(*c1)
        o.begin_p_picture(qp + 6 * (bd - 8))
        dt_np = np.uint8 if bd == 8 else np.uint16
        rec = (np.zeros((mb_h * 16, mb_w * 16), dt_np), np.zeros((mb_h * 8, mb_w * 8), dt_np), np.zeros((mb_h * 8, mb_w * 8), dt_np))
        n_cpu, t_cpu = 0, 0.0
        while t_cpu < min(args.cpu_seconds, 10.0):
            t0 = time.perf_counter()
            o.code_inter(qp + 6 * (bd - 8), decs_h[0], rec)
            t_cpu += time.perf_counter() - t0
            n_cpu += 1
        line["cpu_baseline"] = {"value": n_cpu * nmb / t_cpu, "unit": "MB/s", "cores": cores, "kind": "port",
                                "sample": f"{n_cpu} P pictures (the ring's first), {cores} threads, {t_cpu:.1f} s"}
        o.close()
    if rank == 0:
        print(json.dumps(line), flush=True)
    for st in stages + ho:
        st.close()


def run_deblock(args, rank, world):
    """The deblocking filter of 1080p reconstructions (h264/deblock.rs, 4:2:0, frame pictures; the encoder's
    slice table: 8 row bands, filtered across their edges), device-resident: one step = restore a pristine
    picture into the working buffers (device copy) + filter it in place. A ring of pictures and records
    larger than L2. The oracle (the reference's raster-order deblock_picture restated, one thread) is timed
    on the host over a bounded sample."""
    import torch
    from ironav_b200.inter import InterStage, cuda_library
    from ironav_b200.synth import dbk_encoder_slices, dbk_planes, dbk_records

    bd = args.bd
    dev = torch.device("cuda", torch.cuda.current_device())
    lib = cuda_library()
    st = InterStage(WIDTH, HEIGHT, lib=lib, bd=bd)
    stream = torch.cuda.Stream()
    st.set_stream(stream.cuda_stream)
    mb_w, mb_h, nmb = st.mb_w, st.mb_h, st.nmb
    ring = max(3, min(args.ring, 40))
    rng = np.random.default_rng(0xDB0C + rank)
    pics, recs = [], []
    for _ in range(ring):
        pics.append(dbk_planes(rng, mb_w, mb_h, bd))
        recs.append(dbk_records(rng, mb_w, mb_h, NSLICES, bd, slice_rows=True)[0])
    slices = dbk_encoder_slices(NSLICES)
    itemsize = pics[0][0].dtype.itemsize
    tv = (lambda a: torch.from_numpy(a.view(np.int16) if itemsize == 2 else a))
    d_y = torch.stack([tv(p[0]) for p in pics]).to(dev)
    d_cb = torch.stack([tv(p[1]) for p in pics]).to(dev)
    d_cr = torch.stack([tv(p[2]) for p in pics]).to(dev)
    d_m = torch.stack([torch.from_numpy(r.view(np.uint8)) for r in recs]).to(dev)
    w_y, w_cb, w_cr = torch.empty_like(d_y[0]), torch.empty_like(d_cb[0]), torch.empty_like(d_cr[0])
    ys, cs = mb_w * 16, mb_w * 8

    def step(i, ev=None):
        t = i % ring
        w_y.copy_(d_y[t])
        w_cb.copy_(d_cb[t])
        w_cr.copy_(d_cr[t])
        if ev is not None:
            ev[0].record(stream)
        st.deblock_device(w_y.data_ptr(), ys, w_cb.data_ptr(), w_cr.data_ptr(), cs, d_m[t].data_ptr(), slices)
        if ev is not None:
            ev[1].record(stream)

    with torch.cuda.stream(stream):
        for i in range(args.warmup):
            step(i)
        clocks = Clocks(int(os.environ.get("LOCAL_RANK", 0)))
        clocks.start()
        t_load = time.perf_counter()
        i = 0
        while time.perf_counter() - t_load < 0.6:
            step(args.warmup + i)
            i += 1
            if i % 8 == 0:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for i in range(args.steps):
            step(args.warmup + i, evs[i])
        e1.record(stream)
        torch.cuda.synchronize()
        clk = clocks.stop()
    st.sync()
    ms = e0.elapsed_time(e1)
    k_ms = float(np.mean([a.elapsed_time(b) for a, b in evs]))
    value = world * nmb * args.steps / (ms * 1e-3)
    bytes_per = 2 * (mb_w * 16 * mb_h * 16 * 3 // 2) * itemsize + nmb * 192  # planes read + written, records read
    hbm = measured_hbm()

    # end to end through the host-buffer call, pinned host memory
    pin = [[torch.from_numpy(a.view(np.int16) if itemsize == 2 else a).pin_memory().numpy() for a in p] for p in pics[:8]]
    pin_m = [torch.from_numpy(r.view(np.uint8)).pin_memory().numpy() for r in recs[:8]]
    ho = InterStage(WIDTH, HEIGHT, lib=lib, bd=bd)
    for i in range(args.warmup):
        lib.ironav_deblock_picture(ho.ctx, pin[i % 8][0].ctypes.data, ys, pin[i % 8][1].ctypes.data, pin[i % 8][2].ctypes.data,
                                   cs, pin_m[i % 8].ctypes.data, slices.ctypes.data, NSLICES)
    t0 = time.perf_counter()
    for i in range(args.steps):
        k = i % 8
        s_ = lib.ironav_deblock_picture(ho.ctx, pin[k][0].ctypes.data, ys, pin[k][1].ctypes.data, pin[k][2].ctypes.data,
                                        cs, pin_m[k].ctypes.data, slices.ctypes.data, NSLICES)
        if s_:
            raise RuntimeError(f"ironav_deblock_picture: {s_}")
    el = time.perf_counter() - t0

    line = {
        "metric": f"1080p deblocking MB/s ({bd}-bit, 4:2:0)", "value": value, "unit": "MB/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u8" if bd == 8 else "u16",
        "data": "synthetic: ramp + per-4x4-block steps + noise; seeded macroblock records (intra/inter, coded blocks, "
                "one/two lists, 8x8 transform, keep macroblocks)",
        "config": {"workload": f"deblock one 1920x1088 {bd}-bit 4:2:0 picture per step (restored from a ring of {ring} "
                               "by a device copy, then filtered in place)", "slices": NSLICES, "mode": "device pointers",
                   "l2": f"ring of {ring} pictures and records (> L2)"},
        "gpu_launches": args.steps,
        "e2e": {"value": world * nmb * args.steps / el, "unit": "MB/s",
                "h2d_bytes_per_step": (mb_w * 16 * mb_h * 16 * 3 // 2) * itemsize + nmb * 192 + NSLICES * 20,
                "d2h_bytes_per_step": (mb_w * 16 * mb_h * 16 * 3 // 2) * itemsize,
                "ms_per_step": 1e3 * el / args.steps, "note": "ironav_deblock_picture on pinned host buffers, one thread"},
        "roofline": {"bound": "hbm", "kernel": f"deblock_kernel<{'uint8_t' if bd == 8 else 'uint16_t'}>",
                     "achieved": bytes_per / (k_ms * 1e-3) / 1e9, "peak": hbm[0], "unit": "GB/s",
                     "frac": bytes_per / (k_ms * 1e-3) / 1e9 / hbm[0], "peak_source": hbm[1], "ms_per_launch": k_ms,
                     "traffic": None,
                     "note": f"latency bound: the macroblock-row wavefront's critical path is mb_w + 2 (mb_h - 1) = "
                             f"{mb_w + 2 * (mb_h - 1)} macroblock steps"},
        "clocks": clk,
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from tests.oracle_lib import oracle_library

        o = InterStage(WIDTH, HEIGHT, lib=oracle_library(), bd=bd)
        n_cpu, t_cpu = 0, 0.0
        while t_cpu < min(args.cpu_seconds, 10.0):
            k = n_cpu % ring
            y, cb, cr = (a.copy() for a in pics[k])
            t0 = time.perf_counter()
            o.lib.ironav_deblock_picture(o.ctx, y.ctypes.data, ys, cb.ctypes.data, cr.ctypes.data, cs, recs[k].ctypes.data,
                                         slices.ctypes.data, NSLICES)
            t_cpu += time.perf_counter() - t0
            n_cpu += 1
        line["cpu_baseline"] = {"value": n_cpu * nmb / t_cpu, "unit": "MB/s", "cores": 1, "kind": "port",
                                "sample": f"{n_cpu} pictures, the oracle's raster-order filter on one thread "
                                          f"(deblock_picture), {t_cpu:.1f} s"}
    if rank == 0:
        print(json.dumps(line), flush=True)
    st.close()
    ho.close()


def ctypes_peak(lib):
    import ctypes

    v = ctypes.c_double()
    f = lib.ironav_measure_int32_peak
    f.argtypes = [ctypes.POINTER(ctypes.c_double)]
    return v.value if f(ctypes.byref(v)) == 0 else None


def replay_kernel_name(form: int, bd: int) -> str:
    t = "uint8_t" if bd == 8 else "uint16_t"
    return f"analyse_kernel<MODE_REPLAY, {t}>" if form == 1 else f"g8::analyse_replay_g8_kernel<{t}, {({2: 16, 3: 4}).get(form, 8)}>"


def measured_hbm():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            return float(json.load(f)["hbm_gbs"]), "MEASURED_PEAKS.json hbm_gbs (measured)"
    except (OSError, KeyError, ValueError):
        return 6650.0, "fallback 6.65 TB/s"


def time_planes(st, fp, stream, torch, n=20):
    evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(n)]
    with torch.cuda.stream(stream):
        for i in range(n):
            st.clear_references()
            evs[i][0].record(stream)
            st.push_reference_device(fp(i % RING), WIDTH, WIDTH, HEIGHT, None)
            evs[i][1].record(stream)
        st.sync()
    return float(np.mean([a.elapsed_time(b) for a, b in evs[3:]]))


def run_e2e(args, st, frames, d_states, nmb, world, torch, dist, dev, stream):
    """The same steps through the host-buffer ABI: every step copies its source, its reference and both
    decision arrays in from pinned host memory and its results out. The calls return when their work is
    done, so the steps are spread over a few host threads, each with its own context and CUDA stream: one
    step's transfers overlap another's kernels. Steps i, i + T, i + 2T ... go to thread i (T threads)."""
    import threading

    from ironav_b200.inter import MBRESULT_DTYPE, InterStage

    n = min(RING, 12)
    nthreads = max(1, args.e2e_threads)
    pin_frames = torch.from_numpy(frames[:n].view(np.int16) if frames.dtype == np.uint16 else frames[:n]).pin_memory()
    pin_states = d_states[:n].cpu().pin_memory()
    fr = pin_frames.numpy()
    stv = pin_states.numpy()
    lib = st.lib
    workers = []
    for k in range(nthreads):
        ws = InterStage(WIDTH, HEIGHT, nslices=NSLICES, lib=lib, bd=args.bd)
        if args.replay_form is not None:
            ws._check(lib.ironav_set_replay_form(ws.ctx, args.replay_form), "ironav_set_replay_form")
        wstream = torch.cuda.Stream()
        ws.set_stream(wstream.cuda_stream)
        out = torch.zeros((nmb * 104,), dtype=torch.uint8).pin_memory()
        workers.append((ws, wstream, out, out.numpy().view(MBRESULT_DTYPE)))
    qpp = qp_prime(args.bd)
    lam, thr = lib.ironav_lambda(qpp), lib.ironav_skip_threshold(qpp)

    def step(w, i):
        ws, _, _, out = workers[w]
        t = 1 + i % (n - 1)
        col = stv[t - 1].ctypes.data if t >= 2 else None
        s = lib.ironav_clear_references(ws.ctx)
        s |= lib.ironav_push_reference(ws.ctx, fr[t - 1].ctypes.data, WIDTH, WIDTH, HEIGHT, col)
        s |= lib.ironav_set_source(ws.ctx, fr[t].ctypes.data, WIDTH)
        s |= lib.ironav_begin_p_picture(ws.ctx, qpp, lam, thr, 1, 0, 0)
        s |= lib.ironav_analyse_picture_replay(ws.ctx, stv[t].ctypes.data, out.ctypes.data)
        if s:
            raise RuntimeError(f"e2e step failed: {s}")

    def run(first, count):
        errors = []

        def worker(w):
            try:
                for i in range(first + w, first + count, nthreads):
                    step(w, i)
            except Exception as e:  # reported after the join
                errors.append(e)

        threads = [threading.Thread(target=worker, args=(w,)) for w in range(nthreads)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        if errors:
            raise errors[0]

    run(0, max(args.warmup, nthreads))
    torch.cuda.synchronize()
    # the timed window is at least E2E_MIN_S of wall clock: K steps, repeated as often as one untimed pass of K
    # steps says that takes (the same count on every rank)
    t0 = time.perf_counter()
    run(args.warmup, args.steps)
    torch.cuda.synchronize()
    once = max_over_ranks(time.perf_counter() - t0, world, dev)
    reps = max(1, int(np.ceil(E2E_MIN_S / max(once, 1e-6))))
    if world > 1:
        dist.barrier()
    t0 = time.perf_counter()
    for k in range(reps):
        run(args.warmup + k * args.steps, args.steps)
    torch.cuda.synchronize()
    el = max_over_ranks(time.perf_counter() - t0, world, dev)
    steps = reps * args.steps
    for ws, *_ in workers:
        ws.close()
    return {"value": world * nmb * steps / el, "unit": "MB/s",
            "h2d_bytes_per_step": 2 * WIDTH * HEIGHT * fr.itemsize + 2 * nmb * 72, "d2h_bytes_per_step": nmb * 104,
            "ms_per_step": 1e3 * el / steps, "host_threads": nthreads, "steps": steps, "seconds": el,
            "note": "host-buffer C ABI calls (each returns when its work is done) from pinned host memory, "
                    f"steps spread over {nthreads} host threads with a context and CUDA stream each; wall clock "
                    f"around {reps} x K steps (at least {E2E_MIN_S} s), max over ranks; above the device-resident value "
                    "when several pictures' copies and kernels overlap on their streams (value runs one stream, step "
                    "after step)"}


def finish(world):
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
