#!/usr/bin/env python3
"""Benchmark of the plain BN254 G1 MSM at N = 2^22 (one JSON line on rank 0).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl b200|reference]

A step is one msm_execute_async over 2^22 points: uniform Montgomery-form
scalars (seed 1) against resident bases k_i * G (k_i from seed 1, generated on
the device).  `value` times K steps with device-resident inputs (bases
256 MiB + scalars 128 MiB, larger than the 126 MB L2, so no flush is needed);
`e2e` times K steps through the same C ABI with the scalars in pinned host
memory and the 254 results written to pinned host memory, copies included.

Both arms print the same `config` and these objects beside the headline:
  "configs"  the other plain configurations, each timed the same way:
             N = 2^12 uniform (seed 0) and N = 2^22 skewed (seed 2: 40 % zero,
             20 % one, 20 % below 2^16, 20 % uniform);
  "batched"  the uneven 64-instance batch (lengths log-uniform in [2^10, 2^22],
             seed 3, over one resident 2^22-point table): the per-execution
             device time (mean, p50, p99) of the batched graph against the
             per-iteration time of the 64-call plain loop; for the reference,
             the 64 calls zero-padded to powers of two (--no-batched skips it).
The b200 arm adds the stage times, the roofline objects, the on-device final
sum, the CPU baseline (the oracle's multithreaded host Pippenger) and
  "serving"  Poisson arrivals of requests with sizes log-uniform in [2^12, 2^23]
             over a resident 2^23-point table and a 16 GiB scratch budget: the
             request server (continuous batching) against a plain loop running
             one request per call, both with latency measured from each
             request's scheduled arrival (p50/p99) and Mpoints/s, at 0.6, 0.9
             and 1.2 times the plain loop's capacity; a sample of both loops'
             results is checked against the oracle after the timed runs
             (--serving-requests, 10,000 per rate by default as in the
             configuration; --no-serving skips it).

--impl reference runs the reference era-bellman-cuda msm_execute_async built
for sm_100a from its own sources (oracle/_ref/libbellman-cuda-ref.so) on the
same inputs: the reference is a CUDA library with no CPU implementation of the
MSM.  That process maps only the reference library: its bases are generated by
a child process (this script with --gen-bases, which uses this repository's
library) and read back from files.

Multi-GPU: one process per GPU (torchrun); the MSM does not shard in the
reference's API, so every rank runs an independent replica (weak scaling) and
the job value is N * 2^22 points over the slowest rank's time.
"""
from __future__ import annotations

import argparse
import json
import os
import shutil
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(REPO, "era-bellman-cuda_b200"))

METRIC = "BN254 MSM Mpoints/s at 2^22 and batched p50/p99 vs plain per-call; bit-exact"
REF_LIB = os.path.join(REPO, "oracle", "_ref", "libbellman-cuda-ref.so")
MEASURED_PEAKS = os.path.join(REPO, "MEASURED_PEAKS.json")
FALLBACK_HBM_GBS = 6650.0
MADD_MULOPS = 2392  # 6 mul (264) + 2 sqr (208) + one a*b - c*d (392) per XYZZ += affine
AFFINE_MULOPS = 1528  # 5 mul (264) + 1 sqr (208) per affine pair sum of the (optional) affine levels
# DRAM bytes (dram__bytes_read.sum + dram__bytes_write.sum) of one accumulate_kernel launch per
# nonzero entry it processes, from the ncu --set full capture of the 2^21 uniform case at
# c = 17 (2.678 GB over 31.46 M entries); a launch's traffic grows with the entries it gathers.
ACC_DRAM_BYTES_PER_ENTRY = 85.1

# (name, distribution, seed, log2 N): the headline and the other plain configurations
HEADLINE = ("config 1", "uniform", 1, 22)
OTHER_CONFIGS = (("config 0", "uniform", 0, 12), ("config 2", "skewed", 2, 22))
BATCH_SEED, BATCH_TABLE_LOG = 3, 22


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["b200", "reference"], default="b200")
    ap.add_argument("--log-n", type=int, default=22, help="log2 N of the headline MSM (profiling of smaller cases)")
    ap.add_argument("--affine-levels", type=int, default=None,
                    help="affine pairing levels of the plain MSMs (msm_b200_set_affine_levels; default: the library's, none)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-configs", action="store_true", help="skip configs 0 and 2")
    ap.add_argument("--no-batched", action="store_true", help="skip the 64-instance batch")
    ap.add_argument("--no-serving", action="store_true", help="skip the serving run")
    ap.add_argument("--serving-requests", type=int, default=10000, help="requests per rate")
    ap.add_argument("--batched-only", action="store_true",
                    help="profiling aid: run only the batched section (--steps executions) and print its object")
    ap.add_argument("--batched-scale", type=int, default=1, help="with --batched-only: divide every instance length by this")
    ap.add_argument("--gen-bases", nargs="+", metavar="ARG",
                    help="child mode: OUT_DIR SEED:LOG_N ... -- write k_i * G (k from seed) as bases_SEED_LOGN.bin")
    return ap.parse_args()


class Dist:
    """Rank bookkeeping; a gloo group only for the barrier and the max of times."""

    def __init__(self, n):
        self.rank = int(os.environ.get("RANK", "0"))
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.local = int(os.environ.get("LOCAL_RANK", "0"))
        self.pg = None
        if self.world > 1:
            import datetime

            import torch.distributed as dist
            dist.init_process_group("gloo", timeout=datetime.timedelta(seconds=120))
            self.pg = dist
        if n != self.world and self.world > 1:
            print(f"warning: --gpus {n} but WORLD_SIZE {self.world}", file=sys.stderr)

    def barrier(self):
        if self.pg:
            self.pg.barrier()

    def max(self, x: float) -> float:
        if not self.pg:
            return x
        import torch
        t = torch.tensor([x], dtype=torch.float64)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def close(self):
        if self.pg:
            self.pg.destroy_process_group()


class ClockSampler:
    """nvidia-smi samples during the timed region (clocks and throttle reasons)."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.idx = gpu_index
        self.proc = None
        self.path = os.path.join(tempfile.gettempdir(), f"bench_clocks_{os.getpid()}.csv")

    def start(self):
        try:
            self.out = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.idx), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                                          "-lms", "200"], stdout=self.out, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self):
        if not self.proc:
            return None
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.out.close()
        sm, mx, reasons = [], [], set()
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for name, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(name)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons), "samples": len(sm)}


def hbm_peak():
    try:
        return float(json.load(open(MEASURED_PEAKS))["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs)"
    except (OSError, KeyError, ValueError):
        return FALLBACK_HBM_GBS, "fallback 6.65 TB/s"


# ---------------------------------------------------------------------------
# bases k_i * G: generated on the device by this repository's library, in this
# process (b200 arm) or in a child process writing files (reference arm)
# ---------------------------------------------------------------------------
def generate_bases(ours, seed: int, n: int, stream) -> int:
    """n bases k_i * G (k_i = synth.base_multipliers(seed, n)) on the device; returns the pointer."""
    import synth
    kd = ours.to_device(synth.base_multipliers(seed, n))
    bd = ours.malloc(n * 64)
    ours.generator_multiples(kd, bd, n, stream)
    ours.stream_synchronize(stream)
    ours.free(kd)
    return bd


def gen_bases_child(args) -> None:
    """--gen-bases OUT_DIR SEED:LOG_N ...: one file of raw Montgomery affine bases per pair."""
    import bellman_cuda as bcm
    out_dir, pairs = args[0], args[1:]
    bc = bcm.BellmanCuda()
    bc.set_device(int(os.environ.get("LOCAL_RANK", "0")))
    stream = bc.stream_create(True)
    for pair in pairs:
        seed, log_n = (int(x) for x in pair.split(":"))
        bd = generate_bases(bc, seed, 1 << log_n, stream)
        bc.from_device(bd, (1 << log_n, 16)).tofile(os.path.join(out_dir, f"bases_{seed}_{log_n}.bin"))
        bc.free(bd)
    bc.stream_destroy(stream)


class ReferenceBases:
    """Bases for the reference arm, made by a child process of this script; the
    reference process itself only reads the files."""

    def __init__(self, pairs, local_rank: int):
        base = "/dev/shm" if os.path.isdir("/dev/shm") and shutil.disk_usage("/dev/shm").free > (3 << 30) else None
        self.dir = tempfile.mkdtemp(prefix="bench_bases_", dir=base)
        env = dict(os.environ, LOCAL_RANK=str(local_rank))
        subprocess.run([sys.executable, os.path.abspath(__file__), "--gen-bases", self.dir, *[f"{s}:{l}" for s, l in pairs]],
                       check=True, env=env)

    def get(self, seed: int, log_n: int) -> np.ndarray:
        return np.fromfile(os.path.join(self.dir, f"bases_{seed}_{log_n}.bin"), dtype=np.uint32).reshape(-1, 16)

    def close(self):
        shutil.rmtree(self.dir, ignore_errors=True)


# ---------------------------------------------------------------------------
# timing helpers (CUDA events on the launching stream)
# ---------------------------------------------------------------------------
def time_steps(bc, stream, k: int, enqueue) -> float:
    """ms per step of k enqueued steps."""
    e0, e1 = bc.event_create(), bc.event_create()
    bc.stream_synchronize(stream)
    bc.event_record(e0, stream)
    for _ in range(k):
        enqueue()
    bc.event_record(e1, stream)
    bc.event_synchronize(e1)
    ms = bc.elapsed_ms(e0, e1) / k
    bc.event_destroy(e0)
    bc.event_destroy(e1)
    return ms


def time_each(bc, stream, k: int, enqueue) -> list:
    """Device time of each of k back-to-back steps (an event between steps), in ms."""
    events = [bc.event_create() for _ in range(k + 1)]
    bc.stream_synchronize(stream)
    bc.event_record(events[0], stream)
    for i in range(k):
        enqueue()
        bc.event_record(events[i + 1], stream)
    bc.event_synchronize(events[k])
    out = [bc.elapsed_ms(events[i], events[i + 1]) for i in range(k)]
    for ev in events:
        bc.event_destroy(ev)
    return out


def dist_summary(ms: list, points: int) -> dict:
    mean = float(np.mean(ms))
    return {"value": round(points / mean / 1e3, 2), "ms": round(mean, 3), "p50_ms": round(float(np.percentile(ms, 50)), 3),
            "p99_ms": round(float(np.percentile(ms, 99)), 3), "samples": len(ms)}


# ---------------------------------------------------------------------------
# the other plain configurations
# ---------------------------------------------------------------------------
def other_configs(bc, pool, stream, bases_of, steps: int, warmup: int, slow_reference: bool) -> list:
    """Configs 0 and 2, device-resident, timed like the headline.  The reference's
    skewed 2^22 MSM takes seconds per call (its per-bucket loop is serial), so the
    reference arm times it over 3 steps after 1 warm-up."""
    import synth
    out = []
    for name, dist, seed, log_n in OTHER_CONFIGS:
        n = 1 << log_n
        scalars, _ = synth.workload(dist, n, seed)
        bases_dev = bases_of(seed, log_n)
        sd = bc.to_device(scalars)
        rd = bc.malloc(254 * 96)
        k, w = (3, 1) if (slow_reference and dist == "skewed") else (steps, warmup)
        for _ in range(w):
            bc.msm(pool, stream, bases_dev, sd, rd, log_n)
        ms = time_steps(bc, stream, k, lambda: bc.msm(pool, stream, bases_dev, sd, rd, log_n))
        out.append({"config": name, "workload": f"plain single MSM, N=2^{log_n}, {dist} Montgomery-form scalars (seed {seed}), resident bases "
                                                f"k_i*G (k_i seed {seed}), device-resident inputs and results",
                    "n": n, "value": round(n / (ms * 1e-3) / 1e6, 3), "unit": "Mpoints/s", "ms_per_step": round(ms, 4), "steps": k, "warmup": w})
        for p in (sd, rd, bases_dev):
            bc.free(p)
    return out


# ---------------------------------------------------------------------------
# CPU baseline (the oracle's multithreaded host Pippenger)
# ---------------------------------------------------------------------------
def cpu_baseline(bc, scalars_all: np.ndarray, bases_dev: int, results_dev: int, target_s: float = 6.0):
    """Multithreaded host Pippenger (the CPU oracle) on a bounded prefix of the
    workload; also the caller-side Horner pass over this run's 254 results on
    one host core, the CPU counterpart of msm_b200_final_sum_async."""
    sys.path.insert(0, os.path.join(REPO, "oracle"))
    import oracle as orc
    subprocess.run(["make", "-s", "-C", os.path.join(REPO, "oracle")], check=True)
    o = orc.Oracle()
    results = bc.from_device(results_dev, (254, 24))
    horner_s = []
    for _ in range(5):
        t0 = time.perf_counter()
        o.horner(results)
        horner_s.append(time.perf_counter() - t0)
    cores = os.cpu_count() or 1
    n = 1 << 14
    best = None
    while True:
        bases = bc.from_device(bases_dev, (n, 16))
        secs, _ = orc.time_cpu_pippenger(o, bases, np.ascontiguousarray(scalars_all[:n]), cores)
        best = (n, secs)
        if secs * 2.5 > target_s or n >= len(scalars_all):
            break
        n <<= 1
    n, secs = best
    return {"value": n / secs / 1e6, "unit": "Mpoints/s", "cores": cores, "kind": "port",
            "sample": f"host Pippenger (oracle/bn254_oracle.c, {cores} threads) over the first 2^{n.bit_length() - 1} points of the same "
                      f"workload, {secs:.2f} s wall",
            "host_horner_ms": round(1e3 * statistics.median(horner_s), 4)}


# ---------------------------------------------------------------------------
# batched (config 3)
# ---------------------------------------------------------------------------
def batched_section(bc, pool, stream, table_dev: int, n_table: int, executions: int, warmup: int, scale: int = 1,
                    reference: bool = False) -> dict:
    """The uneven 64-instance batch (lengths log-uniform in [2^10, 2^22], seed 3;
    even instances uniform, odd ones skewed; prefixes of one resident 2^22-point
    table): the device time of each execution of the batched graph against each
    iteration of 64 sequential plain calls (for the reference: 64 calls padded
    with zero scalars to powers of two)."""
    import synth
    lengths = [max(1, int(x) // scale) for x in synth.batch_lengths(BATCH_SEED, 64)]
    work = [s for _, s in synth.batch_workload(BATCH_SEED, lengths)]
    points = sum(lengths)
    out = {"workload": "64 MSMs, lengths log-uniform in [2^10, 2^22] (seed 3), even instances uniform scalars, odd ones the skewed mix, "
                       "prefixes of one resident 2^22-point base table", "instances": 64, "points": points}
    if not reference:
        table = bc.base_table_create(table_dev, n_table, stream)
        sd = [bc.to_device(w) for w in work]
        rd = [bc.malloc(254 * 96) for _ in lengths]
        batch = bc.batch_create(table, lengths)
        scratch, kernels, entries = bc.batch_info(batch)
        for _ in range(warmup):
            bc.batch_execute(batch, sd, rd, stream)
        batched = time_each(bc, stream, executions, lambda: bc.batch_execute(batch, sd, rd, stream))

        def plain():
            for n, s_, r in zip(lengths, sd, rd):
                bc.check(bc.msm_any(pool, stream, table_dev, s_, r, n), "msm_b200_execute_async")

        for _ in range(warmup):
            plain()
        loop = time_each(bc, stream, executions, plain)
        out.update({"unit": "Mpoints/s", **dist_summary(batched, points), "plain_per_call": dist_summary(loop, points),
                    "speedup_vs_plain_per_call": round(float(np.mean(loop)) / float(np.mean(batched)), 3),
                    "graph_kernels": kernels, "entries": entries, "scratch_gib": round(scratch / 2**30, 2),
                    "table_gib": round(bc.base_table_bytes(table) / 2**30, 2)})
        bc.batch_destroy(batch)
        bc.base_table_destroy(table)
        for p_ in sd + rd:
            bc.free(p_)
    else:  # the reference: one call per instance, zero-padded to the next power of two
        padded = []
        for w in work:
            logn = max(0, (len(w) - 1).bit_length())
            full = np.zeros((1 << logn, 8), np.uint32)
            full[: len(w)] = w
            padded.append((logn, bc.to_device(full)))
        rd = bc.malloc(254 * 96)

        def plain():
            for logn, s_ in padded:
                bc.msm(pool, stream, table_dev, s_, rd, logn)

        for _ in range(warmup):
            plain()
        loop = time_each(bc, stream, executions, plain)
        out["plain_per_call"] = {**dist_summary(loop, points), "note": "64 reference msm_execute_async calls, each zero-padded to a power of two"}
        for _, p_ in padded:
            bc.free(p_)
        bc.free(rd)
    return out


# ---------------------------------------------------------------------------
# serving (config 4)
# ---------------------------------------------------------------------------
def serving_section(bc, pool, stream, requests: int, rates_rel=(0.6, 0.9, 1.2), checks: int = 8) -> dict:
    """Config 4: Poisson arrivals (seed 4), sizes log-uniform in [2^12, 2^23],
    scalars half uniform and half skewed (device-resident slices of two
    2^23-point pools), over a resident 2^23-point table with a 16 GiB scratch
    budget.  The server (continuous batching) against a plain loop that runs
    one request per call in arrival order; rates are multiples of the plain
    loop's measured capacity.  Latency of every request, in both loops, runs
    from its scheduled arrival to its result being ready."""
    import threading
    import synth
    sys.path.insert(0, os.path.join(REPO, "oracle"))
    import oracle as orc
    n_table = 1 << 23
    k_table = synth.base_multipliers(4, n_table)
    kd = bc.to_device(k_table)
    table_dev = bc.malloc(n_table * 64)
    bc.generator_multiples(kd, table_dev, n_table, stream)
    bc.stream_synchronize(stream)
    bc.free(kd)
    table = bc.base_table_create(table_dev, n_table, stream)
    host_pools = {"uniform": synth.uniform_scalars(40, n_table), "skewed": synth.skewed_scalars(41, n_table)}
    pools = {d: bc.to_device(a) for d, a in host_pools.items()}
    rng = np.random.Generator(np.random.PCG64(np.random.SeedSequence([4, 5])))
    sizes = np.rint(np.exp2(rng.uniform(12, 23, requests))).astype(np.int64)
    offsets = [int(rng.integers(0, n_table - n + 1)) for n in sizes]
    dists = ["uniform" if j % 2 == 0 else "skewed" for j in range(requests)]
    src = [pools[d] + 32 * off for d, off in zip(dists, offsets)]
    results_plain = bc.malloc(requests * 254 * 96)
    results_server = bc.malloc(requests * 254 * 96)
    res_p = [results_plain + j * 254 * 96 for j in range(requests)]
    res_s = [results_server + j * 254 * 96 for j in range(requests)]
    points = int(sizes.sum())

    # plain capacity: back-to-back calls over the first requests, no arrivals
    probe = min(requests, 2000)
    for j in range(min(8, requests)):
        bc.msm_any(pool, stream, table_dev, src[j], res_p[j], int(sizes[j]))
    bc.stream_synchronize(stream)
    t0 = time.perf_counter()
    for j in range(probe):
        bc.msm_any(pool, stream, table_dev, src[j], res_p[j], int(sizes[j]))
    bc.stream_synchronize(stream)
    # requests per second of the probe, scaled to the mean request size of the whole run
    capacity = probe / (time.perf_counter() - t0) * (float(sizes[:probe].sum()) / probe) / (points / requests)

    def pct(lat):
        return {"p50_ms": round(float(np.percentile(lat, 50)), 3), "p99_ms": round(float(np.percentile(lat, 99)), 3)}

    out = {"workload": f"{requests} requests per rate, Poisson arrivals (seed 4), sizes log-uniform in [2^12, 2^23], half uniform / half "
                       "skewed scalars, resident 2^23-point table, 16 GiB scratch budget",
           "requests": requests, "points": points, "plain_capacity_rps": round(capacity, 1),
           "latency": "from each request's scheduled arrival to its result being ready, both loops", "rates": []}
    server = bc.server_create(table, 16 << 30, streams=4, max_group=16)
    for rel in rates_rel:
        rate = rel * capacity
        gaps = np.random.Generator(np.random.PCG64(np.random.SeedSequence([4, int(rel * 1000)]))).exponential(1.0 / rate, requests)
        # plain loop: one call per request, in arrival order
        lat = np.zeros(requests)
        start = time.perf_counter() + 0.01
        arrival = start + np.cumsum(gaps)
        for j in range(requests):
            while time.perf_counter() < arrival[j]:
                pass
            bc.msm_any(pool, stream, table_dev, src[j], res_p[j], int(sizes[j]))
            bc.stream_synchronize(stream)
            lat[j] = (time.perf_counter() - arrival[j]) * 1e3
        plain_span = time.perf_counter() - start
        # server: a producer submits at the arrival times (recording how late it
        # was), this thread collects in order; latency = lateness + the
        # server's own submit-to-done time
        tickets = [None] * requests
        late = np.zeros(requests)
        start = time.perf_counter() + 0.01
        arrival = start + np.cumsum(gaps)

        def producer():
            for j in range(requests):
                while time.perf_counter() < arrival[j]:
                    pass
                late[j] = time.perf_counter() - arrival[j]
                tickets[j] = bc.server_submit(server, src[j], int(sizes[j]), res_s[j])

        th = threading.Thread(target=producer)
        th.start()
        th.join()
        slat, last = np.zeros(requests), 0.0
        groups, first_submit = [], None
        for j in range(requests):
            rc, times = bc.server_wait(server, tickets[j])
            bc.check(rc, "msm_b200_server_wait")
            slat[j] = late[j] * 1e3 + (times.done_us - times.submit_us) / 1e3
            first_submit = times.submit_us - late[j] * 1e6 if first_submit is None else first_submit
            last = max(last, times.done_us)
            groups.append(times.group_size)
        server_span = (last - first_submit) / 1e6
        out["rates"].append({"rate_rps": round(rate, 1), "rate_vs_plain_capacity": rel,
                             "server": {"mpoints_s": round(points / server_span / 1e6, 2), **pct(slat), "mean_group": round(float(np.mean(groups)), 2)},
                             "plain": {"mpoints_s": round(points / plain_span / 1e6, 2), **pct(lat)}})
    stats = bc.server_stats(server)
    out["server_groups"] = stats.groups
    out["max_inflight_groups"] = stats.max_inflight_groups
    bc.server_destroy(server)
    # results of the last rate, both loops, against the checksum oracle: the two
    # largest requests and a seeded sample of the rest
    subprocess.run(["make", "-s", "-C", os.path.join(REPO, "oracle")], check=True)
    o = orc.Oracle()
    order = np.argsort(-sizes)
    sample = list(order[:2]) + list(np.random.Generator(np.random.PCG64(44)).choice(order[2:], max(0, checks - 2), replace=False))
    ok = 0
    for j in sample:
        n, off = int(sizes[j]), offsets[j]
        want = o.msm_checksum(np.ascontiguousarray(k_table[:n]), np.ascontiguousarray(host_pools[dists[j]][off:off + n]))
        got_p = o.horner(bc.from_device(res_p[j], (254, 24)))
        got_s = o.horner(bc.from_device(res_s[j], (254, 24)))
        ok += int(got_p == want) + int(got_s == want)
    out["checked"] = {"requests": len(sample), "results_equal_to_oracle": ok, "of": 2 * len(sample),
                      "what": "plain-loop and server results of the last rate, checksum oracle, outside the timed runs"}
    for p_ in (results_plain, results_server, *pools.values()):
        bc.free(p_)
    bc.base_table_destroy(table)
    bc.free(table_dev)
    return out


# ---------------------------------------------------------------------------
def headline(bc, pool, stream, bases_dev: int, scalars: np.ndarray, n: int, log_n: int, args, dist: Dist):
    """Device-resident steps (value) and end-to-end steps through pinned host memory (e2e)."""
    scalars_dev = bc.to_device(scalars)
    results_dev = bc.malloc(254 * 96)

    def step_device():
        bc.msm(pool, stream, bases_dev, scalars_dev, results_dev, log_n)

    for _ in range(max(args.warmup, 3)):
        step_device()
    bc.stream_synchronize(stream)
    clocks = ClockSampler(dist.local)
    dist.barrier()
    clocks.start()
    ms_local = time_steps(bc, stream, args.steps, step_device)
    clock_info = clocks.stop()
    ms = dist.max(ms_local)

    host_scalars, hs_ptr = bc.pinned_array(scalars.shape)
    host_scalars[...] = scalars
    host_results, hr_ptr = bc.pinned_array((254, 24))

    def step_e2e():
        bc.msm(pool, stream, bases_dev, hs_ptr, hr_ptr, log_n)

    for _ in range(2):
        step_e2e()
    dist.barrier()
    e2e_ms = dist.max(time_steps(bc, stream, args.steps, step_e2e))
    bc.free_host(hs_ptr)
    bc.free_host(hr_ptr)
    return ms, e2e_ms, clock_info, scalars_dev, results_dev


def base_line(dist: Dist, args, n: int, ms: float, e2e_ms: float, clock_info) -> dict:
    name, workload, seed, _ = HEADLINE
    log_n = args.log_n
    line = {
        "metric": METRIC,
        "value": round(dist.world * n / (ms * 1e-3) / 1e6, 3),
        "unit": "Mpoints/s",
        "n_gpus": dist.world,
        "steps": args.steps,
        "warmup": max(args.warmup, 3),
        "ms_per_step": round(ms, 4),
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "u32",
        "data": "synthetic",
        "config": {
            "workload": f"plain single MSM, N=2^{log_n}, {workload} Montgomery-form scalars (seed {seed}), "
                        f"resident bases k_i*G (k_i seed {seed}), device-resident inputs and results",
            "n": n,
            "l2": f"no flush: inputs larger than L2 (bases {n * 64 >> 20} MiB + scalars {n * 32 >> 20} MiB per step)",
            "parallelism": f"replicas x{dist.world}",
        },
        "e2e": {"value": round(dist.world * n / (e2e_ms * 1e-3) / 1e6, 3), "unit": "Mpoints/s", "ms_per_step": round(e2e_ms, 4),
                "h2d_bytes_per_step": n * 32, "d2h_bytes_per_step": 254 * 96},
    }
    if clock_info:
        line["clocks"] = clock_info
    return line


def run_reference(args, dist: Dist) -> None:
    import bellman_cuda as bcm
    import synth
    if not os.path.exists(REF_LIB):
        if dist.rank == 0:
            print(json.dumps({"impl": "reference", "unavailable": "reference sm_100a build oracle/_ref/libbellman-cuda-ref.so absent "
                                                                  "(build it with `make -C oracle ref REF=<reference tree>`)"}))
        return
    _, workload, seed, _ = HEADLINE
    log_n = args.log_n
    n = 1 << log_n
    pairs = [(seed, log_n)]
    extras = dist.rank == 0 and dist.world == 1
    if extras and not args.no_configs:
        pairs += [(s, l) for _, _, s, l in OTHER_CONFIGS]
    if extras and not args.no_batched:
        pairs.append((BATCH_SEED, BATCH_TABLE_LOG))
    files = ReferenceBases(pairs, dist.local)  # child process; nothing of ours is mapped here
    try:
        bc = bcm.BellmanCuda(REF_LIB)
        bc.set_device(dist.local)
        bc.ff_set_up(25, 14)
        bc.msm_set_up()
        pool = bc.mem_pool_create(dist.local)
        stream = bc.stream_create(True)
        bases_dev = bc.to_device(files.get(seed, log_n))
        scalars, _ = synth.workload(workload, n, seed)
        ms, e2e_ms, clock_info, scalars_dev, results_dev = headline(bc, pool, stream, bases_dev, scalars, n, log_n, args, dist)
        line = base_line(dist, args, n, ms, e2e_ms, clock_info)
        line["impl"] = "reference"
        line["what"] = "the reference's msm_execute_async built for sm_100a from its own sources (oracle/_ref/libbellman-cuda-ref.so)"
        for p in (scalars_dev, results_dev, bases_dev):
            bc.free(p)
        if extras and not args.no_configs:
            line["configs"] = other_configs(bc, pool, stream, lambda s, l: bc.to_device(files.get(s, l)), args.steps, max(args.warmup, 3), True)
        if extras and not args.no_batched:
            table_dev = bc.to_device(files.get(BATCH_SEED, BATCH_TABLE_LOG))
            line["batched"] = batched_section(bc, pool, stream, table_dev, 1 << BATCH_TABLE_LOG, 3, 1, reference=True)
            bc.free(table_dev)
        if dist.rank == 0:
            print(json.dumps(line))
    finally:
        files.close()


def run_b200(args, dist: Dist) -> None:
    import bellman_cuda as bcm
    import synth
    bc = bcm.BellmanCuda()
    bc.set_device(dist.local)
    bc.msm_set_up()
    if args.affine_levels is not None:
        bc.set_affine_levels(args.affine_levels)
    pool = bc.mem_pool_create(dist.local)
    stream = bc.stream_create(True)
    if args.batched_only:
        table_dev = generate_bases(bc, BATCH_SEED, (1 << BATCH_TABLE_LOG) // args.batched_scale, stream)
        print(json.dumps(batched_section(bc, pool, stream, table_dev, (1 << BATCH_TABLE_LOG) // args.batched_scale, args.steps,
                                         max(args.warmup, 3), args.batched_scale)))
        bc.free(table_dev)
        return
    _, workload, seed, _ = HEADLINE
    log_n = args.log_n
    n = 1 << log_n
    scalars, _ = synth.workload(workload, n, seed)
    bases_dev = generate_bases(bc, seed, n, stream)
    ms, e2e_ms, clock_info, scalars_dev, results_dev = headline(bc, pool, stream, bases_dev, scalars, n, log_n, args, dist)
    line = base_line(dist, args, n, ms, e2e_ms, clock_info)
    line["impl"] = "b200"

    # ---- stage times over K more steps (events recorded by the library) ----
    events = [[bc.event_create() for _ in range(7)] for _ in range(args.steps)]
    stage_ms = np.zeros(6)
    launches = 0
    bc.stream_synchronize(stream)
    for s in range(args.steps):
        launches = bc.msm_staged(pool, stream, bases_dev, scalars_dev, results_dev, n, events[s])
    bc.stream_synchronize(stream)
    for s in range(args.steps):
        stage_ms += [bc.elapsed_ms(events[s][i], events[s][i + 1]) for i in range(6)]
        for ev in events[s]:
            bc.event_destroy(ev)
    stage_ms /= args.steps
    prof = bc.msm_profiled(pool, stream, bases_dev, scalars_dev, results_dev, n)
    # pipe peak: the better of independent mad.lo and paired lo/hi carry chains
    peak = max(bc.mul_throughput(4), bc.mul_throughput(1))
    montmul_rate = bc.mul_throughput(2)
    madd_rate = bc.mul_throughput(3)
    acc_s = stage_ms[3] * 1e-3
    # XYZZ madds, plus the pair sums of the affine levels when a caller turned them on
    achieved = (prof.madds * MADD_MULOPS + prof.affine_additions * AFFINE_MULOPS) / acc_s
    line["gpu_launches"] = launches * args.steps
    line["tuning"] = {"window_bits": prof.window_bits, "windows": prof.windows, "affine_levels": prof.affine_levels}
    line["stages_ms"] = {name: round(float(v), 4) for name, v in zip(bcm.MsmB200Profile.STAGES, stage_ms)}
    line["roofline"] = {
        "bound": "imad",
        "kernel": "accumulate_kernel",
        "achieved": round(achieved / 1e12, 3),
        "peak": round(peak / 1e12, 3),
        "unit": "T mul-instr/s",
        "frac": round(achieved / peak, 4),
        "traffic": round(ACC_DRAM_BYTES_PER_ENTRY * prof.nonzero_entries),
        "traffic_source": "ncu capture at 2^21 (dram__bytes_read.sum + dram__bytes_write.sum per launch), scaled by the nonzero "
                          "entries of this launch",
        "work": f"{prof.madds} XYZZ+affine additions x {MADD_MULOPS} 32-bit multiply instructions"
                + (f" + {prof.affine_additions} affine pair sums x {AFFINE_MULOPS}" if prof.affine_levels else ""),
        "peak_source": "measured in this run: max of msm_b200_measure_mul_throughput kinds 4 (independent mad.lo) and 1 (paired "
                       "mad.lo.cc/madc.hi.cc chains), i.e. ~64 multiply instructions per clock per SM",
        "probe_montmul_frac": round(montmul_rate / peak, 4),
        "probe_madd_frac": round(madd_rate / peak, 4),
    }
    hbm, hbm_src = hbm_peak()
    passes = (prof.window_bits - 1 + 7) // 8  # 8-bit radix passes over keys of c - 1 bits
    sort_bytes = (n * 32 + prof.windows * n * 8) + passes * (prof.windows * n * 16)
    sort_s = (stage_ms[0] + stage_ms[1]) * 1e-3
    line["roofline_hbm"] = {"kernels": "digits + sort", "achieved": round(sort_bytes / sort_s / 1e9, 1), "peak": hbm, "unit": "GB/s",
                            "frac": round(sort_bytes / sort_s / 1e9 / hbm, 4), "peak_source": hbm_src,
                            "bytes": f"32 B scalar + 8 B/entry digit write; 16 B/entry (8 read + 8 write) per radix pass, {passes} passes"}
    # ---- the optional on-device final reduction of the 254 results ---------
    point_dev = bc.malloc(80)  # sizeof(msm_b200_affine_point)

    def step_final_sum():
        bc.check(bc.final_sum_async(results_dev, point_dev, stream), "msm_b200_final_sum_async")

    step_final_sum()
    line["final_sum"] = {"ms": round(time_steps(bc, stream, args.steps, step_final_sum), 4),
                         "what": "msm_b200_final_sum_async: sum 2^i R_i of the 254 results as one canonical affine point, on "
                                 "the device (a cluster of eight blocks; latency-bound: 142 dependent doublings, one inversion)"}
    bc.free(point_dev)
    extras = dist.rank == 0 and dist.world == 1
    if extras and not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_baseline(bc, scalars, bases_dev, results_dev)
    for p in (scalars_dev, results_dev, bases_dev):
        bc.free(p)
    if extras and not args.no_configs:
        line["configs"] = other_configs(bc, pool, stream, lambda s, l: generate_bases(bc, s, 1 << l, stream), args.steps,
                                        max(args.warmup, 3), False)
    if extras and not args.no_batched:
        table_dev = generate_bases(bc, BATCH_SEED, 1 << BATCH_TABLE_LOG, stream)
        line["batched"] = batched_section(bc, pool, stream, table_dev, 1 << BATCH_TABLE_LOG, max(20, args.steps), 2)
        bc.free(table_dev)
    if extras and not args.no_serving:
        line["serving"] = serving_section(bc, pool, stream, args.serving_requests)
    if dist.rank == 0:
        print(json.dumps(line))


def main():
    args = parse()
    if args.gen_bases:
        gen_bases_child(args.gen_bases)
        return
    dist = Dist(args.gpus)
    try:
        if args.impl == "reference":
            run_reference(args, dist)
        else:
            run_b200(args, dist)
    finally:
        dist.close()


if __name__ == "__main__":
    main()
