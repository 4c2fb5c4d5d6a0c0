#!/usr/bin/env python
"""Benchmark of the Zindex query hot path on B200.

Workload (the batched k-mer query): 256 colours with genome lengths
log-uniform in 1-10 Mbp, each genome 70% i.i.d. uniform ACGT and 30% copied
from 50 seeded 100 kbp core segments; index k=31, H=4, b=8 built by the host
builder; query 1,000,000 reads of 150 bp (70% sampled from random colours with
0.5% substitutions, 30% uniform random). Seeded synthetic data stand in for
real collections (there is no network).

One step = one aggregate query pass over the whole read batch:
  value : batch resident in HBM, one CUDA-graph replay per step (pack, tile
          plan, fused extraction+probe kernel, counter reduction).
  e2e   : the same query through the C ABI with host buffers (pinned), H2D of
          bases + offsets and D2H of the per-colour counts inside each step.
Both report query seeds/s (whole job, all GPUs). With --gpus N each rank holds
a full index replica and queries its own read batch (weak scaling, no
collective on the data path).

--impl reference times the CPU restatement of the reference query (the
reference is Rust and cannot be built here) on all host cores, on a bounded
sample of the same workload, with the reference's own lookup speed measures
(blocks of 32 keys, rows prefetched 4 keys ahead, AVX2 fingerprint screens).
"""
from __future__ import annotations

import argparse
import fcntl
import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

# Workloads: c2 (the default line) and the other configurations, each as
# synthetic genomes (zx_build --synth kind:colors:min:max:seed), index options,
# the query batch (zx_synth reads) and the long records of the served mix.
CONFIGS = {
    "c2": {
        "workload": {"workload": "batched-kmer-query", "colors": 256,
                     "genome_len_bp": [1_000_000, 10_000_000],
                     "genome_model": "70% iid + 30% core-pool", "k": 31, "hashes": 4,
                     "fingerprint_bits": 8, "index_mode": "kmers", "reads": 1_000_000,
                     "read_len_bp": 150, "sourced": 0.7, "substitutions": 0.005,
                     "genome_seed": 1, "read_seed": 7},
        "synth": "pool:256:1000000:10000000:1", "build": ["-k", "31", "-H", "4", "-b", "8"],
        "reads": ["--kind", "short", "--reads", "1000000", "--length", "150", "--sourced", "0.7",
                  "--subst", "0.005"],
    },
    "c1": {
        "workload": {"workload": "plain-kmer-small", "colors": 10, "genome_len_bp": [2_000_000, 2_000_000],
                     "genome_model": "iid uniform", "k": 31, "hashes": 4, "fingerprint_bits": 8,
                     "index_mode": "kmers", "reads": 100, "read_len_bp": 1000,
                     "query": "record 0 copied from genome 0, 99 iid records", "genome_seed": 1},
        "synth": "uniform:10:2000000:2000000:1", "build": ["-k", "31", "-H", "4", "-b", "8"],
        "reads": ["--kind", "fragment", "--reads", "100", "--length", "1000"],
    },
    "c3": {
        "workload": {"workload": "batched-minimizer-uneven", "colors": 2048,
                     "genome_len_bp": [500_000, 8_000_000],
                     "genome_model": "70% iid + 30% core-pool", "k": 49, "m": 31, "hashes": 3,
                     "fingerprint_bits": 16, "index_mode": "minimizers", "reads": 200_000,
                     "read_len_bp": "lognormal median 2000, clipped 100-100000", "sourced": 0.8,
                     "substitutions": 0.01, "n_runs": 0.1,
                     "index_build": "zx_build --device (the GPU builder)"},
        "synth": "pool:2048:500000:8000000:1",
        "build": ["-i", "minimizers", "-k", "49", "-m", "31", "-H", "3", "-b", "16", "--device"],
        "reads": ["--kind", "long", "--reads", "200000", "--length", "2000", "--sourced", "0.8",
                  "--subst", "0.01", "--n-runs", "0.1"],
    },
    "c4s": {
        "workload": {"workload": "served-wide-rows-scaled", "colors": 16384,
                     "genome_len_bp": [20_000, 120_000],
                     "genome_model": "70% iid + 30% core-pool", "k": 31, "hashes": 8,
                     "fingerprint_bits": 4, "index_mode": "kmers", "reads": 20_000,
                     "read_len_bp": 150, "sourced": 0.6, "substitutions": 0.005,
                     "scaled": "genome lengths 1-6 Mbp scaled down 50x (a fast stand-in for c4); "
                               "rows are the full 8 KiB",
                     "index_build": "zx_build --device (the GPU builder)"},
        "synth": "pool:16384:20000:120000:1", "build": ["-k", "31", "-H", "8", "-b", "4", "--device"],
        "reads": ["--kind", "short", "--reads", "20000", "--length", "150", "--sourced", "0.6",
                  "--subst", "0.005"],
        # 64 KiB of rows per seed: fewer served requests keep the run bounded.
        "served": {"closed": 100, "open": 300, "rate": 200.0},
    },
    "c4": {
        "workload": {"workload": "served-large-resident-index", "colors": 16384,
                     "genome_len_bp": [1_000_000, 6_000_000],
                     "genome_model": "70% iid + 30% core-pool", "k": 31, "hashes": 8,
                     "fingerprint_bits": 4, "index_mode": "kmers", "reads": 50_000,
                     "read_len_bp": 150, "sourced": 0.6, "substitutions": 0.005,
                     "index_build": "zx_build --device (the GPU builder)"},
        "synth": "pool:16384:1000000:6000000:1",
        "build": ["-k", "31", "-H", "8", "-b", "4", "--device"],
        "reads": ["--kind", "short", "--reads", "50000", "--length", "150", "--sourced", "0.6",
                  "--subst", "0.005"],
        "served": {"closed": 100, "open": 300, "rate": 200.0},
        # 16,384 dense counts per read: a bounded per-record sample.
        "per_record_reads": 5_000,
    },
}
CONFIG = CONFIGS["c2"]
WORKLOAD = CONFIG["workload"]
METRIC = "query seeds/s"
# Per-record form: reads counted one by one, and the compact report threshold.
PER_RECORD_READS = 200_000
PER_RECORD_CPU_READS = 20_000
PER_RECORD_MIN_RATIO = 0.5
LIB = ROOT / "zindex_b200" / "_lib"
PEAKS = ROOT / "MEASURED_PEAKS.json"
FALLBACK_HBM_GBS = 6650.0


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def dist_env():
    return (int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)),
            int(os.environ.get("LOCAL_RANK", 0)))


def build_native():
    from zindex_b200.build import build

    build()
    subprocess.run(["make", "-s", "-C", str(ROOT / "oracle")], check=True)


def _synth_genome_args(cfg):
    kind, colors, lo, hi, seed = cfg["synth"].split(":")
    return ["--genome-kind", kind, "--colors", colors, "--min-len", lo, "--max-len", hi,
            "--seed", seed]


def prepare(cache: Path, rank: int, name: str = "c2"):
    """Index (built once per cache dir, file-locked) and this rank's reads."""
    cfg = CONFIGS[name]
    cache.mkdir(parents=True, exist_ok=True)
    index = cache / f"index-{name}"
    with open(cache / ".lock", "w") as lk:
        fcntl.flock(lk, fcntl.LOCK_EX)
        if not (index / "manifest.json").exists():
            t0 = time.time()
            subprocess.run([str(LIB / "zx_build"), "--synth", cfg["synth"], "-o", str(index),
                            *cfg["build"], "-q"], check=True)
            log(f"built index in {time.time() - t0:.1f}s")
        reads = cache / f"reads-{name}-r{rank}"
        if not Path(str(reads) + ".offsets").exists():
            subprocess.run([str(LIB / "zx_synth"), "reads", *_synth_genome_args(cfg),
                            "--read-seed", str(7 + rank), *cfg["reads"], "--format", "raw",
                            "--out", str(reads)], check=True)
        long = cache / f"long-{name}-r{rank}"
        if not Path(str(long) + ".offsets").exists():
            # Long records for the served request mix: lognormal lengths,
            # median 30 kbp, clipped to 100 bp-100 kbp, 60% sourced.
            subprocess.run([str(LIB / "zx_synth"), "reads", "--kind", "long",
                            *_synth_genome_args(cfg), "--read-seed", str(101 + rank), "--reads",
                            "400", "--length", "30000", "--sourced", "0.6", "--subst", "0.005",
                            "--format", "raw", "--out", str(long)], check=True)
    bases = np.fromfile(str(reads) + ".bases", dtype=np.uint8)
    offsets = np.fromfile(str(reads) + ".offsets", dtype=np.uint64)
    return index, bases, offsets


def over_ranks(dist, device, value: float, op: str) -> float:
    """`value` reduced over the ranks ("max" or "sum"); itself on one process."""
    if dist is None or not dist.is_initialized() or dist.get_world_size() == 1:
        return value
    import torch

    t = torch.tensor([float(value)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX if op == "max" else dist.ReduceOp.SUM)
    return float(t.item())


def job_rate(dist, device, units: float, seconds: float) -> float:
    """Whole-job throughput: the units of every rank over the slowest rank's
    time (the timed region ends when the last rank ends)."""
    return over_ranks(dist, device, units, "sum") / over_ranks(dist, device, seconds, "max")


def long_pool(cache: Path, rank: int, name: str = "c2"):
    long = cache / f"long-{name}-r{rank}"
    return (np.fromfile(str(long) + ".bases", dtype=np.uint8),
            np.fromfile(str(long) + ".offsets", dtype=np.uint64))


def launches_per_step(ix, nbases: int, records: int) -> int:
    """Kernels one batched query launches (all compiled into libzindex_b200.so):
    pack, count_tiles, the two kernels of the CUB tile scan and fill_tiles (one
    kernel for small batches); then the fused query kernel and, with shared
    counters, the counter reduction, once or once per round of a split
    minimizer query; or, for the wide-row form, per round the extraction, the
    sort of ordered rounds (bucket count, scan and twice bin places and tile
    scatter), the wide probe and, with ordered rounds, the window probe (of
    the two probes the one that the round's key count does not select returns
    at once). Batches of up to 2^28 bases are one round."""
    lc, info = ix.launch(), ix.info
    probe = 1 + (1 if lc["smem_counters"] else 0)
    tiles_bound = nbases // 256 + records + nbases // 16384 + 1
    split = lc.get("split") and info.index_mode == 1 and lc["planes"] == 1 and lc["stage_bytes"] == 0
    if lc.get("wide"):
        plan = 1 if records <= 4096 and nbases <= (1 << 18) else 5
        rounds = 1 if nbases <= (1 << 28) else -(-tiles_bound // 262144)
        return plan + rounds * (2 + (6 if lc.get("order") else 0) + (1 if lc.get("order") == 1 else 0))
    if records <= 4096 and nbases <= (1 << 20) and not split:
        # Small batches: one block packs and plans, then the fused kernel
        # (adding into the caller's counters for up to 1,024 colours).
        return 1 + 1 + (1 if lc["smem_counters"] and ix.colors > 1024 else 0)
    plan = 5
    if split:
        rounds = -(-tiles_bound // 262144)
        return plan + rounds * (1 + probe)
    return plan + probe


def records_fasta(cache: Path, rank: int, name: str, bases, offsets, n: int) -> Path:
    """The first n reads as a FASTA file with identifiers r0, r1, ... (the
    per-record report's input), written once per cache dir."""
    path = cache / f"records-{name}-r{rank}-{n}.fa"
    if not path.exists():
        tmp = Path(str(path) + f".tmp{os.getpid()}")
        with open(tmp, "wb") as f:
            for r in range(n):
                f.write(b">r%d\n" % r)
                f.write(bases[int(offsets[r]): int(offsets[r + 1])].tobytes() + b"\n")
        os.replace(tmp, path)
    return path


def make_requests(bases, offsets, lbases, loffsets, n, seed):
    """Served request mix: half are 1-10,000 reads of 150 bp, half 1-10 long
    records (lognormal, median 30 kbp), drawn from the read pools."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        if rng.random() < 0.5:
            b, o, k = bases, offsets, int(rng.integers(1, 10001))
        else:
            b, o, k = lbases, loffsets, int(rng.integers(1, 11))
        r = len(o) - 1
        k = min(k, r)
        st = int(rng.integers(0, max(1, r - k)))
        oo = o[st: st + k + 1] - o[st]
        out.append((b[int(o[st]): int(o[st + k])], np.ascontiguousarray(oo)))
    return out


def planned_form(ix, bases, offsets, seeds, step_ms, e2e_ms):
    """The learned planner (trained on the GPU on the committed autotuner rows)
    ranks every candidate launch for this batch; its top predictions and the
    default are timed on the batch and the fastest is kept, and it picks the
    cut. Exhaustive autotuning over the same candidates is timed alongside as
    the measure of the regret; the default launch gives the gain.
    step_ms(launch) times device steps under a launch."""
    from zindex_b200 import planner as pl
    from zindex_b200 import tuning as tn

    rows, _ = pl.load_rows()
    planner = pl.Planner(seed=1)
    t0 = time.perf_counter()
    loss = planner.fit(rows)
    train_s = time.perf_counter() - t0
    default = dict(ix.default_launch(), blocks=0)
    lengths = np.diff(offsets.astype(np.int64))
    feats = tn.Autotuner.features(ix, lengths, seeds)
    # The network's candidates are the fused kernel's launches; an index whose
    # default is the wide-row form has that default as one more candidate.
    fused = dict(ix.default_fused_launch(), blocks=0)
    cands = [dict(fused, **l, stage_bytes=0, wide=0) for l in tn.REGISTER_LAUNCHES]
    if default["wide"]:
        cands.append(default)
    timed = {}

    def timed_ms(launch):
        key = pl.launch_key(dict(launch, cut=1))
        if key not in timed:
            try:
                timed[key] = step_ms(launch)
            except Exception:  # e.g. more shared memory than a block may use
                timed[key] = float("inf")
        return timed[key]

    t0 = time.perf_counter()
    short = planner.shortlist(feats, cands, default)
    pick = min(short, key=timed_ms)
    cuts = planner.shortlist(feats, [dict(pick, cut=c) for c in tn.CUTS],
                             dict(pick, cut=default["cut"]), 1, e2e=True)
    pick = min(cuts, key=e2e_ms)
    plan_s = time.perf_counter() - t0
    for launch in cands:  # exhaustive: every candidate
        timed_ms(launch)
    best_key = min(timed, key=timed.get)
    t_pick = timed_ms(pick)
    t_default = timed_ms(default)
    return pick, {
        "chosen": {k: pick[k] for k in ("team", "warps", "min_blocks", "planes", "cut", "wide")},
        "ms_per_step": t_pick, "default_ms_per_step": t_default,
        "exhaustive_best_ms_per_step": timed[best_key],
        "exhaustive_best": dict((k, v) for k, v in best_key
                                if k in ("team", "warps", "min_blocks", "planes", "wide")),
        "regret": t_pick / timed[best_key] - 1.0, "gain_over_default": t_default / t_pick,
        "timed": len(short), "cuts_timed": len(cuts), "candidates": len(cands),
        "train_rows": len(rows),
        "train_loss": loss, "train_s_on_gpu": train_s, "plan_and_verify_s": plan_s,
    }


def served_form(zx, ix, requests_closed, requests_open, rate):
    """Closed loop (all requests queued at once: served throughput) and an open
    Poisson arrival stream at `rate` requests/s (latency percentiles)."""
    out = {}
    with zx.Server(ix, slots=3) as server:
        for b, o in requests_closed[:20]:  # warm-up
            server.wait(server.submit(b, o))
        server.stats(reset=True)
        t0 = time.perf_counter()
        tickets = [server.submit(b, o) for b, o in requests_closed]
        seeds = sum(server.wait(t)[1] for t in tickets)
        dt = time.perf_counter() - t0
        st = server.stats(reset=True)
        out["closed_loop"] = {"requests": len(tickets), "seconds": dt, "seeds_per_s": seeds / dt,
                              "bases_per_s": st["bases"] / dt, "batches": st["batches"],
                              "p50_ms": st["p50_s"] * 1e3, "p99_ms": st["p99_s"] * 1e3}
        dt, seeds, st = poisson_run(server, requests_open, rate, 5)
        out["poisson"] = {"rate_req_per_s": rate, "requests": len(requests_open), "seconds": dt,
                          "seeds_per_s": seeds / dt, "batches": st["batches"],
                          "p50_ms": st["p50_s"] * 1e3, "p99_ms": st["p99_s"] * 1e3,
                          "max_ms": st["max_s"] * 1e3,
                          "server_device_bytes": st["device_bytes"]}
    return out


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
        return self

    def __exit__(self, *exc):
        self.lines = []
        if self.proc:
            time.sleep(0.25)
            self.proc.terminate()
            out, _ = self.proc.communicate(timeout=10)
            self.lines = [l for l in out.splitlines() if l.strip()]

    def summary(self):
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in getattr(self, "lines", []):
            f = [x.strip() for x in l.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


def hbm_peak():
    try:
        p = json.loads(PEAKS.read_text())
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


def query_roofline(ix, seeds: int, nbases: int, kernel_ms: float) -> dict:
    """What bounds the timed sequence (ix.last_kernel_ms: everything between
    the tile plan and the counters). Batches whose row reads are four times
    the rows take the window probe, which copies each window of rows once and
    gathers every seed's rows from shared memory: its bound is 128 bytes per
    clock and SM. Other batches read the rows from HBM or L2 in the wide probe
    or the fused kernel: their bound is the copy rate. The sequence's other
    kernels (extraction, sort) are part of the time and move none of these
    bytes. No DRAM traffic is captured for a whole batch: traffic is null."""
    import torch

    info, launch = ix.info, ix.launch()
    rec_bytes = 8 if info.abandoned_hashes else 0
    row_bytes = seeds * info.gather_bytes_per_seed
    alg = row_bytes + seeds * rec_bytes + nbases * 3 // 8
    # The same gather in whole 32-byte DRAM sectors (each row touch costs its sectors).
    sector = (seeds * (info.gather_sector_bytes_per_seed + (32 if rec_bytes else 0))
              + nbases * 3 // 8)
    seconds = kernel_ms / 1e3
    common = {"unit": "GB/s", "kernel_ms": kernel_ms, "algorithmic_bytes_per_launch": int(alg),
              "gather_bytes_per_seed": int(info.gather_bytes_per_seed),
              "sector_bytes_per_seed": int(info.gather_sector_bytes_per_seed), "traffic": None}
    if launch["wide"] and launch["order"] == 1 and row_bytes >= 4 * info.resident_bytes:
        prop = torch.cuda.get_device_properties(torch.cuda.current_device())
        mhz = nvidia_smi_max_sm_mhz()
        peak = prop.multi_processor_count * 128 * mhz * 1e6 / 1e9
        achieved = row_bytes / seconds / 1e9
        return dict(common, bound="shared memory", achieved=achieved, peak=peak,
                    frac=achieved / peak,
                    peak_kind=f"128 B x {prop.multi_processor_count} SMs x {mhz:.0f} MHz",
                    kernel="extract_dense_kernel, key sort, window_probe_kernel")
    peak, kind = hbm_peak()
    achieved = alg / seconds / 1e9
    kernel = ("extract_dense_kernel, key sort, wide_probe_kernel" if launch["wide"] else
              "findere_query_kernel or fused_query_kernel" if info.index_mode == 3 else
              "fused_query_kernel")
    return dict(common, bound="hbm", achieved=achieved, peak=peak, frac=achieved / peak,
                peak_kind=kind, kernel=kernel, sector_achieved=sector / seconds / 1e9,
                sector_frac=sector / seconds / 1e9 / peak)


def nvidia_smi_max_sm_mhz() -> float:
    try:
        out = subprocess.run(["nvidia-smi", "--query-gpu=clocks.max.sm",
                              "--format=csv,noheader,nounits"], capture_output=True, text=True,
                             timeout=30, check=True).stdout
        return float(out.split()[0])
    except Exception:
        return 1965.0


class CpuOracle:
    """The oracle (CPU restatement of the reference query) with its index
    resident in host memory, timed on all host cores. The timed queries take
    its fast lookup (the reference's lookup_batch blocks, 4-ahead row
    prefetch and AVX2 fingerprint screens; the same counts as the scalar
    checker) where the index allows it: kind "port-simd", else "port"."""

    def __init__(self, index):
        import ctypes
        from ctypes import POINTER, c_char_p, c_double, c_int, c_size_t, c_uint64, c_void_p

        self.ct = ctypes
        lib = ctypes.CDLL(str(ROOT / "oracle" / "_build" / "liboracle.so"))
        lib.oracle_open.argtypes = [c_char_p, c_int, POINTER(c_void_p)]
        lib.oracle_open.restype = c_int
        lib.oracle_close.argtypes = [c_void_p]
        lib.oracle_query_handle.argtypes = [c_void_p, c_void_p, POINTER(c_uint64), c_size_t, c_int,
                                            POINTER(c_uint64), c_size_t, POINTER(c_uint64),
                                            POINTER(c_double)]
        lib.oracle_query_handle.restype = c_int
        lib.oracle_query_handle_fast.argtypes = lib.oracle_query_handle.argtypes
        lib.oracle_query_handle_fast.restype = c_int
        lib.oracle_fast_serves.argtypes = [c_void_p]
        lib.oracle_fast_serves.restype = c_int
        lib.oracle_last_error.restype = c_char_p
        self.lib = lib
        self.h = c_void_p()
        if lib.oracle_open(str(index).encode(), 1, ctypes.byref(self.h)):
            raise RuntimeError(lib.oracle_last_error().decode())
        self.cores = os.cpu_count() or 1
        self.fast = bool(lib.oracle_fast_serves(self.h))
        self.kind = "port-simd" if self.fast else "port"

    def run(self, bases, offsets, n, colors, checker=False):
        """(seeds, seconds, counts) of the first n records; checker=True takes
        the scalar lookup (the parity checker) instead of the fast one."""
        if not 0 < n <= len(offsets) - 1:
            raise ValueError(f"oracle sample of {n} records outside a batch of {len(offsets) - 1}")
        ct = self.ct
        off = np.ascontiguousarray(offsets[: n + 1])
        counts = np.zeros(colors, dtype=np.uint64)
        total, secs = ct.c_uint64(), ct.c_double()
        fast = self.fast and not checker
        fn = self.lib.oracle_query_handle_fast if fast else self.lib.oracle_query_handle
        rc = fn(self.h, bases.ctypes.data_as(ct.c_void_p),
                                          off.ctypes.data_as(ct.POINTER(ct.c_uint64)), n, self.cores,
                                          counts.ctypes.data_as(ct.POINTER(ct.c_uint64)), colors,
                                          ct.byref(total), ct.byref(secs))
        if rc:
            raise RuntimeError(self.lib.oracle_last_error().decode())
        return total.value, secs.value, counts

    def sized(self, bases, offsets, colors, target_s):
        n = min(20000, len(offsets) - 1)  # a probe run, within the batch
        seeds, secs, _ = self.run(bases, offsets, n, colors)
        n = int(min(len(offsets) - 1, max(n, n * target_s / max(secs, 1e-3))))
        seeds, secs, counts = self.run(bases, offsets, n, colors)
        # A whole batch that runs in well under a second: median of repeats.
        if n == len(offsets) - 1 and secs < 0.2:
            reps = [secs] + [self.run(bases, offsets, n, colors)[1]
                             for _ in range(int(min(200, 1.0 / max(secs, 1e-4))))]
            secs = statistics.median(reps)
        return seeds, secs, counts, n

    def records_report(self, path, min_ratio, compact):
        """(report bytes, seconds) of the per-record report on all host cores."""
        ct = self.ct
        f = self.lib.oracle_records_report_handle
        f.argtypes = [ct.c_void_p, ct.c_char_p, ct.c_double, ct.c_int, ct.c_int, ct.c_char_p,
                      ct.c_size_t, ct.POINTER(ct.c_size_t), ct.POINTER(ct.c_double)]
        f.restype = ct.c_int
        n, secs = ct.c_size_t(), ct.c_double()
        args = (self.h, str(path).encode(), float(min_ratio), int(compact), self.cores)
        if f(*args, None, 0, ct.byref(n), ct.byref(secs)):
            raise RuntimeError(self.lib.oracle_last_error().decode())
        buf = ct.create_string_buffer(max(1, n.value))
        if f(*args, buf, n.value, ct.byref(n), ct.byref(secs)):
            raise RuntimeError(self.lib.oracle_last_error().decode())
        return buf.raw[: n.value], secs.value

    def close(self):
        self.lib.oracle_close(self.h)


def cpu_baseline(index, bases, offsets, colors, target_s=15.0):
    """seeds/s of the oracle on a bounded prefix of the read batch."""
    orc = CpuOracle(index)
    seeds, secs, counts, n = orc.sized(bases, offsets, colors, target_s)
    orc.close()
    return {"value": seeds / secs, "unit": "seeds/s", "cores": orc.cores, "kind": orc.kind,
            "sample": f"first {n} of the {len(offsets) - 1:,} query records ({seeds} seeds), query only "
                      f"(index load excluded), {secs:.2f}s"}, n, counts


# Configurations measured beside the default line (their batched step, kernel
# roofline and an oracle parity sample), and the reads of the parity sample.
OTHER_CONFIGS = {"c3": 300, "c4s": 2000}


def other_config(zx, torch, name, cache: Path, steps: int):
    """The batched step of another configuration: index (GPU builder) and
    reads prepared like the default line's, device-resident batch, `steps`
    timed steps (inputs larger than L2), the probe's kernel time against the
    copy peak, and the first reads' counts against the oracle's."""
    cfg = CONFIGS[name]
    index_dir, bases, offsets = prepare(cache, 0, name)
    records = len(offsets) - 1
    dev = torch.device("cuda", 0)
    with zx.Index(index_dir) as ix:
        info = ix.info
        d_bases = torch.from_numpy(bases).to(dev)
        d_off = torch.from_numpy(offsets.view(np.int64)).to(dev)
        d_counts = torch.zeros(ix.colors, dtype=torch.int64, device=dev)
        d_total = torch.zeros(1, dtype=torch.int64, device=dev)
        stream = torch.cuda.current_stream(dev)

        def step(graph=True):
            d_counts.zero_()
            d_total.zero_()
            ix.query_device(d_bases.data_ptr(), len(bases), d_off.data_ptr(), records,
                            d_counts.data_ptr(), d_total.data_ptr(), stream=stream.cuda_stream,
                            use_graph=graph)

        for _ in range(3):
            step()
        torch.cuda.synchronize(dev)
        seeds = int(d_total.item())
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(steps):
            step()
        e1.record(stream)
        torch.cuda.synchronize(dev)
        ms = e0.elapsed_time(e1) / steps
        ix.set_timing(True)
        kms = []
        for _ in range(3):
            step(graph=False)
            kms.append(ix.last_kernel_ms())
        ix.set_timing(False)
        kernel_ms = statistics.median(kms)
        roofline = query_roofline(ix, seeds, len(bases), kernel_ms)
        n = min(OTHER_CONFIGS[name], records)
        got, got_total = ix.query_records(bases[: int(offsets[n])], offsets[: n + 1])
        launch = ix.launch()
    orc = CpuOracle(index_dir)
    _, _, want = orc.run(bases, offsets, n, len(got), checker=True)
    orc.close()
    return {"workload": cfg["workload"], "value": seeds / (ms / 1e3), "unit": "seeds/s",
            "ms_per_step": ms, "steps": steps, "seeds_per_step": seeds,
            "roofline": roofline,
            "launch": launch, "resident_bytes": int(info.resident_bytes),
            "parity_vs_oracle_sample": bool(np.array_equal(got, want)),
            "parity_sample_reads": n}


def reference_arm(args):
    rank, world, local = dist_env()
    if rank != 0:
        return
    build_native()
    index, bases, offsets = prepare(Path(args.cache), 0, args.config)
    orc = CpuOracle(index)
    colors = json.loads((index / "manifest.json").read_text())["colors"].__len__()
    per_step = max(1.0, 60.0 / max(1, args.steps + args.warmup))
    n = None
    vals = []
    for i in range(args.warmup + args.steps):
        if n is None:
            seeds, secs, _, n = orc.sized(bases, offsets, colors, per_step)
        else:
            seeds, secs, _ = orc.run(bases, offsets, n, colors)
        if i >= args.warmup:
            vals.append(seeds / secs)
    orc.close()
    base = {"unit": "seeds/s", "cores": orc.cores, "kind": orc.kind,
            "sample": f"first {n} of the {len(offsets) - 1:,} query records per step (the rate "
                      f"on that prefix), query only (index load excluded)"}
    value = statistics.median(vals)
    base = dict(base, value=value)
    line = {"metric": METRIC, "value": value, "unit": "seeds/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": None, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "u64", "data": "synthetic", "impl": "reference",
            "config": dict(WORKLOAD, config=args.config),
            "cpu_baseline": base,
            "e2e": {"value": value, "unit": "seeds/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def ours(args):
    import torch
    import torch.distributed as dist

    rank, world, local = dist_env()
    if world > 1:
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=600))
    if rank == 0 or world == 1:
        build_native()
    if world > 1:
        dist.barrier()
    import zindex_b200 as zx

    index_dir, bases, offsets = prepare(Path(args.cache), rank, args.config)
    if args.reads:
        offsets = offsets[: args.reads + 1].copy()
        bases = bases[: int(offsets[-1])].copy()
        WORKLOAD["reads"] = args.reads
    records = len(offsets) - 1
    dev = torch.device("cuda", local)
    torch.cuda.set_device(dev)
    torch.zeros(1, device=dev)  # the CUDA context exists before the load is timed
    t_load = time.perf_counter()
    ix = zx.Index(index_dir, device=local)
    load_s = time.perf_counter() - t_load
    info = ix.info
    file_bytes = sum(p.stat().st_size for p in Path(index_dir).iterdir() if p.is_file())
    # Device-resident batch.
    d_bases = torch.from_numpy(bases).to(dev)
    d_off = torch.from_numpy(offsets.view(np.int64)).to(dev)
    d_counts = torch.zeros(ix.colors, dtype=torch.int64, device=dev)
    d_total = torch.zeros(1, dtype=torch.int64, device=dev)
    stream = torch.cuda.current_stream(dev)

    def step(graph=True):
        d_counts.zero_()
        d_total.zero_()
        ix.query_device(d_bases.data_ptr(), len(bases), d_off.data_ptr(), records,
                        d_counts.data_ptr(), d_total.data_ptr(), stream=stream.cuda_stream,
                        use_graph=graph)

    for _ in range(max(3, args.warmup)):
        step()
    torch.cuda.synchronize(dev)
    seeds = int(d_total.item())
    counts_dev = d_counts.cpu().numpy().astype(np.uint64)
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize(dev)
    # An index and batch that fit the 126 MB L2 are timed step by step with
    # the L2 flushed (a 256 MiB write) before each step, outside the events.
    flush = info.resident_bytes + len(bases) * 2 < (126 << 20)
    scrub = torch.empty(256 << 20, dtype=torch.uint8, device=dev) if flush else None
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clocks:
        if flush:
            ms = 0.0
            for _ in range(args.steps):
                scrub.fill_(1)
                e0.record(stream)
                step()
                e1.record(stream)
                torch.cuda.synchronize(dev)
                ms += e0.elapsed_time(e1)
            ms /= args.steps
        else:
            e0.record(stream)
            for _ in range(args.steps):
                step()
            e1.record(stream)
            torch.cuda.synchronize(dev)
            ms = e0.elapsed_time(e1) / args.steps
    if world > 1:
        dist.barrier()
    ddist = dist if world > 1 else None
    value = job_rate(ddist, dev, seeds, ms / 1e3)
    bases_rate = job_rate(ddist, dev, len(bases), ms / 1e3)
    ms = over_ranks(ddist, dev, ms, "max")
    launches = launches_per_step(ix, len(bases), records) * args.steps

    log("stage: kernel timing")
    # The query's kernels after the tile plan, timed alone with CUDA events on
    # their launch stream.
    ix.set_timing(True)
    kms = []
    for _ in range(max(3, min(args.steps, 10))):
        step(graph=False)
        kms.append(ix.last_kernel_ms())
    ix.set_timing(False)
    kernel_ms = statistics.median(kms)
    roofline = query_roofline(ix, seeds, len(bases), kernel_ms)

    log("stage: end to end")
    # End to end through the C ABI with pinned host buffers.
    h_bases = torch.from_numpy(bases).pin_memory()
    h_off = torch.from_numpy(offsets.view(np.int64)).pin_memory()
    hb, ho = h_bases.numpy(), h_off.numpy().view(np.uint64)
    for _ in range(2):
        c_e2e, t_e2e = ix.query_records(hb, ho)
    times = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        c_e2e, t_e2e = ix.query_records(hb, ho)
        times.append(time.perf_counter() - t0)
    e2e_s = statistics.median(times)
    e2e_rate = job_rate(ddist, dev, seeds, e2e_s)
    assert t_e2e == seeds and np.array_equal(c_e2e, counts_dev), "e2e and device paths disagree"

    log("stage: planned form")
    # Planned form: launch and cut chosen by the learned planner.
    def step_ms(launch, reps=3):
        ix.set_launch(**launch)
        step()
        torch.cuda.synchronize(dev)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(reps):
            step()
        b.record(stream)
        torch.cuda.synchronize(dev)
        return a.elapsed_time(b) / reps

    def e2e_ms(launch, reps=3):
        ix.set_launch(**launch)
        ix.query_records(hb, ho)
        ts = []
        for _ in range(reps):
            t0 = time.perf_counter()
            ix.query_records(hb, ho)
            ts.append(time.perf_counter() - t0)
        return statistics.median(ts) * 1e3

    default_launch = ix.launch()
    # Ordered wide-row rounds against extraction order (same launch otherwise).
    unordered = None
    if default_launch.get("wide") and default_launch.get("order"):
        unordered = seeds / (step_ms(dict(default_launch, order=0)) / 1e3)
        ix.set_launch(**default_launch)
    pick, planned = planned_form(ix, bases, offsets, seeds, step_ms, e2e_ms)
    ix.set_launch(**pick)
    times = []
    for _ in range(max(3, args.steps // 2)):
        t0 = time.perf_counter()
        c_pl, t_pl = ix.query_records(hb, ho)
        times.append(time.perf_counter() - t0)
    assert t_pl == seeds and np.array_equal(c_pl, counts_dev), "planned launch changed the counts"
    planned["seeds_per_s"] = seeds / (planned["ms_per_step"] / 1e3)
    planned["e2e_seeds_per_s"] = seeds / statistics.median(times)
    ix.set_launch(**default_launch)

    log("stage: served form")
    # Served form: request mix through the continuous-batching server.
    lb, lo = long_pool(Path(args.cache), rank, args.config)
    sv = CONFIG.get("served", {"closed": 400, "open": 1000, "rate": 200.0})
    served = served_form(zx, ix, make_requests(bases, offsets, lb, lo, sv["closed"], 11 + rank),
                         make_requests(bases, offsets, lb, lo, sv["open"], 23 + rank), sv["rate"])

    log("stage: query file")
    # The drop-in's own path: zx_query_file on the whole batch as a FASTA file
    # (page cache): parsing, host-to-device copies, the query and the counts.
    qfile = records_fasta(Path(args.cache), rank, args.config, bases, offsets, records)
    ix.query_file(qfile)
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        c_file, t_file, _ = ix.query_file(qfile)
        times.append(time.perf_counter() - t0)
    assert t_file == seeds and np.array_equal(c_file, counts_dev), "file and device paths disagree"
    query_file = {"seeds_per_s": seeds / statistics.median(times),
                  "seconds": statistics.median(times), "file_bytes": qfile.stat().st_size,
                  "note": "zx_query_file of the batch as FASTA (one record per read, in the page "
                          "cache): read, parse, copy, query, counts back"}

    log("stage: plain form")
    # Plain form: one record per launch, on a prefix.
    n_plain = min(4000, records)
    pb = bases[: int(offsets[n_plain])]
    po = offsets[: n_plain + 1]
    t0 = time.perf_counter()
    _, plain_seeds = ix.query_records(pb, po, plain=True)
    plain_rate = plain_seeds / (time.perf_counter() - t0)

    log("stage: per-record form")
    # Per-record form (`query --records`): each read counted alone. Counts of
    # every read through zx_query_per_record (host buffers, copies inside the
    # timed region), then the compact report of a FASTA file end to end
    # (reading, counting, formatting, writing to /dev/null).
    n_rec = min(CONFIG.get("per_record_reads", PER_RECORD_READS), records)
    rb, ro = bases[: int(offsets[n_rec])], offsets[: n_rec + 1]
    pr_counts, pr_totals = ix.query_per_record(rb, ro)
    agg_counts, agg_total = ix.query_records(rb, ro)
    assert (int(pr_totals.sum()) == agg_total and
            np.array_equal(pr_counts.sum(axis=0, dtype=np.uint64), agg_counts)), \
        "per-record counts do not add up to the aggregate"
    # Page-locked inputs and outputs, as a throughput-minded caller passes them.
    p_bases = torch.from_numpy(rb).pin_memory().numpy()
    p_off = torch.from_numpy(ro.view(np.int64)).pin_memory().numpy().view(np.uint64)
    p_counts = torch.zeros((n_rec, ix.colors), dtype=torch.int64).pin_memory().numpy().view(np.uint64)
    p_totals = torch.zeros(n_rec, dtype=torch.int64).pin_memory().numpy().view(np.uint64)
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        ix.query_per_record(p_bases, p_off, counts=p_counts, totals=p_totals)
        times.append(time.perf_counter() - t0)
    pr_s = statistics.median(times)
    assert np.array_equal(p_counts, pr_counts) and np.array_equal(p_totals, pr_totals)
    fasta = records_fasta(Path(args.cache), rank, args.config, bases, offsets, n_rec)
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        ix.query_records_report(fasta, os.devnull, min_ratio=PER_RECORD_MIN_RATIO, fmt="compact")
        times.append(time.perf_counter() - t0)
    rep_s = statistics.median(times)
    # The reference's default report: TSV rows for every colour of every read.
    n_tsv = min(n_rec, PER_RECORD_CPU_READS)
    tsv_fasta = records_fasta(Path(args.cache), rank, args.config, bases, offsets, n_tsv)
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        ix.query_records_report(tsv_fasta, os.devnull, min_ratio=0.0, fmt="tsv")
        times.append(time.perf_counter() - t0)
    tsv_s = statistics.median(times)
    per_record = {
        "reads": n_rec, "seeds": agg_total,
        "counts_reads_per_s": n_rec / pr_s, "counts_seeds_per_s": agg_total / pr_s,
        "report_reads_per_s": n_rec / rep_s,
        "report_tsv_all_colours_reads_per_s": n_tsv / tsv_s,
        "report_tsv_sample_reads": n_tsv,
        "report": f"compact, min_ratio {PER_RECORD_MIN_RATIO}, {fasta.stat().st_size} B FASTA "
                  "read, counted and formatted per call",
        "d2h_bytes_per_call": int(8 * n_rec * (ix.colors + 1)),
    }

    if rank == 0:
        cb = None
        parity = None
        if world == 1 and not args.no_cpu_baseline:
            log("stage: cpu baseline")
            cb, n_cpu, cpu_counts = cpu_baseline(index_dir, bases, offsets, ix.colors)
            c_part, _ = ix.query_records(bases[: int(offsets[n_cpu])], offsets[: n_cpu + 1])
            parity = bool(np.array_equal(c_part, cpu_counts))
            # Per-record report on the host cores, on a bounded sample of reads.
            n_s = min(n_rec, PER_RECORD_CPU_READS)
            sample = records_fasta(Path(args.cache), rank, args.config, bases, offsets, n_s)
            orc = CpuOracle(index_dir)
            want, secs = orc.records_report(sample, PER_RECORD_MIN_RATIO, True)
            orc.close()
            got_path = Path(args.cache) / f"records-gpu-{os.getpid()}.txt"
            ix.query_records_report(sample, got_path, min_ratio=PER_RECORD_MIN_RATIO, fmt="compact")
            per_record["cpu_baseline"] = {
                "value": n_s / secs, "unit": "reads/s", "cores": orc.cores, "kind": "port",
                "sample": f"compact report of the first {n_s} reads, {secs:.2f}s"}
            per_record["parity_vs_oracle_sample"] = got_path.read_bytes() == want
            orc = CpuOracle(index_dir)
            want_tsv, secs_tsv = orc.records_report(sample, 0.0, False)
            orc.close()
            ix.query_records_report(sample, got_path, min_ratio=0.0, fmt="tsv")
            per_record["cpu_baseline_tsv_all_colours"] = {
                "value": n_s / secs_tsv, "unit": "reads/s", "cores": orc.cores, "kind": "port",
                "sample": f"TSV report, every colour, of the first {n_s} reads, {secs_tsv:.2f}s"}
            per_record["parity_vs_oracle_sample_tsv"] = got_path.read_bytes() == want_tsv
            got_path.unlink()
        line = {
            "metric": METRIC, "value": value, "unit": "seeds/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u64",
            "data": "synthetic",
            "config": dict(WORKLOAD, config=args.config),
            "run": {"seeds_per_step": seeds, "bases_per_step": int(len(bases)),
                    "parallelism": f"replicas{world}",
                    "l2": ("L2 flushed (256 MiB write) before each timed step" if flush else
                           "no flush: index and reads exceed the 126 MB L2"),
                    "launch": ix.launch()},
            "bases_per_s": bases_rate,
            "e2e": {"value": e2e_rate, "unit": "seeds/s",
                    "h2d_bytes_per_step": int(len(bases) + 8 * (records + 1)),
                    "d2h_bytes_per_step": int(8 * ix.colors + 8)},
            "roofline": dict(roofline, traffic_unit="GB",
                             l2_resident=bool(info.resident_bytes < (126 << 20))),
            "forms": {"plain_seeds_per_s": plain_rate, "batched_seeds_per_s": value / world,
                      "served_seeds_per_s": served["closed_loop"]["seeds_per_s"],
                      "planned_seeds_per_s": world * planned["seeds_per_s"],
                      "unordered_seeds_per_s": unordered,
                      "served": served, "planned": planned, "per_record": per_record},
            "query_file": query_file,
            "index_load": {"seconds": load_s, "banks_s": info.load_banks_s,
                           "recovery_s": info.load_recovery_s, "file_bytes": file_bytes,
                           "resident_bytes": int(info.resident_bytes),
                           "resident_gb_per_s": info.resident_bytes / load_s / 1e9,
                           "note": "zx_open: manifest; bank frames read (page cache) and "
                                   "zstd-decoded on the host cores into a pinned ring whose "
                                   "pieces are copied to HBM while later frames decode; the "
                                   "recovery map decoded concurrently"},
            "gpu_launches": launches,
            "clocks": clocks.summary(),
            "cpu_baseline": cb,
            "parity_vs_oracle_sample": parity,
        }
        if world == 1 and args.config == "c2" and not args.no_other_configs:
            ix.close()
            ix = None
            others = {}
            for name in OTHER_CONFIGS:
                log(f"stage: {name}")
                torch.cuda.empty_cache()
                try:
                    others[name] = other_config(zx, torch, name, Path(args.cache),
                                                max(3, min(args.steps, 5)))
                except Exception as e:  # reported, never hides the default line
                    others[name] = {"error": f"{type(e).__name__}: {e}"}
            line["other_configs"] = others
        print(json.dumps(line), flush=True)
    if ix is not None:
        ix.close()
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser(description=__doc__.splitlines()[0])
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--cache", default=os.environ.get("ZX_BENCH_CACHE", "/tmp/zx_bench"))
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-other-configs", action="store_true",
                    help="default line only (no c3 / c4s measurements beside it)")
    ap.add_argument("--config", choices=sorted(CONFIGS), default="c2",
                    help="workload: c2 (default line) or another configuration")
    ap.add_argument("--reads", type=int, default=None,
                    help="query only the first N reads (smaller case for profiler captures)")
    ap.add_argument("--slice", type=int, default=None,
                    help="profiler case: three plain launches over the first N reads, no timing")
    ap.add_argument("--serve-sweep", action="store_true",
                    help="serving rate sweep: p50/p99 latency against the offered Poisson rate "
                         "and the sustainable request rate of the config (one JSON line)")
    args = ap.parse_args()
    global CONFIG, WORKLOAD
    CONFIG = CONFIGS[args.config]
    WORKLOAD = dict(CONFIG["workload"])
    if args.warmup < 3:
        args.warmup = 3
    if args.slice:
        profile_slice(args)
    elif args.serve_sweep:
        serve_sweep(args)
    elif args.impl == "reference":
        reference_arm(args)
    else:
        ours(args)


def poisson_run(server, requests, rate, seed):
    """Requests submitted at Poisson arrivals of `rate` per second; returns
    the seconds from the first arrival to the last completion, the seeds and
    the server's latency statistics."""
    rng = np.random.default_rng(seed)
    arrivals = np.cumsum(rng.exponential(1.0 / rate, len(requests)))
    tickets = [None] * len(requests)
    server.stats(reset=True)
    start = time.perf_counter()

    def submitter():
        for i, (b, o) in enumerate(requests):
            delay = start + arrivals[i] - time.perf_counter()
            if delay > 0:
                time.sleep(delay)
            tickets[i] = server.submit(b, o)

    th = threading.Thread(target=submitter)
    th.start()
    th.join()
    seeds = sum(server.wait(t)[1] for t in tickets)
    return time.perf_counter() - start, seeds, server.stats(reset=True)


# A rate is sustained when the p99 latency stays within this many times the
# p50 service time of a request served alone and the server completes at
# least SUSTAIN_FRACTION of the offered rate.
SUSTAIN_LATENCY = 10.0
SUSTAIN_FRACTION = 0.9


def serve_sweep(args):
    """Serving rate sweep on the config's request mix (half 1-10,000 short
    reads, half 1-10 long records): the service time of a request alone, the
    closed-loop capacity, then open Poisson streams at fractions of that
    capacity and at the config's stated rate. The sustainable rate is the
    highest swept rate at which the p99 latency stays within SUSTAIN_LATENCY
    x the alone-p50 and completions keep up with arrivals."""
    import torch

    build_native()
    import zindex_b200 as zx

    cache = Path(args.cache)
    index_dir, bases, offsets = prepare(cache, 0, args.config)
    lb, lo = long_pool(cache, 0, args.config)
    sv = CONFIG.get("served", {"closed": 400, "open": 1000, "rate": 200.0})
    pool = make_requests(bases, offsets, lb, lo, 400, 31)
    out = {"config": dict(WORKLOAD), "mix": "half 1-10,000 reads of the batch, half 1-10 long "
           "records (lognormal, median 30 kbp)", "sustain_rule": {
               "p99_within_alone_p50_x": SUSTAIN_LATENCY, "completed_over_offered_min":
               SUSTAIN_FRACTION}}
    with zx.Index(index_dir) as ix, zx.Server(ix, slots=3) as server:
        out["launch"] = ix.launch()
        for b, o in pool[:10]:  # warm-up
            server.wait(server.submit(b, o))
        alone = []
        for b, o in pool[10:50]:
            alone.append(server.wait(server.submit(b, o))[2])
        alone_p50 = float(np.median(alone))
        out["alone"] = {"requests": len(alone), "p50_ms": alone_p50 * 1e3,
                        "p99_ms": float(np.percentile(alone, 99)) * 1e3}
        server.stats(reset=True)
        t0 = time.perf_counter()
        tickets = [server.submit(b, o) for b, o in pool[:sv["closed"]]]
        seeds = sum(server.wait(t)[1] for t in tickets)
        dt = time.perf_counter() - t0
        capacity = len(tickets) / dt
        out["closed_loop"] = {"requests": len(tickets), "req_per_s": capacity,
                              "seeds_per_s": seeds / dt}
        rates = sorted({round(capacity * f, 1) for f in (0.2, 0.4, 0.6, 0.8, 0.9, 1.0, 1.1)} |
                       {float(sv["rate"])})
        rows, sustained = [], 0.0
        for i, rate in enumerate(rates):
            n = int(min(len(pool), max(60, rate * 4)))
            reqs = [pool[j % len(pool)] for j in range(n)]
            dt, seeds, st = poisson_run(server, reqs, rate, 100 + i)
            achieved = st["completed"] / dt
            ok = st["p99_s"] <= SUSTAIN_LATENCY * alone_p50 and achieved >= SUSTAIN_FRACTION * rate
            if ok:
                sustained = max(sustained, rate)
            rows.append({"offered_req_per_s": rate, "requests": n, "completed_req_per_s": achieved,
                         "seeds_per_s": seeds / dt, "p50_ms": st["p50_s"] * 1e3,
                         "p99_ms": st["p99_s"] * 1e3, "max_ms": st["max_s"] * 1e3,
                         "batches": st["batches"], "sustained": bool(ok)})
        out["rates"] = rows
        out["sustainable_req_per_s"] = sustained
        out["stated_rate_req_per_s"] = float(sv["rate"])
    print(json.dumps({"serve_sweep": out}))


def profile_slice(args):
    """A small case of the workload for an ncu capture: the first N reads of
    the batch, queried three times without graphs (the third launch of each
    kernel is the one to capture), then the seed count."""
    import torch

    build_native()
    import zindex_b200 as zx
    from zindex_b200.tuning import DeviceBatch

    index_dir, bases, offsets = prepare(Path(args.cache), 0, args.config)
    offsets = offsets[: args.slice + 1].copy()
    bases = bases[: int(offsets[-1])].copy()
    with zx.Index(index_dir) as ix:
        batch = DeviceBatch(bases, offsets, ix.colors)
        for _ in range(3):
            batch.run(ix, torch.cuda.current_stream(), use_graph=False)
        torch.cuda.synchronize()
        print(json.dumps({"slice_reads": args.slice, "bases": int(len(bases)),
                          "seeds": int(batch.d_total.item()), "launch": ix.launch()}))


if __name__ == "__main__":
    main()
