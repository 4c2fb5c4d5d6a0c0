"""The work that users of zindex_b200 have it do, as cases that can be timed.

A case names an index (seed mode, hashes, fingerprint bits, colours, genome
lengths), a batch of records and the public call that queries it:

  device      Index.query_device: a batch resident on the GPU, counted into the
              caller's counters (a pipeline that keeps its reads on the GPU)
  segments    Index.query_segments: several requests coalesced into one launch
              (a service that manages its own buffers)
  host        Index.query_records: records in host memory, counts back (the call
              behind `zorindex query`)
  per_record  Index.query_per_record: every record's own counts (`query --records`)

Indexes are built by zx_build from its seeded synthetic genomes (the core-pool
model of the benchmark: 70 % i.i.d. bases, 30 % copied from 50 shared segments),
and records are drawn from the same genomes with substitutions, plus random
ones. An index depends on the case alone and is opened once per process: a
user's program keeps it resident and queries it with batch after batch. The
records of a batch depend on the seed.
"""
from __future__ import annotations

import functools
import math
import subprocess
import tempfile
from pathlib import Path

import numpy as np
import torch

import zindex_b200 as zx

# The batched k-mer workload's options with its genome lengths scaled down ten
# times (0.4 GB of rows: still several times the L2), so that building it is quick.
READS_INDEX = dict(mode="kmers", k=31, hashes=4, bits=8, colors=256, shortest=100_000,
                   longest=1_000_000)
NO_RECORDS = dict(short=0, short_len=150, long=0, long_median=2000, sourced=0.7, subst=0.005,
                  n_runs=0.0)


def listed():
    return [
        # The smallest call: one read against a resident index, where launches are the cost.
        dict(NO_RECORDS, name="one-read", call="device", **READS_INDEX, short=1),
        # A small FASTA against ten genomes (the benchmark's c1): rows in L2, 97,000 seeds.
        dict(NO_RECORDS, name="small-file", call="device", mode="kmers", k=31, hashes=4, bits=8,
             colors=10, shortest=2_000_000, longest=2_000_000, short=100, short_len=1000,
             sourced=0.01, subst=0.0),
        # A sequencing run's reads in one batch (the benchmark's c2, its default workload).
        dict(NO_RECORDS, name="batched-reads", call="device", **READS_INDEX, short=1_000_000),
        # The same kind of batch handed over in host memory and counted end to end.
        dict(NO_RECORDS, name="host-reads", call="host", **READS_INDEX, short=250_000),
        # Few colours, so narrow rows, and a ragged mix of reads (the geometry sweep's c64).
        dict(NO_RECORDS, name="few-colors", call="device", mode="kmers", k=31, hashes=4, bits=8,
             colors=64, shortest=1_000_000, longest=4_000_000, short=100_000, long=5_000),
        # Long reads of very uneven length against a minimizer index (the benchmark's c3,
        # genomes and records scaled down): windows with N runs, 16-bit fingerprints.
        dict(NO_RECORDS, name="minimizers-long", call="device", mode="minimizers", k=49, m=31,
             hashes=3, bits=16, colors=2048, shortest=50_000, longest=800_000, long=40_000,
             sourced=0.8, subst=0.01, n_runs=0.1),
        # A sampled index (one 49-mer in 16) and the sweep's mixed batch.
        dict(NO_RECORDS, name="modimizers-mix", call="device", mode="modimizers", k=49,
             sampling=16, hashes=4, bits=8, colors=512, shortest=100_000, longest=1_000_000,
             short=100_000, long=5_000),
        # Run-length filtered matching (findere k31 z10) on the sweep's mixed batch.
        dict(NO_RECORDS, name="findere-mix", call="device", mode="findere", k=31, z=10, hashes=4,
             bits=8, colors=128, shortest=100_000, longest=1_000_000, short=50_000, long=2_500),
        # A collection of 16,384 small genomes: 8 KiB rows of 4-bit fields (the benchmark's c4s).
        dict(NO_RECORDS, name="many-colors", call="device", mode="kmers", k=31, hashes=8, bits=4,
             colors=16384, shortest=20_000, longest=120_000, short=20_000, sourced=0.6),
        # Requests of a service answered together: half of them up to 10,000 reads, half up to
        # ten long records (the benchmark's served mix).
        dict(NO_RECORDS, name="served-requests", call="segments", **READS_INDEX, requests=32,
             short=80_000, long=90, long_median=30_000, sourced=0.6),
        # The per-record report's counts: every read for itself, into page-locked buffers.
        dict(NO_RECORDS, name="per-record", call="per_record", **READS_INDEX, short=20_000),
        # Randstrobemer seeds: both strands of every read are linked and counted.
        dict(NO_RECORDS, name="randstrobemers", call="host", mode="kmers", strobes=True, k=21,
             hashes=4, bits=8, colors=64, shortest=100_000, longest=1_000_000, short=20_000,
             long=200),
    ]


def draw(rng):
    """One more case: any index geometry of the supported ranges under any of the calls."""
    mode = rng.choice(["kmers"] * 6 + ["minimizers"] * 2 + ["modimizers", "findere"])
    case = dict(NO_RECORDS, mode=mode, hashes=rng.choice([2, 3, 4, 4, 8, 16]),
                bits=rng.choice([1, 2, 4, 8, 8, 16, 32]))
    if mode == "kmers":
        case.update(k=rng.choice([21, 25, 31, 45]))
    elif mode == "minimizers":
        k, m = rng.choice([(31, 21), (49, 31)])
        case.update(k=k, m=m)
    elif mode == "modimizers":
        case.update(k=rng.choice([31, 49]), sampling=16)
    else:
        case.update(k=31, z=10)
    colors = int(round(math.exp(rng.uniform(math.log(10), math.log(16384)))))
    if mode == "findere":
        colors = min(colors, 2000)
    bases = (10e6 if mode == "findere" else 60e6) * rng.uniform(0.5, 1.0)
    shortest = int(min(2_000_000, max(2_000, bases / colors / 4)))
    case.update(colors=colors, shortest=shortest, longest=shortest * 8)
    # Records up to 40 GB of row reads (1.5e9 field compares where every hit is counted one by
    # one), over the logarithm down to a single read.
    most = min(20e6, 40e9 / row_bytes(case))
    if case["bits"] < 4 or mode == "findere":
        most = min(most, 1.5e9 / colors)
    seeds = math.exp(rng.uniform(math.log(120), math.log(most)))
    windows = seeds / density(case)
    length = rng.choice([150, 150, 151, 250, 1000])
    reads = max(1, int(windows / (length - case["k"] + 1)))
    share = rng.choice([0.0, 0.0, 0.5])
    case.update(call=rng.choice(["device"] * 4 + ["host", "segments", "per_record"]),
                short_len=length, sourced=rng.uniform(0.5, 0.9), subst=rng.choice([0.0, 0.005, 0.01]),
                n_runs=rng.choice([0.0, 0.1]))
    if case["call"] == "per_record":
        reads = min(reads, max(1, 20_000_000 // colors))
    case["short"] = max(1, int(reads * (1.0 - share)))
    case["long"] = int(reads * share * length / (case["long_median"] * 1.65))
    if case["call"] == "segments":
        case["requests"] = max(1, min(rng.randint(1, 64), case["short"]))
    return case


# ---- what a case costs at least --------------------------------------------
def row_bytes(case):
    """Fingerprint bytes of a seed's rows."""
    return case["hashes"] * math.ceil(case["colors"] * case["bits"] / 8)


def density(case):
    """Seeds per window."""
    if case["mode"] == "minimizers":
        return 2.0 / (case["k"] - case["m"] + 2)
    return 1.0 / case["sampling"] if case["mode"] == "modimizers" else 1.0


def work(case):
    span = case["k"]
    long_len = case["long_median"] * math.exp(0.5)
    records = case["short"] + case["long"]
    bases = case["short"] * case["short_len"] + case["long"] * long_len
    seeds = max(0.0, bases - records * (span - 1)) * density(case)
    strands = 2 if case.get("strobes") else 1
    # The filters' fingerprints at one cell per key: read once, or only the seeds' rows.
    keys = float(genome_lengths(case).sum()) * density(case)
    rows = min(keys * case["bits"] / 8, strands * seeds * row_bytes(case))
    rows_out = {"segments": case.get("requests", 1), "per_record": records}.get(case["call"], 1)
    return {"bytes": bases + 8.0 * (records + 1) + rows + 8.0 * rows_out * (case["colors"] + 1),
            "flops": 0.0}


def exact(case, seed):
    """Every output is a whole number: compared as it is."""
    return None


# ---- genomes (the synthetic collections of zx_build --synth) ----------------
GENOME_SEED = 1
BLOCK, CORES = 100_000, 50


def _wrap(v):
    return (v & (1 << 64) - 1) - (1 << 64 if v >> 63 & 1 else 0)


def _splitmix_int(x):
    m = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & m
    x = (x ^ x >> 30) * 0xBF58476D1CE4E5B9 & m
    x = (x ^ x >> 27) * 0x94D049BB133111EB & m
    return x ^ x >> 31


def _shr(x, n):
    return (x >> n) & ((1 << 64 - n) - 1)


def _splitmix(x):
    x = x + _wrap(0x9E3779B97F4A7C15)
    x = (x ^ _shr(x, 30)) * _wrap(0xBF58476D1CE4E5B9)
    x = (x ^ _shr(x, 27)) * _wrap(0x94D049BB133111EB)
    return x ^ _shr(x, 31)


def genome_lengths(case):
    lo, hi, n = case["shortest"], case["longest"], case["colors"]
    if lo == hi:
        return np.full(n, lo, dtype=np.int64)
    u = np.array([(_splitmix_int(GENOME_SEED ^ _splitmix_int(0x6C656E67746800 + g)) >> 11) * 2.0**-53
                  for g in range(n)])
    return np.floor(np.exp(math.log(lo) + u * (math.log(hi) - math.log(lo)))).astype(np.int64)


def _genome_codes(g, p):
    """2-bit base codes at positions p of genomes g (core-pool model)."""
    block, off = p // BLOCK, p % BLOCK
    r = _splitmix(_splitmix_int_tensor(GENOME_SEED ^ 0x626C6F636B, p.device) ^ (g << 24) ^ block)
    # r % 1000 of the unsigned value.
    low = torch.remainder(_shr(r, 1) % 500 * 2 + (r & 1), 1000)
    core = _shr(r, 32) % CORES
    shared = off ^ _splitmix(_wrap(GENOME_SEED ^ 0x636F7265) ^ (core << 40))
    own = p ^ _splitmix(_wrap(GENOME_SEED ^ 0x67656E6F6D) ^ (g << 20))
    return _splitmix(torch.where(low < 300, shared, own)) & 3


def _splitmix_int_tensor(v, device):
    return torch.tensor(_wrap(_splitmix_int(v)), dtype=torch.int64, device=device)


@functools.lru_cache(maxsize=4)
def _open_index(options):
    """The index of a case, built by the command-line builder and made resident."""
    case = dict(options)
    with tempfile.TemporaryDirectory() as work:
        out = Path(work) / "index"
        # (Equal lengths: still the core-pool model, as the records assume.)
        args = ["--synth", f"pool:{case['colors']}:{case['shortest']}:{case['longest']}:{GENOME_SEED}",
                "-o", str(out), "-q", "-i", case["mode"], "-k", str(case["k"]),
                "-H", str(case["hashes"]), "-b", str(case["bits"])]
        for key, flag in (("m", "-m"), ("z", "-z"), ("sampling", "-d")):
            if key in case:
                args += [flag, str(case[key])]
        if case.get("strobes"):
            args.append("-r")
        elif case["mode"] != "findere":
            args.append("--device")
        subprocess.run([str(Path(zx.LIB_DIR) / "zx_build"), *args], check=True)
        return zx.Index(out)


def open_index(case):
    keys = ("mode", "k", "m", "z", "sampling", "strobes", "hashes", "bits", "colors", "shortest",
            "longest")
    return _open_index(tuple((key, case[key]) for key in keys if key in case))


def make_records(case, seed):
    """(bases uint8, offsets int64) on the GPU: the short reads, then the long ones."""
    dev = torch.device("cuda")
    rng = torch.Generator(device=dev)
    rng.manual_seed(seed)
    n_short, n_long = case["short"], case["long"]
    lengths = torch.full((n_short + n_long,), case["short_len"], dtype=torch.int64, device=dev)
    if n_long:
        z = torch.randn(n_long, generator=rng, device=dev, dtype=torch.float64)
        lengths[n_short:] = (torch.exp(math.log(case["long_median"]) + z)).clamp(100, 100_000).long()
    n = n_short + n_long
    genomes = torch.from_numpy(genome_lengths(case)).to(dev)
    sourced = torch.rand(n, generator=rng, device=dev) < case["sourced"]
    g = torch.randint(0, case["colors"], (n,), generator=rng, device=dev)
    lengths = torch.where(sourced, torch.minimum(lengths, genomes[g]), lengths)
    at = (torch.rand(n, generator=rng, device=dev, dtype=torch.float64)
          * (genomes[g] - lengths + 1).clamp(min=1)).long()
    n_at = (torch.rand(n, generator=rng, device=dev, dtype=torch.float64) * lengths).long()
    n_len = torch.randint(1, 51, (n,), generator=rng, device=dev)
    n_len = torch.where(torch.rand(n, generator=rng, device=dev) < case["n_runs"], n_len, 0)
    offsets = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    offsets[1:] = torch.cumsum(lengths, 0)
    nbases = int(offsets[-1])
    bases = torch.empty(nbases, dtype=torch.uint8, device=dev)
    acgt = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=dev)
    step = 1 << 24
    for a in range(0, nbases, step):
        i = torch.arange(a, min(nbases, a + step), device=dev)
        r = torch.searchsorted(offsets, i, right=True) - 1
        p = i - offsets[r]
        code = _genome_codes(g[r], at[r] + p)
        other = torch.randint(0, 4, i.shape, generator=rng, device=dev)
        code = torch.where(sourced[r], code, other)
        wrong = torch.rand(i.shape, generator=rng, device=dev) < case["subst"]
        code = torch.where(wrong, (code + 1 + other % 3) & 3, code)
        b = acgt[code]
        bases[a:a + step] = torch.where((p >= n_at[r]) & (p < n_at[r] + n_len[r]), ord("N"), b)
    return bases, offsets


def prepare(case, seed):
    ix = open_index(case)
    bases, offsets = make_records(case, seed)
    records = offsets.numel() - 1
    state = {"call": case["call"], "ix": ix, "records": records, "nbases": bases.numel()}
    if case["call"] in ("host", "per_record"):
        state.update(bases=bases.cpu().numpy(), offsets=offsets.cpu().numpy().view(np.uint64))
        if case["call"] == "per_record":
            # Page-locked results, as query_per_record's documentation suggests.
            state["keep"] = [torch.zeros((records, ix.colors), dtype=torch.int64, pin_memory=True),
                             torch.zeros(records, dtype=torch.int64, pin_memory=True)]
            state["counts"], state["totals"] = (t.numpy().view(np.uint64) for t in state["keep"])
        return state
    state.update(bases=bases, offsets=offsets)
    rows = 1
    if case["call"] == "segments":
        # Half of the requests share the short reads, half the long records.
        rows = case["requests"]
        rng = np.random.default_rng(seed)
        halves = [(rows + 1) // 2, rows // 2] if case["long"] and rows > 1 else [rows, 0]
        cuts, first = [0], 0
        for requests, n in zip(halves, (case["short"], case["long"])):
            if halves[1] == 0:
                n = records
            if requests:
                cuts += sorted(rng.integers(0, n + 1, requests - 1) + first) + [first + n]
                first += n
        state["segments"] = np.array(cuts, dtype=np.uint64)
    state["counts"] = torch.zeros((rows, ix.colors), dtype=torch.int64, device="cuda")
    state["total"] = torch.zeros(rows, dtype=torch.int64, device="cuda")
    return state


def run(state):
    ix, call = state["ix"], state["call"]
    if call == "host":
        counts, total = ix.query_records(state["bases"], state["offsets"])
        return {"counts": counts, "total": total}
    if call == "per_record":
        counts, totals = ix.query_per_record(state["bases"], state["offsets"],
                                             counts=state["counts"], totals=state["totals"])
        return {"counts": counts, "totals": totals}
    state["counts"].zero_()
    state["total"].zero_()
    stream = torch.cuda.current_stream().cuda_stream
    args = (state["bases"].data_ptr(), state["nbases"], state["offsets"].data_ptr(), state["records"])
    out = (state["counts"].data_ptr(), state["total"].data_ptr(), stream)
    if call == "segments":
        ix.query_segments(*args, state["segments"], *out)
    else:
        ix.query_device(*args, *out)
    return {"counts": state["counts"], "total": state["total"]}
