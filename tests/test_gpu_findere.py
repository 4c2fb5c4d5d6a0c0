"""Findere by position masks (kernels/findere.cuh) against the oracle where it
can go wrong: run lengths around the counters' widths and the 128-position
stretches, rows from one chunk to the widest, every fingerprint width, size
classes, hash partitions, long s-mers, invalid bases, recovered origins, and
the indexes it leaves to the per-hit form (a multi-member group, 2-bit fields,
wider rows). Counts are whole numbers: equality."""
import numpy as np
import pytest

import helpers
from helpers import build_index, dna, sample_reads

pytestmark = pytest.mark.gpu

CASES = [
    dict(colors=10, H=4, b=8, k=31, z=10),
    dict(colors=10, H=3, b=8, k=25, z=0),
    dict(colors=60, H=2, b=16, k=32, z=7),                   # 8 hits: a counter's width exactly
    dict(colors=60, H=4, b=32, k=33, z=8),
    dict(colors=130, H=5, b=4, k=31, z=3, max_size="16KiB"),  # hash partitions
    dict(colors=300, H=4, b=8, k=160, z=127),                # runs as long as a stretch
    dict(colors=60, H=4, b=8, k=160, z=128),
    dict(colors=40, H=4, b=8, k=250, z=224),                 # the longest runs
    dict(colors=20, H=4, b=8, k=60, z=10),                   # s-mers of 50 bases
    dict(colors=480, H=3, b=8, k=31, z=10),                  # 30 chunks and more over the classes
    dict(colors=700, H=3, b=8, k=31, z=10),                  # too wide
    dict(colors=40, H=4, b=2, k=31, z=10),
    dict(colors=40, H=4, b=8, k=31, z=10, groups="0,1,2"),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_findere_matches_oracle(gpu, oracle, tmp_path, case):
    import zindex_b200 as zx

    case = dict(case)
    colors = case.pop("colors")
    lengths = [1500 if c % 3 == 0 else (3000 if c % 3 == 1 else 6000) for c in range(colors)]
    (tmp_path / "g").mkdir()
    genomes, lines = [dna(n, 71 + c) for c, n in enumerate(lengths)], []
    for c, g in enumerate(genomes):
        p = tmp_path / "g" / f"g{c}.fa"
        helpers.write_fasta(p, [g])
        lines.append(f"g{c}\t{p}")
    (tmp_path / "fof.tsv").write_text("\n".join(lines) + "\n")
    ix = build_index(tmp_path / "fof.tsv", tmp_path / "index", mode="findere", min_docs=1, **case)
    rng = np.random.default_rng(3)
    reads = sample_reads(genomes, rng, 150, 300, subst=0.01, n_runs=0.2)
    reads += sample_reads(genomes, rng, 6, 1400, sourced=1.0, subst=0.001) + [b"A" * 700, b"ACGT" * 60]
    bases, offsets = zx.pack_records(reads)
    with zx.Index(ix) as index:
        for recover in (True, False):
            want, want_total = oracle.query_records(ix, bases, offsets, recover=recover)
            for launch in ({}, {"smem_counters": 0, "warps": 2}):
                index.set_launch(**launch)
                got, total = index.query_records(bases, offsets, recover=recover)
                assert total == want_total
                np.testing.assert_array_equal(got, want)
        index.set_launch()
        counts, totals = index.query_per_record(bases, offsets)
        np.testing.assert_array_equal(counts.sum(axis=0), oracle.query_records(ix, bases, offsets)[0])
        for r in (0, 40, len(reads) - 2):
            one = zx.pack_records([reads[r]])
            want, want_total = oracle.query_records(ix, *one)
            np.testing.assert_array_equal(counts[r], want)
            assert totals[r] == want_total
