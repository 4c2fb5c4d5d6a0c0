"""The window probe (kernels/window_probe.cuh) against the oracle at the sizes
where it can go wrong: every slice width a remainder can take, hash counts of
each unroll and of none, segments from 16 to 1,024 cells, hash partitions,
multi-member groups, batches at the key count where it takes over, and keys
that all fall into one bucket. Counts are whole numbers: equality."""
import numpy as np
import pytest

import helpers
from helpers import build_index, dna, sample_reads

pytestmark = pytest.mark.gpu

CASES = [
    dict(colors=250, H=2, b=8, k=25),                     # 16 chunks, ragged last field
    dict(colors=300, H=4, b=8, k=31, seg=16),             # 16 + 2 + 1 chunks, short segments
    dict(colors=700, H=3, b=4, k=25, groups="0,1,2;7,9"),
    dict(colors=260, H=8, b=16, k=31, max_size="256KiB"),  # hash partitions
    dict(colors=300, H=5, b=32, k=25, max_size="1MiB"),
    dict(colors=600, H=16, b=8, k=31),
    dict(colors=270, H=32, b=8, k=21),
    dict(colors=300, H=4, b=8, k=31, seg=256),            # four-chunk slices
    dict(colors=300, H=3, b=8, k=31, seg=1024),           # one-chunk slices
    dict(colors=300, H=4, b=8, k=31, seg=4096),           # no window fits: the wide probe
]


def _index(base, colors, **opts):
    lengths = [2000 if c % 3 == 0 else (4000 if c % 3 == 1 else 9000) for c in range(colors)]
    (base / "g").mkdir()
    lines = []
    for c, n in enumerate(lengths):
        p = base / "g" / f"g{c}.fa"
        helpers.write_fasta(p, [dna(n, 31 + c)])
        lines.append(f"g{c}\t{p}")
    (base / "fof.tsv").write_text("\n".join(lines) + "\n")
    build_index(base / "fof.tsv", base / "index", min_docs=1, **opts)
    return base / "index", [dna(n, 31 + c) for c, n in enumerate(lengths)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_window_probe_matches_oracle(gpu, oracle, tmp_path, case):
    import zindex_b200 as zx

    ix, genomes = _index(tmp_path, **case)
    rng = np.random.default_rng(5)
    batches = [sample_reads(genomes, rng, 3000, 150, n_runs=0.1),
               sample_reads(genomes, rng, 1, 150),
               [b"A" * 9000] * 20 + sample_reads(genomes, rng, 400, 150),  # one k-mer over and over
               [genomes[2][:2000]] * 200]
    with zx.Index(ix) as index:
        for recover in (True, False):
            for reads in batches:
                bases, offsets = zx.pack_records(reads)
                want, want_total = oracle.query_records(ix, bases, offsets, recover=recover)
                got, total = index.query_records(bases, offsets, recover=recover)
                assert total == want_total
                np.testing.assert_array_equal(got, want)


def test_window_probe_around_its_threshold(gpu, oracle, tmp_path):
    """Batches growing through the key count from which windows are used."""
    import zindex_b200 as zx

    ix, genomes = _index(tmp_path, colors=256, H=4, b=8, k=31)
    rng = np.random.default_rng(6)
    with zx.Index(ix) as index:
        for reads in (10, 50, 100, 130, 150, 200, 400, 800):
            bases, offsets = zx.pack_records(sample_reads(genomes, rng, reads, 151))
            want, want_total = oracle.query_records(ix, bases, offsets)
            got, total = index.query_records(bases, offsets)
            assert total == want_total
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("case", [dict(colors=64, H=4, b=8, k=31), dict(colors=9, H=3, b=16, k=25),
                                  dict(colors=30, H=2, b=4, k=45, groups="0,1;5,6"),
                                  dict(colors=100, H=8, b=8, mode="modimizers", k=31, d=4),
                                  dict(colors=100, H=4, b=8, mode="minimizers", k=31, m=21)],
                         ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_dense_batches_of_narrow_rows(gpu, oracle, tmp_path, case):
    """Batches past 1 MiB of an index that defaults to the fused kernel: the
    window probe, and the fused kernel itself once a launch names it."""
    import zindex_b200 as zx

    ix, genomes = _index(tmp_path, **case)
    reads = sample_reads(genomes, np.random.default_rng(8), 8000, 151, n_runs=0.05)
    bases, offsets = zx.pack_records(reads)
    assert len(bases) > 1 << 20
    with zx.Index(ix) as index:
        assert not index.launch()["wide"]
        for recover in (True, False):
            want, want_total = oracle.query_records(ix, bases, offsets, recover=recover)
            for cut in (1, 4):  # chunks past and below 1 MiB
                index.set_launch(cut=cut)
                got, total = index.query_records(bases, offsets, recover=recover)
                assert total == want_total
                np.testing.assert_array_equal(got, want)
        index.set_launch(planes=0)
        got, total = index.query_records(bases, offsets, recover=False)
        assert total == want_total
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("colors", [300, 40])
def test_page_locked_chunks_join_one_list(gpu, oracle, tmp_path, colors):
    """Host batches in page-locked memory: the chunks' seeds are probed
    together, and a record whose offsets decrease is still reported."""
    import torch

    import zindex_b200 as zx

    ix, genomes = _index(tmp_path, colors=colors, H=4, b=8, k=31)
    reads = sample_reads(genomes, np.random.default_rng(9), 24000, 150, n_runs=0.05)
    reads += sample_reads(genomes, np.random.default_rng(10), 40, 3000)
    bases, offsets = zx.pack_records(reads)
    want, want_total = oracle.query_records(ix, bases, offsets)
    locked = torch.from_numpy(bases).pin_memory().numpy()
    with zx.Index(ix) as index:
        for cut in (1, 2, 3, 4):
            index.set_launch(cut=cut)
            got, total = index.query_records(locked, offsets)
            assert total == want_total
            np.testing.assert_array_equal(got, want)
        bad = offsets.copy()
        bad[1001] = bad[1003]  # record 1001 ends before it starts
        with pytest.raises(zx.ZxError) as err:
            index.query_records(locked, bad)
        assert err.value.code == 1
        got, total = index.query_records(locked, offsets)
        assert total == want_total
        np.testing.assert_array_equal(got, want)


def test_more_buckets_than_a_block_counts(gpu, oracle, tmp_path):
    """A class of 2^17 segments: 2^18 buckets, counted in L2."""
    import subprocess

    import zindex_b200 as zx

    subprocess.run([str(helpers.ZX_BUILD), "--synth", "uniform:2:6000000:6000000:5", "-o",
                    str(tmp_path / "index"), "-q", "-k", "31", "-H", "4", "-b", "8", "--device"],
                   check=True)
    genomes = [np.frombuffer(dna(6_000_000, 5 + c), dtype=np.uint8) for c in range(2)]
    rng = np.random.default_rng(4)
    reads = [genomes[i % 2][at: at + 10_000] for i, at in enumerate(rng.integers(0, 5_990_000, 1900))]
    bases = np.concatenate(reads)
    offsets = np.arange(len(reads) + 1, dtype=np.uint64) * 10_000
    with zx.Index(tmp_path / "index") as index:
        got, total = index.query_records(bases, offsets)
        index.set_launch(cut=1)
        once, total_once = index.query_records(bases, offsets)
    want, want_total = oracle.query_records(tmp_path / "index", bases, offsets)
    assert total == total_once == want_total
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(once, want)
