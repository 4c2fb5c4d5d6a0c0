"""Batches past the size that is sorted and probed as one list, against the
oracle: chunks and records of both sides of it in one host call."""
import numpy as np
import pytest

import helpers
from helpers import build_index, dna, make_genomes, sample_reads

pytestmark = pytest.mark.gpu


def _narrow_index(tmp_path, colors=40, length=5000):
    fof = make_genomes(tmp_path / "g", colors, length, 31)
    return (build_index(fof, tmp_path / "index", k=31, H=4, b=8, min_docs=1),
            [dna(length, 31 + c) for c in range(colors)])


def test_records_past_and_below_the_round_limit(gpu, oracle, tmp_path):
    """A record above the limit beside chunks, and records, that are dense."""
    import zindex_b200 as zx

    ix, genomes = _narrow_index(tmp_path)
    rng = np.random.default_rng(11)
    long = b"".join(sample_reads(genomes, rng, 16000, 150))  # 2.4e6 bases
    reads = sample_reads(genomes, rng, 10500, 150, n_runs=0.05)
    bases, offsets = zx.pack_records([long] + reads)
    chunks = np.searchsorted(offsets, [len(bases) // 3, len(bases) // 3 * 2])
    sizes = np.diff(np.concatenate(([0], offsets[chunks], offsets[-1:])).astype(np.int64))
    assert sizes[0] > 2 << 20 > sizes[2] > 1 << 20
    want, want_total = oracle.query_records(ix, bases, offsets)
    two, two_offsets = zx.pack_records([long, long[:1_500_000]])
    want_two, want_two_total = oracle.query_records(ix, two, two_offsets)
    with zx.Index(ix) as index:
        assert not index.launch()["wide"]
        index.set_round_bases(2 << 20)
        got, total = index.query_records(bases, offsets)
        assert total == want_total
        np.testing.assert_array_equal(got, want)
    with zx.Index(ix) as index:
        index.set_round_bases(2 << 20)
        got, total = index.query_records(two, two_offsets, plain=True)
        assert total == want_two_total
        np.testing.assert_array_equal(got, want_two)
