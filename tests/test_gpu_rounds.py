"""Batches that are sorted and probed as one list, and those past that size or
without memory for it, against the oracle; the planner's and the lists' bounds
under offsets that go back; workspaces after a failed allocation."""
import numpy as np
import pytest

import helpers
from helpers import build_index, dna, make_genomes, sample_reads

pytestmark = pytest.mark.gpu


def _lists_held(index) -> int:
    """Bytes of the key lists that the index holds (it gives them back)."""
    import torch

    before = torch.cuda.mem_get_info()[0]
    index.set_round_bases(0)
    return torch.cuda.mem_get_info()[0] - before


def _narrow_index(tmp_path, colors=240, length=3000):
    fof = make_genomes(tmp_path / "g", colors, length, 31)
    return (build_index(fof, tmp_path / "index", k=31, H=4, b=8, min_docs=1),
            [dna(length, 31 + c) for c in range(colors)])


def test_records_past_and_below_the_round_limit(gpu, oracle, tmp_path):
    """A record above the limit beside chunks, and records, that are dense."""
    import zindex_b200 as zx

    ix, genomes = _narrow_index(tmp_path)
    rng = np.random.default_rng(11)
    long = b"".join(sample_reads(genomes, rng, 34000, 150))  # 5.1e6 bases
    reads = sample_reads(genomes, rng, 22000, 150, n_runs=0.05)
    bases, offsets = zx.pack_records([long] + reads)
    cuts = np.searchsorted(offsets, [len(bases) // 4, len(bases) // 4 * 3])
    sizes = np.diff(np.concatenate(([0], offsets[cuts], offsets[-1:])).astype(np.int64))
    # (The last chunk is dense; the middle one is not.)
    assert sizes[0] > 4 << 20 > sizes[2] > 2_000_000 and sizes[1] < 1_270_000
    want, want_total = oracle.query_records(ix, bases, offsets)
    two, two_offsets = zx.pack_records([long, long[:3_000_000]])
    want_two, want_two_total = oracle.query_records(ix, two, two_offsets)
    # (Without a limit: dense chunks on both sides of one that is not.)
    for limit in (4 << 20, 0):
        with zx.Index(ix) as index:
            assert not index.launch()["wide"]
            index.set_round_bases(limit)
            got, total = index.query_records(bases, offsets)
            assert total == want_total
            np.testing.assert_array_equal(got, want)
            assert _lists_held(index) >= 16 * sizes[2]
    with zx.Index(ix) as index:
        index.set_round_bases(4 << 20)
        got, total = index.query_records(two, two_offsets, plain=True)
        assert total == want_two_total
        np.testing.assert_array_equal(got, want_two)
        assert _lists_held(index) >= 16 * 3_000_000


@pytest.mark.parametrize("opts", [dict(), dict(mode="findere", k=31, z=10), dict(homopolymer=True),
                                  dict(mode="minimizers", k=31, m=21)],
                         ids=["kmers", "findere", "homopolymer", "minimizers"])
@pytest.mark.parametrize("colors", [12, 270], ids=["narrow", "wide"])
def test_overlapping_records_stay_inside_the_lists(gpu, oracle, tmp_path, opts, colors):
    """Offsets that go back to 0 again and again: every other record is the
    whole batch, so the records hold many times the batch's tiles and seeds.
    They are reported, no count is higher than those records' own, and the
    index keeps answering correctly."""
    import torch

    import zindex_b200 as zx

    fof = make_genomes(tmp_path / "g", colors, 3000, 31)
    ix = build_index(fof, tmp_path / "index", **{**dict(k=31, H=4, b=8, min_docs=1), **opts})
    genomes = [dna(3000, 31 + c) for c in range(colors)]
    rng = np.random.default_rng(12)
    dev = torch.device("cuda", 0)
    with zx.Index(ix) as index:
        for nbases, records in ((300_000, 3001), (1_500_000, 801)):
            reads = sample_reads(genomes, rng, nbases // 150, 150)
            bases, offsets = zx.pack_records(reads)
            one = np.array([0, len(bases)], dtype=np.uint64)
            want, want_total = oracle.query_records(ix, bases, one)
            bad = np.zeros(records + 1, dtype=np.int64)
            bad[1::2] = len(bases)
            whole = (records + 1) // 2  # records that are the whole batch
            d_b = torch.from_numpy(bases).to(dev)
            d_bad = torch.from_numpy(bad).to(dev)
            counts = torch.zeros(index.colors, dtype=torch.int64, device=dev)
            total = torch.zeros(1, dtype=torch.int64, device=dev)
            args = (d_b.data_ptr(), len(bases), d_bad.data_ptr(), records, counts.data_ptr(),
                    total.data_ptr())
            calls = [lambda: index.query_device(*args, use_graph=False)]
            if "homopolymer" not in opts:
                calls.append(lambda: index.query_device_noalloc(*args))
            for call in calls:
                counts.zero_()
                total.zero_()
                call()
                torch.cuda.synchronize(dev)
                with pytest.raises(zx.ZxError) as err:
                    index.query_status()
                assert err.value.code == 1
                assert 0 < int(total) <= whole * want_total
                assert np.all(counts.cpu().numpy() <= whole * want.astype(np.int64))
            got, got_total = index.query_records(bases, one)
            assert got_total == want_total
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("opts", [dict(k=31), dict(k=45), dict(mode="minimizers", k=25, m=21)],
                         ids=["short", "long", "minimizers"])
def test_a_full_key_list_has_no_holes(gpu, tmp_path, opts):
    """Records that overlap fill the key list. The list's old keys (all in the
    first genome) must not come back - seeds of random bases hit no 32-bit
    fingerprint - and it is full to the last place in every run."""
    import torch

    import zindex_b200 as zx

    fof = make_genomes(tmp_path / "g", 64, 3000, 31)
    ix = build_index(fof, tmp_path / "index", **{**dict(H=4, b=32, min_docs=1), **opts})
    rng = np.random.default_rng(13)
    dev = torch.device("cuda", 0)
    nbases, records = 1_500_000, 160_001
    # (The list has a quarter more room than the batch that made it.)
    hits = np.frombuffer(dna(3000, 31) * (nbases * 5 // 4 // 3000), dtype=np.uint8)
    misses = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, nbases)]
    # Records of 1 to 200 windows, so that small ones still fit where larger
    # ones no longer do.
    bad = np.empty(records + 1, dtype=np.int64)
    bad[0::2] = rng.integers(0, 30, len(bad[0::2]))
    bad[1::2] = bad[0::2] + rng.integers(45, 245, len(bad[1::2]))
    d_bad = torch.from_numpy(bad).to(dev)
    one = torch.tensor([0, len(hits)], dtype=torch.int64, device=dev)
    with zx.Index(ix) as index:
        assert index.launch()["wide"]
        counts = torch.zeros(index.colors, dtype=torch.int64, device=dev)
        total = torch.zeros(1, dtype=torch.int64, device=dev)
        out = (counts.data_ptr(), total.data_ptr())
        d_hits, d_misses = torch.from_numpy(hits.copy()).to(dev), torch.from_numpy(misses).to(dev)
        totals = []
        for i in range(40):
            if i:
                index.query_device(d_hits.data_ptr(), len(hits), one.data_ptr(), 1, *out,
                                   use_graph=False)
            counts.zero_()
            total.zero_()
            index.query_device(d_misses.data_ptr(), nbases, d_bad.data_ptr(), records, *out,
                               use_graph=False)
            torch.cuda.synchronize(dev)
            with pytest.raises(zx.ZxError):
                index.query_status()
            totals.append(int(total))
            assert int(counts.sum()) == 0
        assert min(totals) == max(totals) >= nbases


@pytest.mark.parametrize("colors", [12, 270], ids=["narrow", "wide"])
def test_a_batch_without_memory_leaves_the_index_usable(gpu, oracle, tmp_path, colors):
    """2^42 bases fit no GPU: ZX_ENOMEM before any base is read, and the calls
    after it, of sizes seen and not seen before, answer correctly."""
    import torch

    import zindex_b200 as zx

    fof = make_genomes(tmp_path / "g", colors, 3000, 31)
    ix = build_index(fof, tmp_path / "index", k=31, H=4, b=8, min_docs=1)
    genomes = [dna(3000, 31 + c) for c in range(colors)]
    batches = [zx.pack_records(sample_reads(genomes, np.random.default_rng(n), n, 150))
               for n in (200, 20, 2000)]
    dev = torch.device("cuda", 0)
    with zx.Index(ix) as index:
        counts = torch.zeros(index.colors, dtype=torch.int64, device=dev)
        total = torch.zeros(1, dtype=torch.int64, device=dev)
        offsets = torch.tensor([0, 100], dtype=torch.int64, device=dev)
        args = (offsets.data_ptr(), 1, counts.data_ptr(), total.data_ptr())
        seg = np.array([0, 1], dtype=np.uint64)
        for bases, offs in batches:
            want, want_total = oracle.query_records(ix, bases, offs)
            for graph in (False, True):
                got, got_total = index.query_records(bases, offs)
                assert got_total == want_total
                np.testing.assert_array_equal(got, want)
                with pytest.raises(zx.ZxError) as err:
                    index.query_device(counts.data_ptr(), 1 << 42, *args, use_graph=graph)
                assert err.value.code == 4
                with pytest.raises(zx.ZxError) as err:
                    index.query_segments(counts.data_ptr(), 1 << 42, *args[:2], seg, *args[2:])
                assert err.value.code == 4
            per, totals = index.query_per_record(bases, offs)
            assert int(totals.sum()) == want_total
            np.testing.assert_array_equal(per.sum(axis=0, dtype=np.uint64), want)


def test_many_hash_partitions_keep_the_bucket_table_small(gpu, oracle, tmp_path):
    """8,192 partitions: sorted by the first hash alone, in 2^16 buckets. One
    read takes no more than ten times its unsorted time (with the partitions in
    the key it was 2^23 buckets, walked by one block in every call)."""
    import subprocess

    import torch

    import zindex_b200 as zx

    subprocess.run([str(helpers.ZX_BUILD), "--synth", "uniform:128:40000:40000:5", "-o",
                    str(tmp_path / "index"), "-q", "-k", "31", "-H", "2", "-b", "16", "-L", "4",
                    "-X", "2KiB"], check=True)
    genomes = [dna(40000, 5 + c) for c in range(128)]
    rng = np.random.default_rng(14)
    dev = torch.device("cuda", 0)
    with zx.Index(tmp_path / "index") as index:
        assert index.info.banks == 8192 and index.launch()["wide"]
        for reads in (1, 300, 20000):
            bases, offsets = zx.pack_records(sample_reads(genomes, rng, reads, 150))
            want, want_total = oracle.query_records(tmp_path / "index", bases, offsets)
            got, total = index.query_records(bases, offsets)
            assert total == want_total
            np.testing.assert_array_equal(got, want)
        d_b = torch.from_numpy(np.frombuffer(genomes[7][:150], dtype=np.uint8).copy()).to(dev)
        d_off = torch.tensor([0, 150], dtype=torch.int64, device=dev)
        counts = torch.zeros(128, dtype=torch.int64, device=dev)
        n = torch.zeros(1, dtype=torch.int64, device=dev)
        stream = torch.cuda.current_stream(dev).cuda_stream

        def micros():
            best = float("inf")
            for _ in range(20):
                first, last = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                first.record()
                for _ in range(50):
                    index.query_device(d_b.data_ptr(), 150, d_off.data_ptr(), 1,
                                       counts.data_ptr(), n.data_ptr(), stream)
                last.record()
                last.synchronize()
                best = min(best, first.elapsed_time(last) * 20)
            return best

        sorted_us = micros()
        index.set_launch(wide=1, order=0)
        plain_us = micros()
        print(f"one read: {sorted_us:.1f} us sorted, {plain_us:.1f} us unsorted")
        assert sorted_us < 10 * plain_us


def test_dense_batches_of_grouped_colours(gpu, oracle, tmp_path):
    """Narrow rows can hold many colours through multi-member groups: with six
    classes and 32 hashes the probe's row table leaves no shared memory for
    9,600 colour counters."""
    import zindex_b200 as zx

    per_class, members = 1600, 50
    lengths = [60, 120, 240, 480, 960, 1920]
    (tmp_path / "g").mkdir()
    lines, groups = [], []
    for i, n in enumerate(lengths):
        first = i * per_class
        for c in range(first, first + per_class):
            p = tmp_path / "g" / f"g{c}.fa"
            helpers.write_fasta(p, [dna(n, 31 + c)])
            lines.append(f"g{c}\t{p}")
        groups += [",".join(map(str, range(a, a + members)))
                   for a in range(first, first + per_class, members)]
    (tmp_path / "fof.tsv").write_text("\n".join(lines) + "\n")
    ix = build_index(tmp_path / "fof.tsv", tmp_path / "index", k=31, H=32, b=8, seg=16, min_docs=1,
                     groups=";".join(groups))
    rng = np.random.default_rng(15)
    genomes = [dna(960, 31 + int(c)) for c in rng.integers(4 * per_class, 5 * per_class, 200)]
    reads = sample_reads(genomes, rng, 300, 150)
    # (Dense by bases that are no seeds.)
    bases, offsets = zx.pack_records([r + b"N" * 60_000 for r in reads])
    want, want_total = oracle.query_records(ix, bases, offsets)
    with zx.Index(ix) as index:
        assert not index.launch()["wide"] and index.info.classes == 6
        index.set_launch(cut=1)
        got, total = index.query_records(bases, offsets)
        assert total == want_total
        np.testing.assert_array_equal(got, want)
        assert _lists_held(index) >= 16 * len(bases)
        index.set_launch(blocks=1000)  # no longer the default: the fused kernel
        got, total = index.query_records(bases, offsets)
        assert total == want_total
        np.testing.assert_array_equal(got, want)


def test_key_lists_come_and_go_with_the_memory(gpu, oracle, tmp_path):
    """Key lists are held while there is room for them: not while 1.4 GB are
    free, again once the memory is back, and no longer when another buffer of
    the index needs theirs."""
    import torch

    import zindex_b200 as zx

    fof = make_genomes(tmp_path / "g", 260, 3000, 31)
    ix = build_index(fof, tmp_path / "index", k=31, H=4, b=8, min_docs=1)
    genomes = [dna(3000, 31 + c) for c in range(260)]
    rng = np.random.default_rng(16)
    reads = sample_reads(genomes, rng, 2000, 150)
    few = zx.pack_records(reads[:50])
    # (20 million bases, most of them no seeds: lists of 400 MB.)
    bases, offsets = zx.pack_records([r + b"N" * (10_000 - len(r)) for r in reads])
    want, want_total = oracle.query_records(ix, bases, offsets)
    per_want = [oracle.query_records(ix, few[0][i * 150:(i + 1) * 150],
                                     np.array([0, 150], dtype=np.uint64))[0] for i in range(50)]
    dev = torch.device("cuda", 0)
    d_b = torch.from_numpy(bases).to(dev)
    d_off = torch.from_numpy(offsets.view(np.int64)).to(dev)
    counts = torch.zeros(260, dtype=torch.int64, device=dev)
    total = torch.zeros(1, dtype=torch.int64, device=dev)

    def free():
        torch.cuda.synchronize(dev)
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info(dev)[0]

    def fill(leave):
        return torch.empty(free() - leave, dtype=torch.uint8, device=dev)

    with zx.Index(ix) as index:
        assert index.launch()["wide"]

        def query():
            counts.zero_()
            total.zero_()
            index.query_device(d_b.data_ptr(), len(bases), d_off.data_ptr(), len(reads),
                               counts.data_ptr(), total.data_ptr(), use_graph=False)
            torch.cuda.synchronize(dev)
            assert int(total) == want_total
            np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint64), want)

        index.query_records(*few)
        filler = fill(1400 << 20)
        query()  # in rounds
        query()
        del filler
        before = free()
        query()
        assert before - free() > 350 << 20
        before = free()
        query()
        assert free() == before
        filler = fill(100 << 20)
        per, totals = index.query_per_record(*few)  # 256 MiB of counters
        np.testing.assert_array_equal(per, np.array(per_want))
        query()  # in rounds again
        del filler
        assert free() > before
        query()


@pytest.mark.parametrize("opts", [dict(k=25, b=8), dict(mode="minimizers", k=25, m=21, b=16)],
                         ids=["kmers", "minimizers"])
def test_several_unsegmented_rounds(gpu, oracle, tmp_path, opts):
    """Three rounds of 2^18 tiles: two key lists in turn, extraction beside the
    probe, every order, windows and the wide probe, against the oracle and
    the batch in one round."""
    import zindex_b200 as zx

    colors = 260 if opts["b"] == 8 else 130
    fof = make_genomes(tmp_path / "g", colors, 3000, 31)
    ix = build_index(fof, tmp_path / "index", H=4, min_docs=1, **opts)
    pool = np.frombuffer(b"".join(dna(3000, 31 + c) for c in range(colors)), dtype=np.uint8)
    rng = np.random.default_rng(17)
    records, length = 600_000, 28
    at = rng.integers(0, len(pool) - length, records)
    bases = pool[at[:, None] + np.arange(length)].copy()
    bases[rng.random(records) < 0.3, 5] = ord("N")
    bases = bases.reshape(-1)
    offsets = np.arange(records + 1, dtype=np.uint64) * length
    with zx.Index(ix) as index:
        for recover in (True, False):
            want, want_total = oracle.query_records(ix, bases, offsets, recover=recover)
            for limit in (1 << 20, 0):
                index.set_round_bases(limit)
                for order in (1, 2, 0):
                    index.set_launch(wide=1, order=order, cut=1)
                    got, total = index.query_records(bases, offsets, recover=recover)
                    assert total == want_total
                    np.testing.assert_array_equal(got, want)


def test_split_rounds_of_a_launch_that_is_not_the_default(gpu, oracle, tmp_path):
    """Split minimizer queries of narrow rows in three rounds: with the default
    launch the batch takes the window probe."""
    import zindex_b200 as zx

    fof = make_genomes(tmp_path / "g", 20, 3000, 31)
    ix = build_index(fof, tmp_path / "index", mode="minimizers", k=25, m=21, H=4, b=8, min_docs=1)
    pool = np.frombuffer(b"".join(dna(3000, 31 + c) for c in range(20)), dtype=np.uint8)
    records, length = 600_000, 27
    at = np.random.default_rng(18).integers(0, len(pool) - length, records)
    bases = pool[at[:, None] + np.arange(length)].reshape(-1).copy()
    offsets = np.arange(records + 1, dtype=np.uint64) * length
    want, want_total = oracle.query_records(ix, bases, offsets)
    with zx.Index(ix) as index:
        for launch in (dict(split=1, min_blocks=3), dict(split=0)):
            index.set_launch(cut=1, **launch)
            assert index.launch() != {**index.default_launch(), "cut": 1}
            got, total = index.query_records(bases, offsets)
            assert total == want_total
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("opts", [dict(k=31, homopolymer=True), dict(k=45, homopolymer=True),
                                  dict(k=21, pattern="##_#_##_#_#_#_##_#_##"),
                                  dict(mode="minimizers", k=21, m=21),
                                  dict(mode="minimizers", k=31, m=15, pattern="#####_###_#####")],
                         ids=lambda o: "-".join(f"{k}{v}" for k, v in o.items()))
@pytest.mark.parametrize("colors", [240, 270])
def test_seed_options_of_dense_batches(gpu, oracle, tmp_path, opts, colors):
    """Homopolymer compression, spaced seeds and every m-mer past 1 MiB: in
    device memory, in chunks from pageable and joined from page-locked memory."""
    import torch

    import zindex_b200 as zx

    fof = make_genomes(tmp_path / "g", colors, 3000, 31)
    ix = build_index(fof, tmp_path / "index", **{**dict(H=4, b=8, min_docs=1), **opts})
    genomes = [dna(3000, 31 + c) for c in range(colors)]
    reads = sample_reads(genomes, np.random.default_rng(19), 14_500, 150, n_runs=0.05)
    reads += [genomes[3][:40] + b"A" * 2000 + genomes[4][:900]] * 20
    # (Every chunk is dense, also by bases that are no seeds.)
    bases, offsets = zx.pack_records([r + b"N" * 2500 for r in reads])
    want, want_total = oracle.query_records(ix, bases, offsets)
    dev = torch.device("cuda", 0)
    with zx.Index(ix) as index:
        assert index.launch()["wide"] == (colors > 250)
        for source in (bases, torch.from_numpy(bases).pin_memory().numpy()):
            got, total = index.query_records(source, offsets)
            assert total == want_total
            np.testing.assert_array_equal(got, want)
            assert _lists_held(index) >= 4 * len(bases)  # 16 a base of a chunk
        d_b = torch.from_numpy(bases).to(dev)
        d_off = torch.from_numpy(offsets.view(np.int64)).to(dev)
        counts = torch.zeros(colors, dtype=torch.int64, device=dev)
        n = torch.zeros(1, dtype=torch.int64, device=dev)
        index.query_device(d_b.data_ptr(), len(bases), d_off.data_ptr(), len(reads),
                           counts.data_ptr(), n.data_ptr(), use_graph=False)
        torch.cuda.synchronize(dev)
        assert int(n) == want_total
        np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint64), want)


def test_dense_batches_only_where_they_are_faster(gpu, tmp_path):
    """One-chunk rows that L2 holds: sorting for the window probe does not pay
    before tens of millions of bases. The default is at most a third slower
    than the fused kernel at 1.3e6 bases (it was twice) and faster at 8e7."""
    import subprocess

    import torch

    import zindex_b200 as zx

    subprocess.run([str(helpers.ZX_BUILD), "--synth", "uniform:10:100000:100000:5", "-o",
                    str(tmp_path / "index"), "-q", "-k", "31", "-H", "4", "-b", "8"], check=True)
    dev = torch.device("cuda", 0)
    acgt = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=dev)
    torch.manual_seed(20)
    with zx.Index(tmp_path / "index") as index:
        counts = torch.zeros(10, dtype=torch.int64, device=dev)
        total = torch.zeros(1, dtype=torch.int64, device=dev)
        stream = torch.cuda.current_stream(dev).cuda_stream

        def micros(bases, offsets):
            best = float("inf")
            for _ in range(20):
                first, last = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                first.record()
                index.query_device(bases.data_ptr(), bases.numel(), offsets.data_ptr(),
                                   offsets.numel() - 1, counts.data_ptr(), total.data_ptr(),
                                   stream, use_graph=False)
                last.record()
                last.synchronize()
                best = min(best, first.elapsed_time(last) * 1e3)
            return best

        ratio = {}
        for records in (8_700, 540_000):
            bases = acgt[torch.randint(0, 4, (records * 150,), device=dev)]
            offsets = torch.arange(records + 1, dtype=torch.int64, device=dev) * 150
            index.set_launch()
            default = micros(bases, offsets)
            index.set_launch(blocks=10_000)  # as many as fit: the default's grid
            fused = micros(bases, offsets)
            print(f"{records * 150} bases: default {default:.0f} us, fused {fused:.0f} us")
            ratio[records] = default / fused
        assert ratio[8_700] < 4 / 3 and ratio[540_000] < 1


@pytest.mark.parametrize("case", [dict(colors=64, H=4, b=8, k=31), dict(colors=9, H=3, b=16, k=25),
                                  dict(colors=30, H=2, b=4, k=45, groups="0,1;5,6"),
                                  dict(colors=5, H=4, b=32, k=31),
                                  dict(colors=100, H=16, b=8, k=31, max_size="256KiB"),
                                  dict(colors=100, H=8, b=8, mode="modimizers", k=31, d=4),
                                  dict(colors=100, H=4, b=8, mode="minimizers", k=31, m=21)],
                         ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_dense_batches_past_their_threshold(gpu, oracle, tmp_path, case):
    """Narrow rows of each width, hash count and seed mode in the window probe:
    batches of 36 million bases, most of them no seeds, whole and in chunks."""
    import torch

    import zindex_b200 as zx

    opts = dict(case)
    colors = opts.pop("colors")
    lengths = [2000 if c % 3 == 0 else (4000 if c % 3 == 1 else 9000) for c in range(colors)]
    genomes = [dna(n, 31 + c) for c, n in enumerate(lengths)]
    (tmp_path / "g").mkdir()
    lines = []
    for c, g in enumerate(genomes):
        p = tmp_path / "g" / f"g{c}.fa"
        helpers.write_fasta(p, [g])
        lines.append(f"g{c}\t{p}")
    (tmp_path / "fof.tsv").write_text("\n".join(lines) + "\n")
    ix = build_index(tmp_path / "fof.tsv", tmp_path / "index", min_docs=1, **opts)
    reads = sample_reads(genomes, np.random.default_rng(21), 8000, 151, n_runs=0.05)
    bases, offsets = zx.pack_records([r + b"N" * 4400 for r in reads])
    locked = torch.from_numpy(bases).pin_memory().numpy()
    with zx.Index(ix) as index:
        assert not index.launch()["wide"]
        for recover in (True, False):
            want, want_total = oracle.query_records(ix, bases, offsets, recover=recover)
            index.set_launch(cut=1)
            got, total = index.query_records(bases, offsets, recover=recover)
            assert total == want_total
            np.testing.assert_array_equal(got, want)
            assert _lists_held(index) >= 16 * len(bases)
            index.set_launch(cut=3)  # joined
            got, total = index.query_records(locked, offsets, recover=recover)
            assert total == want_total
            np.testing.assert_array_equal(got, want)
            assert _lists_held(index) >= 16 * len(bases)


@pytest.mark.parametrize("colors", [12, 270], ids=["narrow", "wide"])
def test_first_graph_of_a_homopolymer_index(gpu, oracle, tmp_path, colors):
    """The compressed batch's buffers are there before the graph is captured."""
    import torch

    import zindex_b200 as zx

    fof = make_genomes(tmp_path / "g", colors, 3000, 31)
    ix = build_index(fof, tmp_path / "index", k=31, H=4, b=8, min_docs=1, homopolymer=True)
    genomes = [dna(3000, 31 + c) for c in range(colors)]
    dev = torch.device("cuda", 0)
    with zx.Index(ix) as index:
        for n in (50, 3000):
            bases, offsets = zx.pack_records(sample_reads(genomes, np.random.default_rng(n), n, 150))
            want, want_total = oracle.query_records(ix, bases, offsets)
            d_b = torch.from_numpy(bases).to(dev)
            d_off = torch.from_numpy(offsets.view(np.int64)).to(dev)
            counts = torch.zeros(colors, dtype=torch.int64, device=dev)
            total = torch.zeros(1, dtype=torch.int64, device=dev)
            for replay in (1, 2):
                index.query_device(d_b.data_ptr(), len(bases), d_off.data_ptr(), n,
                                   counts.data_ptr(), total.data_ptr(), use_graph=True)
                torch.cuda.synchronize(dev)
                assert int(total) == replay * want_total
                np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint64), replay * want)
