"""The bounded waits of the single-pass scans and radix passes: a launch whose
first tile is left out gives up after its poll limit, the call returns an
error, and the context goes on working.  The launches of a pipeline are taken
one after another (the context counts those of several tiles)."""
import numpy as np
import pytest

from trinityrnaseq_gb300 import (Context, DeBruijnGraphs, KmerTable, Normalization, ReadSet, coverage_stats,
                                 native, synth)
from trinityrnaseq_gb300.kmer import count_bins

pytestmark = pytest.mark.gpu


def reads(n, length, seed, fastq=False, mate=1):
    rng = np.random.default_rng(seed)
    genome = rng.choice(np.frombuffer(b"ACGT", np.uint8), 60_000)
    out = []
    for i, p in enumerate(rng.integers(0, genome.size - length, n)):
        s = genome[p:p + length].tobytes()
        out.append(b"@q%07d/%d\n%s\n+\n%s\n" % (i, mate, s, b"I" * length) if fastq else b">q%07d/%d\n%s\n" % (i, mate, s))
    return b"".join(out)


def count(c):
    t = KmerTable(c, 25, True)
    rs = ReadSet(c, reads(6_000, 80, 1))
    t.add(rs)
    return [t.dump_fasta(1), *t.dump(1), *coverage_stats(t, rs)]


def large_sort(c):
    """Pairs enough for the larger tiles (1024 pairs per SM and more)."""
    keys = np.random.default_rng(2).permutation(np.arange(400_000, dtype=np.uint64) * np.uint64(2_654_435_761))
    t = KmerTable(c, 25, False)
    t.load_pairs(keys, np.ones(keys.size, np.uint32))
    return list(t.dump(1))


def prep(c):
    return [ReadSet(c, reads(9_000, 40, 3, True)).to_fasta(1)]


def normalize(c):
    """Names that fit one packed key, and (with a number repeated) the order by the whole line."""
    out = []
    for n, twice in ((6_000, False), (5_000, True)):
        sides = [ReadSet(c, reads(n, 30, 4, True, m) + (reads(3, 30, 4, True, m) if twice else b"")) for m in (1, 2)]
        size = sides[0].n_reads
        stats = (np.full(size, 9, np.uint32), np.full(size, 9.5, np.float32), np.full(size, 0.5, np.float32))
        nm = Normalization(c, sides[0], stats, sides[1], stats, 50, 1, 10_000)
        out += [nm.accs(), nm.table(), nm.extract(sides[0])]
    return out


def de_bruijn(c):
    rng = np.random.default_rng(5)
    recs = [b">s_%d\n%s\n" % (i, rng.choice(np.frombuffer(b"ACGT", np.uint8), 60).tobytes()) for i in range(9_000)]
    return [DeBruijnGraphs(c, b"".join(recs), 24).text()]


def bins(c):
    parts = [reads(400, 60, 10 + i) for i in range(40)]
    off = np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.uint64)
    text, at, kmers = count_bins(c, b"".join(parts), off, 25, True, 1)
    return [bytes(text), np.asarray(at), kmers]


def same(a, b):
    return len(a) == len(b) and all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("work,least", [(count, 8), (large_sort, 5), (prep, 1), (normalize, 8), (de_bruijn, 3), (bins, 6)])
def test_every_wait_that_runs_out_is_reported(ctx, monkeypatch, work, least):
    want = work(ctx)
    other = KmerTable(ctx, 25, True)   # memory of another context beside the one that fails
    other.count_text(synth.transcriptome_reads(seed=3, n_reads=3000))
    before = other.dump_fasta(1)
    failed = 0
    for which in range(1, 200):
        monkeypatch.setenv("TRINKMER_WAIT_TEST", f"{which} 2000")
        with Context(ctx.device) as c:
            monkeypatch.delenv("TRINKMER_WAIT_TEST")
            try:
                got = work(c)
            except native.TrinkmerError as err:
                failed += 1
                assert err.status == native.TK_E_CUDA and "ran out" in str(err), str(err)
                got = work(c)   # the next call on the same context
                assert same(got, want)
            else:
                assert same(got, want)   # fewer launches than `which`
                break
    assert least <= failed < 198, failed
    assert other.dump_fasta(1) == before
