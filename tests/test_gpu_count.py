"""GPU parity of parsing (K1), counting (K2), histo/dump (K3/K4) and
catalogue loading against the CPU oracle, through the C ABI.  Integer work:
bit-exact."""
import numpy as np
import pytest

from trinityrnaseq_gb300 import KmerTable, ReadSet, native, synth
from tests.helpers import dict_to_arrays, kmer_counter_to_canonical, read_gz

pytestmark = pytest.mark.gpu


def gpu_count(ctx, text, k=25, canonical=True, capacity=0):
    t = KmerTable(ctx, k, canonical, capacity)
    t.count_text(text)
    return t


def assert_pairs(got, want):
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("name", ["edge", "bulk"])
def test_parse_matches_fasta_reader(ctx, golden, name):
    text = (golden / f"{name}.fa").read_bytes()
    rs = ReadSet(ctx, text)
    want = [l.split(b"\t") for l in (golden / f"{name}.fasta_reader.tsv").read_bytes().split(b"\n") if l]
    assert rs.n_reads == len(want)
    assert rs.accessions() == [w[0] for w in want]
    assert rs.sequences() == [w[1].upper() for w in want]


def test_parse_fastq(ctx, golden):
    rs = ReadSet(ctx, (golden / "edge.fq").read_bytes())
    assert rs.format == native.TK_FMT_FASTQ
    want = (golden / "edge.fastQ_to_fastA.fa").read_bytes().split(b"\n")
    assert rs.sequences() == [l for l in want[1::2] if l or True][:rs.n_reads]


@pytest.mark.parametrize("name", ["edge", "bulk"])
def test_count_matches_reference_perl_counter(ctx, golden, name):
    text = (golden / f"{name}.fa").read_bytes()
    want = dict_to_arrays(kmer_counter_to_canonical(read_gz(golden / f"{name}.kmer_counter.txt.gz")))
    assert_pairs(gpu_count(ctx, text).dump(1), want)


@pytest.mark.parametrize("k", [1, 5, 17, 24, 25, 31])
@pytest.mark.parametrize("canonical", [True, False])
def test_count_parity_k(ctx, oracle, golden, k, canonical):
    text = (golden / "edge.fa").read_bytes() + (golden / "bulk.fa").read_bytes()
    assert_pairs(gpu_count(ctx, text, k, canonical).dump(1), oracle.count(text, k, canonical))


def test_count_parity_transcriptome_1M(ctx, oracle):
    """Single-end 76-nt transcriptome workload at full size (1M reads)."""
    text = synth.transcriptome_reads(seed=1, n_reads=1_000_000).tobytes()
    t = gpu_count(ctx, text)
    want = oracle.count(text, 25, True)
    got = t.dump(1)
    assert_pairs(got, want)
    d, total, cap = t.info()
    assert d == len(want[0]) and total == int(want[1].sum()) == 52_000_000
    np.testing.assert_array_equal(t.histo(1, 10000), oracle.histo(want[1], 1, 10000))
    for L in (1, 2):
        assert t.dump_fasta(L) == oracle.dump(want[0], want[1], 25, L)


def test_count_fastq_pairs_with_n(ctx, oracle):
    left, right = synth.gene_pairs(seed=9, n_genes=300, n_pairs=20000, n_rate=0.01)
    text = left.tobytes() + right.tobytes()
    assert_pairs(gpu_count(ctx, text).dump(1), oracle.count(text, 25, True))


def test_batches_add_up(ctx, oracle):
    a = synth.transcriptome_reads(seed=3, n_reads=30000).tobytes()
    b = synth.transcriptome_reads(seed=4, n_reads=50000).tobytes()
    t = KmerTable(ctx, 25, True)
    t.count_text(a)
    t.count_text(b)
    assert_pairs(t.dump(1), oracle.count(a + b, 25, True))


def test_add_many_equals_concatenation(ctx, oracle):
    a = synth.transcriptome_reads(seed=13, n_reads=40000).tobytes()
    b, c = synth.gene_pairs(seed=14, n_genes=400, n_pairs=30000)
    sets = [ReadSet(ctx, x) for x in (a, b.tobytes(), b"", c.tobytes())]
    t = KmerTable(ctx, 25, True)
    t.add_many(sets)
    assert_pairs(t.dump(1), oracle.count(a + b.tobytes() + c.tobytes(), 25, True))
    # a second multi-set pass into the now non-empty table
    t.add_many(sets[:2])
    assert_pairs(t.dump(1), oracle.count(a + b.tobytes() + c.tobytes() + a + b.tobytes(), 25, True))


def test_large_partitioned_table(ctx, oracle):
    """Enough distinct k-mers for a multi-partition table (> 2M slots)."""
    text = synth.transcriptome_reads(seed=15, n_transcripts=4000, n_reads=600_000, err=0.02).tobytes()
    t = gpu_count(ctx, text)
    d, total, cap = t.info()
    assert cap > (1 << 21)
    assert_pairs(t.dump(1), oracle.count(text, 25, True))


def test_overflow_and_growth_are_exact(ctx, oracle):
    """Eight reprobes at up to 0.6 load: many inserts overflow, the table
    doubles and the overflow list is re-inserted; the counts stay exact."""
    text = synth.transcriptome_reads(seed=5, n_reads=3000).tobytes()
    ctx.set_reprobes(8)
    try:
        t = gpu_count(ctx, text, capacity=1024)
        got = t.dump(1)
    finally:
        ctx.set_reprobes(4096)
    assert_pairs(got, oracle.count(text, 25, True))


def test_empty_and_degenerate_inputs(ctx):
    for text in (b"", b"\n\n  \n", b">a\n\n>b\nNNNNNNNNNNNNNNNNNNNNNNNNNNNNNN\n", b">only_header"):
        t = gpu_count(ctx, text)
        k, c = t.dump(1)
        assert len(k) == 0
        assert t.dump_fasta(1) == b""
        assert int(t.histo().sum()) == 0


def test_malformed_fastq_is_an_error(ctx):
    with pytest.raises(native.TrinkmerError) as ei:
        ReadSet(ctx, b"@r1\nACGT\n+\nIIII\n@r2\nACGT\nIIII\n")
    assert ei.value.status == native.TK_E_PARSE
    with pytest.raises(native.TrinkmerError):
        ReadSet(ctx, b"@r1\nACGT\nXX\nIIII\n")


def test_load_dump_roundtrip(ctx, oracle, golden):
    text = (golden / "bulk.fa").read_bytes() + synth.transcriptome_reads(seed=8, n_reads=20000).tobytes()
    keys, counts = oracle.count(text, 25, True)
    d2 = oracle.dump(keys, counts, 25, 2)
    t = KmerTable(ctx, 25, True)
    t.load_dump_fasta(d2)
    assert_pairs(t.dump(1), oracle.load_dump(d2, 25, True))
    # a non-canonical dump loaded canonically merges strands
    kf, cf = oracle.count(text, 25, False)
    df = oracle.dump(kf, cf, 25, 1)
    t2 = KmerTable(ctx, 25, True)
    t2.load_dump_fasta(df)
    assert_pairs(t2.dump(1), oracle.load_dump(df, 25, True))


def test_load_pairs(ctx, oracle, golden):
    text = (golden / "bulk.fa").read_bytes()
    keys, counts = oracle.count(text, 25, True)
    t = KmerTable(ctx, 25, True)
    t.load_pairs(keys, counts)
    t.load_pairs(keys, counts)
    assert_pairs(t.dump(1), (keys, counts * 2))


def test_bad_dump_is_an_error(ctx):
    t = KmerTable(ctx, 25, True)
    with pytest.raises(native.TrinkmerError) as ei:
        t.load_dump_fasta(b">3\nACGTACGTACGTACGTACGTACGTA\n>x\nACGTACGTACGTACGTACGTACGTA\n")
    assert ei.value.status == native.TK_E_PARSE


def test_range_build_fallback_when_deferred_list_overruns(native_built, oracle):
    """A fresh table is built range by range in shared memory; keys whose probe
    leaves their range are deferred.  With the deferred list capped at one
    entry the build overruns it, the table is emptied and counted with global
    atomics instead: the result must not change."""
    import os
    import subprocess
    import sys
    code = (
        "import numpy as np, sys\n"
        "from trinityrnaseq_gb300 import Context, KmerTable, synth\n"
        "left, right = synth.gene_pairs(seed=41, n_genes=2000, n_pairs=300000, fastq=False)\n"
        "t = KmerTable(Context(0), 25, True)\n"
        "t.count_text(left.tobytes() + right.tobytes())\n"
        "sys.stdout.buffer.write(t.dump_fasta(1))\n")
    env = dict(os.environ, TRINKMER_DEFER_CAP="1")
    capped = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, timeout=600)
    assert capped.returncode == 0, capped.stderr[-2000:]
    left, right = synth.gene_pairs(seed=41, n_genes=2000, n_pairs=300000, fastq=False)
    keys, counts = oracle.count(left.tobytes() + right.tobytes(), 25, True)
    assert capped.stdout == oracle.dump(keys, counts, 25, 1)


def test_block_cache_trim_and_zero_cap(native_built, ctx, oracle):
    """Large blocks are cached per context after they are freed; tk_ctx_trim
    gives them back, and a zero cap (TRINKMER_BLOCK_CACHE_GB=0) frees them at
    once.  Counting is unchanged either way."""
    import os
    import subprocess
    import sys
    left, right = synth.gene_pairs(seed=43, n_genes=3000, n_pairs=1_500_000, fastq=False)
    t = KmerTable(ctx, 25, True)
    t.count_text(left.tobytes() + right.tobytes())
    assert t.info(distinct=False)[2] * 16 >= 256 << 20   # the table is a cached-size block
    t.free()
    free_before, _ = ctx.mem_info()
    ctx.trim()
    free_after, _ = ctx.mem_info()
    assert free_after >= free_before
    code = ("import sys\n"
            "from trinityrnaseq_gb300 import Context, KmerTable, synth\n"
            "left, right = synth.gene_pairs(seed=43, n_genes=3000, n_pairs=200000, fastq=False)\n"
            "t = KmerTable(Context(0), 25, True)\n"
            "t.count_text(left.tobytes() + right.tobytes())\n"
            "sys.stdout.buffer.write(t.dump_fasta(2))\n")
    p = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, TRINKMER_BLOCK_CACHE_GB="0"),
                       capture_output=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    left, right = synth.gene_pairs(seed=43, n_genes=3000, n_pairs=200000, fastq=False)
    keys, counts = oracle.count(left.tobytes() + right.tobytes(), 25, True)
    assert p.stdout == oracle.dump(keys, counts, 25, 2)


def pieces_of(texts, n):
    from trinityrnaseq_gb300 import kmer
    out = []
    for a in texts:
        cuts = kmer.split_records(a, n)
        out += [a[int(cuts[i]):int(cuts[i + 1])] for i in range(n)]
    return out


def test_count_texts_equals_parse_then_add(ctx, oracle):
    """tk_table_count_texts: each host text's first counting pass runs as soon
    as it is parsed (per-text key buffers, the partitions read as one segment
    of each); the counts and the read sets equal parse_many + add_many."""
    left, right = synth.gene_pairs(seed=61, n_genes=1500, n_pairs=200000, fastq=True, n_rate=0.005)
    pieces = pieces_of((left, right), 3)
    pieces.insert(2, np.zeros(0, dtype=np.uint8))   # an empty text among them
    whole = left.tobytes() + right.tobytes()
    t = KmerTable(ctx, 25, True)
    sets = t.count_texts(pieces)
    assert_pairs(t.dump(1), oracle.count(whole, 25, True))
    ref = ReadSet.parse_many(ctx, pieces)
    assert [r.n_reads for r in sets] == [r.n_reads for r in ref]
    for a, b in zip(sets, ref):
        assert a.accessions() == b.accessions() and a.sequences() == b.sequences()
    # counted again into the now filled table (the atomic path over several key buffers)
    t.count_texts(pieces[:3])
    assert_pairs(t.dump(1), oracle.count(whole + b"".join(p.tobytes() for p in pieces[:3]), 25, True))


def test_count_texts_beyond_one_pass_of_sets(ctx, oracle):
    """More texts than one counting pass takes (64): parsed, then counted in groups."""
    text = synth.transcriptome_reads(seed=62, n_reads=70000).tobytes()
    arr = np.frombuffer(text, dtype=np.uint8)
    pieces = pieces_of((arr,), 70)
    t = KmerTable(ctx, 25, True)
    sets = t.count_texts(pieces)
    assert len(sets) == 70 and sum(r.n_reads for r in sets) == 70000
    assert_pairs(t.dump(1), oracle.count(text, 25, True))


def test_multi_set_partitioned_table_and_deferred_fallback(native_built, oracle):
    """Several read sets into a multi-partition table, by ranges and, with the
    deferred list capped at one entry, by the atomic fallback: both exact."""
    import os
    import subprocess
    import sys
    code = (
        "import sys\n"
        "from trinityrnaseq_gb300 import Context, KmerTable, ReadSet, synth\n"
        "ctx = Context(0)\n"
        "text = synth.transcriptome_reads(seed=63, n_transcripts=4000, n_reads=600_000, err=0.02).tobytes()\n"
        "q = len(text) // 3\n"
        "cut = [0, text.index(b'\\n>', q) + 1, text.index(b'\\n>', 2 * q) + 1, len(text)]\n"
        "sets = [ReadSet(ctx, text[cut[i]:cut[i + 1]]) for i in range(3)]\n"
        "t = KmerTable(ctx, 25, True)\n"
        "t.add_many(sets)\n"
        "assert t.info()[2] > (1 << 21)\n"
        "sys.stdout.buffer.write(t.dump_fasta(1))\n")
    text = synth.transcriptome_reads(seed=63, n_transcripts=4000, n_reads=600_000, err=0.02).tobytes()
    keys, counts = oracle.count(text, 25, True)
    want = oracle.dump(keys, counts, 25, 1)
    for cap in (None, "1"):
        env = dict(os.environ)
        if cap:
            env["TRINKMER_DEFER_CAP"] = cap
        run = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, timeout=600)
        assert run.returncode == 0, run.stderr[-2000:]
        assert run.stdout == want, cap


def test_count_texts_error_leaves_the_context_usable(ctx, oracle):
    """A malformed text among the pieces fails the call (no read set is
    returned, the key buffers of the texts before it are freed); the context
    and a new table still count exactly afterwards."""
    good = synth.transcriptome_reads(seed=64, n_reads=20000).tobytes()
    bad = b"@r1\nACGT\n+\nIIII\n@r2\nACGT\n"
    t = KmerTable(ctx, 25, True)
    with pytest.raises(native.TrinkmerError):
        t.count_texts([np.frombuffer(good, dtype=np.uint8), np.frombuffer(bad, dtype=np.uint8)])
    t2 = KmerTable(ctx, 25, True)
    sets = t2.count_texts([np.frombuffer(good, dtype=np.uint8)])
    assert sets[0].n_reads == 20000
    assert_pairs(t2.dump(1), oracle.count(good, 25, True))


@pytest.mark.parametrize("n", [3, 1 << 21, (1 << 21) + 1])
@pytest.mark.parametrize("dirty", [False, True])
def test_sizes_read_back_or_bounded(ctx, oracle, n, dirty):
    """Small FASTA inputs and small sets get buffers of the largest size they
    can need, larger ones (above 2^22 lines, 2^24 positions) of the size read
    back: n records of seven bases lie below, at and above both lines.  A space
    in one sequence line has the codes packed a second time."""
    rng = np.random.default_rng(71)
    rec = np.empty((n, 11), dtype=np.uint8)
    rec[:, :] = np.frombuffer(b">r\n.......\n", dtype=np.uint8)
    rec[:, 3:10] = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, (n, 7), dtype=np.uint8)]
    if dirty:
        rec[n // 2, 6] = ord(" ")
    text = rec.tobytes()
    rs = ReadSet(ctx, text)
    assert rs.n_reads == n
    t = KmerTable(ctx, 5, True)
    t.add(rs)
    clean = text.replace(b" ", b"")
    assert_pairs(t.dump(1), oracle.count(clean, 5, True))
    if n < 10:
        assert rs.sequences() == [clean.split(b"\n")[2 * i + 1] for i in range(n)]


def line_mix(seed, n, lens, fastq, blank=0.0, lower=True):
    """Records of the given sequence-line lengths (FASTA: up to three lines a record, blank lines among them)."""
    rng = np.random.default_rng(seed)
    out, seqs = [], []
    letters = np.frombuffer(b"ACGTACGTACGTNacgtnR" if lower else b"ACGTACGTACGTN", dtype=np.uint8)
    for i in range(n):
        rows = [letters[rng.integers(0, len(letters), int(L))].tobytes()
                for L in rng.choice(lens, 1 if fastq else int(rng.integers(0, 4)))]
        if fastq and i == n - 1:
            rows = [b"ACGTA"]   # (an empty last quality line would be trimmed with the text's trailing whitespace)
        seq = b"".join(rows)
        seqs.append(seq.upper())
        if fastq:
            out.append(b"@r%d x\n%s\n+\n%s\n" % (i, seq, b"I" * len(seq)))
        else:
            body = b"".join(r + b"\n" + b"\n" * int(blank * rng.integers(0, 40)) for r in rows)
            out.append(b">r%d\n%s" % (i, body))
    return b"".join(out), seqs


@pytest.mark.parametrize("shift", [0, 1, 7])
@pytest.mark.parametrize("fastq", [False, True])
@pytest.mark.parametrize("case", ["reads", "short", "blank", "long", "clean"])
def test_copied_lines_and_codes(ctx, oracle, case, fastq, shift):
    """Sequence lines into the read array and its codes, in tiles of 8192
    positions and pieces of 32: lines around the size of a piece, more lines in
    a tile than are held at a time (512), blank lines among them, lines over
    several tiles, lower-case and N, texts at odd addresses on the GPU."""
    import torch
    n, lens, blank = {"reads": (2500, [31, 32, 33, 64, 76, 100], 0), "short": (9000, [0, 1, 2, 5], 0),
                      "blank": (1500, [0, 3, 40], 1.0), "long": (9, [8191, 8192, 8193, 20000, 70000], 0),
                      "clean": (2500, [76], 0)}[case]
    text, seqs = line_mix(81, n, lens, fastq, blank, case != "clean")
    dev = torch.zeros(len(text) + shift, dtype=torch.uint8, device="cuda:0")
    dev[shift:] = torch.frombuffer(bytearray(text), dtype=torch.uint8).to("cuda:0")
    torch.cuda.synchronize()
    rs = ReadSet(ctx, dev.data_ptr() + shift, len(text), device=True)
    assert rs.n_reads == n
    assert rs.sequences() == seqs
    t = KmerTable(ctx, 5, True)
    t.add(rs)
    assert_pairs(t.dump(1), oracle.count(text, 5, True))


@pytest.mark.parametrize("shift", [0, 1, 3, 7])
@pytest.mark.parametrize("fastq", [False, True])
def test_accessions_of_every_length(ctx, fastq, shift):
    """First header tokens of 0 to 40 bytes, ended by each kind of whitespace, by
    the line's end and by the text's, at every alignment of the text's words."""
    import torch
    seps = [b"", b" x", b"\tx", b"\r", b"\x0bx", b"\x0cx", b" ", b"\x0e y", b"\x80\x89\xa0 z"]
    names, out = [], []
    for i in range(41 * len(seps)):
        name = (b"abcdefghijklmnopqrstuvwxyz/123456789_.:-|"[:i % 41])
        sep = seps[i // 41]
        cut = name + sep.split(b" ")[0] if sep[:1] in (b"\x0e", b"\x80") else name
        names.append(cut)
        out.append((b"@%s%s\nACGT\n+\nIIII\n" if fastq else b">%s%s\nACGT\n") % (name, sep))
    if not fastq:
        out.append(b">last_one")
        names.append(b"last_one")
    text = b"".join(out)
    dev = torch.zeros(len(text) + shift, dtype=torch.uint8, device="cuda:0")
    dev[shift:] = torch.frombuffer(bytearray(text), dtype=torch.uint8).to("cuda:0")
    torch.cuda.synchronize()
    rs = ReadSet(ctx, dev.data_ptr() + shift, len(text), device=True)
    noff, nlen = np.zeros(rs.n_reads, np.uint64), np.zeros(rs.n_reads, np.uint32)
    ctx.check(rs.lib.tk_reads_names(rs.h, noff.ctypes.data, nlen.ctypes.data), "names")
    assert [text[int(o):int(o) + int(n)] for o, n in zip(noff, nlen)] == names
    assert rs.max_len == 4


@pytest.mark.parametrize("k", [1, 2, 15, 16, 25, 31])
@pytest.mark.parametrize("canonical", [True, False])
def test_loaded_kmers_at_every_offset_of_the_codes(ctx, k, canonical):
    """A catalogue's k-mers are cut from the codes at records' starts, k + 1
    positions apart; a letter that is no base is refused wherever it stands."""
    rng = np.random.default_rng(k)
    n = min(4 ** k, 300)
    mers = sorted({"".join(rng.choice(list("ACGT"), k)) for _ in range(n)})
    lines = [">%d\n%s\n" % (i + 1, m if i % 3 else m.lower()) for i, m in enumerate(mers)]
    want = {}
    for i, m in enumerate(mers):
        rc = m[::-1].translate(str.maketrans("ACGT", "TGCA"))
        key = min(m, rc) if canonical else m
        want[key] = want.get(key, 0) + i + 1
    t = KmerTable(ctx, k, canonical)
    t.load_dump_fasta("".join(lines).encode())
    got = t.dump(1)
    code = lambda m: sum("ACGT".index(c) << (2 * (k - 1 - i)) for i, c in enumerate(m))
    assert dict(zip(got[0].tolist(), got[1].tolist())) == {code(m): c for m, c in want.items()}
    for at in {0, k // 2, k - 1}:
        m = mers[-1][:at] + "N" + mers[-1][at + 1:]
        with pytest.raises(native.TrinkmerError):
            KmerTable(ctx, k, canonical).load_dump_fasta(("".join(lines) + ">1\n%s\n>2\n%s\n" % (m, mers[0])).encode())


def fasta_of(seqs, gap):
    """Records of seqs with gap(i) blank lines after record i."""
    return b"".join(b">r%d x\n%s\n%s" % (i, s, b"\n" * gap(i)) for i, s in enumerate(seqs))


@pytest.mark.parametrize("gap", [4090, 4094, 4095, 4096, 4097, 9000, 40_000])
@pytest.mark.parametrize("at", [0, 1, 70, 119])
def test_parse_many_blank_lines_at_one_place(ctx, gap, at):
    """Lines without positions: a tile of the read array may hold any number of them."""
    rng = np.random.default_rng(gap + at)
    seqs = [bytes(rng.choice(np.frombuffer(b"ACGTacgtN", np.uint8), int(n))) for n in rng.integers(0, 400, 120)]
    rs = ReadSet(ctx, fasta_of(seqs, lambda i: gap if i == at else 0))
    assert rs.sequences() == [s.upper() for s in seqs]
    assert rs.accessions() == [b"r%d" % i for i in range(120)]


@pytest.mark.parametrize("n", [2047, 2048, 2049, 12_289])
@pytest.mark.parametrize("lens", [(0,), (1,), (0, 1, 0, 40), (3, 0, 0, 0, 900), (2, 0, 0, 0, 0, 0, 0, 1)])
@pytest.mark.parametrize("fastq", [False, True])
def test_parse_short_and_empty_records(ctx, n, lens, fastq):
    rng = np.random.default_rng(n)
    letters = rng.choice(np.frombuffer(b"ACGTN", np.uint8), 20_000).tobytes()
    seqs = [letters[i % 7000:i % 7000 + lens[i % len(lens)]] for i in range(n)] + [b"ACGTACGTAC"]
    if fastq:
        text = b"".join(b"@r%d/1\n%s\n+\n%s\n" % (i, s, b"I" * len(s)) for i, s in enumerate(seqs))
    else:
        text = b"".join(b">r%d/1\n%s\n" % (i, s) for i, s in enumerate(seqs))
    rs = ReadSet(ctx, text)
    assert rs.sequences() == seqs
    k = KmerTable(ctx, 5, False)
    k.add(rs)   # the 2-bit codes made beside the letters
    want = {}
    for s in seqs:
        for j in range(len(s) - 4):
            w = s[j:j + 5]
            if b"N" not in w:
                want[w.decode()] = want.get(w.decode(), 0) + 1
    assert_pairs(k.dump(1), dict_to_arrays(want))


def test_blank_lines_do_not_hold_up_the_parser(ctx):
    """3M blank lines in one place cost about what their bytes cost (one block
    that walked them took 80 times the parse without them)."""
    import time
    rng = np.random.default_rng(3)
    seqs = [s.tobytes() for s in rng.choice(np.frombuffer(b"ACGT", np.uint8), (100_000, 100))]

    def best(text):
        out = []
        for _ in range(6):
            t0 = time.perf_counter()
            ReadSet(ctx, text).free()
            out.append(time.perf_counter() - t0)
        return min(out)

    plain = best(fasta_of(seqs, lambda i: 0))
    blank = best(fasta_of(seqs, lambda i: 3_000_000 if i == 50_000 else 0))
    assert blank < 6 * plain, (blank, plain)


def test_count_a_partition_of_more_than_2_32_keys(ctx):
    """Deep reads over few k-mers: one table slice, 4.6G windows in one call.
    Counted by ranges like any other call (the same launches per read set and
    three more), every count a multiple of the one set's."""
    import torch
    if torch.cuda.mem_get_info()[0] < 150 << 30:
        pytest.skip("needs 150 GB of GPU memory")
    g = torch.Generator().manual_seed(4)
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8)
    genome = letters[torch.randint(0, 4, (60_000,), generator=g)].cuda()
    at = torch.randint(0, 60_000 - 100, (3_000_000,), generator=g).cuda()
    reads = genome[at[:, None] + torch.arange(100, device="cuda")]
    n = at.numel()
    text = torch.cat([torch.tensor(list(b">r\n"), dtype=torch.uint8, device="cuda").expand(n, 3), reads,
                      torch.full((n, 1), 10, dtype=torch.uint8, device="cuda")], 1).reshape(-1)
    torch.cuda.synchronize()
    rs = ReadSet(ctx, text.data_ptr(), text.numel(), device=True)
    launches, pairs = [], []
    for times in (2, 3, 20):
        t = KmerTable(ctx, 25, True)
        before = ctx.kernel_launches
        t.add_many([rs] * times)
        launches.append(ctx.kernel_launches - before)
        keys, counts = t.dump(1)
        pairs.append((keys, counts // times))
        assert not (counts % times).any()
        assert t.info()[1] == times * n * 76
        t.free()
    assert 20 * n * 76 > 1 << 32 and launches[2] - launches[0] == 18 * (launches[1] - launches[0])
    for p in pairs[1:]:
        assert_pairs(p, pairs[0])
    rs.free()
    del text, reads
    torch.cuda.empty_cache()
    ctx.trim()


def test_count_runs_of_equal_keys(ctx):
    """One-window reads, every k-mer many times in a row, in table slices short
    enough that some runs lie at the end of a range: whole warps add one key."""
    rng = np.random.default_rng(12)
    kmers = np.unique(rng.choice(np.frombuffer(b"ACGT", np.uint8), (20_000, 25)), axis=0)
    times = rng.choice([1, 31, 127, 128, 129, 200, 700], kmers.shape[0])
    at = np.repeat(np.arange(kmers.shape[0]), times)
    rows = np.concatenate([np.full((at.size, 1), ord(">"), np.uint8), np.full((at.size, 1), 10, np.uint8), kmers[at],
                           np.full((at.size, 1), 10, np.uint8)], axis=1)
    t = gpu_count(ctx, rows.tobytes(), canonical=False)
    code = np.zeros(kmers.shape[0], np.uint64)
    for j in range(25):
        code = code * np.uint64(4) + np.searchsorted(np.frombuffer(b"ACGT", np.uint8), kmers[:, j]).astype(np.uint64)
    order = np.argsort(code)
    assert_pairs(t.dump(1), (code[order], times[order].astype(np.uint32)))
    assert t.info()[:2] == (kmers.shape[0], int(times.sum()))


@pytest.mark.parametrize("unit", [b"A", b"AC", b"ACGT", b"ACGTTGCAAC"])
def test_count_repeats_beside_ordinary_reads(ctx, oracle, unit):
    rng = np.random.default_rng(len(unit))
    genome = rng.choice(np.frombuffer(b"ACGT", np.uint8), 30_000)
    recs = [b">a\n" + (unit * 100)[i % len(unit):][:100] + b"\n" for i in range(20_000)]
    for p in rng.integers(0, 29_900, 20_000):
        recs.append(b">b\n" + genome[p:p + 100].tobytes() + b"\n")
    for mixed in (False, True):
        text = b"".join([recs[i] for i in rng.permutation(len(recs))] if mixed else recs)
        assert_pairs(gpu_count(ctx, text).dump(1), oracle.count(text, 25, True))
