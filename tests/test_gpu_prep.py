"""FASTQ -> FASTA read prep on the GPU (tk_reads_to_fasta, bin/seqtk-trinity)
against util/support_scripts/fastQ_to_fastA.pl's own output (golden fixtures)
and the oracle's restatement of it, byte for byte."""
import random
import subprocess

import pytest

from trinityrnaseq_gb300 import ReadSet, native, synth
from trinityrnaseq_gb300.build import BIN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fixture,append,rev", [
    ("prep.fa", -1, False), ("prep.a1.fa", 1, False), ("prep.rev.fa", -1, True), ("prep.a2rev.fa", 2, True)])
def test_prep_matches_reference_script(ctx, golden, fixture, append, rev):
    rs = ReadSet(ctx, (golden / "prep.fq").read_bytes())
    assert rs.to_fasta(append, revcomp=rev) == (golden / fixture).read_bytes()


def test_prep_edge_fastq(ctx, golden):
    rs = ReadSet(ctx, (golden / "edge.fq").read_bytes())
    assert rs.to_fasta() == (golden / "edge.fastQ_to_fastA.fa").read_bytes()


def test_prep_dirty_records(ctx, golden):
    rs = ReadSet(ctx, (golden / "prep_dirty.fq").read_bytes())
    assert rs.to_fasta(ignore_dirty=True) == (golden / "prep_dirty.ignore.fa").read_bytes()
    with pytest.raises(native.TrinkmerError) as e:
        rs.to_fasta()
    assert e.value.status == native.TK_E_PARSE


@pytest.mark.parametrize("append,rev,if_missing", [(1, False, True), (2, True, True), (-1, True, False), (7, False, False)])
def test_prep_parity_200k_pairs(ctx, oracle, append, rev, if_missing):
    left, _ = synth.gene_pairs(seed=51, n_genes=500, n_pairs=200000, fastq=True)
    text = left.tobytes()
    flags = (oracle.FA_REV if rev else 0) | (oracle.FA_IF_MISSING if if_missing else 0)
    want = oracle.fastq_to_fasta(text, append, flags)
    assert ReadSet(ctx, text).to_fasta(append, revcomp=rev, if_missing=if_missing) == want


@pytest.mark.parametrize("crlf", [False, True])
@pytest.mark.parametrize("append,rev", [(1, False), (12, True)])
def test_prep_record_shapes(ctx, oracle, crlf, append, rev):
    """Headers with and without further fields, names of 0 to 40 bytes, sequences of 0 to 70, qualities of another
    length or blank, '+' lines that repeat the name, and a last record without a newline; with CRs (the set's lines
    are then searched) and without."""
    rng = random.Random(7)
    recs = []
    for i in range(1500):
        name = "".join(rng.choice("abcXYZ019:/_") for _ in range(rng.choice([0, 1, 2, 13, 40]))) + rng.choice(["", "/1", "/2"])
        rest = rng.choice(["", "", " 1:N:0:ATC", " 2:Y:0", "\t1:", " x 1:", "  "])
        n = rng.choice([0, 1, 15, 16, 17, 33, 70])
        seq = "0" if n == 1 and rng.random() < 0.3 else "".join(rng.choice("ACGTNacgtRYKM") for _ in range(n))
        q = "I" * (n + rng.choice([0, 0, 0, 0, 1])) if rng.random() < 0.95 else " " * n
        recs.append(f"@{name}{rest}\n{seq}\n+{rng.choice(['', name])}\n{q}\n")
    text = "".join(recs + ["@last\nACGTAC\n+\nIIIIII"])
    if crlf:
        text = text.replace("\n", "\r\n")
    text = text.encode()
    flags = oracle.FA_IGNORE_DIRTY | (oracle.FA_REV if rev else 0)
    want = oracle.fastq_to_fasta(text, append, flags)
    assert ReadSet(ctx, text).to_fasta(append, revcomp=rev, ignore_dirty=True) == want


def test_prep_rejects_fasta_input(ctx, golden):
    rs = ReadSet(ctx, (golden / "edge.fa").read_bytes())
    with pytest.raises(native.TrinkmerError) as e:
        rs.to_fasta()
    assert e.value.status == native.TK_E_INVAL


def test_seqtk_trinity_cli(native_built, oracle, golden, tmp_path):
    """The command line Trinity runs: `cat f.fq | seqtk-trinity seq -A -R 2 [-r] -`."""
    fq = (golden / "prep.fq").read_bytes()
    for args, flags in ((["-R", "2"], oracle.FA_IF_MISSING), (["-R", "1", "-r"], oracle.FA_IF_MISSING | oracle.FA_REV)):
        p = subprocess.run([str(BIN / "seqtk-trinity"), "seq", "-A", *args, "-"], input=fq, capture_output=True,
                           timeout=300)
        assert p.returncode == 0, p.stderr
        assert p.stdout == oracle.fastq_to_fasta(fq, int(args[1]), flags)
    bad = subprocess.run([str(BIN / "seqtk-trinity"), "seq", "-A", str(golden / "prep_dirty.fq")], capture_output=True,
                         timeout=300)
    assert bad.returncode != 0 and b"improperly formatted" in bad.stderr
