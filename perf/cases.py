"""The work a Trinity run gives this package, as cases to time.

Each case is one call sequence a user's program makes through the package's
public entry points: counting reads (jellyfish count, histo, dump), per-read
coverage statistics (fastaToKmerCoverageStats), the normalization's selection
and extraction, read-to-component assignment (ReadsToTranscripts), the
components' de Bruijn graphs (FastaToDeBruijn), the per-bin catalogues of the
assembly's second phase, the FASTQ -> FASTA read prep, and a whole
normalization job.  Large texts are resident in GPU memory as they are after
an upload; the small and the batched calls take host text and return host
text, as the executables do.

The inputs are reads drawn from a synthetic transcriptome (genes of a few
isoforms made of shared exons, log-normal expression, both strands,
substitutions, a few N), written as FASTA or FASTQ records.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from trinityrnaseq_gb300 import kmer
from trinityrnaseq_gb300.kmer import (Context, DeBruijnGraphs, KmerTable, Normalization, ReadSet, ReadsToTranscripts,
                                      coverage_stats_into)

DEV = "cuda:0"
_context = None


def context() -> Context:
    """The process's one context (a program makes one and keeps it)."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


# ---------------------------------------------------------------- cases

def listed():
    return [
        # one read bin of the assembly's second phase: a few thousand reads in, its k-mer catalogue out
        {"name": "count one bin", "op": "count", "reads": 2000, "length": 76, "mates": 1, "fastq": False, "host": True,
         "k": 25, "canonical": True, "ragged": False, "min_count": 1},
        # single-end 76-nt FASTA of a small experiment, strand-specific
        {"name": "count 1M single", "op": "count", "reads": 1_000_000, "length": 76, "mates": 1, "fastq": False,
         "host": False, "k": 25, "canonical": False, "ragged": False, "min_count": 1},
        # paired 100-nt FASTQ of a full experiment: the k-mer catalogue both Inchworm and the normalization use
        {"name": "count 5M pairs", "op": "count", "reads": 5_000_000, "length": 100, "mates": 2, "fastq": True,
         "host": False, "k": 25, "canonical": True, "ragged": False, "min_count": 2},
        # the coverage pass of those reads against their own catalogue
        {"name": "coverage 5M pairs", "op": "coverage", "reads": 5_000_000, "length": 100, "mates": 2, "fastq": True,
         "k": 25, "canonical": True, "ragged": False},
        # quality-trimmed longer reads of every length up to 600 nt, k = 31
        {"name": "coverage ragged", "op": "coverage", "reads": 300_000, "length": 600, "mates": 1, "fastq": False,
         "k": 31, "canonical": True, "ragged": True},
        # fastaToKmerCoverageStats as the normalization script starts it: a dumped catalogue and a FASTA file
        {"name": "catalogue stats 400K", "op": "catalogue", "reads": 400_000, "length": 100, "k": 25,
         "canonical": True, "ragged": False},
        # the normalization after the statistics: name sort, pair merge, selection, both mates' records
        {"name": "normalize 2M pairs", "op": "normalize", "reads": 2_000_000, "length": 100, "k": 25,
         "canonical": True, "max_cov": 50},
        # reads to components of an Inchworm bundle, the bundle's table built in the call
        {"name": "assign 3M reads", "op": "assign", "reads": 3_000_000, "length": 100, "contigs": 30_000, "k": 25,
         "strand": False, "ragged": False},
        # the components' de Bruijn graphs
        {"name": "de Bruijn 30K contigs", "op": "debruijn", "contigs": 30_000, "K": 24, "strand": False},
        # the second phase's bins in one batch, power-law sizes
        {"name": "bins 2000", "op": "bins", "bins": 2000, "length": 100, "k": 25, "canonical": True},
        # read prep of one mate file
        {"name": "fastq to fasta 3M", "op": "prep", "reads": 3_000_000, "length": 100, "append": 1, "revcomp": False,
         "ragged": False},
        # a whole normalization job of a small sample: both mates parsed, counted, dumped, covered, selected, extracted
        {"name": "normalize job 50K pairs", "op": "job", "reads": 50_000, "length": 100, "k": 25, "canonical": True,
         "max_cov": 30},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["count", "count", "count", "coverage", "coverage", "catalogue", "normalize", "assign", "debruijn",
                     "bins", "prep", "job"])
    k = rng.choice([25, 25, 25, 21, 31])
    length = rng.choice([50, 76, 100, 101, 125, 150])
    ragged = rng.random() < 0.3
    canonical = rng.random() < 0.7
    if op == "count":
        if rng.random() < 0.3:
            return {"op": op, "reads": _log_int(rng, 500, 20_000), "length": length, "mates": 1, "fastq": False,
                    "host": True, "k": k, "canonical": canonical, "ragged": ragged, "min_count": 1}
        mates = rng.choice([1, 2])
        return {"op": op, "reads": _log_int(rng, 20_000, 3_000_000), "length": length, "mates": mates,
                "fastq": mates == 2 or rng.random() < 0.5, "host": False, "k": k, "canonical": canonical,
                "ragged": ragged, "min_count": rng.choice([1, 2])}
    if op == "coverage":
        if rng.random() < 0.4:
            return {"op": op, "reads": _log_int(rng, 5_000, 300_000), "length": rng.randint(160, 600), "mates": 1,
                    "fastq": False, "k": k, "canonical": canonical, "ragged": True}
        return {"op": op, "reads": _log_int(rng, 20_000, 3_000_000), "length": length, "mates": 2, "fastq": True,
                "k": k, "canonical": canonical, "ragged": ragged}
    if op == "catalogue":
        return {"op": op, "reads": _log_int(rng, 10_000, 400_000), "length": length, "k": k, "canonical": canonical,
                "ragged": ragged}
    if op == "normalize":
        return {"op": op, "reads": _log_int(rng, 20_000, 2_000_000), "length": min(length, 100), "k": 25,
                "canonical": canonical, "max_cov": rng.choice([30, 50, 200])}
    if op == "assign":
        return {"op": op, "reads": _log_int(rng, 20_000, 2_500_000), "length": length,
                "contigs": _log_int(rng, 500, 30_000), "k": 25, "strand": not canonical, "ragged": ragged}
    if op == "debruijn":
        return {"op": op, "contigs": _log_int(rng, 500, 30_000), "K": rng.choice([24, 24, 30]), "strand": not canonical}
    if op == "bins":
        return {"op": op, "bins": _log_int(rng, 20, 2000), "length": min(length, 100), "k": k, "canonical": canonical}
    if op == "prep":
        return {"op": op, "reads": _log_int(rng, 20_000, 2_000_000), "length": length, "append": rng.choice([1, 2]),
                "revcomp": rng.random() < 0.3, "ragged": ragged}
    return {"op": op, "reads": _log_int(rng, 5_000, 300_000), "length": min(length, 125), "k": 25,
            "canonical": canonical, "max_cov": rng.choice([30, 50])}


# ---------------------------------------------------------------- synthetic inputs

BASES = b"ACGT"


class Draws:
    """Random numbers on the GPU from one seed."""

    def __init__(self, seed: int):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)

    def uniform(self, *shape, dtype=torch.float32):
        return torch.rand(*shape, generator=self.g, device=DEV, dtype=dtype)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device=DEV)

    def integers(self, lo: int, hi: int, *shape, dtype=torch.int64):
        return torch.randint(lo, hi, shape, generator=self.g, device=DEV, dtype=dtype)


def _pieces(start, length):
    """Indices start[i], start[i] + 1, ... (length[i] of them) for every i, one after another."""
    before = torch.cumsum(length, 0) - length
    return torch.repeat_interleave(start - before, length) + torch.arange(int(length.sum()), device=DEV)


class Transcripts:
    """Genes of 8 exons and 3 isoforms (each with about 70% of the gene's exons), and each isoform's share of the reads."""

    def __init__(self, r: Draws, genes: int, exon: float = 150.0):
        n_ex, n_iso = 8, 3
        ex_len = (exon * torch.exp(0.6 * r.normal(genes, n_ex))).clamp(40, 12 * exon).long()
        ex_off = torch.cumsum(ex_len.view(-1), 0) - ex_len.view(-1)
        pool = r.integers(0, 4, int(ex_len.sum()), dtype=torch.uint8)
        has = r.uniform(genes, n_iso, n_ex) < 0.7
        has[:, 0, :] = True                      # the first isoform has every exon
        gene, iso, ex = has.nonzero(as_tuple=True)
        at = gene * n_ex + ex
        piece_len = ex_len.view(-1)[at]
        self.codes = pool[_pieces(ex_off[at], piece_len)]
        n_tx = genes * n_iso
        self.length = torch.zeros(n_tx, dtype=torch.int64, device=DEV).index_add_(0, gene * n_iso + iso, piece_len)
        self.start = torch.cumsum(self.length, 0) - self.length
        weight = torch.exp(1.5 * r.normal(n_tx)).double() * self.length
        self.cum = torch.cumsum(weight / weight.sum(), 0)

    def pick(self, r: Draws, n: int):
        return torch.searchsorted(self.cum, r.uniform(n, dtype=torch.float64)).clamp_max(self.length.numel() - 1)


def _genes_for(reads: int) -> int:
    return max(8, min(20_000, reads // 100))


def _substitute(r: Draws, codes, err: float, n_rate: float):
    """Base codes with substitutions at rate err and N (code 4) at rate n_rate."""
    u = r.uniform(*codes.shape)
    other = (codes + r.integers(1, 4, *codes.shape, dtype=torch.uint8)) & 3
    codes = torch.where(u < err, other, codes)
    return torch.where(u > 1.0 - n_rate, torch.full_like(codes, 4), codes)


def _codes_of(tx: Transcripts, r: Draws, start, step, length, width: int, err: float, n_rate: float):
    """Reads as base codes (n x width, columns past a read's length unspecified): bases start, start + step, ... of
    the transcripts, complemented when step is -1."""
    out = torch.empty(start.numel(), width, dtype=torch.uint8, device=DEV)
    col = torch.arange(width, device=DEV)
    last = tx.codes.numel() - 1
    for a in range(0, start.numel(), 1_000_000):
        s = slice(a, min(a + 1_000_000, start.numel()))
        at = (start[s, None] + step[s, None] * torch.minimum(col[None, :], length[s, None] - 1)).clamp_(0, last)
        c = tx.codes[at]
        c = torch.where(step[s, None] < 0, 3 - c, c)
        out[s] = _substitute(r, c, err, n_rate)
    return out


def _read_codes(case, seed):
    """[(codes, lengths)] of each mate of a case's reads."""
    r = Draws(seed)
    n, width = case["reads"], case["length"]
    long_reads = width > 160
    tx = Transcripts(r, _genes_for(n), 450.0 if long_reads else 150.0)
    n_rate = 0.0001
    err = 0.005 if case.get("mates", 2) == 1 else 0.01
    t = tx.pick(r, n)
    tl = tx.length[t]
    if case.get("mates", 2) == 2:
        frag = (300 + 50 * r.normal(n)).long().clamp_min(width)
    else:
        frag = torch.full((n,), width, dtype=torch.int64, device=DEV)
    frag = torch.minimum(frag, tl)
    left = tx.start[t] + (r.uniform(n, dtype=torch.float64) * (tl - frag + 1)).long()
    flip = r.uniform(n) < 0.5
    fwd = torch.where(flip, -1, 1)
    sides = [(torch.where(flip, left + frag - 1, left), fwd), (torch.where(flip, left, left + frag - 1), -fwd)]
    out = []
    for start, step in sides[:case.get("mates", 2)]:
        length = torch.minimum(torch.full_like(frag, width), frag)
        if case.get("ragged"):
            kept = torch.where(r.uniform(n) < (0.1 if long_reads else 0.6), 1.0, r.uniform(n))
            length = torch.maximum((length * kept).long(), torch.minimum(length, torch.full_like(length, 20)))
        out.append((_codes_of(tx, r, start, step, length, width, err, n_rate), length))
    return out


def _decimal(n: int, digits: int):
    """0 .. n-1 as fixed-width decimal text (n x digits)."""
    i = torch.arange(n, device=DEV)
    return torch.stack([(i // 10 ** (digits - 1 - d)) % 10 for d in range(digits)], 1).to(torch.uint8) + ord("0")


def _text(codes, length, fastq: bool, mate: int, ragged: bool):
    """The reads as FASTA or FASTQ text: a uint8 tensor on the GPU, names r0000000000/1, ..."""
    n, width = codes.shape
    letters = torch.tensor(list(b"ACGTN"), dtype=torch.uint8, device=DEV)

    def const(s: bytes):
        return torch.tensor(list(s), dtype=torch.uint8, device=DEV).expand(n, len(s))

    head = torch.cat([const(b"@r" if fastq else b">r"), _decimal(n, 10), const(b"/%d\n" % mate)], 1)
    seq = letters[codes.long()] if n * width < 100_000_000 else torch.cat(
        [letters[c.long()] for c in codes.split(1_000_000)])
    parts = [head, seq, const(b"\n")]
    if fastq:
        parts += [const(b"+\n"), torch.full_like(seq, ord("I")), const(b"\n")]
    rows = torch.cat(parts, 1)
    if not ragged and bool((length == width).all()):
        return rows.reshape(-1)
    inside = torch.arange(width, device=DEV)[None, :] < length[:, None]
    on = torch.ones(n, 1, dtype=torch.bool, device=DEV)
    keep = [on.expand(n, head.shape[1]), inside, on]
    if fastq:
        keep += [on.expand(n, 2), inside, on]
    return rows[torch.cat(keep, 1)]


def _pinned(text) -> np.ndarray:
    """A page-locked host copy of a text."""
    t = text if isinstance(text, torch.Tensor) else torch.from_numpy(np.frombuffer(text, dtype=np.uint8).copy())
    h = torch.empty(t.numel(), dtype=torch.uint8, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _bundle(r: Draws, contigs: int):
    """(bundle text on the GPU, contig bases): records >s_<c> of 1-40 contigs joined by X, as Chrysalis bundles them."""
    lens = (400.0 * torch.exp(0.5 * r.normal(contigs))).clamp(200, 6000).long()
    comp = torch.sort((r.uniform(contigs) ** 1.5 * max(1, contigs // 3)).long()).values
    codes = r.integers(0, 4, int(lens.sum()), dtype=torch.uint8)
    start = torch.cumsum(lens, 0) - lens
    # some contigs repeat a stretch of the one before them (isoforms of one gene)
    again = ((r.uniform(contigs) < 0.3) & (torch.arange(contigs, device=DEV) > 0)).nonzero().view(-1)
    part = torch.minimum(lens[again], lens[again - 1]) // 2
    codes[_pieces(start[again], part)] = codes[_pieces(start[again - 1], part)]
    h_codes = np.frombuffer(BASES, dtype=np.uint8)[codes.cpu().numpy()]
    cut = np.append(start.cpu().numpy(), h_codes.size)
    out, last = [], -1
    for i, c in enumerate(comp.tolist()):
        out.append(b"X" if c == last else (b"\n>s_%d\n" % c if out else b">s_%d\n" % c))
        out.append(h_codes[cut[i]:cut[i + 1]].tobytes())
        last = c
    out.append(b"\n")
    return b"".join(out), codes, start, lens


class State:
    """What a program holds before a call: its inputs, handles and output buffers."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _room(n) -> torch.Tensor:
    """An output buffer in GPU memory, zero past what a call writes."""
    return torch.zeros(int(n), dtype=torch.uint8, device=DEV)


def _host_room(n) -> torch.Tensor:
    return torch.zeros(int(n), dtype=torch.uint8, pin_memory=True)


def _dump_bytes(windows: float, k: int, min_count: int) -> int:
    """More than the dump of a read set with so many windows takes."""
    return int(windows * (0.3 if min_count > 1 else 0.6) * (k + 5)) + 65536


def _windows_of(case, mates: int) -> int:
    return case["reads"] * mates * max(1, case["length"] - case["k"] + 1)


def _stats_room(n: int):
    return [torch.empty(n, dtype=d, device=DEV) for d in (torch.int32, torch.float32, torch.float32)]


def _select_room(case):
    n = case["reads"]
    return {"accs": _room(n * 12), "left": _room(n * _record_bytes(case["length"], True)),
            "right": _room(n * _record_bytes(case["length"], True))}


def _parse(text) -> ReadSet:
    if isinstance(text, torch.Tensor):
        return ReadSet(context(), text.data_ptr(), text.numel(), device=True)
    return ReadSet(context(), text)


def prepare(case, seed):
    op = case["op"]
    if op in ("count", "coverage", "catalogue", "normalize", "prep", "job"):
        mates = {"catalogue": 1, "prep": 1, "normalize": 2, "job": 2}.get(op, case.get("mates"))
        fastq = case.get("fastq", op in ("normalize", "prep", "job"))
        sides = _read_codes(dict(case, mates=mates), seed)
        texts = [_text(c, ln, fastq, i + 1, bool(case.get("ragged"))) for i, (c, ln) in enumerate(sides)]
        torch.cuda.synchronize()
        if op == "count":
            size = _dump_bytes(_windows_of(case, mates), case["k"], case["min_count"])
            if case["host"]:
                return State(case=case, texts=[_pinned(t) for t in texts], dump=_host_room(size))
            return State(case=case, texts=texts, dump=_room(size))
        if op == "prep":
            return State(case=case, texts=texts, out=_room(case["reads"] * _record_bytes(case["length"] + 2, False)))
        if op == "job":
            return State(case=case, texts=texts, dump=_room(_dump_bytes(_windows_of(case, 2), case["k"], 2)),
                         stats=[_stats_room(case["reads"]) for _ in texts], out=_select_room(case))
        sets = [_parse(t) for t in texts]
        table = KmerTable(context(), case["k"], case["canonical"])
        table.add_many(sets)
        if op == "catalogue":
            dump = table.dump_fasta(2)
            return State(case=case, reads=_pinned(texts[0]), dump=_pinned(dump))
        stats = [_stats_room(s.n_reads) for s in sets]
        st = State(case=case, texts=texts, sets=sets, table=table, stats=stats)
        if op == "normalize":
            for s, b in zip(sets, stats):
                coverage_stats_into(table, s, *[x.data_ptr() for x in b])
            context().synchronize()
            table.free()
            st.out = _select_room(case)
        return st
    r = Draws(seed)
    if op == "debruijn":
        bundle, _, _, _ = _bundle(r, case["contigs"])
        text = torch.from_numpy(np.frombuffer(bundle, dtype=np.uint8).copy()).to(DEV)
        torch.cuda.synchronize()
        return State(case=case, bundle=text, out=_room(case["contigs"] * 700 * (case["K"] + 18)))
    if op == "assign":
        bundle, codes, start, lens = _bundle(r, case["contigs"])
        tx = Transcripts.__new__(Transcripts)
        tx.codes, tx.start, tx.length = codes, start, lens
        n, width = case["reads"], case["length"]
        weight = torch.exp(1.5 * r.normal(lens.numel())).double() * lens
        tx.cum = torch.cumsum(weight / weight.sum(), 0)
        t = tx.pick(r, n)
        left = start[t] + (r.uniform(n, dtype=torch.float64) * (lens[t] - width + 1)).long()
        flip = (r.uniform(n) < 0.5) & (not case["strand"])
        length = torch.full((n,), width, dtype=torch.int64, device=DEV)
        if case["ragged"]:
            length = torch.where(r.uniform(n) < 0.6, length, (length * r.uniform(n)).long().clamp_min(20))
        reads = _codes_of(tx, r, torch.where(flip, left + width - 1, left), torch.where(flip, -1, 1), length, width,
                          0.01, 0.0001)
        text = _text(reads, length, False, 1, case["ragged"])
        out = [torch.empty(n, dtype=torch.int32, device=DEV) for _ in range(3)]
        torch.cuda.synchronize()
        return State(case=case, bundle=_pinned(bundle), text=text, out=out)
    # bins: reads per bin by a power law (exponent 1.8, 50 .. 20,000), each bin from its own few transcripts
    n_bins, width = case["bins"], case["length"]
    u = (torch.randperm(n_bins, generator=r.g, device=DEV).double() + 0.5) / n_bins
    lo, hi = 50.0 ** -0.8, 20_000.0 ** -0.8
    per_bin = ((lo + u * (hi - lo)) ** (-1 / 0.8)).long()
    tx = Transcripts(r, n_bins)
    n = int(per_bin.sum())
    of = torch.repeat_interleave(torch.arange(n_bins, device=DEV), per_bin)
    t = of * 3 + r.integers(0, 3, n)
    t = torch.where(tx.length[t] >= width, t, of * 3)
    left = tx.start[t] + (r.uniform(n, dtype=torch.float64) * (tx.length[t] - width + 1)).long()
    flip = r.uniform(n) < 0.5
    length = torch.full((n,), width, dtype=torch.int64, device=DEV)
    reads = _codes_of(tx, r, torch.where(flip, left + width - 1, left), torch.where(flip, -1, 1), length, width, 0.01,
                      0.0001)
    text = _text(reads, length, False, 1, False)
    record = text.numel() // n
    off = np.zeros(n_bins + 1, dtype=np.uint64)
    off[1:] = np.cumsum(per_bin.cpu().numpy()).astype(np.uint64) * record
    windows = float((per_bin * (width - case["k"] + 1)).sum())
    room = _host_room(_dump_bytes(windows * 0.6 + 3000.0 * n_bins, case["k"], 1))
    return State(case=case, text=_pinned(text), off=off, out=room.numpy())


# ---------------------------------------------------------------- one pass

def _dump(table: KmerTable, min_count: int, room: torch.Tensor):
    """The table's dump as text in the buffer (GPU or host memory) and its length."""
    n = table.dump_fasta_len(min_count)
    table.dump_fasta_into(min_count, room.data_ptr(), room.numel(), device=room.is_cuda)
    return {"histo": table.histo().astype(np.int64), "dump": room, "dump_bytes": n}


def _select(sets, stats, max_cov: int, room):
    """The selected accs and both mates' selected records (in GPU memory)."""
    nm = Normalization(context(), sets[0], [x.data_ptr() for x in stats[0]], sets[1],
                       [x.data_ptr() for x in stats[1]], max_cov, 1, 10000, device=True)
    nm.ctx.check(nm.lib.tk_norm_accs(nm.h, 1, room["accs"].data_ptr(), room["accs"].numel()), "tk_norm_accs")
    sizes = [nm.accs_len] + [nm.extract_into(reads, room[side].data_ptr(), room[side].numel(), device=True)
                             for side, reads in zip(("left", "right"), sets)]
    return dict(room, bytes=np.array(sizes, dtype=np.int64),
                counts=np.array([nm.counts[f] for f in ("rows", "selected", "aberrant", "below_min")], dtype=np.int64))


def run(s):
    case = s.case
    op = case["op"]
    ctx = context()
    if op == "count":
        table = KmerTable(ctx, case["k"], case["canonical"])
        if case["host"]:
            table.count_text(s.texts[0])
        else:
            table.add_many([_parse(t) for t in s.texts])
        return _dump(table, case["min_count"], s.dump)
    if op == "coverage":
        for reads, b in zip(s.sets, s.stats):
            coverage_stats_into(s.table, reads, *[x.data_ptr() for x in b])
        ctx.synchronize()
        return [{"median": b[0], "mean": b[1], "stdev": b[2]} for b in s.stats]
    if op == "catalogue":
        table = KmerTable(ctx, case["k"], case["canonical"])
        table.load_dump_fasta(s.dump)
        med, mean, sd = kmer.coverage_stats(table, ReadSet(ctx, s.reads))
        return [{"median": med.astype(np.int64), "mean": mean, "stdev": sd}]
    if op == "normalize":
        return _select(s.sets, s.stats, case["max_cov"], s.out)
    if op == "assign":
        z = ReadsToTranscripts(ctx, s.bundle, case["k"], case["strand"])
        reads = _parse(s.text)
        z.assign_into(reads, *[x.data_ptr() for x in s.out])
        ctx.synchronize()
        ids = np.zeros(case["contigs"], dtype=np.int64)
        ids[:z.n_records] = z.component_ids
        return {"rec": s.out[0], "hits": s.out[1], "nwin": s.out[2], "ids": ids}
    if op == "debruijn":
        g = DeBruijnGraphs(ctx, s.bundle.data_ptr(), case["K"], case["strand"], s.bundle.numel(), device=True)
        g.text_into(s.out.data_ptr(), s.out.numel(), device=True)
        return {"text": s.out, "bytes": g.text_len, "components": g.n_components, "nodes": g.n_nodes}
    if op == "bins":
        text, off, kmers = kmer.count_bins(ctx, s.text, s.off, case["k"], case["canonical"], 1, s.out)
        return {"text": s.out, "bytes": text.size, "off": off.astype(np.int64), "kmers": kmers}
    if op == "prep":
        reads = _parse(s.texts[0])
        n = reads.fasta_into(s.out.data_ptr(), s.out.numel(), case["append"], case["revcomp"], if_missing=True,
                             device=True)
        ctx.synchronize()
        return {"text": s.out, "bytes": n}
    # job
    table = KmerTable(ctx, case["k"], case["canonical"])
    sets = [_parse(t) for t in s.texts]
    table.add_many(sets)
    dump = _dump(table, 2, s.dump)
    for reads, b in zip(sets, s.stats):
        coverage_stats_into(table, reads, *[x.data_ptr() for x in b])
    picked = _select(sets, s.stats, case["max_cov"], s.out)
    return {"dump": dump, "picked": picked, "stats": [{"median": b[0], "mean": b[1], "stdev": b[2]} for b in s.stats]}


# ---------------------------------------------------------------- bytes and 64-bit values

def _record_bytes(width: int, fastq: bool) -> int:
    return 15 + width + 1 + ((2 + width + 1) if fastq else 0)


def work(case):
    """Bytes of one pass: the input text, tables the call is given, and its outputs, each once (a k-mer table or
    catalogue holds about a third of the reads' windows as distinct k-mers)."""
    op, width = case["op"], case.get("length", 0)
    k = case.get("k", 25)
    kept = 0.65 if case.get("ragged") else 1.0
    n = case.get("reads", 0) * case.get("mates", 2 if op in ("normalize", "job") else 1)
    win = n * max(1.0, width * kept - k + 1)
    text_fa, text_fq = n * _record_bytes(int(width * kept), False), n * _record_bytes(int(width * kept), True)
    if op == "count":
        b = (text_fq if case["fastq"] else text_fa) + win / 3 * (k + 5) / case["min_count"]
    elif op == "coverage":
        b = win / 4 + win / 3 * 12 + n * 12
    elif op == "catalogue":
        b = text_fa + win / 6 * (k + 5) + n * 12
    elif op == "normalize":
        b = n * 12 + text_fq
    elif op == "assign":
        b = text_fa + case["contigs"] * 450 + n * 12
    elif op == "debruijn":
        b = case["contigs"] * 450 * 45
    elif op == "bins":
        b = case["bins"] * 470 * (_record_bytes(width, False) + (width - k + 1) / 3 * (k + 5))
    elif op == "prep":
        b = text_fq + text_fa
    else:
        b = text_fq * 2 + win / 6 * (k + 5) + n * 12
    return {"bytes": float(b), "flops": 0.0}


def _windows(codes, length, k: int, canonical: bool):
    """(keys, valid) of every window of the reads: n x (width - k + 1)."""
    n, width = codes.shape
    m = width - k + 1
    fw = torch.zeros(n, m, dtype=torch.int64, device=DEV)
    rc = torch.zeros_like(fw)
    bad = torch.zeros(n, m, dtype=torch.bool, device=DEV)
    for j in range(k):
        c = codes[:, j:j + m].long()
        bad |= c > 3
        c = c & 3
        fw = (fw << 2) | c
        rc = rc | ((3 - c) << (2 * j))
    ok = ~bad & (torch.arange(m, device=DEV)[None, :] + k <= length[:, None])
    return (torch.minimum(fw, rc) if canonical else fw), ok


def exact(case, seed):
    """The coverage statistics' mean and stdev in 64 bits (the other outputs are whole numbers and bytes)."""
    op = case["op"]
    if op not in ("coverage", "catalogue", "job"):
        return None
    mates = {"catalogue": 1, "job": 2}.get(op, case.get("mates"))
    k = case["k"]
    if case["reads"] * mates * max(1, case["length"] - k + 1) > 900_000_000:
        return None
    sides = _read_codes(dict(case, mates=mates), seed)
    step = max(1, 60_000_000 // case["length"])
    keys = []
    for codes, length in sides:
        for a in range(0, codes.shape[0], step):
            w, ok = _windows(codes[a:a + step], length[a:a + step], k, case["canonical"])
            keys.append(w[ok])
    keys = torch.sort(torch.cat(keys)).values
    first = torch.ones(keys.numel(), dtype=torch.bool, device=DEV)
    first[1:] = keys[1:] != keys[:-1]
    at = first.nonzero().view(-1)
    distinct = keys[at]
    count = torch.diff(at, append=torch.tensor([keys.numel()], device=DEV)).double()
    del keys, first, at
    stats = []
    for codes, length in sides:
        means, sds = [], []
        for a in range(0, codes.shape[0], step):
            w, ok = _windows(codes[a:a + step], length[a:a + step], k, case["canonical"])
            v = count[torch.searchsorted(distinct, w).clamp_max(distinct.numel() - 1)] * ok
            n = ok.sum(1).clamp_min(1).double()
            mean = v.sum(1) / n
            dev = (v - mean[:, None]) * ok
            means.append(mean)
            sds.append(torch.sqrt((dev * dev).sum(1) / n))
        stats.append({"median": None, "mean": torch.cat(means), "stdev": torch.cat(sds)})
    if op == "job":
        return {"dump": None, "picked": None, "stats": stats}
    return stats
