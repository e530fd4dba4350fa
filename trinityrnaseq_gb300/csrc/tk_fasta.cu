// tk_fasta.cu -- FASTQ -> FASTA read prep on the GPU: the conversion Trinity
// runs before counting (`seqtk-trinity seq -A -R {1,2} [-r]`, Trinity:2745-2805),
// whose executable spec is util/support_scripts/fastQ_to_fastA.pl:60-118.
//
// Input is a parsed FASTQ read set (tk_reads_parse has checked the 4-line
// structure: '@' header, '+' third line).  One thread per record finds the
// record's four lines in the device copy of the text and applies the
// script's rules:
//   * only the header loses its CRs; sequence and quality lines lose just
//     their "\n" (a CRLF sequence keeps its CR, as the script prints it);
//   * a record is clean when its sequence is non-empty and not "0", and its
//     quality line holds a non-space byte and is as long as the sequence;
//   * name = first whitespace-separated field after '@' (empty if the header
//     starts with whitespace); "/1" or "/2" is added when another field
//     follows, the name does not end in /1 or /2 and that field starts "1:"
//     or "2:" (Casava 1.8); then "/append" (every name, the script's -a, or
//     with TK_FA_IF_MISSING only names not ending in /1 or /2);
//   * TK_FA_REVCOMP maps each byte through ACGTacgtyrkmYRKMUu ->
//     TGCAtgcarymkRYMKAa in reverse order (PerlLib/Nuc_translator.pm:286-292).
// Pass 1 sizes every record's output (0 for a skipped record), a scan places
// them, pass 2 writes ">" name suffix "\n" sequence "\n".
#include "tk_text.cuh"

#include <algorithm>

#include <string>

namespace tk {

constexpr int FA_THREADS = 256;

__device__ __forceinline__ bool pl_ws(uint32_t c) { return c == ' ' || c - 9u < 5u; }

__device__ __forceinline__ uint8_t rc_letter(uint8_t c) {
    switch (c) {
        case 'A': return 'T'; case 'C': return 'G'; case 'G': return 'C'; case 'T': return 'A';
        case 'a': return 't'; case 'c': return 'g'; case 'g': return 'c'; case 't': return 'a';
        case 'y': return 'r'; case 'r': return 'y'; case 'k': return 'm'; case 'm': return 'k';
        case 'Y': return 'R'; case 'R': return 'Y'; case 'K': return 'M'; case 'M': return 'K';
        case 'U': return 'A'; case 'u': return 'a';
        default: return c;
    }
}

__device__ __forceinline__ uint64_t line_end(const char *__restrict__ t, uint64_t len, uint64_t p) {
    while (p < len && t[p] != '\n') p++;
    return p;
}

// decimal digits of v (v >= 0)
__device__ __forceinline__ uint32_t n_digits(uint32_t v) {
    uint32_t d = 1;
    while (v >= 10) { v /= 10; d++; }
    return d;
}

struct FaRec {
    uint64_t name0, name1;   // header bytes [name0, name1) hold the first field (CRs skipped when copied)
    uint32_t name_len;       // the field's length without CRs
    uint64_t seq0;           // sequence line
    uint32_t seq_len;        // bytes before its "\n", CRs included
    uint32_t suffix;         // 0 none, else the Casava mate digit ('1' or '2')
    bool ends12;             // the name ends in /1 or /2
    bool clean;
};

// The header line of the record at `at`: its first field and mate suffix.
__device__ FaRec fa_header(const char *__restrict__ t, uint64_t len, uint64_t at) {
    FaRec f;
    const uint64_t he = line_end(t, len, at);
    // first field of the header (after '@'), CRs removed before splitting
    uint64_t p = at + 1;
    uint32_t nl = 0;
    uint8_t last = 0, prev = 0;
    while (p < he) {
        const uint8_t c = (uint8_t)t[p];
        if (c != '\r') {
            if (pl_ws(c)) break;
            prev = last;
            last = c;
            nl++;
        }
        p++;
    }
    f.name0 = at + 1;
    f.name1 = p;
    f.name_len = nl;
    f.ends12 = nl >= 2 && prev == '/' && (last == '1' || last == '2');
    // the next field: "1:" or "2:" adds the mate suffix
    while (p < he && (pl_ws((uint8_t)t[p]) || t[p] == '\r')) p++;
    f.suffix = 0;
    if (p < he && !f.ends12) {
        uint8_t a = 0, b = 0;
        uint64_t q = p;
        while (q < he && t[q] == '\r') q++;
        if (q < he) a = (uint8_t)t[q++];
        while (q < he && t[q] == '\r') q++;
        if (q < he) b = (uint8_t)t[q];
        if ((a == '1' || a == '2') && b == ':') f.suffix = a;
    }
    f.seq0 = he + 1;
    return f;
}

// The record's sequence length is set; its quality line is [q0, qe): whether it is clean.
__device__ __forceinline__ bool fa_clean(const char *__restrict__ t, uint64_t len, const FaRec &f, uint64_t q0, uint64_t qe) {
    const uint64_t sl = f.seq_len, ql = qe > q0 ? qe - q0 : 0;
    if (!(f.seq0 < len && q0 <= len && sl > 0 && !(sl == 1 && t[f.seq0] == '0') && ql == sl)) return false;
    bool ns = false;
    for (uint64_t i = q0; i < qe && !ns; i++) ns = !pl_ws((uint8_t)t[i]);
    return ns;
}

// What the parser knows of a record of a read set whose sequence lines hold
// no whitespace: the sequence line is the read's length long, and the quality
// line ends one byte before the next record (the last record's is searched).
struct FaSet {
    const char *text;
    uint64_t len;
    const uint64_t *name_off;
    const uint32_t *name_len;
    const uint64_t *rd_off;
    uint64_t n;
    bool plain;
};

// Record r.  With a plain set only the '+' line and, when the header has more
// than its first field, the header are searched byte by byte.
__device__ FaRec fa_get(const FaSet &s, uint64_t r) {
    const char *t = s.text;
    const uint64_t name0 = s.name_off[r];
    const uint32_t nl = s.name_len[r];
    const uint64_t after = name0 + nl;   // the first whitespace after the name
    FaRec f;
    if (s.plain && after < s.len && t[after] == '\n') {
        f.name0 = name0;
        f.name1 = after;
        f.name_len = nl;
        f.ends12 = nl >= 2 && t[after - 2] == '/' && (t[after - 1] == '1' || t[after - 1] == '2');
        f.suffix = 0;
        f.seq0 = after + 1;
    } else {
        f = fa_header(t, s.len, name0 - 1);
    }
    const uint64_t sl = s.plain ? s.rd_off[r + 1] - s.rd_off[r] - 1
                                : (f.seq0 < s.len ? line_end(t, s.len, f.seq0) - f.seq0 : 0);
    f.seq_len = (uint32_t)sl;
    const uint64_t q0 = line_end(t, s.len, f.seq0 + sl + 1) + 1;
    const uint64_t qe = s.plain && r + 1 < s.n ? s.name_off[r + 1] - 2 : line_end(t, s.len, q0);
    f.clean = fa_clean(t, s.len, f, q0, qe);
    return f;
}

__device__ __forceinline__ uint32_t fa_suffix_len(const FaRec &f, int append, int flags) {
    uint32_t n = f.suffix ? 2u : 0u;
    if (append >= 0 && !((flags & TK_FA_IF_MISSING) && (f.ends12 || f.suffix))) n += 1u + n_digits((uint32_t)append);
    return n;
}

__global__ void k_fa_len(FaSet s, int append, int flags, uint32_t *__restrict__ out_len,
                         unsigned long long *__restrict__ first_bad) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= s.n) return;
    const FaRec f = fa_get(s, r);
    if (!f.clean) {
        out_len[r] = 0;
        if (!(flags & TK_FA_IGNORE_DIRTY)) atomicMin(first_bad, (unsigned long long)r);
        return;
    }
    out_len[r] = 1u + f.name_len + fa_suffix_len(f, append, flags) + 1u + f.seq_len + 1u;
}

// A warp takes 32 consecutive records: each lane finds its record, stores the
// bytes around the name and the sequence, and the warp then copies the 32
// names and the 32 sequences in aligned 16-byte words (copy_group); reverse
// complements and names holding CRs are written byte by byte.  Bound by
// memory (the text read and written once).  3M records of 100 nt: a thread per
// record storing its bytes one by one took 3.18 ms, after 1.14 ms of k_fa_len
// walking all four lines byte by byte.
__global__ void __launch_bounds__(FA_THREADS) k_fa_write(FaSet s, ParseGeom g, int append, int flags,
                                                        const uint64_t *__restrict__ out_off, char *__restrict__ out) {
    __shared__ uint8_t rc[256];
    if (flags & TK_FA_REVCOMP) {
        for (int i = threadIdx.x; i < 256; i += FA_THREADS) rc[i] = rc_letter((uint8_t)i);
        __syncthreads();
    }
    const unsigned lane = lane_id();
    const uint64_t warps = (uint64_t)gridDim.x * (FA_THREADS / 32);
    for (uint64_t r0 = ((uint64_t)blockIdx.x * (FA_THREADS / 32) + (threadIdx.x >> 5)) * 32; r0 < s.n; r0 += warps * 32) {
        const uint64_t r = r0 + lane;
        uint64_t name_src = 0, name_dst = 0, seq_src = 0, seq_dst = 0;
        uint32_t name_n = 0, seq_n = 0;
        if (r < s.n && out_off[r + 1] != out_off[r]) {
            const FaRec f = fa_get(s, r);
            uint64_t o = out_off[r];
            out[o++] = '>';
            name_src = f.name0;
            name_dst = o;
            if (f.name1 - f.name0 == f.name_len) {
                name_n = f.name_len;
            } else {   // CRs inside the name are dropped
                uint64_t q = o;
                for (uint64_t p = f.name0; p < f.name1; p++)
                    if (s.text[p] != '\r') out[q++] = s.text[p];
            }
            o += f.name_len;
            if (f.suffix) {
                out[o++] = '/';
                out[o++] = (char)f.suffix;
            }
            if (append >= 0 && !((flags & TK_FA_IF_MISSING) && (f.ends12 || f.suffix))) {
                out[o++] = '/';
                const uint32_t d = n_digits((uint32_t)append);
                uint32_t v = (uint32_t)append;
                for (uint32_t i = 0; i < d; i++) {
                    out[o + d - 1 - i] = (char)('0' + v % 10);
                    v /= 10;
                }
                o += d;
            }
            out[o++] = '\n';
            seq_src = f.seq0;
            seq_dst = o;
            seq_n = f.seq_len;
            out[o + seq_n] = '\n';
        }
        uint8_t *ob = reinterpret_cast<uint8_t *>(out);
        copy_group(g, name_src, name_dst, name_n, ob);
        if (flags & TK_FA_REVCOMP) {
            for (int i = 0; i < 32; i++) {
                const uint32_t n = __shfl_sync(0xffffffffu, seq_n, i);
                const uint64_t src = __shfl_sync(0xffffffffu, seq_src, i), dst = __shfl_sync(0xffffffffu, seq_dst, i);
                for (uint32_t j = lane; j < n; j += 32) ob[dst + j] = rc[(uint8_t)s.text[src + n - 1 - j]];
            }
        } else {
            copy_group(g, seq_src, seq_dst, seq_n, ob);
        }
    }
}

// FASTA text of a FASTQ read set into *d_text (device, caller frees with dfree).
int reads_fasta(tk_reads *r, int append, int flags, char **d_text, uint64_t *text_len) {
    tk_ctx *c = r->ctx;
    *d_text = nullptr;
    *text_len = 0;
    const uint64_t n = r->n_reads;
    uint32_t *lens = nullptr;
    uint64_t *offs = nullptr;
    unsigned long long *bad = nullptr;
    TK_TRY(dmalloc(c, (void **)&lens, (n ? n : 1) * 4, "fasta record lengths"));
    int e = dmalloc(c, (void **)&offs, (n + 1) * 8, "fasta record offsets");
    if (!e) e = dmalloc(c, (void **)&bad, 8, "fasta first bad record");
    if (!e) e = cuda_check(c, cudaMemsetAsync(bad, 0xFF, 8, c->stream), "bad reset");
    const unsigned grid = (unsigned)((n + FA_THREADS - 1) / FA_THREADS);
    const FaSet set{r->d_text, r->text_len, r->d_name_off, r->d_name_len, r->d_rd_off, n, r->plain_seq};
    if (!e && n) {
        k_fa_len<<<grid, FA_THREADS, 0, c->stream>>>(set, append, flags, lens, bad);
        c->launches++;
        e = check_launch(c, "fasta lengths");
    }
    unsigned long long hbad = ~0ULL;
    uint64_t total = 0;
    if (!e && n) e = scan_excl_u32_to_u64(c, lens, offs, n, &total);   // synchronises
    if (!e) e = cuda_check(c, cudaMemcpyAsync(&hbad, bad, 8, cudaMemcpyDeviceToHost, c->stream), "bad d2h");
    if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "fasta sync");
    if (!e && hbad != ~0ULL)
        e = set_err(c, TK_E_PARSE, "FASTQ input: improperly formatted entry (record " + std::to_string(hbad + 1) + ")");
    if (!e && n) {
        cudaMemcpyAsync(offs + n, &total, 8, cudaMemcpyHostToDevice, c->stream);
        e = dmalloc(c, (void **)d_text, total ? total : 1, "fasta text");
        if (!e && total) {
            ParseGeom g{};
            g.text = r->d_text;
            g.len = r->text_len;
            g.vec = ((uintptr_t)r->d_text & 15u) == 0;
            k_fa_write<<<std::min(grid, (unsigned)c->sm_count * 32), FA_THREADS, 0, c->stream>>>(set, g, append, flags, offs,
                                                                                                *d_text);
            c->launches++;
            e = check_launch(c, "fasta write");
        }
    }
    if (!e) *text_len = total;
    dfree(c, lens);
    dfree(c, offs);
    if (bad) dfree(c, bad);
    if (e && *d_text) {
        dfree(c, *d_text);
        *d_text = nullptr;
    }
    return e;
}

}  // namespace tk
