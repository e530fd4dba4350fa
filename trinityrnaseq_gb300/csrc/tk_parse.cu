// tk_parse.cu -- K1: FASTA/FASTQ text -> device read set.
//
// The text is split into lines and records entirely on the GPU with tiled,
// coalesced passes (each thread owns 32 consecutive bytes, read as two 16-byte
// vectors; a block owns an 8 KB tile):
//   A1  newlines per tile                 -> scan -> first line of every tile
//   A2  newline positions (line ends)
//   L   line kinds: FASTA '>' header / sequence; FASTQ line index mod 4,
//       with the '@' and '+' checks of a 4-line record; header lines are
//       scanned into a record index per line
//   C   every 32 positions of seq from the line (or lines) that hold them,
//       upper-cased, with their 2-bit codes
//   N   accession (first header token) and read length per record
// and, when a sequence line holds whitespace, instead of C
//   B1  emitted bases per tile (sequence-line bytes that are not whitespace)
//   B2  emit: base -> seq[emit_prefix + record] upper-cased; a header's first
//       byte records its read's start
// Semantics follow PerlLib/Fasta_reader.pm:45-73 (records start at '>' lines,
// sequence = following lines with whitespace removed), Sequence->new at
// PerlLib/Fasta_reader.pm:107-118 (accession = first whitespace token), and the
// 4-line record checks of util/support_scripts/fastQ_to_fastA.pl:80-92.
#include "tk_text.cuh"

#include <algorithm>

namespace tk {

constexpr int PT_THREADS = 256;
constexpr int PT_BYTES = 32;
constexpr uint64_t PT_TILE = (uint64_t)PT_THREADS * PT_BYTES;

enum LineKind : uint8_t { LK_SKIP = 0, LK_HDR = 1, LK_SEQ = 2 };

// ' ', '\t', '\n', '\v', '\f', '\r' (9..13)
__device__ __forceinline__ bool is_ws(uint32_t c) { return c == ' ' || c - 9u < 5u; }

struct Bytes32 {
    uint32_t w[8];
    __device__ __forceinline__ uint32_t get(int i) const { return (w[i >> 2] >> ((i & 3) * 8)) & 0xFFu; }
};

// 32 bytes at p (p is 16-byte aligned relative to an aligned base when `vec`)
__device__ __forceinline__ Bytes32 load32(const char *__restrict__ text, uint64_t len, uint64_t p, bool vec) {
    Bytes32 b;
    if (vec && p + 32 <= len) {
        uint4 a = __ldg(reinterpret_cast<const uint4 *>(text + p));
        uint4 c = __ldg(reinterpret_cast<const uint4 *>(text + p + 16));
        b.w[0] = a.x; b.w[1] = a.y; b.w[2] = a.z; b.w[3] = a.w;
        b.w[4] = c.x; b.w[5] = c.y; b.w[6] = c.z; b.w[7] = c.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            uint32_t v = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint64_t q = p + (uint64_t)(i * 4 + j);
                uint32_t by = q < len ? (uint32_t)(uint8_t)text[q] : 0u;
                v |= by << (8 * j);
            }
            b.w[i] = v;
        }
    }
    return b;
}

// ---- bounds: first non-whitespace byte and one past the last one
__global__ void k_bounds(const char *__restrict__ text, uint64_t len, unsigned long long *out) {
    __shared__ unsigned long long found;
    if (threadIdx.x == 0) found = ~0ULL;
    __syncthreads();
    for (uint64_t base = 0; base < len; base += blockDim.x) {
        uint64_t p = base + threadIdx.x;
        if (p < len && !is_ws((uint8_t)text[p])) atomicMin(&found, (unsigned long long)p);
        __syncthreads();
        if (found != ~0ULL) break;
        __syncthreads();
    }
    unsigned long long S = found;
    __syncthreads();
    if (threadIdx.x == 0) found = 0;
    __syncthreads();
    if (S != ~0ULL) {
        for (uint64_t base = 0; base < len; base += blockDim.x) {
            uint64_t q = base + threadIdx.x;
            if (q < len) {
                uint64_t p = len - 1 - q;
                if (!is_ws((uint8_t)text[p])) atomicMax(&found, (unsigned long long)(p + 1));
            }
            __syncthreads();
            if (found != 0) break;
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) {
        out[0] = S == ~0ULL ? len : S;
        out[1] = S == ~0ULL ? len : found;
        out[2] = S == ~0ULL ? 0 : (uint8_t)text[S];
    }
}

// Bit i set when byte p+i (p = this thread's first byte) is a '\n' inside
// [S, E).  Per 4-byte word the equal bytes are found with the exact
// zero-byte test and their top bits gathered by one multiply.
__device__ __forceinline__ uint32_t newline_bits(const ParseGeom &g, const Bytes32 &b, uint64_t p) {
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const uint32_t v = b.w[q] ^ 0x0A0A0A0Au;
        const uint32_t z = ~((((v & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | v)) & 0x80808080u;   // bit 7 of each '\n' byte
        m |= ((((z >> 7) * 0x00204081u) >> 21) & 0xFu) << (4 * q);                     // byte b -> bit b
    }
    if (p < g.S) m &= g.S - p >= 32 ? 0u : ~0u << (g.S - p);
    if (p + 32 > g.E) m &= g.E <= p ? 0u : (g.E - p >= 32 ? ~0u : (1u << (g.E - p)) - 1u);
    return m;
}

// ---- A1: newlines per tile, and each thread's newline bits for A2
// (the parsed range still on the GPU, as k_bounds found it)
__global__ void k_tile_newlines(ParseGeom g, const unsigned long long *__restrict__ bounds, uint32_t *__restrict__ tile_nl,
                                uint32_t *__restrict__ nl_bits) {
    __shared__ uint32_t sm[PT_THREADS / 32 + 1];
    g.S = bounds[0];
    g.E = bounds[1];
    uint64_t p = (uint64_t)blockIdx.x * PT_TILE + (uint64_t)threadIdx.x * PT_BYTES;
    Bytes32 b = load32(g.text, g.len, p, g.vec);
    const uint32_t m = newline_bits(g, b, p);
    nl_bits[(uint64_t)blockIdx.x * PT_THREADS + threadIdx.x] = m;
    uint32_t tot;
    block_excl_scan<uint32_t>(__popc(m), sm, &tot);
    if (threadIdx.x == 0) tile_nl[blockIdx.x] = tot;
}

// ---- A2: line ends, from the newline bits (1/8 of the text's bytes)
__global__ void k_line_ends(ParseGeom g, const uint32_t *__restrict__ nl_bits, const uint64_t *__restrict__ tile_line0,
                            uint64_t *__restrict__ line_end) {
    __shared__ uint32_t sm[PT_THREADS / 32 + 1];
    const uint64_t p = (uint64_t)blockIdx.x * PT_TILE + (uint64_t)threadIdx.x * PT_BYTES;
    uint32_t m = nl_bits[(uint64_t)blockIdx.x * PT_THREADS + threadIdx.x];
    uint32_t tot;
    uint64_t line = tile_line0[blockIdx.x] + block_excl_scan<uint32_t>(__popc(m), sm, &tot);
    while (m) {
        line_end[line++] = p + (uint32_t)(__ffs(m) - 1);
        m &= m - 1;
    }
}

// ---- L: line kinds.  FASTQ errors record the first offending line.
__global__ void k_line_kinds(ParseGeom g, const uint64_t *__restrict__ line_end, uint64_t n_lines, int fastq,
                             uint8_t *__restrict__ kind, uint32_t *__restrict__ is_hdr, uint32_t *__restrict__ len,
                             uint32_t *__restrict__ err) {
    uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_lines) return;
    uint64_t ls = j == 0 ? g.S : line_end[j - 1] + 1;
    uint64_t le = line_end[j];
    uint32_t first = le > ls ? (uint8_t)g.text[ls] : 0u;
    uint8_t kd;
    uint32_t h = 0;
    if (!fastq) {
        h = first == '>';
        kd = h ? LK_HDR : LK_SEQ;
    } else {
        uint32_t m = (uint32_t)(j & 3);
        if (m == 0) {
            h = 1;
            kd = LK_HDR;
            if (first != '@') { atomicExch(&err[DE_PARSE], 1u); atomicMin(&err[DE_PARSE + 1], (uint32_t)(j + 1)); }
        } else if (m == 1) {
            kd = LK_SEQ;
        } else {
            kd = LK_SKIP;
            if (m == 2 && first != '+') { atomicExch(&err[DE_PARSE], 1u); atomicMin(&err[DE_PARSE + 1], (uint32_t)(j + 1)); }
        }
    }
    kind[j] = kd;
    is_hdr[j] = h;
    // fast path: bytes the line emits if sequence lines hold no whitespace
    // besides their newline (checked while copying); k_line_records clears
    // lines that precede the first record
    len[j] = kd == LK_SEQ ? (uint32_t)(le - ls) : 0u;
}

// record index per line (~0 before the first header) and header line per record
__global__ void k_line_records(const uint32_t *__restrict__ is_hdr, uint64_t *__restrict__ line_rec_io, uint64_t n_lines,
                               uint64_t *__restrict__ hdr_line, uint32_t *__restrict__ len,
                               const uint32_t *__restrict__ wait_err) {
    uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_lines || *wait_err) return;   // (the scan gave up: nothing to store by)
    uint64_t incl = line_rec_io[j] + is_hdr[j];   // exclusive scan + own flag
    if (is_hdr[j]) hdr_line[incl - 1] = j;
    line_rec_io[j] = incl == 0 ? ~0ULL : incl - 1;
    if (incl == 0) len[j] = 0u;
}

// FASTQ: line j belongs to record j >> 2, whose header is line 4r
__global__ void k_fastq_records(uint64_t *__restrict__ line_rec, uint64_t n_lines, uint64_t *__restrict__ hdr_line) {
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_lines) return;
    line_rec[j] = j >> 2;
    if ((j & 3) == 0) hdr_line[j >> 2] = j;
}

// The accession of the header line [ls, le): where the first whitespace after
// its first byte is (le if there is none), and that first byte.  Aligned
// 8-byte words of the text, byte by byte at its ends: every load of a warp
// touches 32 headers, so that fewer loads are what counts.
__device__ __forceinline__ uint64_t accession_end(const ParseGeom &g, uint64_t ls, uint64_t le, uint32_t &first) {
    first = 0;
    if (ls >= le) return ls + 1;   // an empty line
    const uintptr_t text = (uintptr_t)g.text, end = text + g.len, at = text + ls;
    uintptr_t w = at & ~(uintptr_t)7;
    uint64_t q = ls + 1;
    if (w >= text) {
        uint64_t skip = ~0ULL << (8 * (uint32_t)(at & 7)) << 8;   // the bytes after the first
        if (w + 8 <= end) first = (uint32_t)(__ldg(reinterpret_cast<const unsigned long long *>(w)) >> (8 * (uint32_t)(at & 7))) & 0xFFu;
        else first = (uint8_t)g.text[ls];
        while (w + 8 <= end) {
            const uint64_t v = __ldg(reinterpret_cast<const unsigned long long *>(w));
            const uint64_t m = (((uint64_t)ws_bytes((uint32_t)(v >> 32)) << 32) | ws_bytes((uint32_t)v)) & skip;
            if (m) return min((uint64_t)(w - text) + (uint64_t)((__ffsll((long long)m) - 1) >> 3), le);
            w += 8;
            skip = ~0ULL;
            q = w - text;
            if (q >= le) return le;
        }
    } else {
        first = (uint8_t)g.text[ls];
    }
    if (q < ls + 1) q = ls + 1;
    while (q < le && !is_ws((uint8_t)g.text[q])) q++;
    return q;
}

// ---- FASTQ: records of four lines, handled per record (no per-line arrays).
// The header line starts with '@' and the third with '+' (the first offending
// line is recorded, as k_line_kinds does); the accession; the sequence line's
// length, and the longest (the reads' lengths if no line holds whitespace).
// A record's line ends are two 16-byte loads, the one before them is the
// neighbouring lane's last.  3M records: 196 us, where a pass over the records for
// the checks and one after the copy for the accessions, byte by byte, took 107
// and 188.
__global__ void k_fq_records(ParseGeom g, const uint64_t *__restrict__ line_end, uint64_t n_reads,
                             uint32_t *__restrict__ seq_len, uint64_t *__restrict__ name_off,
                             uint32_t *__restrict__ name_len, uint32_t *__restrict__ err) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t j = 4 * min(r, n_reads - 1);
    const ulonglong2 e01 = __ldg(reinterpret_cast<const ulonglong2 *>(line_end + j));
    const ulonglong2 e23 = __ldg(reinterpret_cast<const ulonglong2 *>(line_end + j + 2));
    uint64_t before = __shfl_up_sync(0xffffffffu, (unsigned long long)e23.y, 1);
    if (lane_id() == 0 && j) before = line_end[j - 1];
    uint32_t L = 0;
    if (r < n_reads) {
        const uint64_t h0 = j == 0 ? g.S : before + 1, h1 = e01.x;
        const uint64_t p0 = e01.y + 1, p1 = e23.x;
        uint32_t fh;
        const uint64_t q = accession_end(g, h0, h1, fh);
        const uint32_t fp = p1 > p0 ? (uint8_t)g.text[p0] : 0u;
        if (fh != '@') { atomicExch(&err[DE_PARSE], 1u); atomicMin(&err[DE_PARSE + 1], (uint32_t)(j + 1)); }
        if (fp != '+') { atomicExch(&err[DE_PARSE], 1u); atomicMin(&err[DE_PARSE + 1], (uint32_t)(j + 3)); }
        name_off[r] = h0 + 1;
        name_len[r] = (uint32_t)(q - (h0 + 1));
        L = (uint32_t)(e01.y - (h1 + 1));
        seq_len[r] = L;
    }
    L = __reduce_max_sync(0xffffffffu, L);
    if (lane_id() == 0 && L) atomicMax(&err[DE_MAXLEN], L);
}

// per-thread walk over its 32 bytes with the line each byte belongs to
struct LineWalk {
    uint64_t line;
    uint8_t kind;
    uint64_t rec;
};

__device__ __forceinline__ void line_info(const uint8_t *__restrict__ kind, const uint64_t *__restrict__ line_rec,
                                          uint64_t line, uint64_t n_lines, LineWalk &w) {
    w.line = line;
    if (line < n_lines) {
        w.kind = kind[line];
        w.rec = line_rec[line];
    } else {
        w.kind = LK_SKIP;
        w.rec = ~0ULL;
    }
}

// ---- B1: emitted bytes per tile
__global__ void k_tile_emits(ParseGeom g, const uint64_t *__restrict__ tile_line0, const uint8_t *__restrict__ kind,
                             const uint64_t *__restrict__ line_rec, uint64_t n_lines, uint32_t *__restrict__ tile_emit) {
    __shared__ uint32_t sm[PT_THREADS / 32 + 1];
    uint64_t p = (uint64_t)blockIdx.x * PT_TILE + (uint64_t)threadIdx.x * PT_BYTES;
    Bytes32 b = load32(g.text, g.len, p, g.vec);
    uint32_t nl = 0;
#pragma unroll
    for (int i = 0; i < PT_BYTES; i++) {
        uint64_t q = p + i;
        nl += (q >= g.S && q < g.E && b.get(i) == '\n');
    }
    uint32_t tot;
    uint64_t line = tile_line0[blockIdx.x] + block_excl_scan<uint32_t>(nl, sm, &tot);
    LineWalk w;
    line_info(kind, line_rec, line, n_lines, w);
    uint32_t em = 0;
    for (int i = 0; i < PT_BYTES; i++) {
        uint64_t q = p + i;
        if (q < g.S || q >= g.E) continue;
        uint32_t c = b.get(i);
        if (c == '\n') {
            line_info(kind, line_rec, w.line + 1, n_lines, w);
            continue;
        }
        em += (w.kind == LK_SEQ && w.rec != ~0ULL && !is_ws(c));
    }
    block_excl_scan<uint32_t>(em, sm, &tot);
    if (threadIdx.x == 0) tile_emit[blockIdx.x] = tot;
}

// ---- B2: write upper-cased bases and read starts
__global__ void k_emit(ParseGeom g, const uint64_t *__restrict__ tile_line0, const uint64_t *__restrict__ tile_emit0,
                       const uint8_t *__restrict__ kind, const uint64_t *__restrict__ line_rec, uint64_t n_lines,
                       uint8_t *__restrict__ seq, uint64_t *__restrict__ rd_off) {
    __shared__ uint32_t sm[PT_THREADS / 32 + 1];
    uint64_t p = (uint64_t)blockIdx.x * PT_TILE + (uint64_t)threadIdx.x * PT_BYTES;
    Bytes32 b = load32(g.text, g.len, p, g.vec);
    uint32_t nl = 0;
#pragma unroll
    for (int i = 0; i < PT_BYTES; i++) {
        uint64_t q = p + i;
        nl += (q >= g.S && q < g.E && b.get(i) == '\n');
    }
    uint32_t tot;
    uint64_t line = tile_line0[blockIdx.x] + block_excl_scan<uint32_t>(nl, sm, &tot);
    LineWalk w;
    line_info(kind, line_rec, line, n_lines, w);
    uint32_t em = 0;
    for (int i = 0; i < PT_BYTES; i++) {
        uint64_t q = p + i;
        if (q < g.S || q >= g.E) continue;
        uint32_t c = b.get(i);
        if (c == '\n') { line_info(kind, line_rec, w.line + 1, n_lines, w); continue; }
        em += (w.kind == LK_SEQ && w.rec != ~0ULL && !is_ws(c));
    }
    uint64_t pos = tile_emit0[blockIdx.x] + block_excl_scan<uint32_t>(em, sm, &tot);
    line_info(kind, line_rec, line, n_lines, w);
    bool nl_before = p > g.S && p - 1 < g.E && g.text[p - 1] == '\n';
    for (int i = 0; i < PT_BYTES; i++) {
        uint64_t q = p + i;
        if (q < g.S || q >= g.E) continue;
        uint32_t c = b.get(i);
        bool line_start = q == g.S || nl_before;
        nl_before = c == '\n';
        if (c == '\n') {
            line_info(kind, line_rec, w.line + 1, n_lines, w);
            continue;
        }
        if (line_start && w.kind == LK_HDR) rd_off[w.rec] = pos + w.rec;
        if (w.kind == LK_SEQ && w.rec != ~0ULL && !is_ws(c)) {
            uint32_t u = (c >= 'a' && c <= 'z') ? c - 32u : c;
            seq[pos + w.rec] = (uint8_t)u;
            pos++;
        }
    }
}

// ---- N: accession and read length per record
__global__ void k_names(ParseGeom g, const uint64_t *__restrict__ hdr_line, int fastq,
                        const uint64_t *__restrict__ line_end, uint64_t n_reads, const uint64_t *__restrict__ rd_off,
                        uint64_t *__restrict__ name_off, uint32_t *__restrict__ name_len, uint32_t *__restrict__ max_len) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t L32 = 0;
    if (r < n_reads) {
        const uint64_t j = fastq ? 4 * r : hdr_line[r];   // FASTQ: the header is line 4r
        const uint64_t ls = j == 0 ? g.S : line_end[j - 1] + 1;
        const uint64_t le = line_end[j];
        uint32_t first;
        name_off[r] = ls + 1;
        name_len[r] = (uint32_t)(accession_end(g, ls, le, first) - (ls + 1));
        const uint64_t L = rd_off[r + 1] - rd_off[r] - 1;
        L32 = (uint32_t)(L > 0xFFFFFFFFull ? 0xFFFFFFFFull : L);
    }
    // one atomic per warp (the longest read of its 32)
    L32 = __reduce_max_sync(0xffffffffu, L32);
    if (lane_id() == 0 && L32) atomicMax(max_len, L32);
}

// 32 positions of the read array as 2-bit codes and invalid-position bits, four
// bytes at a time.  Bits 1 and 2 of an upper-case A, C, T, G count 0..3 (code:
// bit 2, then bit 1 ^ bit 2) and the letter is 0x41 with those bits in, but for
// T (bit 2 without bit 1), 0x11 off: a byte that differs is invalid.  The four
// codes, and the four invalid bits, are gathered to the top of a word by one
// multiply each, whose other terms fall on lower bits of their own.
// Returns whether an invalid byte was none of 'N', 'J', '\n' and 0x0E (the
// bytes that are 0x0A under the mask 0xBB): only then can a byte be a lower-case
// letter, or whitespace inside a line.
__device__ __forceinline__ bool pack32(const uint32_t (&w)[8], uint64_t &code, uint32_t &bad) {
    uint32_t other = 0, m[8];
    bad = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const uint32_t s1 = w[q] >> 1, s2 = w[q] >> 2;
        const uint32_t x = ((s1 ^ s2) & 0x01010101u) | (s1 & 0x02020202u);
        const uint32_t t = s2 & ~s1 & 0x01010101u;
        const uint32_t d = ((w[q] & 0xF9F9F9F9u) ^ 0x41414141u) ^ t ^ (t << 4);
        const uint32_t nz = (d | ((d & 0x7F7F7F7Fu) + 0x7F7F7F7Fu)) & 0x80808080u;   // bit 7 of each differing byte
        const uint32_t dn = (w[q] & 0xBBBBBBBBu) ^ 0x0A0A0A0Au;
        other |= nz & (dn | ((dn & 0x7F7F7F7Fu) + 0x7F7F7F7Fu));
        bad = __funnelshift_l((nz >> 7) * 0x80402010u, bad, 4);                      // position 4q at bit 31
        m[q] = x * 0x40100401u;                                                        // position 4q at bits 31, 30
    }
    // the top byte of each product, the first positions at the top
    const uint32_t hi = __byte_perm(__byte_perm(m[3], m[2], 0x0073), __byte_perm(m[1], m[0], 0x0073), 0x5410);
    const uint32_t lo = __byte_perm(__byte_perm(m[7], m[6], 0x0073), __byte_perm(m[5], m[4], 0x0073), 0x5410);
    code = ((uint64_t)hi << 32) | lo;
    return other != 0u;
}

// The codes of the whole read array: thread j converts positions 32j .. 32j+31
// (j = -1 .. n_words-1; the 64 '\n' bytes around `seq` make word -1 all invalid).
// After the byte-wise emit, and for a text without reads; otherwise
// k_seq_tiles has the bases in registers and makes their codes itself.
__global__ void k_pack_codes(const uint8_t *__restrict__ seq, int64_t n_words, uint64_t *__restrict__ codes,
                             uint32_t *__restrict__ inv) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - 1;
    if (j >= n_words) return;
    const uint4 *v = reinterpret_cast<const uint4 *>(seq + 32 * j);
    const uint4 a = v[0], b = v[1];
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint64_t code;
    uint32_t bad;
    pack32(w, code, bad);
    codes[j] = code;
    inv[j] = bad;
}

// ---- fast path, copy.  The read array is cut into tiles of 8192 positions, a
// block each, 32 consecutive positions a thread.  The lines (FASTA) or records
// (FASTQ) that hold the sequence are numbered along it: line j begins at
// start(j) and holds line_len[j] bases, position start(j+1) - 1 is a separator
// if it is not a base; k_line_tiles writes which line each tile begins in.
template <bool FASTQ>
struct SeqLines {
    const uint64_t *line_end, *line_rec, *line_out;   // (line_rec: FASTA)
    const uint32_t *line_len;
    uint64_t n, S, seq_len;
    __device__ __forceinline__ uint64_t start(uint64_t j) const {
        if (j >= n) return seq_len;
        if (FASTQ) return line_out[j] + j;
        const uint64_t rec = line_rec[j];
        return line_out[j] + (rec == ~0ULL ? 0 : rec);   // (lines before the first record are empty)
    }
    __device__ __forceinline__ uint64_t src(uint64_t j) const {
        return FASTQ ? line_end[4 * j] + 1 : j == 0 ? S : line_end[j - 1] + 1;
    }
};

constexpr int ST_THREADS = 256;
constexpr int ST_BLOCKS = 6;         // an SM: 42 registers a thread
constexpr uint32_t ST_TILE = ST_THREADS * 32;
constexpr uint32_t ST_LINES = 512;   // lines of a tile held in shared memory at a time
// Lines of a tile from which each thread looks its lines up in memory instead:
// blank lines and empty records take few positions or none, so there is no
// bound to a tile's lines, and one block would go through all of them (2.4 us for
// 512: 400,000 reads with 300,000 blank lines in one place 1.69 ms against 0.25
// this way, with 100,000 empty records among them 0.49 against 0.30).  Reads of four
// bases have 3300 lines a tile; from 1024 to 8192 lines the time is the same.
constexpr uint32_t ST_DENSE = 8 * ST_LINES;

// Per line: its record's start, and the tiles whose first position it holds.
template <bool FASTQ>
__global__ void k_line_tiles(SeqLines<FASTQ> L, const uint8_t *__restrict__ kind, uint64_t *__restrict__ rd_off,
                             uint64_t *__restrict__ tile_line) {
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= L.n) return;
    const uint64_t s = L.start(j), e = L.start(j + 1);
    if (FASTQ) rd_off[j] = s;
    else if (kind[j] == LK_HDR) rd_off[L.line_rec[j]] = s;
    for (uint64_t t = (s + ST_TILE - 1) / ST_TILE; t * ST_TILE < e; t++) tile_line[t] = j;
}

// x = v from byte a (0..31) on
__device__ __forceinline__ void lay_from(uint32_t (&x)[8], const uint32_t (&v)[8], uint32_t a) {
#pragma unroll
    for (int w = 0; w < 8; w++) {
        const uint32_t from = __funnelshift_lc(0u, ~0u, (uint32_t)max((int)(8 * a) - 32 * w, 0));
        x[w] = (x[w] & ~from) | (v[w] & from);
    }
}

// Copies the sequence lines, upper-cased and with a '\n' after every read, and
// makes their 2-bit codes.  A thread finds the line of its first position by a
// binary search over the tile's lines in shared memory, loads the 32 text bytes
// around each stretch of a line (three aligned 16-byte loads and shifts), lays
// each next stretch over the words from its first position on, and stores
// whole 32-byte pieces.  A byte that may be a lower-case letter or whitespace
// (pack32) takes the slower way of upper-casing; whitespace sets *ws_seen and the
// byte-wise path redoes the emit.  The bytes around seq become '\n' too.
// Bound by instructions and, for each block, by three dependent
// loads before its first base: 3M reads of 100 nt took 377 us with 4 blocks to
// an SM, 287 with 5, 262 with 6, 380 with 7 (spills).  The warps that copied 32
// lines in aligned 16-byte words, the fill of the array with '\n' and the pass
// that made the codes took 286 and 118 us for them, and the fill's 330 MB.
template <bool FASTQ>
__global__ void __launch_bounds__(ST_THREADS, ST_BLOCKS) k_seq_tiles(const char *__restrict__ text, uint64_t len, SeqLines<FASTQ> L,
                                                         const uint64_t *__restrict__ tile_line, uint64_t n_words,
                                                         uint8_t *__restrict__ seq, uint64_t seq_bytes,
                                                         uint64_t *__restrict__ codes, uint32_t *__restrict__ inv,
                                                         uint32_t *__restrict__ ws_seen) {
    __shared__ uint32_t s_start[ST_LINES + 1], s_end[ST_LINES];
    __shared__ int64_t s_delta[ST_LINES];   // text position of a base less its place in seq
    const uint64_t T0 = (uint64_t)blockIdx.x * ST_TILE;
    const uint32_t q0 = threadIdx.x * 32u;
    const uint32_t sep[8] = {0x0A0A0A0Au, 0x0A0A0A0Au, 0x0A0A0A0Au, 0x0A0A0A0Au,
                             0x0A0A0A0Au, 0x0A0A0A0Au, 0x0A0A0A0Au, 0x0A0A0A0Au};
    uint32_t x[8], held = 0;                // held: positions that are bases
#pragma unroll
    for (int w = 0; w < 8; w++) x[w] = sep[w];
    // lays the bases of a line on [q, e) of the tile (e past the thread's last position: cut there)
    auto lay_line = [&](uint32_t q, uint32_t e, int64_t delta) {
        // the text byte that would lie at this thread's first position
        const int64_t at = (int64_t)(T0 + q0) + delta;
        const uint32_t a = q - q0;
        const uintptr_t p = (uintptr_t)text + (uintptr_t)at, p16 = p & ~(uintptr_t)15;
        uint32_t v[8];
        if (p16 >= (uintptr_t)text && p16 + 48 <= (uintptr_t)text + len) {
            const uint4 *u = reinterpret_cast<const uint4 *>(p16);
            const uint4 u0 = __ldg(u), u1 = __ldg(u + 1), u2 = __ldg(u + 2);
            uint32_t t[12] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w, u2.x, u2.y, u2.z, u2.w};
            if (p & 8) {
#pragma unroll
                for (int w = 0; w < 10; w++) t[w] = t[w + 2];
            }
            if (p & 4) {
#pragma unroll
                for (int w = 0; w < 9; w++) t[w] = t[w + 1];
            }
            const uint32_t sh = 8u * (uint32_t)(p & 3);
#pragma unroll
            for (int w = 0; w < 8; w++) v[w] = __funnelshift_r(t[w], t[w + 1], sh);
        } else {   // at an end of the text
#pragma unroll
            for (int w = 0; w < 8; w++) {
                v[w] = 0;
                for (uint32_t i4 = 0; i4 < 4; i4++) {
                    const uint32_t o = 4 * w + i4;
                    if (o >= a && q0 + o < e) v[w] |= (uint32_t)(uint8_t)text[at + o] << (8 * i4);
                }
            }
        }
        lay_from(x, v, a);
        if (e < q0 + 32u) lay_from(x, sep, e - q0);
        held |= (e - q0 >= 32u ? ~0u : (1u << (e - q0)) - 1u) & (~0u << a);
    };
    if (T0 < L.seq_len) {
        const uint32_t lim = (uint32_t)min((uint64_t)ST_TILE, L.seq_len - T0);
        const uint32_t qe = min(q0 + 32u, lim);
        const uint64_t first = tile_line[blockIdx.x];
        const uint64_t last = T0 + ST_TILE < L.seq_len ? tile_line[blockIdx.x + 1] : L.n - 1;
        uint32_t q = q0;
        if (last - first >= ST_DENSE) {
            // a line at a time from memory: the last line that begins at or before q
            uint64_t i = first, hi = last + 1;
            while (hi - i > 1) {
                const uint64_t mid = (i + hi) >> 1;
                if (L.start(mid) <= T0 + q) i = mid;
                else hi = mid;
            }
            while (q < qe) {
                const uint64_t s = L.start(i), e = s + L.line_len[i];
                if (e > T0 + q) lay_line(q, (uint32_t)min(e - T0, (uint64_t)qe), (int64_t)L.src(i) - (int64_t)s);
                q = (uint32_t)min(L.start(i + 1) - T0, (uint64_t)qe);
                uint64_t step = 1;   // on to the line of the new q, in doubling steps and back
                while (i + step <= last && L.start(i + step) <= T0 + q) {
                    i += step;
                    step *= 2;
                }
                for (; step; step >>= 1)
                    if (i + step <= last && L.start(i + step) <= T0 + q) i += step;
            }
        }
        for (uint64_t c0 = first; last - first < ST_DENSE && c0 <= last; c0 += ST_LINES) {
            const uint32_t m = (uint32_t)min((uint64_t)ST_LINES, last - c0 + 1);
            if (c0 != first) __syncthreads();
            for (uint32_t i = threadIdx.x; i <= m; i += ST_THREADS) {
                const uint64_t j = c0 + i, s = L.start(j);
                s_start[i] = s <= T0 ? 0u : (uint32_t)min(s - T0, (uint64_t)ST_TILE);
                if (i < m) {
                    const uint64_t e = s + L.line_len[j];
                    s_end[i] = e <= T0 ? 0u : (uint32_t)min(e - T0, (uint64_t)ST_TILE);
                    s_delta[i] = (int64_t)L.src(j) - (int64_t)s;
                }
            }
            __syncthreads();
            const uint32_t stop = min(qe, s_start[m]);
            if (q < stop) {
                uint32_t i = 0, hi = m;   // the last line that begins at or before q
                while (hi - i > 1) {
                    const uint32_t mid = (i + hi) >> 1;
                    if (s_start[mid] <= q) i = mid;
                    else hi = mid;
                }
                while (q < stop) {
                    while (s_start[i + 1] <= q) i++;
                    const uint32_t e = min(s_end[i], qe);
                    if (e > q) lay_line(q, e, s_delta[i]);
                    q = min(s_start[i + 1], stop);
                }
            }
        }
    }
    const uint64_t word = T0 / 32 + threadIdx.x;
    if (word < n_words) {
        uint64_t code;
        uint32_t bad;
        if (pack32(x, code, bad)) {
            bool ws = false;
#pragma unroll
            for (int w = 0; w < 8; w++) {
                const uint32_t in = ((((held >> (4 * w)) & 0xFu) * 0x00204081u) & 0x01010101u) * 0xFFu;
                x[w] = (upcase_word((x[w] & in) | (0x41414141u & ~in), ws) & in) | (0x0A0A0A0Au & ~in);
            }
            if (ws) *ws_seen = 1u;   // (an atomic per line of a CRLF text took four times the copy)
            pack32(x, code, bad);
        }
        uint4 *o = reinterpret_cast<uint4 *>(seq + 32 * word);
        o[0] = make_uint4(x[0], x[1], x[2], x[3]);
        o[1] = make_uint4(x[4], x[5], x[6], x[7]);
        codes[word] = code;
        inv[word] = bad;
    }
    if (blockIdx.x == 0) {
        if (threadIdx.x < SEQ_PAD / 4) reinterpret_cast<uint32_t *>(seq - SEQ_PAD)[threadIdx.x] = 0x0A0A0A0Au;
        for (uint64_t i = 32 * n_words + threadIdx.x; i < seq_bytes; i += ST_THREADS) seq[i] = (uint8_t)'\n';
        if (threadIdx.x == 0) {
            uint64_t code;
            uint32_t bad;
            pack32(sep, code, bad);
            codes[-1] = code;
            inv[-1] = bad;
        }
    }
}

// Component id of every bundle record: the integer after "s_" in its
// accession, else the record ordinal.  (Parsed on the host, a bundle in GPU
// memory had its whole text copied back for them: 0.87 of 2.59 ms for 14 MB.)
__global__ void k_component_ids(const char *__restrict__ text, const uint64_t *__restrict__ name_off,
                                const uint32_t *__restrict__ name_len, uint64_t n, uint64_t *__restrict__ ids) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const char *h = text + name_off[i];
    const uint32_t L = name_len[i];
    uint64_t id = i;
    if (L > 2 && h[0] == 's' && h[1] == '_' && h[2] >= '0' && h[2] <= '9') {
        id = 0;
        for (uint32_t j = 2; j < L && h[j] >= '0' && h[j] <= '9'; j++) id = id * 10 + (uint64_t)(h[j] - '0');
    }
    ids[i] = id;
}

static inline unsigned grid_for(uint64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

int component_ids(tk_ctx *c, const tk_reads *b, uint64_t *d_ids) {
    if (b->n_reads == 0) return TK_OK;
    k_component_ids<<<grid_for(b->n_reads, 256), 256, 0, c->stream>>>(b->d_text, b->d_name_off, b->d_name_len, b->n_reads,
                                                                       d_ids);
    c->launches++;
    return check_launch(c, "component ids");
}

constexpr uint64_t PARSE_FEW_LINES = 1ull << 22;   // 32 MB of header lines; a round trip is 1% of their 1.2 ms

static uint64_t code_words(const tk_reads *r) { return (r->seq_len + 31) / 32 + 1; }   // without word -1

static int alloc_codes(tk_ctx *c, tk_reads *r) {
    const uint64_t words = code_words(r) + 1;   // incl. word -1
    const uint64_t inv_words = (words + 1) & ~1ULL;
    TK_TRY(dmalloc(c, (void **)&r->d_pack_alloc, words * 8 + inv_words * 4, "2-bit codes"));
    r->d_codes = r->d_pack_alloc + 1;
    r->d_inv = reinterpret_cast<uint32_t *>(r->d_pack_alloc + words) + 1;
    return TK_OK;
}

// r->d_codes / r->d_inv from r->d_seq
static int pack_reads(tk_ctx *c, tk_reads *r) {
    TK_TRY(alloc_codes(c, r));
    const uint64_t n = code_words(r);
    k_pack_codes<<<grid_for(n + 1, 256), 256, 0, c->stream>>>(r->d_seq, (int64_t)n, const_cast<uint64_t *>(r->d_codes),
                                                              const_cast<uint32_t *>(r->d_inv));
    c->launches++;
    return check_launch(c, "2-bit codes");
}

template <bool FASTQ>
static int copy_sequences(tk_ctx *c, tk_reads *r, const SeqLines<FASTQ> &L, const uint8_t *kind, uint64_t seq_bytes) {
    TK_TRY(alloc_codes(c, r));
    const uint64_t words = code_words(r), tiles = (words * 32 + ST_TILE - 1) / ST_TILE;
    uint64_t *tile_line = nullptr;
    TK_TRY(dmalloc(c, (void **)&tile_line, tiles * 8, "sequence tiles"));
    k_line_tiles<FASTQ><<<grid_for(L.n, 256), 256, 0, c->stream>>>(L, kind, r->d_rd_off, tile_line);
    k_seq_tiles<FASTQ><<<(unsigned)tiles, ST_THREADS, 0, c->stream>>>(
        r->d_text, r->text_len, L, tile_line, words, r->d_seq, seq_bytes, const_cast<uint64_t *>(r->d_codes),
        const_cast<uint32_t *>(r->d_inv), c->d_err + DE_WS);
    c->launches += 2;
    dfree(c, tile_line);
    return check_launch(c, "sequence copy");
}

int parse_reads(tk_ctx *c, tk_reads *r) {
    const char *text = r->d_text;
    uint64_t len = r->text_len;
    unsigned long long *d_bounds = nullptr;
    cudaEvent_t ev;
    prof_begin(c, TK_KID_PARSE, &ev);
    // What the host has to know comes back at three synchronisations: the
    // parsed range and the lines; the reads and their bases; whether sequence
    // lines held whitespace, and the longest read.  (A round trip takes about
    // 10 us, one bin of 2000 reads 600.)
    TK_TRY(dmalloc(c, (void **)&d_bounds, 4 * sizeof(unsigned long long), "parse bounds"));   // [3]: records
    k_bounds<<<1, 256, 0, c->stream>>>(text, len, d_bounds);
    c->launches++;
    volatile unsigned long long *hb = reinterpret_cast<volatile unsigned long long *>(c->h_stage);
    int e = TK_OK;
    ParseGeom g;
    g.text = text;
    g.len = len;
    g.S = g.E = 0;
    g.vec = ((uintptr_t)text & 15u) == 0;
    r->format = TK_FMT_NONE;
    int fastq = 0;

    const uint64_t all_tiles = (len + PT_TILE - 1) / PT_TILE;
    uint64_t n_tiles = 0;
    uint32_t *tile_nl = nullptr, *tile_em = nullptr, *is_hdr = nullptr, *nl_bits = nullptr;
    uint64_t *tile_line0 = nullptr, *tile_emit0 = nullptr, *line_end = nullptr, *line_rec = nullptr, *hdr_line = nullptr;
    uint32_t *line_len = nullptr;
    uint64_t *line_out = nullptr;
    uint8_t *kind = nullptr;
    uint32_t *d_maxlen = c->d_err + DE_MAXLEN;
    uint64_t n_nl = 0, n_lines = 0, n_reads = 0, n_emit = 0;
    std::vector<void *> tmp;
    auto alloc = [&](void **p, size_t bytes, const char *what) {
        int ee = dmalloc(c, p, bytes ? bytes : 16, what);
        if (!ee) tmp.push_back(*p);
        return ee;
    };
    do {
        if (all_tiles == 0) break;
        if ((e = alloc((void **)&tile_nl, all_tiles * 4, "tile newlines"))) break;
        if ((e = alloc((void **)&tile_line0, (all_tiles + 1) * 8, "tile lines"))) break;
        if ((e = alloc((void **)&nl_bits, all_tiles * PT_THREADS * 4, "newline bits"))) break;
        k_tile_newlines<<<(unsigned)all_tiles, PT_THREADS, 0, c->stream>>>(g, d_bounds, tile_nl, nl_bits);
        c->launches++;
        if ((e = cuda_check(c, cudaMemcpyAsync(c->h_stage, d_bounds, 24, cudaMemcpyDeviceToHost, c->stream), "bounds d2h"))) break;
        if ((e = scan_excl_u32_to_u64(c, tile_nl, tile_line0, all_tiles, &n_nl))) break;   // syncs
        g.S = hb[0];
        g.E = hb[1];
        if (g.S >= g.E) break;   // nothing but whitespace
        n_tiles = all_tiles;
        r->format = hb[2] == '@' ? TK_FMT_FASTQ : TK_FMT_FASTA;
        fastq = r->format == TK_FMT_FASTQ;
        n_lines = n_nl + 1;
        if ((e = alloc((void **)&line_end, n_lines * 8, "line ends"))) break;
        k_line_ends<<<(unsigned)n_tiles, PT_THREADS, 0, c->stream>>>(g, nl_bits, tile_line0, line_end);
        c->launches++;
        if ((e = cuda_check(c, cudaMemcpyAsync(line_end + n_nl, &g.E, 8, cudaMemcpyHostToDevice, c->stream), "line end"))) break;
        if (fastq && (n_lines & 3) != 0) {
            e = set_err(c, TK_E_PARSE, "FASTQ input: " + std::to_string(n_lines) + " lines is not a multiple of 4");
            break;
        }
        if ((e = cuda_check(c, cudaMemsetAsync(c->d_err, 0, DE_COUNT * 4, c->stream), "err reset"))) break;
        uint32_t big = 0xFFFFFFFFu;
        cudaMemcpyAsync(c->d_err + DE_PARSE + 1, &big, 4, cudaMemcpyHostToDevice, c->stream);
        uint32_t herr[2] = {0, 0};
        if (fastq) {
            // 4-line records, handled per record: checks and sequence lengths,
            // their scan gives every read's place in seq
            n_reads = n_lines / 4;
            if ((e = alloc((void **)&line_len, n_reads * 4, "sequence lengths"))) break;
            if ((e = dmalloc(c, (void **)&r->d_name_off, n_reads * 8, "name offsets"))) break;
            if ((e = dmalloc(c, (void **)&r->d_name_len, n_reads * 4, "name lengths"))) break;
            k_fq_records<<<grid_for(n_reads, 256), 256, 0, c->stream>>>(g, line_end, n_reads, line_len, r->d_name_off,
                                                                        r->d_name_len, c->d_err);
            c->launches++;
            if ((e = cuda_check(c, cudaMemcpyAsync(herr, c->d_err + DE_PARSE, 8, cudaMemcpyDeviceToHost, c->stream), "err d2h"))) break;
            if ((e = alloc((void **)&line_out, (n_reads + 1) * 8, "sequence offsets"))) break;
            if ((e = scan_excl_u32_to_u64(c, line_len, line_out, n_reads, &n_emit))) break;   // syncs
            if (herr[0]) {
                e = set_err(c, TK_E_PARSE, "FASTQ input: malformed record at line " + std::to_string(herr[1]));
                break;
            }
            break;
        }
        if ((e = alloc((void **)&kind, n_lines, "line kinds"))) break;
        if ((e = alloc((void **)&is_hdr, n_lines * 4, "header flags"))) break;
        if ((e = alloc((void **)&line_rec, n_lines * 8, "line records"))) break;
        if ((e = alloc((void **)&line_len, n_lines * 4, "line lengths"))) break;
        k_line_kinds<<<grid_for(n_lines, 256), 256, 0, c->stream>>>(g, line_end, n_lines, fastq, kind, is_hdr, line_len,
                                                                     c->d_err);
        c->launches++;
        // few lines: room for a record at each instead of a round trip for their number
        const bool few = n_lines <= PARSE_FEW_LINES;
        if (few) e = scan_excl_u32_to_u64_async(c, is_hdr, line_rec, n_lines, (uint64_t *)d_bounds + 3);
        else e = scan_excl_u32_to_u64(c, is_hdr, line_rec, n_lines, &n_reads);   // syncs
        if (e) break;
        if ((e = alloc((void **)&hdr_line, ((few ? n_lines : n_reads) + 1) * 8, "header lines"))) break;
        k_line_records<<<grid_for(n_lines, 256), 256, 0, c->stream>>>(is_hdr, line_rec, n_lines, hdr_line, line_len,
                                                                      c->d_err + DE_COUNT);
        c->launches++;
        if ((e = alloc((void **)&line_out, (n_lines + 1) * 8, "line outputs"))) break;
        if (few && (e = cuda_check(c, cudaMemcpyAsync(c->h_stage, d_bounds + 3, 8, cudaMemcpyDeviceToHost, c->stream), "records d2h"))) break;
        if ((e = scan_excl_u32_to_u64(c, line_len, line_out, n_lines, &n_emit))) break;   // syncs
        if (few) n_reads = hb[0];
    } while (0);
    dfree(c, d_bounds);
    if (e) {
        for (void *p : tmp) dfree(c, p);
        return e;
    }
    r->n_reads = n_reads;
    r->n_bases = n_emit;
    r->seq_len = n_emit + n_reads;
    uint64_t seq_alloc = ((r->seq_len + 2 * SEQ_PAD + 15) / 16) * 16 + 16;
    e = dmalloc(c, (void **)&r->d_seq_alloc, seq_alloc, "packed reads");
    if (!e) e = dmalloc(c, (void **)&r->d_rd_off, (n_reads + 1) * 8, "read offsets");
    if (!e && !r->d_name_off) e = dmalloc(c, (void **)&r->d_name_off, (n_reads ? n_reads : 1) * 8, "name offsets");
    if (!e && !r->d_name_len) e = dmalloc(c, (void **)&r->d_name_len, (n_reads ? n_reads : 1) * 4, "name lengths");
    if (!e) {
        r->d_seq = r->d_seq_alloc + SEQ_PAD;
        if (!n_tiles) cudaMemsetAsync(c->d_err, 0, DE_COUNT * 4, c->stream);   // whitespace seen, the longest read
        uint64_t tail = r->seq_len;
        cudaMemcpyAsync(r->d_rd_off + n_reads, &tail, 8, cudaMemcpyHostToDevice, c->stream);
        uint32_t ws_seen = 0;
        // accessions and read lengths (unless k_fq_records had them), and what the host reads back
        auto finish = [&](bool names) -> int {
            if (n_tiles && n_reads && names) {
                k_names<<<grid_for(n_reads, 256), 256, 0, c->stream>>>(g, hdr_line, fastq, line_end, n_reads, r->d_rd_off,
                                                                       r->d_name_off, r->d_name_len, d_maxlen);
                c->launches++;
            }
            TK_CUDA(c, cudaMemcpyAsync(c->h_stage, c->d_err + DE_WS, 8, cudaMemcpyDeviceToHost, c->stream));
            TK_CUDA(c, cudaStreamSynchronize(c->stream));
            TK_TRY(wait_status(c));
            const volatile uint32_t *h = reinterpret_cast<volatile uint32_t *>(c->h_stage);
            ws_seen = h[0];
            r->max_len = h[1];
            return TK_OK;
        };
        const uint64_t seq_bytes = seq_alloc - SEQ_PAD;
        if (n_tiles && n_reads && fastq) {
            e = copy_sequences(c, r, SeqLines<true>{line_end, nullptr, line_out, line_len, n_reads, g.S, r->seq_len}, nullptr, seq_bytes);
        } else if (n_tiles && n_reads) {
            e = copy_sequences(c, r, SeqLines<false>{line_end, line_rec, line_out, line_len, n_lines, g.S, r->seq_len}, kind, seq_bytes);
        } else {
            cudaMemsetAsync(r->d_seq_alloc, '\n', seq_alloc, c->stream);
            e = pack_reads(c, r);
        }
        if (!e) e = finish(!fastq);
        r->plain_seq = fastq && !ws_seen;
        if (!e && ws_seen) {
            // some sequence line holds spaces, tabs or CRs: redo the emit byte by byte
            do {
                if (fastq) {
                    // the byte-wise emit works from the per-line arrays
                    if ((e = alloc((void **)&kind, n_lines, "line kinds"))) break;
                    if ((e = alloc((void **)&is_hdr, n_lines * 4, "header flags"))) break;
                    if ((e = alloc((void **)&line_rec, n_lines * 8, "line records"))) break;
                    uint32_t *ll = nullptr;
                    uint64_t *hl = nullptr;
                    if ((e = alloc((void **)&ll, n_lines * 4, "line lengths"))) break;
                    if ((e = alloc((void **)&hl, (n_reads + 1) * 8, "header lines"))) break;
                    k_line_kinds<<<grid_for(n_lines, 256), 256, 0, c->stream>>>(g, line_end, n_lines, fastq, kind, is_hdr,
                                                                                 ll, c->d_err);
                    k_fastq_records<<<grid_for(n_lines, 256), 256, 0, c->stream>>>(line_rec, n_lines, hl);
                    c->launches += 2;
                }
                if ((e = alloc((void **)&tile_em, n_tiles * 4, "tile emits"))) break;
                if ((e = alloc((void **)&tile_emit0, (n_tiles + 1) * 8, "tile emit offsets"))) break;
                k_tile_emits<<<(unsigned)n_tiles, PT_THREADS, 0, c->stream>>>(g, tile_line0, kind, line_rec, n_lines, tile_em);
                c->launches++;
                if ((e = scan_excl_u32_to_u64(c, tile_em, tile_emit0, n_tiles, &n_emit))) break;
                r->n_bases = n_emit;
                r->seq_len = n_emit + n_reads;
                tail = r->seq_len;
                cudaMemsetAsync(r->d_seq_alloc, '\n', seq_alloc, c->stream);
                cudaMemcpyAsync(r->d_rd_off + n_reads, &tail, 8, cudaMemcpyHostToDevice, c->stream);
                k_emit<<<(unsigned)n_tiles, PT_THREADS, 0, c->stream>>>(g, tile_line0, tile_emit0, kind, line_rec, n_lines,
                                                                       r->d_seq, r->d_rd_off);
                c->launches++;
                dfree(c, r->d_pack_alloc);   // of the lines as they were
                r->d_pack_alloc = nullptr;
                cudaMemsetAsync(d_maxlen, 0, 4, c->stream);
                if (!(e = pack_reads(c, r))) e = finish(true);
            } while (0);
        }
    }
    for (void *p : tmp) dfree(c, p);
    prof_end(c, TK_KID_PARSE, ev, r->text_len);
    return e;
}

}  // namespace tk
