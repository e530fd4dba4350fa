// tk_text.cuh -- the parsed text's geometry, upper-casing, and copying
// stretches of the input text with whole warps (the FASTA writer).
#pragma once
#include "tk_internal.cuh"

namespace tk {

struct ParseGeom {
    const char *text;
    uint64_t len;
    uint64_t S, E;        // parsed byte range (leading/trailing whitespace trimmed)
    bool vec;
};

// Byte mask of the bytes [a, b) of a 4-byte word (0 <= a, b <= 4).
__device__ __forceinline__ uint32_t byte_mask(int a, int b) {
    return b > a ? (0xFFFFFFFFu >> (32 - 8 * (b - a))) << (8 * a) : 0u;
}

// The 16 bytes at offset so of a line of n bytes starting at text position
// S, as four words, and per word the mask of its bytes inside the line
// (bytes outside it read as 'A').  Five aligned 4-byte loads and funnel
// shifts when the text is aligned and they lie inside it, byte loads
// otherwise.
__device__ __forceinline__ void line_word16(const ParseGeom &g, uint64_t S, int64_t so, uint32_t n, uint32_t (&x)[4],
                                            uint32_t (&in)[4]) {
    const int64_t rest = (int64_t)n - so;                    // bytes [lo, hi) are in the line
    const int lo = so < 0 ? (so < -16 ? 16 : (int)-so) : 0;
    const int hi = rest < 16 ? (rest < 0 ? 0 : (int)rest) : 16;
#pragma unroll
    for (int q = 0; q < 4; q++) in[q] = byte_mask(min(max(lo - 4 * q, 0), 4), min(max(hi - 4 * q, 0), 4));
    const int64_t a = (int64_t)S + so;
    if (g.vec && a >= 0 && (uint64_t)((a & ~3LL) + 20) <= g.len) {
        const uint32_t *p = reinterpret_cast<const uint32_t *>(g.text + (a & ~3LL));
        const uint32_t sh = 8u * (uint32_t)(a & 3);
        uint32_t w[5];
#pragma unroll
        for (int i = 0; i < 5; i++) w[i] = __ldg(p + i);
#pragma unroll
        for (int q = 0; q < 4; q++) x[q] = (__funnelshift_r(w[q], w[q + 1], sh) & in[q]) | (0x41414141u & ~in[q]);
        return;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        x[q] = 0;
        for (int i = 0; i < 4; i++) {
            const int64_t o = so + 4 * q + i;
            const uint32_t c = (o >= 0 && o < (int64_t)n) ? (uint8_t)g.text[S + o] : 0x41u;
            x[q] |= c << (8 * i);
        }
    }
}

// Bit 7 of each byte of a word that is whitespace (' ' or 9..13).
__device__ __forceinline__ uint32_t ws_bytes(uint32_t x) {
    const uint32_t t = x & 0x7F7F7F7Fu, sp = x ^ 0x20202020u;
    const uint32_t zsp = ~(((sp & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | sp);
    const uint32_t rng = (t + 0x77777777u) & ~(t + 0x72727272u) & ~x;
    return (zsp | rng) & 0x80808080u;
}

// Upper-cases a word of bases; notes whether it held whitespace.
__device__ __forceinline__ uint32_t upcase_word(uint32_t x, bool &ws) {
    const uint32_t t = x & 0x7F7F7F7Fu;
    // bit 7 of each byte that is a-z
    const uint32_t lower = (t + 0x1F1F1F1Fu) & ~(t + 0x05050505u) & ~x & 0x80808080u;
    ws |= ws_bytes(x) != 0u;
    return x ^ (lower >> 2);
}

// The warp copies the lines its lanes hold (lane l: text[src, src + len) to
// seq + dst; len 0 = none).  The output is cut into the aligned 16-byte words the
// lines touch; the warp numbers the words of its 32 lines one after another (a scan
// of each line's word count) and each lane takes every 32nd, so the lanes stay
// busy whatever the line lengths; a lane finds its word's line by a binary
// search over the lanes' first word numbers.  A word wholly inside its line
// is one 16-byte store; the first and last word of a line (shared with the
// separator and the neighbouring line) are stored byte by byte.  seq is
// 16-byte aligned.
__device__ __forceinline__ void copy_group(const ParseGeom &g, uint64_t src, uint64_t dst, uint32_t len,
                                           uint8_t *__restrict__ seq) {
    const unsigned lane = lane_id();
    const uint32_t nw = len ? (uint32_t)(((dst + len + 15) >> 4) - (dst >> 4)) : 0u;
    uint32_t incl = nw;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (unsigned)o) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t first = incl - nw;   // this lane's line's first word number
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t t = base + lane;
        // the last lane whose first word number is <= t: its line holds word t
        // (a line without words shares its first number with the next line)
        int i = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const uint32_t f = __shfl_sync(0xffffffffu, first, (i + step) & 31);
            if (i + step < 32 && f <= t) i += step;
        }
        const uint64_t s_i = __shfl_sync(0xffffffffu, src, i);
        const uint64_t d_i = __shfl_sync(0xffffffffu, dst, i);
        const uint32_t n_i = __shfl_sync(0xffffffffu, len, i);
        const uint32_t f_i = __shfl_sync(0xffffffffu, first, i);
        if (t >= total) continue;
        const uint64_t out = (d_i & ~15ULL) + 16ull * (t - f_i);   // the word's first output byte
        const int64_t so = (int64_t)out - (int64_t)d_i;            // its offset in the line
        uint32_t x[4], in[4];
        line_word16(g, s_i, so, n_i, x, in);
        uint8_t *o = seq + out;
        if (so >= 0 && so + 16 <= (int64_t)n_i) {
            *reinterpret_cast<uint4 *>(o) = make_uint4(x[0], x[1], x[2], x[3]);
        } else {
            // a line's first or last word: whole 4-byte pieces inside the
            // line as words, the piece cut by a line end byte by byte
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (in[q] == 0xFFFFFFFFu) {
                    reinterpret_cast<uint32_t *>(o)[q] = x[q];
                } else if (in[q]) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if ((in[q] >> (8 * i)) & 0xFFu) o[4 * q + i] = (uint8_t)(x[q] >> (8 * i));
                }
            }
        }
    }
}

}  // namespace tk
