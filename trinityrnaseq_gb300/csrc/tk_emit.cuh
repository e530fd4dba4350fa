// tk_emit.cuh -- text formatting by blocks: every thread writes its line into the
// block's shared-memory buffer and the block stores the lines' bytes together.
#pragma once
#include "tk_internal.cuh"

namespace tk {

__device__ __forceinline__ uint32_t dec_digits(uint32_t v) {
    uint32_t d = 1;
    while (v >= 10) { v /= 10; d++; }
    return d;
}

// v in decimal at p (d = its digits); returns the byte after it
__device__ __forceinline__ char *put_dec(char *p, uint32_t v, uint32_t d) {
    for (uint32_t i = d; i >= 1; i--) {
        p[i - 1] = (char)('0' + v % 10);
        v /= 10;
    }
    return p + d;
}

// The letters of four 2-bit codes (the first in the top two of eight bits),
// the first letter in the low byte.
__device__ __forceinline__ uint32_t base_letters(uint32_t b) {
    const uint32_t sel = (b >> 6) | (b & 0x30u) | ((b & 0x0Cu) << 6) | ((b & 3u) << 12);
    return __byte_perm(0x54474341u, 0u, sel);   // "ACGT"
}

// The k bases of a key and a newline at p (shared memory, any alignment): byte
// stores up to the first aligned word, words of four letters from there on.
__device__ __forceinline__ void put_kmer_line(char *p, uint64_t key, int k) {
    const uint64_t x = key << (64 - 2 * k);                           // the first base in the top bits
    const int a = (int)((4u - ((uint32_t)(uintptr_t)p & 3u)) & 3u);   // bytes before the first aligned word
    const uint32_t head = base_letters((uint32_t)(x >> 56));
#pragma unroll
    for (int i = 0; i < 3; i++)
        if (i < a && i < k) p[i] = (char)(head >> (8 * i));
    if (k > a) {
        const uint64_t y = x << (2 * a);
        const int words = (k - a) >> 2, rest = (k - a) & 3;
        uint32_t *q = reinterpret_cast<uint32_t *>(p + a);
#pragma unroll
        for (int w = 0; w < (MAX_K + 3) / 4; w++)
            if (w < words) q[w] = base_letters((uint32_t)(y >> (56 - 8 * w)) & 0xFFu);
        const uint32_t tail = base_letters((uint32_t)((y << (8 * words & 63)) >> 56));
#pragma unroll
        for (int i = 0; i < 3; i++)
            if (i < rest) p[a + 4 * words + i] = (char)(tail >> (8 * i));
    }
    p[k] = '\n';
}

// Stores the n bytes the block's threads wrote at buf + (w0 & 15) to out + w0
// in aligned 16-byte pieces (buf and out 16-byte aligned); the first and the
// last piece, shared with other blocks' lines, byte by byte.
__device__ __forceinline__ void block_store(const char *buf, char *__restrict__ out, uint64_t w0, uint32_t n) {
    const uint32_t lo = (uint32_t)(w0 & 15), hi = lo + n;
    char *o = out + (w0 & ~15ULL);
    for (uint32_t c = threadIdx.x * 16; c < hi; c += blockDim.x * 16) {
        if (c >= lo && c + 16 <= hi) {
            *reinterpret_cast<uint4 *>(o + c) = *reinterpret_cast<const uint4 *>(buf + c);
        } else {
            for (uint32_t b = max(c, lo); b < min(c + 16, hi); b++) o[b] = buf[b];
        }
    }
}

}  // namespace tk
