// tk_windows.cuh -- windows of k bases cut from the 2-bit codes, a stretch of
// positions per thread (the counting passes and the bundle's table).
#pragma once
#include "tk_internal.cuh"

namespace tk {

// Windows of the 2-bit code form of a packed read array.  A thread owns the
// 32 window end positions [32w, 32w + 32); the 64 positions [32w - 32, 32w + 32)
// (code words w-1 and w, invalid bits likewise) hold every base those windows
// use (k <= 31).  Each window is cut out of the 128-bit code pair with one
// funnel shift, its reverse complement out of the pair's reverse complement,
// and it is valid when none of its k positions has its invalid bit set.
// Calls f(key, i) for every valid window, in order of its end position 32w + i;
// i from I0 up to I1.
template <bool CANON, int I0 = 0, int I1 = 32, typename F>
__device__ __forceinline__ void thread_windows(const uint64_t *__restrict__ codes, const uint32_t *__restrict__ inv,
                                               uint64_t w, bool active, int k, F &&f) {
    uint64_t hi = 0, lo = 0, m = ~0ULL;
    if (active) {
        hi = __ldg(codes + w - 1);
        lo = __ldg(codes + w);
        m = ((uint64_t)__ldg(inv + w - 1) << 32) | __ldg(inv + w);
    }
    // bit b of `bad`: some position among bits b .. b+k-1 of m (position
    // 32w - 32 + x sits at bit 63 - x) is not A/C/G/T
    uint64_t bad = 0, span = m;
    int sh = 0;
#pragma unroll
    for (int l = 0; l < 5; l++) {
        if (k & (1 << l)) {
            bad |= span >> sh;
            sh += 1 << l;
        }
        span |= span >> (1 << l);
    }
    // reverse complement of the 64 positions: complement, then reverse the
    // order of the 2-bit groups
    uint64_t rhi = __brevll(~lo), rlo = __brevll(~hi);
    rhi = ((rhi >> 1) & 0x5555555555555555ULL) | ((rhi & 0x5555555555555555ULL) << 1);
    rlo = ((rlo >> 1) & 0x5555555555555555ULL) | ((rlo & 0x5555555555555555ULL) << 1);
    const uint64_t kmask = (1ULL << (2 * k)) - 1;
#pragma unroll
    for (int i = I0; i < I1; i++) {
        if ((bad >> (31 - i)) & 1ULL) continue;
        // forward: the window ends at position 32 + i of the 64
        const int s = 62 - 2 * i;
        const uint64_t fw = (s ? ((lo >> s) | (hi << (64 - s))) : lo) & kmask;
        uint64_t key = fw;
        if (CANON) {
            // reverse complement: it ends where the window starts, 33 + i - k
            const int r = 66 + 2 * i - 2 * k;   // 4 .. 126
            const uint64_t rc = (r >= 64 ? (rhi >> (r - 64)) : ((rlo >> r) | (rhi << (64 - r)))) & kmask;
            key = rc < fw ? rc : fw;
        }
        f(key, i);
    }
}

}  // namespace tk
