// tk_r2t.cu -- K6: Chrysalis ReadsToTranscripts read-to-component assignment
// (called at Trinity:2237-2251).
//
// Build: the bundle (one '>s_<component>' record per component, contigs
// joined by 'X', util/support_scripts/add_LR_reads_to_iworm_bundle.pl:19-47)
// is parsed like reads; every window of k A/C/G/T bases is inserted with
// value = (its end position, its record index) through a 64-bit atomicMin, so
// a k-mer held by several records belongs to the first of them whatever the
// insertion order, and the table also says where it first occurs.
//
// Assign, by alignment (k_r2t_align): one thread per read.  The first of a few
// windows that the bundle holds (they share no base) gives a place in the
// bundle; the whole read is compared with the bundle there, 32 bases at a time,
// and every window without a difference has the same owner, as long as no
// earlier record owns the bundle's k-mer there (a bit per bundle position).
// What is left are mostly windows over a sequencing error, whose k-mers the
// bundle does not have: a warp takes the left windows of its 32 reads one per
// lane, and a small filter of the bundle's k-mers that stays in L2 answers for
// most of them.  A read of 100 bases then costs one or two random table
// accesses instead of 76.  Reads whose windows belong to more than one record,
// or with more than 128 windows, are left to the per-window kernel.  The bits
// and the filter are built by the first read set that has as many bases as
// the bundle.
//
// Assign, per window (k_r2t_assign): one warp per read packs the read's bases
// 2 bits each into shared memory, cuts each lane's windows out of it, looks
// them up, sorts the record indices in registers and takes the longest run:
// the record with most votes, ties to the smaller index.  Reads with more than
// 256 windows use one block and a global scratch slab.
#include "tk_windows.cuh"
#include "tk_warp.cuh"

#include <algorithm>

namespace tk {

constexpr int RT_THREADS = 256;
constexpr int RT_SPAN = 32;
constexpr uint32_t RT_WARP_MAX = 256;

int parse_reads(tk_ctx *c, tk_reads *r);
int table_alloc_init(tk_table *t, uint64_t capacity, uint64_t init_val);

// the record holding position p: the largest r with rd_off[r] <= p
__device__ __forceinline__ uint64_t r2t_record_of(const uint64_t *__restrict__ rd_off, uint64_t n_rec, uint64_t p) {
    uint64_t lo = 0, hi = n_rec;
    while (hi - lo > 1) {
        const uint64_t mid = (lo + hi) >> 1;
        if (__ldg(rd_off + mid) <= p) lo = mid; else hi = mid;
    }
    return lo;
}

// Calls f(key, end position, record) for every window of the bundle ending in
// the thread's 32 positions.
template <bool CANON, typename F>
__device__ __forceinline__ void bundle_windows(const uint64_t *__restrict__ codes, const uint32_t *__restrict__ inv,
                                               uint64_t w, uint64_t n, const uint64_t *__restrict__ rd_off, uint64_t n_rec,
                                               int k, F &&f) {
    const uint64_t p0 = w * RT_SPAN;
    uint64_t rec = 0, next = 0;
    if (p0 < n) {
        rec = r2t_record_of(rd_off, n_rec, p0);
        next = __ldg(rd_off + rec + 1);
    }
    thread_windows<CANON>(codes, inv, w, p0 < n, k, [&](uint64_t key, int i) {
        while (p0 + i >= next && rec + 1 < n_rec) next = __ldg(rd_off + ++rec + 1);
        f(key, p0 + i, (uint32_t)rec);
    });
}

// Bound by the atomics into a table larger than L2: one CAS per window, 23 G/s
// on GB300 (13.6M windows 0.55 ms).
template <bool CANON>
__global__ void __launch_bounds__(RT_THREADS) k_r2t_build(const uint64_t *__restrict__ codes,
                                                         const uint32_t *__restrict__ inv, uint64_t n,
                                                         const uint64_t *__restrict__ rd_off, uint64_t n_rec, int k,
                                                         DevTable t, int max_probes, uint32_t *__restrict__ err,
                                                         unsigned long long *__restrict__ distinct) {
    const uint64_t w = (uint64_t)blockIdx.x * RT_THREADS + threadIdx.x;
    uint32_t added = 0;
    bundle_windows<CANON>(codes, inv, w, n, rd_off, n_rec, k, [&](uint64_t key, uint64_t e, uint32_t rec) {
        // positions past 2^32 - 2 only order the records (no index is built over such a bundle)
        const uint64_t pos = e < 0xFFFFFFFEull ? e : 0xFFFFFFFEull;
        if (!tbl_min(t, key, pos << 32 | rec, max_probes, &added)) atomicExch(&err[DE_OVERFLOW], 1u);
    });
    added = warp_sum(added);
    if (lane_id() == 0 && added) atomicAdd(distinct, (unsigned long long)added);
}

// ---- the index of the alignment path

__device__ __forceinline__ unsigned long long filter_bits(uint64_t h) { return (1ULL << (h & 63)) | (1ULL << ((h >> 6) & 63)); }
__device__ __forceinline__ uint64_t filter_word(uint64_t h, uint64_t mask) { return (h >> 32) & mask; }

// foreign[j] bit 31-i: an earlier record owns the k-mer of the window ending
// at 32j + i; and the filter's bits of every k-mer.
template <bool CANON>
__global__ void __launch_bounds__(RT_THREADS) k_r2t_index(const uint64_t *__restrict__ codes,
                                                         const uint32_t *__restrict__ inv, uint64_t n,
                                                         const uint64_t *__restrict__ rd_off, uint64_t n_rec, int k,
                                                         DevTable t, uint32_t *__restrict__ foreign,
                                                         unsigned long long *__restrict__ filter, uint64_t filter_mask) {
    const uint64_t w = (uint64_t)blockIdx.x * RT_THREADS + threadIdx.x;
    uint32_t bits = 0;
    bundle_windows<CANON>(codes, inv, w, n, rd_off, n_rec, k, [&](uint64_t key, uint64_t e, uint32_t rec) {
        if (tbl_get2<uint32_t>(t, key, false, PAD_VAL) != rec) bits |= 0x80000000u >> (e & 31);
        const uint64_t h = mix64(key);
        atomicOr(&filter[filter_word(h, filter_mask)], filter_bits(h));
    });
    if (w * RT_SPAN < n) foreign[w] = bits;
}

// 32 positions from p on, the first in the top bits (p >= -32)
__device__ __forceinline__ uint64_t codes_at(const uint64_t *__restrict__ codes, int64_t p) {
    const int64_t q = p >> 5;
    const int s = 2 * (int)(p & 31);
    const uint64_t hi = __ldg(codes + q);
    return s ? (hi << s) | (__ldg(codes + q + 1) >> (64 - s)) : hi;
}
__device__ __forceinline__ uint32_t bits_at(const uint32_t *__restrict__ w, int64_t p) {
    const int64_t q = p >> 5;
    return __funnelshift_l(__ldg(w + q + 1), __ldg(w + q), (uint32_t)(p & 31));
}

struct R2tIndex {
    const uint64_t *codes;
    const uint32_t *inv, *foreign;
    const unsigned long long *filter;
    uint64_t filter_mask;
    const uint64_t *rd_off;  // the bundle's records
    uint64_t len;            // positions of the bundle
};
constexpr uint32_t RT_ALIGN_MAX = 128;   // windows of a read the alignment path takes (two 64-bit masks)

// A mask over a read's windows or positions, bit j of (a, b, c) = number j.
struct Bits192 {
    uint64_t a, b, c;
};

__device__ __forceinline__ Bits192 low_bits(uint32_t n) {   // n <= 128
    return {n >= 64 ? ~0ULL : (1ULL << n) - 1, n > 64 ? ~0ULL >> (128 - n) : 0ULL, 0ULL};
}

// Windows (bit w: positions w .. w+k-1) that hold a marked position.
__device__ __forceinline__ Bits192 windows_over(Bits192 m, int k) {
    Bits192 r{0, 0, 0};
    int sh = 0;
#pragma unroll
    for (int l = 0; l < 5; l++) {
        if (k & (1 << l)) {
            r.a |= sh ? (m.a >> sh) | (m.b << (64 - sh)) : m.a;
            r.b |= sh ? (m.b >> sh) | (m.c << (64 - sh)) : m.b;
            sh += 1 << l;
        }
        const int d = 1 << l;
        m.a |= (m.a >> d) | (m.b << (64 - d));
        m.b |= (m.b >> d) | (m.c << (64 - d));
        m.c |= m.c >> d;
    }
    return r;
}

// Word i (numbers 32i .. 32i+31) of a mask
__device__ __forceinline__ void set_word(Bits192 &m, int i, uint32_t w) {
    const uint64_t v = (uint64_t)w << (32 * (i & 1));
    if (i < 2) m.a |= v;
    else if (i < 4) m.b |= v;
    else m.c |= v;
}

// bit j: base j (of 32, the first in the top two bits) of x is not zero
__device__ __forceinline__ uint32_t base_mask(uint64_t x) {
    x = (x | x >> 1) & 0x5555555555555555ULL;
    x = (x | x >> 1) & 0x3333333333333333ULL;
    x = (x | x >> 2) & 0x0F0F0F0F0F0F0F0FULL;
    x = (x | x >> 4) & 0x00FF00FF00FF00FFULL;
    x = (x | x >> 8) & 0x0000FFFF0000FFFFULL;
    return __brev((uint32_t)(x | x >> 16));
}

// What the table says of the window starting at p: (end position << 32) |
// record, ~0 when the bundle does not have it.  The filter is asked first.
template <bool CANON>
__device__ __forceinline__ uint64_t bundle_lookup(const R2tIndex &ix, const DevTable &t, uint64_t fw, int k) {
    uint64_t key = fw;
    if (CANON) {
        const uint64_t rc = kmer_revcomp(fw, k);
        key = rc < fw ? rc : fw;
    }
    const uint64_t h = mix64(key);
    const unsigned long long fb = filter_bits(h);
    if ((__ldg(ix.filter + filter_word(h, ix.filter_mask)) & fb) != fb) return ~0ULL;
    return tbl_get2<uint64_t>(t, key, true, ~0ULL);
}

constexpr uint32_t RT_LEFT = 1024;   // left windows a warp lists at a time (32 of each read)

// A thread per read (see the head of the file).  3M reads of 100 nt against
// 13.6M bundle k-mers: 1.02 ms (ALU 74% busy), and 0.12 for the reads left over;
// with every thread walking its own open windows, extending to the first
// difference, 1.44 (a lane whose read has errors kept its warp); the per-window
// kernel takes 7.68, bound by its 76 random accesses per read at 38-44 G/s.
template <bool CANON>
__global__ void __launch_bounds__(RT_THREADS, 4) k_r2t_align(R2tIndex ix, DevTable t, const uint64_t *__restrict__ codes,
                                                            const uint32_t *__restrict__ inv,
                                                            const uint64_t *__restrict__ rd_off, uint64_t n_reads, int k,
                                                            int32_t *__restrict__ rec, uint32_t *__restrict__ hits,
                                                            uint32_t *__restrict__ nwin_out, uint32_t *__restrict__ rest,
                                                            unsigned long long *__restrict__ rest_n) {
    __shared__ uint16_t s_left[RT_THREADS / 32][RT_LEFT];   // (lane << 7) | window
    __shared__ uint32_t s_votes[RT_THREADS], s_other[RT_THREADS];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const uint64_t r = (uint64_t)blockIdx.x * RT_THREADS + threadIdx.x;
    uint64_t start = 0, nw = 0;
    if (r < n_reads) {
        start = rd_off[r];
        const uint64_t L = rd_off[r + 1] - start - 1;
        nw = L >= (uint64_t)k ? L - k + 1 : 0;
        nwin_out[r] = (uint32_t)nw;
    }
    const bool too_long = nw > RT_ALIGN_MAX;
    const uint32_t nwin = too_long ? 0u : (uint32_t)nw;
    uint32_t owner = PAD_VAL, votes = 0;
    uint64_t left_a = 0, left_b = 0;
    if (nwin) {
        const int words = (int)((nwin + k - 1 + 31) / 32);   // of the read's bases, 1 .. 5
        Bits192 bad{0, 0, 0};                                // positions that are not A/C/G/T
        for (int i = 0; i < words; i++) set_word(bad, i, __brev(bits_at(inv, (int64_t)start + 32 * i)));
        const Bits192 all = low_bits(nwin);
        const Bits192 nb = windows_over(bad, k);
        left_a = all.a & ~nb.a;
        left_b = all.b & ~nb.b;
        // the first window among 0, k, 2k, ... and the last that the bundle holds
        uint64_t hit = ~0ULL, fw = 0;
        uint32_t w = 0;
        for (;;) {
            if (((w < 64 ? left_a >> w : left_b >> (w - 64)) & 1ULL)) {
                fw = codes_at(codes, (int64_t)(start + w)) >> (64 - 2 * k);
                hit = bundle_lookup<CANON>(ix, t, fw, k);
                if (hit != ~0ULL) break;
            }
            if (w == nwin - 1) break;
            w = min(w + (uint32_t)k, nwin - 1);
        }
        if (hit != ~0ULL) {
            owner = (uint32_t)hit;
            const int64_t e = (int64_t)(hit >> 32), s0 = e - k + 1;   // the bundle's window: positions s0 .. e
            const bool forward = !CANON || codes_at(ix.codes, s0) >> (64 - 2 * k) == fw;
            Bits192 diff = bad, foreign{0, 0, 0};
            for (int i = 0; i < words; i++) {
                // the bundle's 32 positions against the read's bases 32i ..: from p up, or p + 31 down
                const int64_t p = forward ? s0 - (int64_t)w + 32 * i : e + (int64_t)w - 32 * i - 31;
                uint32_t d = ~0u;
                if (p >= -32 && p < (int64_t)ix.len) {
                    uint64_t bw = codes_at(ix.codes, p);
                    uint32_t bi = bits_at(ix.inv, p);
                    if (forward) bi = __brev(bi);
                    else bw = kmer_revcomp(bw, 32);
                    d = bi | base_mask(bw ^ codes_at(codes, (int64_t)start + 32 * i));
                }
                set_word(diff, i, d);
                // windows 32i .. end at the bundle's positions from f up, or f + 31 down
                const int64_t f = forward ? p + k - 1 : p;
                if (i < 4 && f >= -32 && f < (int64_t)ix.len) {
                    const uint32_t b = bits_at(ix.foreign, f);
                    set_word(foreign, i, forward ? __brev(b) : b);
                }
            }
            // only the windows whose place lies in the owner's record (the next
            // record may go on where the read does)
            const int64_t r_lo = (int64_t)ix.rd_off[owner], r_hi = (int64_t)ix.rd_off[owner + 1] - 2;   // its first and last position
            const int64_t w_lo = forward ? r_lo - s0 + (int64_t)w : e + (int64_t)w - r_hi;
            const int64_t w_hi = forward ? r_hi - e + (int64_t)w : s0 + (int64_t)w - r_lo;
            const Bits192 upto = low_bits((uint32_t)min(w_hi + 1, (int64_t)RT_ALIGN_MAX));
            const Bits192 below = low_bits((uint32_t)max(w_lo, (int64_t)0));
            const Bits192 over = windows_over(diff, k);
            const uint64_t ma = all.a & upto.a & ~below.a & ~over.a & ~foreign.a;
            const uint64_t mb = all.b & upto.b & ~below.b & ~over.b & ~foreign.b;
            votes = __popcll(ma) + __popcll(mb);
            left_a &= ~ma;
            left_b &= ~mb;
        }
    }
    s_votes[threadIdx.x] = 0;
    s_other[threadIdx.x] = 0;
    __syncwarp();
    // the left windows of the warp's reads, listed and taken one per lane
    uint16_t *list = s_left[warp];
    while (__any_sync(0xffffffffu, (left_a | left_b) != 0)) {
        const uint32_t mine = min(32u, (uint32_t)(__popcll(left_a) + __popcll(left_b)));
        const uint32_t incl = warp_incl_scan(mine), total = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t at = incl - mine;
        for (uint32_t j = 0; j < mine; j++) {
            uint32_t w;
            if (left_a) {
                w = (uint32_t)__ffsll((long long)left_a) - 1;
                left_a &= left_a - 1;
            } else {
                w = 63u + (uint32_t)__ffsll((long long)left_b);
                left_b &= left_b - 1;
            }
            list[at++] = (uint16_t)(lane << 7 | w);
        }
        __syncwarp();
        for (uint32_t i = lane; i < ((total + 31) & ~31u); i += 32) {
            const uint32_t item = i < total ? list[i] : 0u, l = item >> 7;
            const uint64_t st = __shfl_sync(0xffffffffu, start, (int)l);
            const uint32_t own = __shfl_sync(0xffffffffu, owner, (int)l);
            if (i >= total) continue;
            const uint64_t hit = bundle_lookup<CANON>(ix, t, codes_at(codes, (int64_t)(st + (item & 127u))) >> (64 - 2 * k), k);
            if (hit == ~0ULL) continue;
            if ((uint32_t)hit == own) atomicAdd(&s_votes[warp * 32 + l], 1u);
            else s_other[warp * 32 + l] = 1u;
        }
        __syncwarp();
    }
    if (r >= n_reads) return;
    votes += s_votes[threadIdx.x];
    if (too_long || s_other[threadIdx.x]) {
        rest[atomicAdd(rest_n, 1ULL)] = (uint32_t)r;   // votes are counted per window
        return;
    }
    rec[r] = votes ? (int32_t)owner : -1;
    hits[r] = votes;
}

template <int S, bool CANON>
__device__ __forceinline__ void r2t_warp_read(DevTable t, const uint8_t *__restrict__ seq, uint64_t start, uint32_t nwin,
                                              int k, uint64_t r, int32_t *__restrict__ rec, uint32_t *__restrict__ hits,
                                              uint64_t *words) {
    const unsigned lane = lane_id();
    const uint32_t span = (nwin + 31) / 32;
    uint32_t v[S];
    auto body = [&](int j, bool valid, uint64_t key) { v[j] = valid ? tbl_get2<uint32_t>(t, key, false, PAD_VAL) : PAD_VAL; };
    // k-mers cut from the read packed in shared memory; reads with another
    // character take the byte path
    if (!lane_windows_packed<S, CANON>(seq, start, nwin, span, k, words, body))
        lane_windows<S, CANON>(seq, start, nwin, span, k, body);
    warp_bitonic_sort<S>(v);
    // longest run of equal values; run start indices by an inclusive max-scan
    uint32_t prev_last = __shfl_up_sync(0xffffffffu, v[S - 1], 1);
    int last_start = -1;
    int st[S];
#pragma unroll
    for (int j = 0; j < S; j++) {
        uint32_t prev = j ? v[j - 1] : prev_last;
        bool is_start = (lane == 0 && j == 0) || v[j] != prev;
        if (is_start) last_start = (int)(lane * S + j);
        st[j] = last_start;
    }
    int carry = last_start;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int x = __shfl_up_sync(0xffffffffu, carry, o);
        if ((int)lane >= o) carry = max(carry, x);
    }
    int before = __shfl_up_sync(0xffffffffu, carry, 1);
    if (lane == 0) before = -1;
    uint64_t best = 0;   // (run length << 32) | (0xFFFFFFFF - value)
#pragma unroll
    for (int j = 0; j < S; j++) {
        int s0 = st[j] < 0 ? before : st[j];
        uint32_t len = (uint32_t)((int)(lane * S + j) - s0 + 1);
        if (v[j] != PAD_VAL) {
            uint64_t cand = ((uint64_t)len << 32) | (uint64_t)(0xFFFFFFFFu - v[j]);
            best = max(best, cand);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0) {
        if (best == 0) {
            rec[r] = -1;
            hits[r] = 0;
        } else {
            rec[r] = (int32_t)(0xFFFFFFFFu - (uint32_t)best);
            hits[r] = (uint32_t)(best >> 32);
        }
    }
}

template <bool CANON>
__global__ void __launch_bounds__(RT_THREADS, 6) k_r2t_assign(DevTable t, const uint8_t *__restrict__ seq,
                                                             const uint64_t *__restrict__ rd_off, uint64_t n_reads,
                                                             int k, int32_t *__restrict__ rec,
                                                             uint32_t *__restrict__ hits, uint32_t *__restrict__ nwin_out,
                                                             const uint32_t *__restrict__ list,
                                                             uint32_t *__restrict__ long_list,
                                                             unsigned long long *__restrict__ long_n) {
    __shared__ uint64_t words[RT_THREADS / 32][12];
    uint64_t *w = words[threadIdx.x >> 5];
    const uint64_t warps = (uint64_t)gridDim.x * (RT_THREADS / 32);
    for (uint64_t i = (uint64_t)blockIdx.x * (RT_THREADS / 32) + (threadIdx.x >> 5); i < n_reads; i += warps) {
        const uint64_t r = list ? list[i] : i;   // n_reads = the list's length, with a list
        const uint64_t start = rd_off[r];
        const uint64_t L = rd_off[r + 1] - start - 1;
        const uint32_t nwin = L >= (uint64_t)k ? (uint32_t)(L - k + 1) : 0u;
        if (lane_id() == 0) nwin_out[r] = nwin;
        if (nwin <= 32) r2t_warp_read<1, CANON>(t, seq, start, nwin, k, r, rec, hits, w);
        else if (nwin <= 64) r2t_warp_read<2, CANON>(t, seq, start, nwin, k, r, rec, hits, w);
        else if (nwin <= 128) r2t_warp_read<4, CANON>(t, seq, start, nwin, k, r, rec, hits, w);
        else if (nwin <= RT_WARP_MAX) r2t_warp_read<8, CANON>(t, seq, start, nwin, k, r, rec, hits, w);
        else if (lane_id() == 0) long_list[atomicAdd(long_n, 1ULL)] = (uint32_t)r;
    }
}

template <bool CANON>
__global__ void __launch_bounds__(RT_THREADS) k_r2t_long(DevTable t, const uint8_t *__restrict__ seq,
                                                        const uint64_t *__restrict__ rd_off,
                                                        const uint32_t *__restrict__ list, uint64_t n_long, int k,
                                                        uint32_t *__restrict__ scratch, uint64_t n2max,
                                                        int32_t *__restrict__ rec, uint32_t *__restrict__ hits) {
    uint32_t *slab = scratch + (uint64_t)blockIdx.x * n2max;
    for (uint64_t i = blockIdx.x; i < n_long; i += gridDim.x) {
        const uint32_t r = list[i];
        const uint64_t start = rd_off[r];
        const uint32_t nwin = (uint32_t)(rd_off[r + 1] - start - 1 - (k - 1));
        uint32_t n2 = 1;
        while (n2 < nwin) n2 <<= 1;
        block_window_values<CANON>(seq, start, nwin, n2, k, slab, [&](uint64_t key) { return tbl_get2<uint32_t>(t, key, false, PAD_VAL); });
        block_bitonic_sort(slab, n2);
        if (threadIdx.x == 0) {
            uint32_t best_len = 0, best_v = PAD_VAL;
            for (uint32_t a = 0; a < n2 && slab[a] != PAD_VAL;) {
                uint32_t b = a;
                while (b < n2 && slab[b] == slab[a]) b++;
                if (b - a > best_len) { best_len = b - a; best_v = slab[a]; }
                a = b;
            }
            rec[r] = best_len ? (int32_t)best_v : -1;
            hits[r] = best_len;
        }
        __syncthreads();
    }
}

int r2t_build(tk_r2t *z, tk_reads *b) {
    tk_ctx *c = z->ctx;
    tk_table *t = z->table;
    uint64_t want = 1024;
    while (want < 2 * std::max<uint64_t>(b->n_bases, 1)) want <<= 1;
    TK_TRY(table_alloc_init(t, want, ~0ULL));
    t->distinct = 0;
    t->distinct_valid = true;
    if (b->n_reads == 0 || b->seq_len == 0) return TK_OK;
    TK_CUDA(c, cudaMemsetAsync(c->d_err, 0, DE_COUNT * 4, c->stream));
    TK_CUDA(c, cudaMemsetAsync(t->d_counters, 0, 8, c->stream));
    const uint64_t n = b->seq_len, per_block = (uint64_t)RT_THREADS * RT_SPAN;
    const unsigned grid = (unsigned)((n + per_block - 1) / per_block);
    cudaEvent_t ev;
    prof_begin(c, TK_KID_R2T_BUILD, &ev);
    if (!z->strand)
        k_r2t_build<true><<<grid, RT_THREADS, 0, c->stream>>>(b->d_codes, b->d_inv, n, b->d_rd_off, b->n_reads, z->k, t->t,
                                                              c->max_probes, c->d_err, t->d_counters);
    else
        k_r2t_build<false><<<grid, RT_THREADS, 0, c->stream>>>(b->d_codes, b->d_inv, n, b->d_rd_off, b->n_reads, z->k, t->t,
                                                               c->max_probes, c->d_err, t->d_counters);
    c->launches++;
    prof_end(c, TK_KID_R2T_BUILD, ev, b->n_bases);
    TK_TRY(check_launch(c, "r2t build"));
    uint32_t herr[DE_COUNT];
    unsigned long long distinct = 0;
    TK_CUDA(c, cudaMemcpyAsync(herr, c->d_err, sizeof(herr), cudaMemcpyDeviceToHost, c->stream));
    TK_CUDA(c, cudaMemcpyAsync(&distinct, t->d_counters, 8, cudaMemcpyDeviceToHost, c->stream));
    TK_CUDA(c, cudaStreamSynchronize(c->stream));
    if (herr[DE_OVERFLOW]) return set_err(c, TK_E_TABLE_FULL, "bundle k-mer table: probe limit reached");
    t->distinct = distinct;
    // the bundle's 2-bit form stays for the alignment path
    z->seq_len = b->seq_len;
    z->n_bases = b->n_bases;
    z->n_records = b->n_reads;
    z->d_pack_alloc = b->d_pack_alloc;
    z->d_codes = b->d_codes;
    z->d_inv = b->d_inv;
    z->d_rd_off = b->d_rd_off;
    b->d_pack_alloc = nullptr;
    b->d_codes = nullptr;
    b->d_inv = nullptr;
    b->d_rd_off = nullptr;
    return TK_OK;
}

void r2t_release(tk_r2t *z) {
    void *p[] = {z->d_pack_alloc, z->d_rd_off, z->d_foreign, z->d_filter};
    for (void *q : p)
        if (q) dfree(z->ctx, q);
}

// The bits and the filter of the alignment path; *ready false when they cannot
// be held (the per-window path then serves).
static int r2t_index(tk_r2t *z, bool *ready) {
    tk_ctx *c = z->ctx;
    *ready = z->d_foreign != nullptr;
    if (*ready || !z->d_codes || z->seq_len >= 0xFFFFFFFEull) return TK_OK;
    uint64_t words = 1024;   // a word per 12 bundle bases or fewer
    while (words * 12 < z->n_bases) words <<= 1;
    const uint64_t n_words = (z->seq_len + 31) / 32 + 2;   // word -1 and one past the last, like inv
    uint32_t *foreign = nullptr;
    unsigned long long *filter = nullptr;
    int e = dmalloc(c, (void **)&foreign, (n_words + 1) * 4, "bundle ownership bits");
    if (!e) e = dmalloc(c, (void **)&filter, words * 8, "bundle k-mer filter");
    if (e) {
        if (foreign) dfree(c, foreign);
        return TK_OK;
    }
    e = cuda_check(c, cudaMemsetAsync(foreign, 0, (n_words + 1) * 4, c->stream), "ownership bits reset");
    if (!e) e = cuda_check(c, cudaMemsetAsync(filter, 0, words * 8, c->stream), "filter reset");
    if (!e) {
        const uint64_t per_block = (uint64_t)RT_THREADS * RT_SPAN;
        const unsigned grid = (unsigned)((z->seq_len + per_block - 1) / per_block);
        cudaEvent_t ev;
        prof_begin(c, TK_KID_R2T_BUILD, &ev);
        if (!z->strand)
            k_r2t_index<true><<<grid, RT_THREADS, 0, c->stream>>>(z->d_codes, z->d_inv, z->seq_len, z->d_rd_off, z->n_records,
                                                                  z->k, z->table->t, foreign + 1, filter, words - 1);
        else
            k_r2t_index<false><<<grid, RT_THREADS, 0, c->stream>>>(z->d_codes, z->d_inv, z->seq_len, z->d_rd_off, z->n_records,
                                                                   z->k, z->table->t, foreign + 1, filter, words - 1);
        c->launches++;
        prof_end(c, TK_KID_R2T_BUILD, ev, z->n_bases);
        e = check_launch(c, "r2t index");
    }
    if (e) {
        dfree(c, foreign);
        dfree(c, filter);
        return e;
    }
    z->d_foreign = foreign;
    z->d_filter = filter;
    z->filter_mask = words - 1;
    *ready = true;
    return TK_OK;
}

int r2t_assign(tk_r2t *z, const tk_reads *rd, int32_t *d_rec, uint32_t *d_hits, uint32_t *d_nwin) {
    tk_ctx *c = z->ctx;
    const uint64_t n = rd->n_reads;
    if (n == 0) return TK_OK;
    const int k = z->k;
    const bool may_long = rd->max_len >= (uint32_t)k && rd->max_len - k + 1 > RT_WARP_MAX;
    uint32_t *long_list = nullptr;
    unsigned long long *long_n = nullptr;
    TK_TRY(dmalloc(c, (void **)&long_n, 8, "long-read count"));
    int e = TK_OK;
    if (may_long) e = dmalloc(c, (void **)&long_list, n * 4, "long-read list");
    if (!e) e = cuda_check(c, cudaMemsetAsync(long_n, 0, 8, c->stream), "long reset");
    // The alignment path, for reads of at most 128 windows on average: from as
    // many read bases as the bundle has on, building its index costs less than
    // it saves (0.3 ms for 13.6M bundle bases against 7.7 -> 1.1 ms for 228M
    // windows); once built, every such read set takes it.
    bool align = rd->n_bases <= n * (uint64_t)(RT_ALIGN_MAX + k - 1);
    uint32_t *rest = nullptr;
    uint64_t n_rest = n;
    if (!e && align) {
        align = z->d_foreign != nullptr;
        if (!align && rd->n_bases >= z->n_bases) e = r2t_index(z, &align);
        if (!e && align && dmalloc(c, (void **)&rest, n * 4, "reads left to the per-window vote")) align = false;
    }
    if (!e && align) {
        const R2tIndex ix{z->d_codes, z->d_inv, z->d_foreign + 1, z->d_filter, z->filter_mask, z->d_rd_off, z->seq_len};
        const unsigned grid = (unsigned)((n + RT_THREADS - 1) / RT_THREADS);
        cudaEvent_t ev;
        prof_begin(c, TK_KID_R2T_ASSIGN, &ev);
        if (!z->strand)
            k_r2t_align<true><<<grid, RT_THREADS, 0, c->stream>>>(ix, z->table->t, rd->d_codes, rd->d_inv, rd->d_rd_off, n, k,
                                                                  d_rec, d_hits, d_nwin, rest, long_n);
        else
            k_r2t_align<false><<<grid, RT_THREADS, 0, c->stream>>>(ix, z->table->t, rd->d_codes, rd->d_inv, rd->d_rd_off, n, k,
                                                                   d_rec, d_hits, d_nwin, rest, long_n);
        c->launches++;
        prof_end(c, TK_KID_R2T_ASSIGN, ev, rd->n_bases);
        e = check_launch(c, "r2t align");
        unsigned long long hr = 0;
        if (!e) e = cuda_check(c, cudaMemcpyAsync(&hr, long_n, 8, cudaMemcpyDeviceToHost, c->stream), "rest n");
        if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "rest sync");
        if (!e) e = cuda_check(c, cudaMemsetAsync(long_n, 0, 8, c->stream), "long reset");
        n_rest = hr;
    }
    if (!e && n_rest) {
        const unsigned grid = (unsigned)std::max<uint64_t>(
            1, std::min<uint64_t>((n_rest + RT_THREADS / 32 - 1) / (RT_THREADS / 32), (uint64_t)c->sm_count * 16));
        cudaEvent_t ev;
        prof_begin(c, TK_KID_R2T_ASSIGN, &ev);
        if (!z->strand)
            k_r2t_assign<true><<<grid, RT_THREADS, 0, c->stream>>>(z->table->t, rd->d_seq, rd->d_rd_off, n_rest, k, d_rec,
                                                                   d_hits, d_nwin, rest, long_list, long_n);
        else
            k_r2t_assign<false><<<grid, RT_THREADS, 0, c->stream>>>(z->table->t, rd->d_seq, rd->d_rd_off, n_rest, k, d_rec,
                                                                    d_hits, d_nwin, rest, long_list, long_n);
        c->launches++;
        prof_end(c, TK_KID_R2T_ASSIGN, ev, align ? 0 : rd->n_bases);
        e = check_launch(c, "r2t assign");
    }
    unsigned long long hl = 0;
    if (!e && may_long) {
        e = cuda_check(c, cudaMemcpyAsync(&hl, long_n, 8, cudaMemcpyDeviceToHost, c->stream), "long n");
        if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "long sync");
    }
    if (!e && hl) {
        uint64_t n2max = 1;
        while (n2max < (uint64_t)(rd->max_len - k + 1)) n2max <<= 1;
        uint64_t grid = std::min<uint64_t>(hl, (uint64_t)c->sm_count * 2);
        uint32_t *scratch = nullptr;
        e = dmalloc(c, (void **)&scratch, grid * n2max * 4, "long-read scratch");
        if (!e) {
            if (!z->strand)
                k_r2t_long<true><<<(unsigned)grid, RT_THREADS, 0, c->stream>>>(z->table->t, rd->d_seq, rd->d_rd_off,
                                                                               long_list, hl, k, scratch, n2max, d_rec,
                                                                               d_hits);
            else
                k_r2t_long<false><<<(unsigned)grid, RT_THREADS, 0, c->stream>>>(z->table->t, rd->d_seq, rd->d_rd_off,
                                                                                long_list, hl, k, scratch, n2max, d_rec,
                                                                                d_hits);
            c->launches++;
            e = check_launch(c, "r2t long");
            dfree(c, scratch);
        }
    }
    if (rest) dfree(c, rest);
    if (long_list) dfree(c, long_list);
    dfree(c, long_n);
    return e;
}

}  // namespace tk
